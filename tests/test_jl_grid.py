"""The JL kernels' grid past one CTA per SM. A CTA may accumulate so many units; sizes that
need more CTAs than SMs get whole waves of them, or the last wave's few would take as long
as the first. Compiled from the library's own header for the host."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "lattica_b200", "csrc")
SMS, BOUND = 148, 2048


@pytest.fixture(scope="module")
def unit_grid(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("jl")
    src, lib = tmp / "g.cpp", tmp / "g.so"
    src.write_text('#include "jl_units.h"\nextern "C" unsigned g(unsigned long long n, int w, '
                   'int s) { return grid::unit_grid(n, w, s); }\n'
                   'extern "C" unsigned long long p(unsigned long long u, unsigned long long n) '
                   '{ return grid::parts_per_launch(u, n); }\n')
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o",
                           str(lib)])
    so = C.CDLL(str(lib))
    fn = so.g
    fn.parts = so.p
    fn.restype, fn.argtypes = C.c_uint, [C.c_ulonglong, C.c_int, C.c_int]
    fn.parts.restype, fn.parts.argtypes = C.c_ulonglong, [C.c_ulonglong, C.c_ulonglong]
    return fn


# r = 64 vectors of n polys of 64 coefficients: 128 n units
@pytest.mark.parametrize("warps", [12, 20])
@pytest.mark.parametrize("n", [1, 2, 100, 2048, 2304, 2358, 2359, 2400, 3072, 4096, 4717, 4718,
                               100000])
def test_whole_waves_within_the_bound(unit_grid, warps, n):
    units = 128 * n
    grid = unit_grid(units, warps, SMS)
    waves = -(-grid // SMS)
    turns = -(-units // (grid * warps))  # of a CTA's warps
    assert grid == units or grid % SMS == 0
    assert turns * warps <= BOUND
    # the SMs' warps are busy for all but the last turn of each wave
    assert waves * turns < units / (SMS * warps) + waves + 1
    assert waves == max(1, -(-units // (BOUND // warps * warps * SMS)))


@pytest.mark.parametrize("warps", [12, 20])
def test_few_units_one_cta_each(unit_grid, warps):
    assert [unit_grid(u, warps, SMS) for u in (1, 2, 147, 148, 149)] == [1, 2, 147, 148, 148]


@pytest.mark.parametrize("per_part", [1, 2, 3, 1 << 20, (1 << 31) - 1, 1 << 31])
@pytest.mark.parametrize("num_parts", [1, 2, 1490, (1 << 32) - 1])
def test_launches_of_32_bit_units(per_part, num_parts, unit_grid):
    """However many parts: every launch's units, and the last turn past them, fit 32 bits."""
    step = unit_grid.parts(per_part, num_parts)
    assert 1 <= step <= num_parts
    units = per_part * step
    for warps in (12, 20):
        assert units + unit_grid(units, warps, SMS) * warps < 1 << 32
    assert unit_grid.parts((1 << 31) + 1, num_parts) == 0
