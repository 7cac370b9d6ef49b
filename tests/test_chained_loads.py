"""Kernels that may start while their predecessor in the stream still runs (those that call
grid_dep_wait) are resident while their inputs are written, so they read them neither with
__ldg nor through a const __restrict__ parameter, which the compiler may turn into the same
read-only load: only the plan's own tables, written before any launch, are read so. Read
from the sources: a stale line of the read-only cache shows in no test's result."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "lattica_b200", "csrc")
TABLES = {"gtw", "wtab", "gtab"}  # twiddles and transform matrices of a plan


def _kernels(text):
    """(name, parameters, body) of the __global__ functions."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\([^()]*(?:\([^()]*\))?[^()]*\)\s*)?"
                         r"(\w+)\s*\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, at = text[m.end():i - 1], text.index("{", i)
        depth, j = 1, at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        yield m.group(1), params, text[at:j]


def _read_only(params, body):
    """What a kernel reads through the read-only path besides the tables."""
    names = re.findall(r"const \w[\w ]*\*\s*__restrict__\s+(\w+)", params)
    return [n for n in names if n not in TABLES] + re.findall(r"__ldg\(", body)


def test_chained_kernels_read_their_inputs_coherently():
    chained = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path, encoding="utf-8") as fh:
            for name, params, body in _kernels(fh.read()):
                if "grid_dep_wait()" in body:
                    chained[name] = _read_only(params, body)
    assert set(chained) >= {"emm_pm_kernel", "ntt_tc_kernel", "ntt_mul_tc_kernel",
                            "sum_inverse_kernel", "vec_partial_kernel", "vec_finish_kernel",
                            "amortize_tc_kernel", "amortize_sum_kernel"}
    assert {k: v for k, v in chained.items() if v} == {}


def test_chained_launches_are_of_kernels_that_wait():
    """Every kernel launched chained waits for its predecessor."""
    waits, launched = set(), set()
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path, encoding="utf-8") as fh:
            text = fh.read()
        waits |= {name for name, _, body in _kernels(text) if "grid_dep_wait()" in body}
        for function in text.split("\n}\n"):
            if "launch_chained(" in function and "launch_chained(void" not in function:
                launched |= set(re.findall(r"launch_chained\(\s*(\w+_kernel)\b", function))
                launched |= set(re.findall(r"\brun\((\w+_kernel)\b", function))
    assert launched and launched <= waits
