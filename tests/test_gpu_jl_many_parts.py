"""A projection over so many parts that its units of work (a part of one column is one) do
not fit 32-bit indices: 2^32 - 1 parts, the most the 32-bit stream number allows. All words
are zero but those of a few parts around the ends of the launches, so the expected row sums
need those parts' keystream blocks alone (RFC 8439, written out here)."""
import ctypes as C
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = 4294966657
M32 = 0xFFFFFFFF


def _block(key, counter, nonce):
    """The ChaCha20 block function of RFC 8439."""
    init = [0x61707865, 0x3320646E, 0x79622D32, 0x6B206574, *struct.unpack("<8I", key), counter,
            nonce, 0, 0]
    x = list(init)

    def quarter(a, b, c, d):
        for p, s, t, r in ((a, b, d, 16), (c, d, b, 12), (a, b, d, 8), (c, d, b, 7)):
            x[p] = (x[p] + x[s]) & M32
            v = x[t] ^ x[p]
            x[t] = (v << r | v >> (32 - r)) & M32

    for _ in range(10):
        for i in range(4):
            quarter(i, 4 + i, 8 + i, 12 + i)
        for i in range(4):
            quarter(i, 4 + (i + 1) % 4, 8 + (i + 2) % 4, 12 + (i + 3) % 4)
    return struct.pack("<16I", *((u + v) & M32 for u, v in zip(x, init)))


def _entries(key, part):
    """Column 0 of a part: rows 0 .. 255, two bits each, 00 -> 1, 01 -> -1, 1x -> 0."""
    raw = np.frombuffer(_block(key, 0, part), np.uint8)
    codes = (raw[:, None] >> np.array([0, 2, 4, 6])) & 3
    return np.array([1, -1, 0, 0])[codes.reshape(-1)]


def test_the_written_out_block_is_the_oracles(oracle):
    key = bytes(range(32))
    one = np.array([[1]], np.uint32)
    want, _ = oracle.jl_project(oracle.Field(Q), key, 256, one, 1, 1, 1, want_flat=False)
    assert np.array_equal(_entries(key, 0) % Q, want)


def test_parts_up_to_the_stream_numbers_end(cuda, oracle):
    import torch
    from lattica_b200 import TwistedNttPlan, _lib
    lib, plan = _lib.load(), TwistedNttPlan(Q, 64)
    num_parts, key = (1 << 32) - 1, bytes((11 * i + 3) & 0xFF for i in range(32))
    x = torch.zeros(num_parts, dtype=torch.int32, device=cuda)
    at = {0: 5, 1: Q - 2, (1 << 31) - 1: 77, 1 << 31: Q - 1, (1 << 31) + 1: 9, num_parts - 1: 123456}
    want = np.zeros(256, dtype=object)
    for part, word in at.items():
        x[part] = word - (1 << 32) if word >= 1 << 31 else word
        want += _entries(key, part).astype(object) * word
    p = torch.empty(256, dtype=torch.int32, device=cuda)
    ws = torch.empty(1 << 16, dtype=torch.uint8, device=cuda)
    sd = (C.c_uint8 * 32).from_buffer_copy(key)
    assert lib.grid_gpu_jl_project_dev(plan.handle, sd, 256, x.data_ptr(), num_parts, 1, 1,
                                       p.data_ptr(), None, ws.data_ptr(), ws.numel(),
                                       torch.cuda.current_stream().cuda_stream) == 0
    assert np.array_equal(p.cpu().numpy().view(np.uint32), (want % Q).astype(np.uint32))
    plan.check_device()
