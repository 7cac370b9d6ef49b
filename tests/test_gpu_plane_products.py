"""The byte-plane products over point-major evaluations at the edges of their tiles:
K around a 128-word chunk and over several splits, witness rows of every length
(rows that are no whole 16-byte units go through the row-wise transform), X rows
around 8, 64 and 128, Y rows around every padding, the largest words (every class
at its largest sum). Every word equals the oracle's."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = 4294966657


def _words(q, shape, seed):
    rng = np.random.default_rng(seed)
    x = rng.integers(0, q, shape, dtype=np.uint64).astype(np.uint32)
    x.reshape(-1)[: x.size // 3] = q - 1
    return x


def _dev(x, cuda):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).to(cuda)


def _host(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("q", [Q, 12289])
@pytest.mark.parametrize("batch,rows,cols", [(1, 1, 1), (8, 16, 127), (9, 17, 129), (1, 33, 515),
                                             (64, 16, 131), (65, 5, 130), (128, 64, 33),
                                             (2, 48, 1030), (70, 49, 257), (3, 64, 2049)])
def test_commit_shapes(cuda, oracle, q, batch, rows, cols):
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.commit import PreparedMatrix
    plan, P = TwistedNttPlan(q, 64), oracle.Plan(q, 64)
    A, s = _words(q, (rows, cols, 64), rows), _words(q, (batch, cols, 64), cols)
    got = PreparedMatrix(plan, _dev(A, cuda), rows, cols).mul_vec(_dev(s, cuda))
    want = P.matvec(A, rows, cols, s, batch, threads=0).reshape(batch, rows, 64)
    assert np.array_equal(_host(got), want)
    plan.check_device()


@pytest.mark.parametrize("r,n", [(1, 1), (3, 127), (16, 129), (17, 5), (32, 258), (33, 131),
                                 (48, 64), (49, 130), (64, 386), (64, 1023)])
def test_gram_and_garbage_h_shapes(cuda, oracle, r, n):
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.labrador import compute_garbage_g, compute_garbage_h
    plan, P = TwistedNttPlan(Q, 64), oracle.Plan(Q, 64)
    S, Phi = _words(Q, (r, n, 64), r), _words(Q, (r, n, 64), n + 1)
    assert np.array_equal(_host(compute_garbage_g(plan, _dev(S, cuda))).reshape(-1),
                          P.gram(S, r, n, threads=0))
    assert np.array_equal(
        _host(compute_garbage_h(plan, _dev(S, cuda), _dev(Phi, cuda))).reshape(-1),
        P.garbage_h(S, Phi, r, n).reshape(-1))
    plan.check_device()


def test_matrix_views_of_any_length(cuda, oracle):
    """A column view's length need not be a multiple of four, its row stride is the
    owning matrix's."""
    import torch
    from lattica_b200 import TwistedNttPlan, _lib
    from lattica_b200.commit import PreparedMatrix
    plan, P, lib = TwistedNttPlan(Q, 64), oracle.Plan(Q, 64), _lib.load()
    rows, cols = 8, 333
    A = _words(Q, (rows, cols, 64), 3)
    M = PreparedMatrix(plan, _dev(A, cuda), rows, cols)
    for n in (130, 131, 333):
        h, nb = C.c_void_p(), C.c_size_t()
        assert lib.grid_gpu_matrix_view(M.handle, n, C.byref(h)) == 0
        lib.grid_gpu_commit_workspace(h, 1, C.byref(nb))
        s = _words(Q, (1, n, 64), n)
        ds, t = _dev(s, cuda), torch.empty((rows, 64), dtype=torch.int32, device=cuda)
        ws = torch.empty(nb.value, dtype=torch.uint8, device=cuda)
        assert lib.grid_gpu_commit_dev(h, ds.data_ptr(), 1, t.data_ptr(), ws.data_ptr(),
                                       ws.numel(), torch.cuda.current_stream().cuda_stream) == 0
        want = P.matvec(np.ascontiguousarray(A[:, :n]), rows, n, s, 1).reshape(rows, 64)
        assert np.array_equal(_host(t), want)
        lib.grid_gpu_matrix_destroy(h)
    plan.check_device()


def test_gram_in_the_least_workspace(cuda, oracle):
    """Rows that are no whole 16-byte units want a slightly larger workspace; in one
    that only holds the plain rows the Gram still runs."""
    import torch
    from lattica_b200 import TwistedNttPlan, _lib
    plan, P, lib = TwistedNttPlan(Q, 64), oracle.Plan(Q, 64), _lib.load()
    r, n = 7, 1021
    S = _words(Q, (r, n, 64), 1)
    dS, nb = _dev(S, cuda), C.c_size_t()
    lib.grid_gpu_gram_workspace(plan.handle, r, n, C.byref(nb))
    want = P.gram(S, r, n, threads=0)
    for less in (0, r * 3 * 64 * 4):
        G = torch.empty((r * (r + 1) // 2, 64), dtype=torch.int32, device=cuda)
        ws = torch.empty(nb.value - less, dtype=torch.uint8, device=cuda)
        assert lib.grid_gpu_gram_dev(plan.handle, dS.data_ptr(), r, n, G.data_ptr(), ws.data_ptr(),
                                     ws.numel(), torch.cuda.current_stream().cuda_stream) == 0
        assert np.array_equal(_host(G).reshape(-1), want)
    plan.check_device()
