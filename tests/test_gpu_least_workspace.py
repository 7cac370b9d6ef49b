"""Calls in less workspace than they ask for. The sizes here are what the gathering products
need on 148 SMs (evaluations of unpadded rows and their partials); the queries return more
where the point-major or the vector products want it. In the smaller workspace a call gives
the same words, and in one that holds not even those it is refused."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q, Q_RING = 4294966657, 4294967291


class Calls:
    def __init__(self, cuda, ring=False):
        import torch
        from lattica_b200 import TwistedNttPlan, _lib
        from lattica_b200.ntt import RingPlan
        self.torch, self.cuda, self.lib = torch, cuda, _lib.load()
        self.q = Q_RING if ring else Q
        self.plan = RingPlan(self.q, 64) if ring else TwistedNttPlan(self.q, 64)
        self.g = torch.Generator(device=cuda).manual_seed(11)
        self.st = torch.cuda.current_stream().cuda_stream

    def word(self, *shape):
        return self.torch.randint(0, self.q, shape, dtype=self.torch.int64, device=self.cuda,
                                  generator=self.g).to(self.torch.int32)

    def matrix(self, rows, cols):
        from lattica_b200.commit import PreparedMatrix
        return PreparedMatrix(self.plan, self.word(rows, cols, 64), rows, cols)

    def same_in(self, query, call, least, *outs):
        """call(ws pointer, bytes) in the workspace the query asks for and in `least` bytes."""
        nb = C.c_size_t()
        assert query(C.byref(nb)) == 0
        results = []
        for size in (nb.value, least):
            ws = self.torch.empty(size + 256, dtype=self.torch.uint8, device=self.cuda)
            for o in outs:
                o.fill_(-1)
            assert call(ws.data_ptr(), size) == 0
            results.append([o.clone() for o in outs])
        assert all(self.torch.equal(a, b) for a, b in zip(*results))
        assert not any(bool((o == -1).all()) for o in outs)
        ws = self.torch.empty(256, dtype=self.torch.uint8, device=self.cuda)
        if least > 512:
            assert call(ws.data_ptr(), 256) == 5  # GRID_ERR_INVALID_PARAMETERS
        self.plan.check_device()


@pytest.mark.parametrize("rows,cols,batch,least", [(64, 4096, 1, 1654784), (16, 8320, 1, 2727936),
                                                   (17, 515, 2, 402944), (9, 1021, 16, 4476928),
                                                   (48, 515, 64, 11583488), (64, 129, 5, 328960)])
def test_commit(cuda, rows, cols, batch, least):
    c = Calls(cuda)
    M, s = c.matrix(rows, cols), c.word(batch, cols, 64)
    t = c.word(batch, rows, 64)
    c.same_in(lambda nb: c.lib.grid_gpu_commit_workspace(M.handle, batch, nb),
              lambda ws, n: c.lib.grid_gpu_commit_dev(M.handle, s.data_ptr(), batch, t.data_ptr(),
                                                      ws, n, c.st), least, t)


@pytest.mark.parametrize("rows,mc,oc,batch,least", [(64, 4096, 4096, 1, 2 * 1654784 + 16384),
                                                    (17, 515, 515, 2, 2 * 402944 + 8704),
                                                    (9, 1021, 1021, 16, 2 * 4476928 + 36864)])
def test_linear_and_bdlop(cuda, rows, mc, oc, batch, least):
    c = Calls(cuda)
    A, B, K = c.matrix(rows, mc), c.matrix(rows, oc), c.matrix(rows, oc)
    m, r = c.word(batch, mc, 64), c.word(batch, oc, 64)
    t, u = c.word(batch, rows, 64), c.word(batch, rows, 64)
    c.same_in(lambda nb: c.lib.grid_gpu_linear_commit_workspace(A.handle, B.handle, batch, nb),
              lambda ws, n: c.lib.grid_gpu_linear_commit_dev(
                  A.handle, B.handle, m.data_ptr(), r.data_ptr(), batch, t.data_ptr(), ws, n, c.st),
              least, t)
    c.same_in(lambda nb: c.lib.grid_gpu_bdlop_workspace(K.handle, A.handle, B.handle, batch, nb),
              lambda ws, n: c.lib.grid_gpu_bdlop_commit_dev(
                  K.handle, A.handle, B.handle, m.data_ptr(), r.data_ptr(), batch, u.data_ptr(),
                  t.data_ptr(), ws, n, c.st), least, u, t)


@pytest.mark.parametrize("ring,r,n,gram,garbage", [
    (False, 64, 1, 16384, 1081344), (False, 30, 1, 7680, 245760),
    (False, 33, 257, 2601984, 5457408), (False, 64, 1021, 18857984, 38699008),
    (True, 17, 5, 139264, 339456), (True, 64, 129, 4775936, 10518528)])
def test_gram_and_garbage_h(cuda, ring, r, n, gram, garbage):
    c = Calls(cuda, ring)
    S, Phi, out = c.word(r, n, 64), c.word(r, n, 64), c.word(r * (r + 1) // 2, 64)
    c.same_in(lambda nb: c.lib.grid_gpu_gram_workspace(c.plan.handle, r, n, nb),
              lambda ws, b: c.lib.grid_gpu_gram_dev(c.plan.handle, S.data_ptr(), r, n,
                                                    out.data_ptr(), ws, b, c.st), gram, out)
    c.same_in(lambda nb: c.lib.grid_gpu_garbage_h_workspace(c.plan.handle, r, n, nb),
              lambda ws, b: c.lib.grid_gpu_garbage_h_dev(c.plan.handle, S.data_ptr(),
                                                         Phi.data_ptr(), r, n, out.data_ptr(), ws,
                                                         b, c.st), garbage, out)


@pytest.mark.parametrize("kappa,r,n,least", [(1, 17, 129, 648192), (16, 64, 129, 3444736),
                                             (9, 30, 1021, 8467456), (16, 33, 515, 5300992)])
def test_round(cuda, kappa, r, n, least):
    c = Calls(cuda)
    A, S = c.matrix(kappa, n), c.word(r, n, 64)
    pairs = r * (r + 1) // 2
    t, g, gl = c.word(r * kappa * 4, 64), c.word(pairs, 64), c.word(pairs * 4, 64)
    p, seed = c.word(256), (C.c_uint8 * 32).from_buffer_copy(bytes(range(32)))
    c.same_in(lambda nb: c.lib.grid_gpu_prover_round_workspace(A.handle, r, 256, nb),
              lambda ws, b: c.lib.grid_gpu_prover_round_dev(
                  A.handle, S.data_ptr(), r, 256, 4, 256, 4, seed, 256, t.data_ptr(), g.data_ptr(),
                  gl.data_ptr(), p.data_ptr(), None, ws, b, c.st), least, t, g, gl, p)


def test_workspace_of_a_longer_view(cuda):
    """One workspace for all column views of a matrix, sized for the longest."""
    c = Calls(cuda)
    M, nb = c.matrix(1, 19000), C.c_size_t()
    assert c.lib.grid_gpu_commit_workspace(M.handle, 1, C.byref(nb)) == 0
    ws = c.torch.empty(nb.value, dtype=c.torch.uint8, device=cuda)
    t, s = c.word(2, 64), c.word(19000, 64)
    view = C.c_void_p()
    assert c.lib.grid_gpu_matrix_view(M.handle, 4096, C.byref(view)) == 0
    big = c.torch.empty(1 << 24, dtype=c.torch.uint8, device=cuda)
    for out, w in zip(t, (big, ws)):
        assert c.lib.grid_gpu_commit_dev(view, s.data_ptr(), 1, out.data_ptr(), w.data_ptr(),
                                         w.numel(), c.st) == 0
    assert c.torch.equal(t[0], t[1])
    c.lib.grid_gpu_matrix_destroy(view)
    c.plan.check_device()
