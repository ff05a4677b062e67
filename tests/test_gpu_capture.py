"""Dense products, LU factors and solves captured into CUDA graphs: the graph has
scratch of its own, whatever the handle's does meanwhile."""
import numpy as np
import pytest

from tests._gpu import need_gpu, own_stream

pytestmark = pytest.mark.gpu


def _gemm(A, B, C):
    from sslablu_gb300 import _lib as L
    nb, M, K = A.shape
    N = B.shape[2]
    L.check(L.lib().slu_gemm_batched(L.handle(), 0, 0, M, N, K, 1.0, L.ptr(A), K, M * K, L.ptr(B), N,
                                     K * N, 0.0, L.ptr(C), N, M * N, nb))


def _lu(A, piv):
    from sslablu_gb300 import _lib as L
    nb, n, _ = A.shape
    L.check(L.lib().slu_lu_factor(L.handle(), n, L.ptr(A), n, n * n, L.ptr(piv), n, nb, None))


def test_products_and_factors_in_a_graph():
    need_gpu()
    import torch
    from sslablu_gb300 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(0)

    def rand(*s):
        return torch.randn(s, generator=g, dtype=torch.float64, device="cuda")
    A, B, P = rand(2, 256, 320), rand(2, 320, 256), rand(3, 300, 300)
    C, F = torch.empty((2, 256, 256), dtype=torch.float64, device="cuda"), torch.empty_like(P)
    piv = torch.empty((3, 300), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    s = own_stream()
    with torch.cuda.stream(s):
        L.sync()          # the handle of the stream exists; its scratch does not
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            _gemm(A, B, C)
            F.copy_(P)
            _lu(F, piv)
        for i in range(3):
            A.copy_(rand(2, 256, 320))
            P.copy_(rand(3, 300, 300))
            graph.replay()
            C1, F1, p1 = C.clone(), F.clone(), piv.clone()
            # the same calls, then larger ones, on the handle's scratch
            _gemm(A, B, C)
            F.copy_(P)
            _lu(F, piv)
            s.synchronize()
            assert torch.equal(C, C1) and torch.equal(F, F1) and torch.equal(piv, p1)
            X = rand(2 + i, 512, 512)
            Y = torch.empty_like(X)
            _gemm(X, X, Y)
            L.sync()
            ref = X[0, :2] @ X[0]
            assert float((Y[0, :2] - ref).abs().max()) < 1e-11 * float(ref.abs().max())


def test_block_solves_in_a_graph():
    need_gpu()
    import torch
    from sslablu_gb300 import _lib as L
    from sslablu_gb300.direct_solve.omsdirectsolve import RedBlackSolver
    m, nblk = 300, 4
    rng = np.random.default_rng(2)
    Z = np.zeros((m, m))
    S = [[0.2 / np.sqrt(m) * rng.standard_normal((m, m)) if i else Z,
          0.2 / np.sqrt(m) * rng.standard_normal((m, m)) if i < nblk - 1 else Z] for i in range(nblk)]
    rb = RedBlackSolver(m)
    rb.factorize(S, None)
    s = own_stream()
    with torch.cuda.stream(s):
        B = torch.from_numpy(rng.standard_normal((m * nblk, 64))).cuda()
        X = B.clone()
        rb._solve_dev(X)          # the solve's vectors exist before the capture
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            X.copy_(B)
            rb._solve_dev(X)
        for n in (256, 512):
            B.copy_(torch.from_numpy(rng.standard_normal((m * nblk, 64))))
            graph.replay()
            got = X.clone()
            X.copy_(B)
            rb._solve_dev(X)
            s.synchronize()
            assert torch.equal(got, X)
            Q = torch.randn((4, n, n), dtype=torch.float64, device="cuda")
            _gemm(Q, Q, torch.empty_like(Q))
            L.sync()
