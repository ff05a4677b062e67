"""Float64 products with few outputs (csrc/kernels_dense.cu), exact on integers."""
import numpy as np
import pytest

from tests._gpu import need_gpu

pytestmark = pytest.mark.gpu


# tiles of 8 x 16, 16 x 16 and 32 x 32, steps of 32 deep, remainders of all
@pytest.mark.parametrize("nb,M,N,K", [(1, 1, 17, 1), (1, 8, 32, 32), (2, 9, 33, 31), (1, 65, 70, 33),
                                      (1, 200, 96, 32), (3, 100, 50, 65), (1, 230, 210, 64),
                                      (4, 31, 20, 130), (9, 128, 33, 20), (2, 7, 5, 300)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_exact_on_integers(nb, M, N, K, ta, tb):
    need_gpu()
    import torch
    from sslablu_gb300 import _lib as L
    assert 2.0 * nb * M * N * K < 2.0e7   # the float64 units, not the residue products
    rng = np.random.default_rng(M + N + K)
    A, B = rng.integers(-999, 999, (nb, M, K)), rng.integers(-999, 999, (nb, K, N))
    C0 = rng.integers(-999, 999, (nb, M, N))

    def dev(x, t):
        return torch.from_numpy(np.ascontiguousarray(x.swapaxes(1, 2) if t else x).astype(float)).cuda()
    for alpha, beta in ((1.0, 0.0), (-1.0, 1.0), (2.0, -3.0)):
        a, b = dev(A, ta), dev(B, tb)
        c = dev(C0, 0) if beta else torch.full((nb, M, N), float("nan"), dtype=torch.float64).cuda()
        L.check(L.lib().slu_gemm_batched(L.handle(), ta, tb, M, N, K, alpha, L.ptr(a), a.shape[2],
                                         M * K, L.ptr(b), b.shape[2], K * N, beta, L.ptr(c), N,
                                         M * N, nb))
        L.sync()
        want = alpha * (A @ B) + (beta * C0 if beta else 0)
        np.testing.assert_array_equal(c.cpu().numpy(), want)
