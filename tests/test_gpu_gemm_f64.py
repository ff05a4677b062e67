"""Float64 products on the tensor cores (crt_gemm.cu) against exact products.

Inputs are integers times powers of two whose products and sums a 64-bit
integer holds, so the reference is exact and the result, which rounds once,
must equal it; Gaussian inputs are held to the bound of the rounding of the
inputs, K 2^-(t+1) (|a|_max |b|_max) with t >= 54 at the depths used."""
import numpy as np
import pytest

from tests._gpu import need_gpu

pytestmark = pytest.mark.gpu


def _gemm(A, B, C, ta, tb, alpha, beta):
    import torch
    from sslablu_gb300 import _lib as L
    nb = C.shape[0]
    M, N = C.shape[1:]
    K = A.shape[1] if ta else A.shape[2]
    L.check(L.lib().slu_gemm_batched(L.handle(), int(ta), int(tb), M, N, K, alpha, L.ptr(A),
                                     A.shape[2], A[0].numel(), L.ptr(B), B.shape[2],
                                     B[0].numel(), beta, L.ptr(C), N, C[0].numel(), nb))
    L.sync()
    return C


# tile edges (128 rows, 16 and 256 columns, 64 and 1024 deep), remainders,
# several chunks of depth, both orientations of both operands
SHAPES = [(1, 64, 2600, 64, 0, 0), (2, 128, 256, 256, 0, 1), (1, 129, 257, 320, 1, 0),
          (3, 333, 97, 385, 1, 1), (1, 200, 65, 1024, 0, 0), (1, 130, 72, 1153, 1, 0),
          (1, 257, 33, 4097, 0, 1), (5, 191, 47, 512, 0, 0), (1, 127, 49, 9000, 1, 1),
          (2, 300, 200, 100, 0, 0), (2, 210, 301, 113, 1, 1), (9, 177, 261, 64, 1, 1)]


@pytest.mark.parametrize("nb,M,N,K,ta,tb", SHAPES)
def test_integer_products_are_exact(nb, M, N, K, ta, tb):
    need_gpu()
    import torch
    assert 2.0 * nb * M * N * K >= 2.0e7
    rng = np.random.default_rng(M + N + K)
    # |sum| <= K 2^22 2^22 < 2^58; row and column scales are powers of two
    A = rng.integers(-2**22, 2**22, (nb, M, K))
    B = rng.integers(-2**22, 2**22, (nb, K, N))
    C0 = rng.integers(-2**20, 2**20, (nb, M, N))
    ref = A @ B - C0
    ra, cb = rng.integers(-40, 40, M), rng.integers(-40, 40, N)
    Af, Bf = np.ldexp(A.astype(float), ra[:, None]), np.ldexp(B.astype(float), cb[None, :])
    Cf = np.ldexp(C0.astype(float), ra[:, None] + cb[None, :])
    want = np.ldexp(ref.astype(float), ra[:, None] + cb[None, :])

    def dev(x, t):
        return torch.from_numpy(np.ascontiguousarray(x.swapaxes(1, 2) if t else x)).cuda()
    got = _gemm(dev(Af, ta), dev(Bf, tb), dev(Cf, 0), ta, tb, 1.0, -1.0).cpu().numpy()
    if K <= 8192:
        prod = np.ldexp((A @ B).astype(float), ra[:, None] + cb[None, :])
        np.testing.assert_array_equal(got, prod - Cf)   # the product and the update round once each
    else:   # accumulated in slices of the depth: one rounding per slice
        np.testing.assert_allclose(got, want, rtol=0, atol=2e-16 * float(np.abs(want).max()) * 3)


@pytest.mark.parametrize("nb,M,N,K,ta,tb", SHAPES[1:6] + SHAPES[9:])
def test_gaussian_products(nb, M, N, K, ta, tb):
    need_gpu()
    import torch
    rng = np.random.default_rng(K)
    A, B = rng.standard_normal((nb, M, K)), rng.standard_normal((nb, K, N))
    rows = np.arange(0, M, 17)
    ref = A[:, rows].astype(np.longdouble) @ B.astype(np.longdouble)
    At = torch.from_numpy(np.ascontiguousarray(A.swapaxes(1, 2) if ta else A)).cuda()
    Bt = torch.from_numpy(np.ascontiguousarray(B.swapaxes(1, 2) if tb else B)).cuda()
    C = torch.full((nb, M, N), float("nan"), dtype=torch.float64, device="cuda")
    got = _gemm(At, Bt, C, ta, tb, 1.0, 0.0).cpu().numpy()[:, rows]
    bound = K * 2.0 ** -54 * np.abs(A).max() * np.abs(B).max()
    assert float(np.abs(got - ref).max()) <= bound


def test_rows_that_are_not_finite():
    """An infinity or NaN in one row or column leaves every other element
    exact and gives the float64 product's infinities and NaN where it acts."""
    need_gpu()
    import torch
    rng = np.random.default_rng(5)
    A = rng.integers(-2**20, 2**20, (1, 192, 320)).astype(float)
    B = rng.integers(-2**20, 2**20, (1, 320, 256)).astype(float)
    A[0, 3, 5], A[0, 7, 1], B[0, 9, 200] = np.inf, np.nan, -np.inf
    A[0, 10], B[0, :, 11] = 0.0, 0.0
    A[0, 12] = np.ldexp(A[0, 12], -1070)     # subnormal results and inputs
    A[0, 13] = np.ldexp(A[0, 13], 960)
    with np.errstate(invalid="ignore"):
        want = A @ B
    C = torch.empty((1, 192, 256), dtype=torch.float64, device="cuda")
    got = _gemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C, 0, 0, 1.0, 0.0)
    np.testing.assert_array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("s", [-1, 1])
def test_residue_sums_at_their_limit(s):
    """Every residue product of one sign at its largest: the float32
    accumulators reach 2^24, where they are still exact."""
    need_gpu()
    import torch
    for e in (56, 55):
        A = torch.full((1, 128, 1024), 2.0 ** e, dtype=torch.float64, device="cuda")
        B = torch.full((1, 1024, 96), s * (2.0 ** e - 128 * (e == 55)), dtype=torch.float64,
                       device="cuda")
        C = torch.empty((1, 128, 96), dtype=torch.float64, device="cuda")
        _gemm(A, B, C, 0, 0, 1.0, 0.0)
        assert bool((C == s * 2.0 ** e * (2.0 ** e - 128 * (e == 55)) * 1024).all())


@pytest.mark.parametrize("nb,M,N,K,ta,tb", [(64, 32, 261, 64, 1, 0), (9, 33, 300, 129, 0, 0),
                                            (40, 63, 65, 70, 0, 1), (70, 47, 33, 100, 1, 1)])
def test_few_rows_are_exact(nb, M, N, K, ta, tb):
    test_integer_products_are_exact(nb, M, N, K, ta, tb)
