"""The SVDs of a compression at their edges: block sizes between the kernel's
row and lane counts, zero and rank-deficient couplings (orthonormal bases all
the same), ranks up to the block size."""
import numpy as np
import pytest

from tests._gpu import need_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(5, 2), (16, 4), (17, 17), (33, 11), (36, 20), (40, 8), (48, 24),
                                 (57, 19), (64, 32), (65, 21), (80, 20), (100, 30), (128, 40),
                                 (131, 16), (160, 48)])
@pytest.mark.parametrize("rank", ["zero", "low", "full"])
def test_two_level_compression(n, k, rank):
    """A 2 x 2 block operator whose off-diagonal blocks have rank 0, about
    k / 3 or k: the compressed operator is exact to rounding, and every U and
    V block has orthonormal columns."""
    need_gpu()
    import torch
    from sslablu_gb300.matAssembly.HBS.HBSnew import HBSMAT, samples_for
    q = {"zero": 0, "low": max(1, k // 3), "full": k}[rank]
    rng = np.random.default_rng(100 * n + q)
    A = np.zeros((2 * n, 2 * n))
    for b in range(2):
        rows, cols = slice(b * n, (b + 1) * n), slice((1 - b) * n, (2 - b) * n)
        A[rows, rows] = rng.standard_normal((n, n)) if rank != "zero" else 0.0
        if q:
            A[rows, cols] = rng.standard_normal((n, q)) @ rng.standard_normal((q, n))
    H = HBSMAT(A, None, False)
    H.set_Nbvec([2, 1])
    H.Nbvec = []
    s = samples_for(k, n, 2)
    Om, Psi = rng.standard_normal((2 * n, s)), rng.standard_normal((2 * n, s))
    H.compress_from_sketches(k, Om, Psi, A @ Om, A.T @ Psi, compute_ULV=False)
    for F in (H.Umats[0], H.Vmats[0]):
        for b in range(2):
            Fb = F[b * n:(b + 1) * n]
            # Gram matrix of k columns, each rounded: k eps times a small factor
            assert np.abs(Fb.T @ Fb - np.eye(k)).max() <= 2e-15 * (n + 4 * k)
    X = torch.from_numpy(rng.standard_normal((2 * n, 3))).cuda()
    got = H.matmat(X).cpu().numpy()
    ref = A @ X.cpu().numpy()
    # the pseudo-inverses of the n x s Gaussian sketch blocks (s >= 2 n) have
    # condition numbers below 20; n roundings each
    assert np.linalg.norm(got - ref) <= 1e-13 * n * max(np.linalg.norm(ref), np.finfo(float).tiny)
    assert np.isfinite(got).all()
