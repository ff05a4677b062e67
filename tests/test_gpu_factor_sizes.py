"""HBS construction and ULV solves at block sizes around the edges of the small
triangular solves and panel kernels, against the dense matrix."""
import numpy as np
import pytest

from tests._gpu import need_gpu

pytestmark = pytest.mark.gpu


def _dense(U, D, V, Nbvec):
    A = D[-1]
    for t in range(len(D) - 2, -1, -1):
        nb, k = Nbvec[t], U[t].shape[1]
        n = D[t].shape[0] // nb
        B = np.zeros((nb * n, nb * n))
        for i in range(nb):
            for j in range(nb):
                b = U[t][i * n:(i + 1) * n] @ A[i * k:(i + 1) * k, j * k:(j + 1) * k] \
                    @ V[t][j * n:(j + 1) * n].T
                B[i * n:(i + 1) * n, j * n:(j + 1) * n] = b
            B[i * n:(i + 1) * n, i * n:(i + 1) * n] += D[t][i * n:(i + 1) * n]
        A = B
    return A


@pytest.mark.parametrize("leaf,k,L,c", [(9, 3, 3, 1), (33, 5, 3, 3), (40, 8, 3, 17), (64, 31, 2, 64),
                                        (65, 16, 3, 5), (128, 20, 2, 33), (131, 64, 2, 4),
                                        (140, 66, 3, 2)])
def test_ulv_solves(leaf, k, L, c):
    need_gpu()
    from sslablu_gb300.matAssembly.HBS.HBSnew import HBSMAT
    from sslablu_gb300.synthetic import random_hbs_factors
    rng = np.random.default_rng(leaf + k)
    U, D, V, Nbvec = random_hbs_factors(k, leaf, L, rng=rng, shift=4.0 * np.sqrt(leaf))
    A = _dense(U, D, V, Nbvec)
    H = HBSMAT()
    H.set_mats(U, D, V, list(Nbvec), fac=2)
    H.compute_ULV()
    b = rng.standard_normal((A.shape[0], c))
    for M, x in ((A, H.solve(b)), (A.T, H.solve(b, mode="T"))):
        # backward error of a backward stable solve: a modest multiple of n u
        r = np.linalg.norm(M @ x - b) / (np.linalg.norm(M, 2) * np.linalg.norm(x))
        assert r < 10 * A.shape[0] * 1.2e-16


@pytest.mark.parametrize("n,k", [(15, 5), (16, 5), (31, 9), (127, 30), (129, 30)])
def test_carried_columns(n, k):
    """Sketch panels either side of the sizes that take the compact WY form."""
    from tests.test_gpu_svd_edges import test_two_level_compression as check
    check(n, k, "full")


@pytest.mark.parametrize("leaf,k,L", [(48, 12, 5), (64, 32, 5), (100, 24, 2), (40, 20, 6)])
def test_compression_levels(leaf, k, L):
    """Compression from sketches at block counts that share panels and sweeps
    between eight, four, two or one CTAs."""
    need_gpu()
    import torch
    from sslablu_gb300.matAssembly.HBS.HBSnew import HBSMAT, samples_for
    from sslablu_gb300.synthetic import random_hbs_factors
    rng = np.random.default_rng(leaf * L + k)
    U, D, V, Nbvec = random_hbs_factors(k, leaf, L, rng=rng, shift=4.0 * np.sqrt(leaf))
    A = _dense(U, D, V, Nbvec)
    N, s = A.shape[0], samples_for(k, leaf, 2)
    H = HBSMAT(A, None, False)
    H.set_Nbvec(list(Nbvec))
    H.Nbvec = []
    Om, Psi = rng.standard_normal((N, s)), rng.standard_normal((N, s))
    H.compress_from_sketches(k, Om, Psi, A @ Om, A.T @ Psi, compute_ULV=True)
    X = rng.standard_normal((N, 3))
    got, ref = H.matmat(torch.from_numpy(X).cuda()).cpu().numpy(), A @ X
    # as the two-level compressions: condition numbers below 20, n roundings a level
    assert np.linalg.norm(got - ref) <= 1e-13 * leaf * L * np.linalg.norm(ref)
    x = H.solve(X)
    assert np.linalg.norm(A @ x - X) <= 1e-12 * leaf * L * np.linalg.norm(A, 2) * np.linalg.norm(x)
