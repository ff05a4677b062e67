"""Batched LU (csrc/lu.cu) at the edges of its panels, outer blocks and
clusters, against LAPACK's pivots and the rounding bound of its own factors."""
import numpy as np
import pytest
import scipy.linalg as sl

from tests._gpu import need_gpu

pytestmark = pytest.mark.gpu


def _factor(A, pad=3):
    """(LU, piv, info) of a batch (nb, n, n) with rows padded by `pad`."""
    import torch
    from sslablu_gb300 import _lib as L
    nb, n, _ = A.shape
    lda = n + pad
    D = torch.full((nb, n, lda), 7.0, dtype=torch.float64, device="cuda")
    D[:, :, :n] = torch.from_numpy(A).cuda()
    piv = torch.empty((nb, n), dtype=torch.int32, device="cuda")
    info = torch.zeros(nb, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    L.check(L.lib().slu_lu_factor(L.handle(), n, L.ptr(D), lda, n * lda, L.ptr(piv), n, nb,
                                  L.ptr(info)))
    L.sync()
    assert bool((D[:, :, n:] == 7.0).all())
    return D[:, :, :n].cpu().numpy(), piv.cpu().numpy(), info.cpu().numpy()


def _check(A, LU, piv):
    """||P A - L U|| within the bound 2 n u |L||U| (Higham, thm 9.3), doubled."""
    n = A.shape[0]
    P = A.copy()
    for i, p in enumerate(piv):
        P[[i, p]] = P[[p, i]]
    Lm, U = np.tril(LU, -1) + np.eye(n), np.triu(LU)
    assert np.abs(np.tril(LU, -1)).max(initial=0.0) <= 1.0
    assert np.linalg.norm(P - Lm @ U) <= 4 * n * 1.2e-16 * np.linalg.norm(np.abs(Lm) @ np.abs(U))


@pytest.mark.parametrize("n,nb", [(1, 2), (2, 1), (31, 3), (32, 1), (33, 2), (64, 9), (127, 2),
                                  (128, 1), (129, 3), (160, 1), (257, 2), (513, 3), (700, 1),
                                  (1025, 2), (2080, 1)])
def test_matches_lapack(n, nb):
    need_gpu()
    A = np.random.default_rng(n).standard_normal((nb, n, n))
    LU, piv, info = _factor(A)
    assert not info.any()
    for a, lu, p in zip(A, LU, piv):
        assert np.array_equal(p, sl.lu_factor(a)[1])
        _check(a, lu, p)


@pytest.mark.parametrize("n,col", [(40, 0), (129, 35), (300, 299), (300, 140)])
def test_zero_columns_and_ties(n, col):
    """A zero pivot is reported (first one) and passed over; of equal entries
    the first row is taken."""
    need_gpu()
    rng = np.random.default_rng(n + col)
    A = rng.standard_normal((2, n, n))
    A[0, :, col] = 0.0
    A[1] = np.sign(A[1])        # entries +-1: ties in the first column
    LU, piv, info = _factor(A)
    assert info[0] == col + 1
    _check(A[0], LU[0], piv[0])
    _check(A[1], LU[1], piv[1])
    assert piv[1, 0] == 0


def test_nan_column_keeps_the_earlier_ones():
    need_gpu()
    n = 150
    A = np.random.default_rng(5).standard_normal((2, n, n))
    ref = _factor(A)
    A[0, :, 70] = np.nan
    LU, piv, _ = _factor(A)
    # rows 0 .. 69 are final before column 70 (later swaps move the rows below)
    assert np.array_equal(LU[0, :70, :64], ref[0][0, :70, :64]) and np.isnan(LU[0, 100, 100])
    assert np.array_equal(piv[0, :70], ref[1][0, :70]) and piv[0, 70] == 70
    assert np.array_equal(LU[1], ref[0][1])
