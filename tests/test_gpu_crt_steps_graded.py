"""Residue tree steps (csrc/crt_step.cu) on operators and right-hand sides whose
scales oppose, against the float64 steps (up to 32 columns)."""
import numpy as np
import pytest

from tests._gpu import need_gpu
from tests.test_gpu_crt_steps import TOL, _calls, _cols, _worst

pytestmark = pytest.mark.gpu


def _graded(leaf, L, k, quad, dr, dc):
    """diag(dr) A diag(dc) for a random HBS operator A in leaf order."""
    from sslablu_gb300.matAssembly.HBS.HBSnew import HBSMAT
    from sslablu_gb300.synthetic import random_hbs_factors
    U, D, V, Nbvec = random_hbs_factors(k, leaf, L, quad=quad, rng=np.random.default_rng(4),
                                        shift=16.0)
    U, D, V = list(U), list(D), list(V)
    U[0] = U[0] * dr[:, None]
    V[0] = V[0] * dc[:, None]
    D[0] = D[0] * dr[:, None] * dc.reshape(-1, 1, leaf).repeat(leaf, 1).reshape(-1, leaf)
    H = HBSMAT()
    H.set_mats(U, D, V, list(Nbvec), fac=4 if quad else 2)
    return H


@pytest.mark.parametrize("leaf,L,k,quad,c", [(64, 5, 32, False, 300), (36, 4, 20, True, 290),
                                             (100, 4, 24, False, 301)])
@pytest.mark.parametrize("decades", [6, 12, 100])
def test_scaled_columns_and_rows(leaf, L, k, quad, c, decades):
    """Products with diag(dr) A diag(dc), the vectors scaled by the inverse: what
    the factors 1/dr leave is A's own product, entry by entry."""
    need_gpu()
    import torch
    N = leaf * (4 if quad else 2) ** (L - 1)
    rng = np.random.default_rng(decades)
    dr, dc = (2.0 ** np.rint(-3.32 * decades * rng.random(N)) for _ in range(2))
    H = _graded(leaf, L, k, quad, dr, dc)
    g = torch.Generator(device="cuda").manual_seed(7)
    B = torch.randn((N, c), generator=g, dtype=torch.float64, device="cuda")
    r, q = (torch.from_numpy(d).cuda()[:, None] for d in (dr, dc))
    for f, left, right in ((H.matmat, r, q), (H.rmatmat, q, r)):
        X = B / right
        assert _worst(f(X) / left, _cols(f, X) / left) < TOL


@pytest.mark.parametrize("leaf,L,k,c", [(64, 5, 32, 300), (48, 6, 8, 900)])
def test_identity_operator(leaf, L, k, c):
    """An operator whose couplings are zero and whose blocks are the identity
    returns its vectors, entries of all sizes next to one another."""
    need_gpu()
    import torch
    from sslablu_gb300.matAssembly.HBS.HBSnew import HBSMAT
    from sslablu_gb300.synthetic import random_hbs_factors
    U, D, V, Nbvec = random_hbs_factors(k, leaf, L, rng=np.random.default_rng(4))
    D = [np.zeros_like(d) for d in D]
    D[0] = np.tile(np.eye(leaf), (D[0].shape[0] // leaf, 1))
    H = HBSMAT()
    H.set_mats(U, D, V, list(Nbvec), fac=2)
    N = D[0].shape[0]
    g = torch.Generator(device="cuda").manual_seed(8)
    B = torch.randn((N, c), generator=g, dtype=torch.float64, device="cuda")
    B[3::7] *= 1e20
    B[5::7] = 0.0
    for f in (H.matmat, H.rmatmat):
        # entries that are 1e20 below others in their block are exact, the rest
        # rounded at 2^-57 of the largest of the block's column
        Y = f(B)
        small = torch.ones(N, dtype=torch.bool)
        small[3::7] = False
        assert torch.equal(Y[small], B[small])
        big = B.abs().reshape(-1, leaf, c).amax(1, keepdim=True)
        assert bool(((Y - B).reshape(-1, leaf, c).abs() <= 2.0 ** -56 * big).all())


def test_not_finite_against_zero():
    """A NaN in the operator meets columns of zeros: NaN, as in float64."""
    need_gpu()
    import torch
    dr = np.ones(64 * 16)
    H = _graded(64, 5, 32, False, dr, dr)
    D = [np.array(d) for d in H.Dmats]
    D[0][100, 7] = np.nan
    H.set_mats(H.Umats, D, H.Vmats, [16, 8, 4, 2, 1], fac=2)
    B = torch.ones((64 * 16, 300), dtype=torch.float64, device="cuda")
    B[:, 5] = 0.0
    for f in (H.matmat, H.rmatmat):
        assert torch.equal(torch.isnan(f(B)), torch.isnan(_cols(f, B)))
