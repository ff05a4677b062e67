"""Solves and applies of many right-hand sides as exact residue products
(csrc/crt_step.cu) against the float64 steps, which have up to 32 columns."""
import numpy as np
import pytest

from tests._gpu import need_gpu

pytestmark = pytest.mark.gpu

TOL = 1e-12   # plain float64 path, as test_gpu_hbs


def _op(leaf, L, k, quad):
    from sslablu_gb300.matAssembly.HBS.HBSnew import HBSMAT
    from sslablu_gb300.synthetic import random_hbs_factors
    U, D, V, Nbvec = random_hbs_factors(k, leaf, L, quad=quad, rng=np.random.default_rng(3),
                                        shift=16.0)
    H = HBSMAT()
    H.set_mats(U, D, V, list(Nbvec), fac=4 if quad else 2)
    H.compute_ULV()
    return H, D[0].shape[0]


def _calls(H):
    return [lambda b: H.solve(b), lambda b: H.solve(b, mode="T"), H.matmat, H.rmatmat]


def _cols(f, B):
    import torch
    return torch.cat([f(B[:, j:j + 32].contiguous()) for j in range(0, B.shape[1], 32)], 1)


def _worst(a, b):
    return float(((a - b).norm(dim=0) / b.norm(dim=0)).max())


# every tile (32, 16 and 8 columns; 128, 64 and split rows), widths off the
# multiples of 16, leaves off the multiples of 8, ragged columns, four children
@pytest.mark.parametrize("leaf,L,k,quad,c", [(64, 7, 32, False, 49), (64, 5, 32, False, 300),
                                             (100, 4, 24, False, 301), (33, 7, 16, False, 300),
                                             (36, 4, 20, True, 290), (128, 4, 20, False, 200),
                                             (60, 5, 27, False, 333), (64, 2, 40, False, 2000)])
def test_matches_float64_steps(leaf, L, k, quad, c):
    need_gpu()
    import torch
    H, N = _op(leaf, L, k, quad)
    g = torch.Generator(device="cuda").manual_seed(1)
    B = torch.randn((N, c), generator=g, dtype=torch.float64, device="cuda")
    for f in _calls(H):
        assert _worst(f(B), _cols(f, B)) < TOL


def test_columns_are_independent():
    """A column's result does not depend on the tiles it falls in, scales with
    powers of two, and one that is not finite leaves the others alone."""
    need_gpu()
    import torch
    H, N = _op(64, 7, 32, False)
    g = torch.Generator(device="cuda").manual_seed(2)
    B = torch.randn((N, 300), generator=g, dtype=torch.float64, device="cuda")
    s = torch.ones(300, dtype=torch.float64, device="cuda")
    s[::3] = 2.0 ** 300
    s[1::3] = 2.0 ** -300
    for f in _calls(H):
        Y = f(B)
        for c in (65, 128):
            assert torch.equal(f(B[:, :c].contiguous()), Y[:, :c])
        assert torch.equal(f(B * s), Y * s)
        X = B.clone()
        X[5, 3] = float("inf")
        X[N - 1, 77] = float("nan")
        X[:, 150] = 0.0
        Z, R = f(X), _cols(f, X)
        assert torch.equal(torch.isfinite(Z), torch.isfinite(R))
        assert bool((Z[:, 150] == 0).all())
        keep = [j for j in range(300) if j not in (3, 77, 150)]
        assert torch.equal(Z[:, keep], Y[:, keep])


def test_plans_and_new_factors():
    """A plan's replay equals the call; a new factorisation makes new images."""
    need_gpu()
    import torch
    H, N = _op(64, 7, 32, False)
    g = torch.Generator(device="cuda").manual_seed(5)
    B = torch.randn((N, 100), generator=g, dtype=torch.float64, device="cuda")
    for mode in ("N", "T"):
        b = torch.empty_like(B)
        plan = H.solve_plan(b, mode=mode)
        for x in (B, 3.0 * B):
            b.copy_(x)
            y = plan()
            torch.cuda.synchronize()
            assert torch.equal(y, H.solve(x, mode=mode))
        plan.close()
    want = [f(B) for f in _calls(H)]
    H.compute_ULV()
    for f, w in zip(_calls(H), want):
        assert torch.equal(f(B), w)
