"""The quotients, reciprocals and roots that the factorisation kernels form by
their own iterations, in ulps against correctly rounded ones over the exponent
range, at the limits of the iterations' ranges too."""
import numpy as np
import pytest

from tests._gpu import need_gpu

pytestmark = pytest.mark.gpu


def _values(rng, lo, hi, count):
    """Mantissas near 1, near 2, short and random ones at exponents lo .. hi, the
    fields 64 and 1980 (where the iterations begin and end) among them."""
    m = 1.0 + rng.random(count)
    m[::7] = 1.0 + np.ldexp(rng.integers(0, 8, m[::7].size).astype(float), -52)
    m[1::7] = 2.0 - np.ldexp(rng.integers(1, 8, m[1::7].size).astype(float), -52)
    m[2::7] = 1.0 + rng.integers(0, 8, m[2::7].size) / 8.0
    e = rng.integers(lo, hi + 1, count)
    edge = [x for x in (62, 63, 64, 65, 1978, 1979, 1980, 1981) if lo <= x - 1023 <= hi]
    if edge:
        e[3::5] = np.resize(np.array(edge) - 1023, e[3::5].size)
    return np.where(rng.random(count) < 0.5, -1.0, 1.0) * np.ldexp(m, e)


def _ulps(x, ref):
    return np.abs(x - ref) / np.spacing(np.abs(ref))


def test_reciprocals_of_pivots():
    """The multiplier l / d of [[d, 1], [l, 1]] for powers of two l <= |d| is the
    reciprocal, scaled: the approximation's error and one rounding."""
    need_gpu()
    import torch
    from sslablu_gb300 import _lib as L
    rng = np.random.default_rng(0)
    d = _values(rng, -1020, 1020, 60000)
    l = np.ldexp(1.0, np.frexp(d)[1] - 1)
    A = np.ones((d.size, 2, 2))
    A[:, 0, 0], A[:, 1, 0] = d, l
    D = torch.from_numpy(A).cuda()
    piv = torch.empty((d.size, 2), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    L.check(L.lib().slu_lu_factor(L.handle(), 2, L.ptr(D), 2, 4, L.ptr(piv), 2, d.size, None))
    L.sync()
    keep = (piv[:, 0] == 0).cpu().numpy()      # (d = -l: a tie, the first row)
    assert keep.all()
    assert _ulps(D[:, 1, 0].cpu().numpy(), l / d).max() <= 1.0


def _operator(D):
    from sslablu_gb300.matAssembly.HBS.HBSnew import HBSMAT
    H = HBSMAT()
    H.set_mats([], [D], [], [1], fac=2)
    H.compute_ULV()
    return H


def test_quotients_of_triangular_solves():
    """Blocks [[d, u], [0, 1]] are their own QR; the solution for the second unit
    vector holds -u / d, for the first 1 / d."""
    need_gpu()
    rng = np.random.default_rng(1)
    for n in (64, 126):
        for lo, hi, ulo, uhi in ((-1020, 1020, 0, 0), (-500, 500, -500, 500), (-962, -958, -3, 60),
                                 (955, 960, -60, 3), (-3, 3, -1020, -950), (-3, 3, 940, 1000)):
            d, u = _values(rng, lo, hi, n // 2), _values(rng, ulo, uhi, n // 2)
            D = np.eye(n)
            i = np.arange(0, n, 2)
            D[i, i], D[i, i + 1] = d, u
            H = _operator(D)
            x = H.solve(np.eye(n))
            q, r = x[i, i + 1], x[i, i]
            with np.errstate(over="ignore", under="ignore"):
                want = -u / d
            ok = np.isfinite(want) & (np.abs(want) > 2.0 ** -1021)
            assert _ulps(q[ok], want[ok]).max() <= 1.0
            assert _ulps(r, 1.0 / d).max() <= 1.0


@pytest.mark.parametrize("e", [-500, -460, -440, -100, 0, 100, 440, 460, 480])
def test_reflectors(e):
    """Columns (a, b): the new diagonal is the norm to 4 u (u for each of: the sum
    of squares, halved by the root; the inverse root and its last step; their
    product), and the reflectors are orthogonal to 8 u."""
    need_gpu()
    rng = np.random.default_rng(2)
    n = 64
    D = np.zeros((n, n))
    i = np.arange(0, n, 2)
    a, b = _values(rng, -8, 8, n // 2), _values(rng, -8, 8, n // 2)
    D[i, i], D[i + 1, i], D[i + 1, i + 1] = np.ldexp(a, e), np.ldexp(b, e), 1.0
    H = _operator(D)
    R, Q = H.Rlist[0], H.Qlist[0]
    exact = np.sqrt(a.astype(np.longdouble) ** 2 + b.astype(np.longdouble) ** 2)
    got = np.ldexp(R[i, i], -e)
    assert (np.sign(got) == -np.sign(a)).all()
    assert float(np.abs(np.abs(got) / exact - 1).max()) <= 4 * 2.0 ** -53
    assert np.abs(Q.T @ Q - np.eye(n)).max() <= 8 * 2.0 ** -53
