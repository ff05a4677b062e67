"""Opposed scales beside a row and a column that are not finite: those are float64
dot products whatever they hold, and must not vouch for the other outputs."""
import numpy as np
import pytest

from tests._gpu import need_gpu
from tests.test_gpu_crt_grading import _product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_opposed_scales_beside_infinities(value):
    need_gpu()
    nb, M, N, K = 6, 96, 130, 256
    rng = np.random.default_rng(9)
    d = 10.0 ** (-10 * np.arange(K) / (K - 1))
    A, B = rng.standard_normal((nb, M, K)) * d, rng.standard_normal((nb, K, N)) / d[:, None]
    A[:, 3], B[:, :, 7] = value, value
    got = _product(A, B)
    rows, cols = np.arange(M) != 3, np.arange(N) != 7
    A, B, got = A[:, rows], B[:, :, cols], got[:, rows][:, :, cols]
    s = np.abs(A) @ np.abs(B)
    err = np.abs(got - A.astype(np.longdouble) @ B.astype(np.longdouble)).astype(float)
    assert (err <= 32 * 4 * K * 2.0 ** -53 * s).all()
