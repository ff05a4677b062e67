"""Batched LU of more rows than a cluster's registers hold (4096): the first
panels in global memory, the rest by clusters."""
import numpy as np
import pytest
import scipy.linalg as sl

from tests._gpu import need_gpu
from tests.test_gpu_lu_edges import _check, _factor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4128, 4161])
def test_first_panels_in_global_memory(n):
    need_gpu()
    A = np.random.default_rng(n).standard_normal((1, n, n))
    if n % 2:
        A[0, :, 20] = 0.0      # a zero pivot in such a panel
    LU, piv, info = _factor(A)
    assert info[0] == (21 if n % 2 else 0)
    if n % 2 == 0:
        assert np.array_equal(piv[0], sl.lu_factor(A[0])[1])
    _check(A[0], LU[0], piv[0])
