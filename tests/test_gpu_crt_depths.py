"""Residue products of depth eight and less (csrc/crt.cuh: scaled operands have
at most 59 bits): trees of rank 1 to 4, whose upper steps are that narrow, and
dense products whose last slice is."""
import numpy as np
import pytest

from tests._gpu import need_gpu
from tests.test_gpu_crt_steps import TOL, _calls, _cols, _op, _worst
from tests.test_gpu_gemm_f64 import _gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf,L,k,quad,c", [(100, 6, 4, False, 128), (64, 7, 4, False, 300),
                                             (64, 7, 3, False, 600), (100, 6, 2, False, 400),
                                             (64, 8, 1, False, 600), (100, 4, 2, True, 300),
                                             (64, 5, 1, True, 300)])
def test_low_rank_trees(leaf, L, k, quad, c):
    need_gpu()
    import torch
    H, N = _op(leaf, L, k, quad)
    g = torch.Generator(device="cuda").manual_seed(k)
    B = torch.randn((N, c), generator=g, dtype=torch.float64, device="cuda")
    for f in _calls(H):
        assert _worst(f(B), _cols(f, B)) < TOL


@pytest.mark.parametrize("K", [8193, 8196, 8200, 16385])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 1)])
def test_short_last_slice(K, ta, tb):
    """Integers whose products and partial sums a float64 holds: exact."""
    need_gpu()
    import torch
    M, N = 64, 48
    rng = np.random.default_rng(K)
    A, B = rng.integers(-2**19, 2**19, (1, M, K)), rng.integers(-2**19, 2**19, (1, K, N))
    A[0, :, 8192:] = -np.abs(A[0, :, 8192:])

    def dev(x, t):
        return torch.from_numpy(np.ascontiguousarray(x.swapaxes(1, 2) if t else x).astype(float)).cuda()
    C = torch.empty((1, M, N), dtype=torch.float64, device="cuda")
    got = _gemm(dev(A, ta), dev(B, tb), C, ta, tb, 1.0, 0.0).cpu().numpy()
    np.testing.assert_array_equal(got, (A @ B).astype(float))
