"""Every tile of the residue steps (csrc/crt_step.cu) against the float64 steps,
on shapes that are known to take them in the stated directions."""
import numpy as np
import pytest

from tests._gpu import need_gpu
from tests.test_gpu_crt_steps import TOL, _op, _worst
from tests.test_gpu_wide_calls import _wide

pytestmark = pytest.mark.gpu

# (solve N, solve T, apply N, apply T) by the residue steps.  Tiles of 32, 16 and
# 8 columns, of up to 128 and 64 rows and split ones, step depths up to 64 and 128,
# leaves and widths off the multiples of 8 and 16, ranks off them, four children
# (operators of two row tiles), two levels, few columns
CASES = [((64, 7, 32, False, 150), (1, 1, 1, 1)), ((64, 5, 32, False, 300), (1, 1, 1, 1)),
         ((100, 4, 24, False, 301), (1, 1, 1, 1)), ((33, 7, 16, False, 900), (1, 1, 1, 1)),
         ((36, 4, 20, True, 290), (1, 0, 1, 1)), ((60, 5, 27, False, 333), (1, 1, 1, 1)),
         ((128, 4, 20, False, 400), (0, 1, 0, 0)), ((64, 2, 40, False, 2000), (1, 0, 1, 1)),
         ((120, 2, 8, False, 1500), (1, 1, 1, 1)), ((96, 5, 32, False, 77), (1, 1, 0, 0)),
         ((41, 5, 13, True, 65), (1, 1, 0, 0)), ((100, 6, 28, False, 90), (1, 1, 1, 1)),
         ((40, 7, 20, False, 200), (1, 1, 0, 0)), ((64, 3, 32, False, 261), (0, 0, 0, 0))]


@pytest.mark.parametrize("shape,paths", CASES)
def test_residue_steps_match_float64_steps(shape, paths):
    need_gpu()
    import torch
    leaf, L, k, quad, c = shape
    H, N = _op(leaf, L, k, quad)
    taken = tuple(_wide(H, solve, trans, c) for solve in (1, 0) for trans in (0, 1))
    assert taken == paths
    g = torch.Generator(device="cuda").manual_seed(1)
    B = torch.randn((N, c), generator=g, dtype=torch.float64, device="cuda")
    for i, (f, trans) in enumerate([(H._dev_solve, False), (H._dev_solve, True),
                                    (H._dev_apply, False), (H._dev_apply, True)]):
        X, Y = f(B, trans), f(B, trans, wide=False)
        assert _worst(X, Y) < TOL
        # products that are rounded once never have all bits of an FMA chain
        assert torch.equal(X, Y) == (not paths[i])
