"""A singular pivot block is reported as such whichever block it is."""
import numpy as np
import pytest

from tests._gpu import need_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver,m,nblk,block", [("rb", 5, 4, 1), ("rb", 40, 4, 2), ("rb", 5, 128, 64),
                                                 ("rb", 5, 128, 127), ("thomas", 40, 3, 2)])
def test_zero_pivot_in_any_block(solver, m, nblk, block):
    need_gpu()
    from sslablu_gb300 import _lib as L
    from sslablu_gb300.direct_solve.omsdirectsolve import BlockTridiagonalSolver, RedBlackSolver
    make = RedBlackSolver if solver == "rb" else BlockTridiagonalSolver
    Z = np.zeros((m, m))
    T = [np.eye(m)] * nblk
    S = [[Z, Z]] * nblk
    ok = make(m)
    ok.factorize(S, T)
    T = list(T)
    T[block] = np.diag([0.0] + [1.0] * (m - 1))
    with pytest.raises(L.SluError) as e:
        make(m).factorize(S, T)
    assert e.value.code == 6 and "zero pivot" in str(e.value)
    make(m).factorize(S, [np.eye(m)] * nblk)     # the status is cleared
    x = np.random.default_rng(0).standard_normal((m * nblk, 2))
    np.testing.assert_allclose(ok.solve(x), x, rtol=1e-14)


def test_one_status_word_per_matrix():
    need_gpu()
    import torch
    from sslablu_gb300 import _lib as L
    nb, n = 70, 6
    A = torch.eye(n, dtype=torch.float64, device="cuda").repeat(nb, 1, 1)
    A[33, 4, 4] = 0.0
    A[69, 0, 0] = 0.0
    piv = torch.empty((nb, n), dtype=torch.int32, device="cuda")
    info = torch.zeros(nb + 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    L.check(L.lib().slu_lu_factor(L.handle(), n, L.ptr(A), n, n * n, L.ptr(piv), n, nb, L.ptr(info)))
    L.sync()
    want = np.zeros(nb + 1, dtype=np.int32)
    want[33], want[69] = 5, 1
    np.testing.assert_array_equal(info.cpu().numpy(), want)
