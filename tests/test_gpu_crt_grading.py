"""Residue products (csrc/crt_gemm.cu) whose operands' scales oppose along the
contraction, and the block solvers on row-graded pivot blocks, where a product
held to the largest entries of its rows and columns alone loses the digits."""
import numpy as np
import pytest

from tests._gpu import need_gpu
from tests.test_gpu_gemm_f64 import _gemm

pytestmark = pytest.mark.gpu


def _product(A, B, ta=0, tb=0):
    import torch

    def dev(x, t):
        return torch.from_numpy(np.ascontiguousarray(x.swapaxes(1, 2) if t else x)).cuda()
    C = torch.full((A.shape[0], A.shape[1], B.shape[2]), float("nan"), dtype=torch.float64,
                   device="cuda")
    return _gemm(dev(A, ta), dev(B, tb), C, ta, tb, 1.0, 0.0).cpu().numpy()


def _check(A, B, got):
    """|error| <= 4 K 2^-53 times the largest sum s = |A||B| of the row and of
    the column (both scaled by the columns' and rows' largest entries), the
    stated bound, and 4 K 2^-57 2^44 s for every output (operands of 55 bits or
    more); plus the last rounding."""
    K = A.shape[2]
    ref = A.astype(np.longdouble) @ B.astype(np.longdouble)
    s = np.abs(A) @ np.abs(B)
    a, b = np.abs(A).max(2, keepdims=True), np.abs(B).max(1, keepdims=True)
    with np.errstate(invalid="ignore", divide="ignore"):
        q = np.nan_to_num(s / (a * b))
    env = np.minimum(q.max(2, keepdims=True), q.max(1, keepdims=True)) * a * b
    err = np.abs(got - ref).astype(float)
    unit = 4 * K * 2.0 ** -53
    assert (err <= unit * env + 2.0 ** -52 * np.abs(ref).astype(float)).all()
    assert (err <= unit * 2.0 ** 40 * s).all()


SHAPES = [(20, 64, 128, 64, 0, 0), (6, 96, 130, 256, 1, 0), (5, 70, 50, 700, 0, 1),
          (3, 65, 66, 1200, 1, 1)]


@pytest.mark.parametrize("nb,M,N,K,ta,tb", SHAPES)
@pytest.mark.parametrize("decades", [0, 4, 8, 12, 200])
def test_opposed_scales(nb, M, N, K, ta, tb, decades):
    need_gpu()
    rng = np.random.default_rng(K + decades)
    d = 10.0 ** (-decades * rng.permutation(K) / (K - 1))
    A, B = rng.standard_normal((nb, M, K)) * d, rng.standard_normal((nb, K, N)) / d[:, None]
    got = _product(A, B, ta, tb)
    _check(A, B, got)
    # here every sum is that of Gaussian operands, within a factor of 32 of all others
    s = np.abs(A) @ np.abs(B)
    err = np.abs(got - A.astype(np.longdouble) @ B.astype(np.longdouble)).astype(float)
    assert (err <= 32 * 4 * K * 2.0 ** -53 * s).all()


@pytest.mark.parametrize("nb,M,N,K,ta,tb", SHAPES)
def test_few_outputs_below_the_rest(nb, M, N, K, ta, tb):
    """Sparse rows against graded columns: single outputs, whole rows and whole
    columns that need their own products."""
    need_gpu()
    rng = np.random.default_rng(K)
    A, B = rng.standard_normal((nb, M, K)), rng.standard_normal((nb, K, N))
    A[:, :M // 2] = 0.0
    for i in range(M // 2):
        A[:, i, i % K] = 1.0
    B[:, 0, ::3] = 1e20          # next to entries of order one in the same column
    B[:, 5] *= 1e-30             # a row that only row 5 of A takes alone
    A[:, M - 1] = 0.0            # products with a zero factor only
    A[:, M - 1, 7], B[:, 7] = 1.0, 0.0
    got = _product(A, B, ta, tb)
    _check(A, B, got)
    assert (got[:, M - 1] == 0.0).all()
    np.testing.assert_array_equal(got[:, 5], B[:, 5])


def test_identity_times_a_graded_column():
    need_gpu()
    A = np.tile(np.eye(64), (60, 1, 1))
    B = np.zeros((60, 64, 48))
    B[:, 0], B[:, 1] = 1e20, 1.0
    np.testing.assert_array_equal(_product(A, B), B)


def _graded_system(m, nblk, decades, rng):
    """Blocks I + (well conditioned), couplings of norm below 1/2, every
    equation scaled by its own power of ten."""
    S, T = [], []
    for i in range(nblk):
        d = 10.0 ** (-decades * rng.permutation(m) / (m - 1))[:, None]
        g = [rng.standard_normal((m, m)) * (0.2 / np.sqrt(m)) for _ in range(3)]
        S.append([d * g[0] if i else np.zeros((m, m)),
                  d * g[1] if i < nblk - 1 else np.zeros((m, m))])
        T.append(d * (np.eye(m) + g[2]))
    return S, T


@pytest.mark.parametrize("solver", ["rb", "thomas"])
@pytest.mark.parametrize("m,decades", [(64, 8), (64, 12), (256, 8), (256, 12), (700, 8), (700, 12)])
def test_row_graded_pivot_blocks(solver, m, decades):
    """Scaling the equations leaves the solution alone: the error stays that of
    the unscaled system, whose condition number is below 10 (row-wise backward
    error of LU with partial pivoting and explicit inverses: growth times m u)."""
    need_gpu()
    from sslablu_gb300.direct_solve.omsdirectsolve import BlockTridiagonalSolver, RedBlackSolver
    nblk = 4
    rng = np.random.default_rng(m + decades)
    S, T = _graded_system(m, nblk, decades, rng)
    x = rng.standard_normal((nblk * m, 33))
    X = x.astype(np.longdouble).reshape(nblk, m, 33)
    b = [T[i] @ X[i] for i in range(nblk)]
    for i in range(nblk):
        if i:
            b[i] = b[i] + S[i][0] @ X[i - 1]
        if i < nblk - 1:
            b[i] = b[i] + S[i][1] @ X[i + 1]
    s = RedBlackSolver(m) if solver == "rb" else BlockTridiagonalSolver(m)
    s.factorize(S, T)
    got = s.solve(np.concatenate(b).astype(float))
    assert np.linalg.norm(got - x) <= 100 * m * 1.2e-16 * np.linalg.norm(x)
