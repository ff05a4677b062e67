"""The entry points that may take the residue steps (`wide`) and those that keep
the float64 steps, with the results that their descriptions promise."""
import ctypes

import numpy as np
import pytest

from tests._gpu import need_gpu
from tests.test_gpu_crt_steps import _op

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def op():
    need_gpu()
    return _op(64, 6, 32, False)


def _rhs(N, c, seed=0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((N, c), generator=g, dtype=torch.float64, device="cuda")


def _wide(H, solve, trans, c):
    from sslablu_gb300 import _lib as L
    out = ctypes.c_int(-1)
    L.check(L.lib().slu_hbs_wide_steps(H._op, solve, trans, c, ctypes.byref(out)))
    return out.value


def _solve(H, B, trans=0):
    from sslablu_gb300 import _lib as L
    X = B.clone()
    c = B.shape[1]
    L.check(L.lib().slu_ulv_solve(L.handle(), H._op, L.ptr(X), c, c, trans))
    return X


def test_where_the_residue_steps_run(op):
    H, N = op
    for solve in (0, 1):
        for trans in (0, 1):
            assert [_wide(H, solve, trans, c) for c in (1, 16, 32)] == [0, 0, 0]
            assert [_wide(H, solve, trans, c) for c in (150, 261, 1000)] == [1, 1, 1]
    # steps deeper than 128, and a single level, keep the float64 steps
    deep, _ = _op(128, 4, 20, False)
    assert _wide(deep, 1, 0, 1000) == 0 and _wide(deep, 0, 0, 1000) == 0
    from sslablu_gb300.matAssembly.HBS.HBSnew import HBSMAT
    root = HBSMAT().set_mats([], [np.eye(64)], [], [1], fac=2)
    assert _wide(root, 0, 0, 1000) == 0


def test_float64_solves_have_the_same_bits(op):
    """slu_ulv_solve of many columns equals itself by narrow pieces, the call
    without allocations, the timed one, slu_ulv_solve_into and its plan."""
    import torch
    from sslablu_gb300 import _lib as L
    H, N = op
    c = 150
    B = _rhs(N, c)
    for trans in (0, 1):
        X = _solve(H, B, trans)
        pieces = torch.cat([_solve(H, B[:, j:j + 32].contiguous(), trans) for j in range(0, c, 32)], 1)
        assert torch.equal(X, pieces)
        Y = B.clone()
        L.check(L.lib().slu_ulv_solve_noalloc(L.handle(), H._op, L.ptr(Y), c, c, trans))
        assert torch.equal(X, Y)
        Z = torch.empty_like(B)
        L.check(L.lib().slu_ulv_solve_into(L.handle(), H._op, L.ptr(B), c, L.ptr(Z), c, c, trans))
        assert torch.equal(X, Z)
        p = ctypes.c_void_p()
        Z.zero_()
        L.check(L.lib().slu_ulv_solve_plan_create(L.handle(), H._op, L.ptr(B), c, L.ptr(Z), c, c, trans,
                                                  ctypes.byref(p)))
        L.check(L.lib().slu_ulv_solve_plan_launch(L.handle(), p, 1))
        L.lib().slu_ulv_solve_plan_destroy(p)
        assert torch.equal(X, Z)
    Y = B.clone()
    n = ctypes.c_int()
    L.check(L.lib().slu_ulv_solve_timed(L.handle(), H._op, L.ptr(Y), c, c, None, None, None, 0,
                                        ctypes.byref(n)))
    assert torch.equal(_solve(H, B), Y)


def test_groups_have_the_bits_of_their_members(op):
    import torch
    from sslablu_gb300 import _lib as L
    from sslablu_gb300.grouped import solve_grouped_device
    H, N = op
    K, M = _op(64, 5, 24, False)
    Bs = [_rhs(N, 150), _rhs(M, 300, 1), _rhs(N, 5, 2)]
    ops = [H, K, H]
    want = [_solve(h, b) for h, b in zip(ops, Bs)]
    got = solve_grouped_device(ops, [b.clone() for b in Bs])
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    tr = (ctypes.c_int * 3)(0, 1, 1)
    oa = (ctypes.c_void_p * 3)(*[h._op for h in ops])
    Ys = [torch.empty_like(b) for b in Bs]
    xp = (ctypes.c_void_p * 3)(*[b.data_ptr() for b in Bs])
    yp = (ctypes.c_void_p * 3)(*[y.data_ptr() for y in Ys])
    ld = (ctypes.c_int * 3)(*[b.shape[1] for b in Bs])
    L.check(L.lib().slu_hbs_apply_grouped(L.handle(), 3, oa, tr, xp, ld, yp, ld, ld))
    for h, b, y, t in zip(ops, Bs, Ys, tr):
        ref, c = torch.empty_like(b), b.shape[1]
        L.check(L.lib().slu_hbs_apply(L.handle(), h._op, t, L.ptr(b), c, L.ptr(ref), c, c))
        assert torch.equal(y, ref)


def test_served_results_do_not_depend_on_the_batch(op):
    import torch
    from sslablu_gb300.serving import Request, SolveServer, hbs_group_solver, hbs_solver
    H, N = op
    rng = np.random.default_rng(3)
    blocks = [rng.standard_normal((N, c)) for c in (64, 3, 90, 41)]
    alone = [H.solve(torch.from_numpy(b[:, :3]).cuda()).cpu().numpy() for b in blocks]
    for group in (None, hbs_group_solver("f64")):
        srv = SolveServer(budget_bytes=1 << 30, workers=1, max_batch_rhs=256, group_solve=group)
        try:
            srv.admit("a", lambda: H, 1, lambda o: hbs_solver(o))
            reqs = [Request("a", b, rid=i) for i, b in enumerate(blocks)]
            srv.run(reqs)
            for r, x in zip(reqs, alone):
                assert r.error is None
                np.testing.assert_array_equal(r.X[:, :3], x)
        finally:
            srv.close()


def test_wide_calls_agree(op):
    """The class's calls are the wide entry points'; a plan replays the call."""
    import torch
    from sslablu_gb300 import _lib as L
    H, N = op
    B = _rhs(N, 261, 4)
    for trans, mode in ((0, "N"), (1, "T")):
        X = torch.empty_like(B)
        L.check(L.lib().slu_ulv_solve_wide(L.handle(), H._op, L.ptr(B), 261, L.ptr(X), 261, 261, trans))
        assert torch.equal(X, H.solve(B, mode=mode))
        assert float((X - _solve(H, B, trans)).norm() / X.norm()) < 1e-12
        plan = H.solve_plan(B, mode=mode)
        assert torch.equal(plan(), X)
        plan.close()
        # in place
        Y = B.clone()
        L.check(L.lib().slu_ulv_solve_wide(L.handle(), H._op, L.ptr(Y), 261, L.ptr(Y), 261, 261, trans))
        assert torch.equal(X, Y)
        L.check(L.lib().slu_hbs_apply_wide(L.handle(), H._op, trans, L.ptr(B), 261, L.ptr(X), 261, 261))
        assert torch.equal(X, H.matmat(B) if mode == "N" else H.rmatmat(B))
