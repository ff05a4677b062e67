"""A kernel that gives up a bounded wait: the next call on the handle, the copy
of a result to the host and a synchronisation report it, once.  The wait is one
of a probe kernel with a short limit, on a barrier nobody arrives at."""
import numpy as np
import pytest

from tests._gpu import need_gpu, own_stream

pytestmark = pytest.mark.gpu


def _give_up(wait=True):
    import torch
    from sslablu_gb300 import _lib as L
    L.sync()
    L.check(L.lib().slu_wait_probe(L.handle(), 100))
    if wait:
        torch.cuda.current_stream().synchronize()


def _raises(f):
    from sslablu_gb300 import _lib as L
    with pytest.raises(L.SluError) as e:
        f()
    assert e.value.code == 7 and "gave up waiting" in str(e.value)


@pytest.fixture(scope="module")
def op():
    need_gpu()
    from tests.test_gpu_crt_steps import _op
    return _op(64, 3, 16, False)


def test_synchronisation(op):
    from sslablu_gb300 import _lib as L
    _give_up(wait=False)
    _raises(L.sync)
    L.sync()


@pytest.mark.parametrize("columns", [1, 40])
@pytest.mark.parametrize("where", ["device", "host", "pinned"])
def test_next_call(op, where, columns):
    import torch
    H, N = op
    b = torch.ones((N, columns), dtype=torch.float64)
    if where == "device":
        b = b.cuda()
    elif where == "pinned":
        b = b.pin_memory()
    else:
        b = b.numpy()
    calls = [H.solve] if where == "pinned" else [H.solve, H.matmat]
    for f in calls:
        want = f(b)
        _give_up()
        _raises(lambda: f(b))
        got = f(b)
        if where != "host":
            torch.cuda.synchronize()
            want, got = want.cpu().numpy(), got.cpu().numpy()
        np.testing.assert_array_equal(got, want)


def test_result_on_the_host(op):
    """The result of the call itself: its copy to the host follows the kernel."""
    import torch
    from sslablu_gb300 import _dev as dv
    H, N = op
    x = H.solve(torch.ones((N, 3), dtype=torch.float64, device="cuda"))
    _give_up(wait=False)      # on the stream of x, before its copy
    _raises(lambda: dv.to_host(x))
    assert np.isfinite(dv.to_host(x)).all()


def test_other_streams_are_not_told(op):
    import torch
    H, N = op
    b = torch.ones((N, 2), dtype=torch.float64, device="cuda")
    _give_up()
    s = own_stream()
    with torch.cuda.stream(s):
        H.solve(b)
    s.synchronize()
    _raises(lambda: H.solve(b))


def test_served_batch(op):
    """A request whose batch gave up waiting completes with the error."""
    import torch
    from sslablu_gb300 import _lib as L
    from sslablu_gb300.serving import Request, SolveServer, hbs_solver
    H, N = op
    srv = SolveServer(budget_bytes=1 << 30, workers=1)
    fail = [True, False]

    def factory(o):
        solve = hbs_solver(o)

        def f(X):
            Y = solve(X)
            if fail.pop(0):
                L.check(L.lib().slu_wait_probe(L.handle(), 100))
            return Y
        return f
    try:
        srv.admit("a", lambda: H, 1, factory)
        bad = srv.run([Request("a", np.ones(N))])[0]
        assert bad.X is None and bad.error.code == 7
        good = srv.run([Request("a", np.ones(N))])[0]
        assert good.error is None
        ref = H.solve(torch.ones((N, 1), dtype=torch.float64, device="cuda")).cpu().numpy()
        np.testing.assert_allclose(good.X, ref, rtol=1e-12)
    finally:
        srv.close()
