"""Memory of the wide calls and of the handle's scratch: counted, bounded, given
back."""
import ctypes

import numpy as np
import pytest

from tests._gpu import need_gpu, own_stream
from tests.test_gpu_crt_steps import _op
from tests.test_gpu_wide_calls import _rhs, _wide

pytestmark = pytest.mark.gpu


def _nbytes(H, which):
    from sslablu_gb300 import _lib as L
    out = ctypes.c_size_t()
    L.check(L.lib().slu_hbs_nbytes(H._op, which, ctypes.byref(out)))
    return out.value


def test_images_are_counted_and_limited():
    need_gpu()
    import torch
    from sslablu_gb300 import _lib as L
    H, N = _op(64, 6, 32, False)
    B = _rhs(N, 261)
    f64 = [H._dev_solve(B, wide=False), H._dev_apply(B, wide=False)]
    assert _nbytes(H, 2) == 0
    # a limit below the need: float64 steps, once refused not tried again
    L.check(L.lib().slu_hbs_set_wide_limit(H._op, 1000))
    for _ in range(2):
        assert torch.equal(H.solve(B), f64[0]) and torch.equal(H.matmat(B), f64[1])
        assert _nbytes(H, 2) == 0
        assert _wide(H, 1, 0, 261) == 0 and _wide(H, 0, 0, 261) == 0
    # a higher one: images, kept, of 32 to 40 bytes per entry of the step operators
    L.check(L.lib().slu_hbs_set_wide_limit(H._op, 1 << 30))
    assert _wide(H, 1, 0, 261) == 1
    assert not torch.equal(H.solve(B), f64[0])
    one = _nbytes(H, 2)
    assert one > 0
    H.solve(B)
    assert _nbytes(H, 2) == one
    H.solve(B, mode="T")
    H.matmat(B)
    H.rmatmat(B)
    assert _nbytes(H, 2) > 3 * one // 2
    # a new factorisation drops those of the solves
    H.compute_ULV()
    assert 0 < _nbytes(H, 2) < 3 * one


def _used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_scratch_is_bounded_and_given_back():
    """24 products of 1024^3 and 24 inverses of 1024 x 1024 within a gigabyte and a
    half of scratch, all of it returned."""
    need_gpu()
    import torch
    from sslablu_gb300 import _lib as L
    nb, n = 24, 1024
    A = torch.randn((nb, n, n), dtype=torch.float64, device="cuda")
    C = torch.empty_like(A)
    s = own_stream()
    with torch.cuda.stream(s):
        L.sync()
        before = _used()
        L.check(L.lib().slu_gemm_batched(L.handle(), 0, 0, n, n, n, 1.0, L.ptr(A), n, n * n, L.ptr(A), n,
                                         n * n, 0.0, L.ptr(C), n, n * n, nb))
        L.sync()
        held = _used() - before
        assert 0 < held < 700 << 20
        L.check(L.lib().slu_trim(L.handle()))
        L.sync()
        assert _used() - before < 64 << 20
    ref = A[23, :3] @ A[23]
    assert float((C[23, :3] - ref).abs().max()) <= 1e-12 * float(ref.abs().max())


def test_all_handles_trimmed():
    """What this thread's handles hold, on whatever streams, is returned; the next
    call allocates anew."""
    need_gpu()
    import torch
    from sslablu_gb300 import _lib as L
    H, N = _op(64, 5, 16, False)
    B = _rhs(N, 40)
    with torch.cuda.stream(own_stream()):
        want = H.solve(B)
        L.sync()
        torch.cuda.synchronize()
        for h in L._handles.handles.values():
            L.check(L.lib().slu_trim(h))
        got = H.solve(B)
        L.sync()
        assert torch.equal(got, want)


def test_inverses_in_pieces():
    """More blocks than one piece holds (LU, inverses and the carried products)."""
    need_gpu()
    from sslablu_gb300.direct_solve.omsdirectsolve import RedBlackSolver
    m, nblk = 700, 32
    rng = np.random.default_rng(1)
    Z = np.zeros((m, m))
    T = [np.eye(m) + rng.standard_normal((m, m)) * (0.2 / np.sqrt(m)) for _ in range(nblk)]
    S = [[rng.standard_normal((m, m)) * (0.2 / np.sqrt(m)) if i else Z,
          rng.standard_normal((m, m)) * (0.2 / np.sqrt(m)) if i < nblk - 1 else Z] for i in range(nblk)]
    s = RedBlackSolver(m)
    s.factorize(S, T)
    x = rng.standard_normal((nblk, m, 2))
    b = np.einsum("iab,ibc->iac", np.array(T), x)
    for i in range(nblk):
        b[i] += (S[i][0] @ x[i - 1] if i else 0) + (S[i][1] @ x[i + 1] if i < nblk - 1 else 0)
    got = s.solve(b.reshape(-1, 2))
    assert np.linalg.norm(got - x.reshape(-1, 2)) <= 100 * m * 1.2e-16 * np.linalg.norm(x)
