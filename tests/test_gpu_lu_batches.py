"""Batches of more matrices than one launch takes (65535)."""
import numpy as np
import pytest

from tests._gpu import need_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nb", [(3, 65536), (4, 140000), (33, 65540)])
def test_many_matrices(n, nb):
    need_gpu()
    import torch
    from sslablu_gb300 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((nb, n, n), generator=g, dtype=torch.float64, device="cuda")
    A[nb - 1, :, 1] = 0.0
    D = A.clone()
    piv = torch.empty((nb, n), dtype=torch.int32, device="cuda")
    info = torch.zeros(nb, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    L.check(L.lib().slu_lu_factor(L.handle(), n, L.ptr(D), n, n * n, L.ptr(piv), n, nb, L.ptr(info)))
    L.sync()
    assert int(info[nb - 1]) == 2 and int((info != 0).sum()) == 1
    P = A.clone()
    i = torch.arange(nb, device="cuda")
    for r in range(n):
        p = piv[:, r].long()
        P[i, r], P[i, p] = P[i, p], P[i, r].clone()
    Lm = torch.tril(D, -1) + torch.eye(n, dtype=torch.float64, device="cuda")
    U = torch.triu(D)
    # ||P A - L U|| <= 2 n u |L||U| (Higham, thm 9.3), doubled
    err, bound = (P - Lm @ U).abs(), Lm.abs() @ U.abs()
    assert bool((err.flatten(1).sum(1) <= 4 * n * 1.2e-16 * bound.flatten(1).sum(1)).all())
