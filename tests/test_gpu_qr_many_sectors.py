"""QR of many sectors at once: the cluster narrows with their number, the factors stay those
of LAPACK (the limits of tests/test_gpu_cluster_factor.py)."""

import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_cluster_factor import EPS

pytestmark = pytest.mark.gpu


# counts at the edges of the widths: 16, 8, 4 and 2 CTAs per sector, one beyond
@pytest.mark.parametrize("count", [8, 9, 16, 17, 36, 37, 74, 75])
@pytest.mark.parametrize("m,n", [(90, 60), (40, 300)])
def test_factors_of_every_sector(m, n, count):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    rt = tb.Runtime(0)
    rule, k = tb.U1FusionRule(), min(m, n)
    leg = lambda d: [tb.GradedSpace(rule, [(q, d) for q in range(count)])]
    plan = rt.fplan(rt.space(rule, leg(m), leg(n)))
    A = np.random.default_rng(count + m).standard_normal((count, m, n))
    a = torch.as_tensor(A.transpose(0, 2, 1).ravel().copy(), device="cuda")
    q, r = (torch.full((count * x,), np.nan, dtype=torch.float64, device="cuda") for x in (m * k, k * n))
    p = lambda t: C.c_void_p(t.data_ptr())
    _lib.call("tnt_qr", rt._h, plan._h, p(a), p(q), p(r), rt.stream())
    Q = q.cpu().numpy().reshape(count, k, m).transpose(0, 2, 1)
    R = r.cpu().numpy().reshape(count, n, k).transpose(0, 2, 1)
    tol = 100 * np.sqrt(k) * EPS
    assert np.linalg.norm(Q @ R - A, axis=(1, 2)).max() <= tol * np.linalg.norm(A, axis=(1, 2)).min()
    assert np.abs(Q.transpose(0, 2, 1) @ Q - np.eye(k)).max() <= tol
    assert np.all(np.tril(R[:, :, :k], -1) == 0) and np.all(np.diagonal(R, axis1=1, axis2=2) >= 0)
