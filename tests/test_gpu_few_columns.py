"""SVD and QR of plans whose every sector has few columns, at the edges of the one-launch rule.

Tolerances of tests/test_gpu_cluster_factor.py; the SVD keeps the engine's range of
magnitudes and, at any rank, an orthonormal short side.
"""

import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_cluster_factor import EPS

pytestmark = pytest.mark.gpu

PLANS = [[(1, 1), (4, 4), (3, 1), (1, 3)], [(2, 1400), (1400, 4), (700, 3)], [(8, 8), (640, 8), (7, 500), (5, 5)],
         [(4, 4)] * 150, [(8, 6)] * 148, [(8, 6)] * 149, [(600, 5), (200, 8), (4, 200), (1, 1400)],
         [(4, 600)] * 40, [(5, 600)] * 80]


def run(kind, shapes, blocks):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    rt = tb.Runtime(0)
    rule = tb.U1FusionRule()
    rows = tb.GradedSpace(rule, [(q, m) for q, (m, _) in enumerate(shapes)])
    cols = tb.GradedSpace(rule, [(q, n) for q, (_, n) in enumerate(shapes)])
    space = rt.space(rule, [rows], [cols])
    plan = rt.fplan(space)
    order = [lab for lab, _, _, _ in space.sectors()]
    host = np.empty(space.size)
    by_label = {lab: i for i, lab in enumerate(sorted(order))}
    index = [by_label[lab] for lab in order]  # charges 0, 1, .. in the order given
    for (_, m, n, off), i in zip(space.sectors(), index):
        host[off: off + m * n] = blocks[i].T.ravel()
    a = torch.as_tensor(host, device="cuda")
    u, s, v = (torch.full((x,), np.nan, dtype=torch.float64, device="cuda") for x in (plan.u_size, plan.s_size,
                                                                                      plan.v_size))
    p = lambda t: C.c_void_p(t.data_ptr())
    args = {"svd": (p(a), p(u), p(s), p(v)), "qr": (p(a), p(u), p(v)), "eigh": (p(a), p(u), p(s), None)}[kind]
    _lib.call(f"tnt_{kind}", rt._h, plan._h, *args, rt.stream())
    u, s, v = (t.cpu().numpy() for t in (u, s, v))
    for (_, m, n, _), rec, i in zip(space.sectors(), plan.records.tolist(), index):
        k = min(m, n)
        yield (blocks[i], u[rec[4]: rec[4] + m * k].reshape(k, m).T, s[rec[5]: rec[5] + k],
               v[rec[6]: rec[6] + k * n].reshape(n, k).T)


@pytest.mark.parametrize("shapes", PLANS)
@pytest.mark.parametrize("rank,scale", [(None, 1.0), (None, 1e200), (1, 1e-200), (2, 1.0), (0, 1.0)])
def test_svd(shapes, rank, scale):
    rng = np.random.default_rng(len(shapes))
    make = lambda m, n: (rng.standard_normal((m, n)) if rank is None
                         else rng.standard_normal((m, rank)) @ rng.standard_normal((rank, n)))
    blocks = [make(m, n) for m, n in shapes]
    for A, u, s, v in run("svd", shapes, [b * scale for b in blocks]):
        m, n = A.shape
        k = min(m, n)
        tol = 100 * np.sqrt(k) * EPS
        B, w = A / scale, s / scale
        ref = np.linalg.svd(B, compute_uv=False)
        assert np.abs(w - ref).max() <= tol * max(ref[0], 1e-300) and np.all(np.diff(w) <= 0)
        assert np.linalg.norm((u * w) @ v - B) <= tol * np.linalg.norm(B)
        short = v if m >= n else u.T
        assert np.abs(short @ short.T - np.eye(k)).max() <= tol


@pytest.mark.parametrize("shapes", PLANS)
def test_qr(shapes):
    rng = np.random.default_rng(len(shapes))
    for A, q, _, r in run("qr", shapes, [rng.standard_normal(s) for s in shapes]):
        k = min(A.shape)
        tol = 100 * np.sqrt(k) * EPS
        assert np.linalg.norm(q @ r - A) <= tol * np.linalg.norm(A)
        assert np.abs(q.T @ q - np.eye(k)).max() <= tol
        assert np.all(np.tril(r[:, :k], -1) == 0) and np.all(r.diagonal() >= 0)
