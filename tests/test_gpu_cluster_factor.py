"""Cluster QR, cluster Jacobi SVD and eigh at the edges of their size classes.

One dense sector per case.  Tolerances: a column goes through about 12 k
rotations (and k reflections) of a few rounding errors each, which add like a
random walk, so factors reconstruct, and values agree with LAPACK, within
100 sqrt(k) eps of the largest scale; pairs count as orthogonal at 4 sqrt(k) eps.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


@pytest.fixture(scope="module")
def rt():
    from tenet_b200 import Runtime

    return Runtime(0)


def factor(rt, kind, A):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    m, n = A.shape
    k = min(m, n)
    rule = tb.U1FusionRule()
    sp = rt.space(rule, [tb.GradedSpace(rule, [(0, m)])], [tb.GradedSpace(rule, [(0, n)])])
    plan = rt.fplan(sp)
    a = torch.as_tensor(np.ascontiguousarray(A.T).ravel(), device="cuda")
    u, s, v = (torch.full((x,), np.nan, dtype=torch.float64, device="cuda") for x in (m * k, k, k * n))
    p = lambda t: C.c_void_p(t.data_ptr())
    if kind == "svd":
        _lib.call("tnt_svd", rt._h, plan._h, p(a), p(u), p(s), p(v), rt.stream())
    elif kind == "qr":
        _lib.call("tnt_qr", rt._h, plan._h, p(a), p(u), p(v), rt.stream())
    else:
        _lib.call("tnt_eigh", rt._h, plan._h, p(a), p(u), p(s), None, rt.stream())
    h = lambda t, r, c: t.cpu().numpy().reshape(c, r).T
    return h(u, m, k), s.cpu().numpy(), h(v, k, n)


def graded(m, n, seed):
    rng = np.random.default_rng(seed)
    k = min(m, n)
    return (rng.standard_normal((m, k)) * 10.0 ** (-4.0 * np.arange(k) / k)) @ rng.standard_normal((k, n)) / np.sqrt(k)


# (rows, columns): one-CTA classes to 32 and 64, clusters to 128, 256, 512 and 608,
# more block pairs than CTAs beyond; panels of 32 reflectors to 640 rows, of 16 to
# 1408, the general kernels beyond; tall and wide sectors take a second QR pass.
SHAPES = [(1, 1), (1, 7), (7, 1), (2, 2), (31, 32), (33, 33), (64, 64), (65, 64), (65, 65), (97, 128), (129, 129),
          (256, 200), (257, 257), (513, 513), (609, 609), (641, 641), (100, 700), (1025, 1030), (1408, 9), (9, 1409)]


@pytest.mark.parametrize("m,n", SHAPES)
def test_svd_size_classes(rt, m, n):
    k = min(m, n)
    tol = 100 * np.sqrt(k) * EPS
    for A in (np.random.default_rng(m + n).standard_normal((m, n)), graded(m, n, m * n)):
        u, s, v = factor(rt, "svd", A)
        ref = np.linalg.svd(A, compute_uv=False)
        assert np.abs(s - ref).max() <= tol * ref[0] and np.all(np.diff(s) <= 0)
        assert np.linalg.norm((u * s) @ v - A) <= tol * np.linalg.norm(A)
        # both sides are orthogonal down to the smallest column above the rounding level
        assert np.abs(u.T @ u - np.eye(k)).max() <= tol and np.abs(v @ v.T - np.eye(k)).max() <= tol
        assert np.all(u[np.abs(u).argmax(0), np.arange(k)] > 0)


@pytest.mark.parametrize("m,n", SHAPES)
def test_qr_size_classes(rt, m, n):
    k = min(m, n)
    A = graded(m, n, m + 3 * n)
    q, _, r = factor(rt, "qr", A)
    tol = 100 * np.sqrt(k) * EPS
    assert np.linalg.norm(q @ r - A) <= tol * np.linalg.norm(A)
    assert np.abs(q.T @ q - np.eye(k)).max() <= tol
    assert np.all(np.tril(r[:, :k], -1) == 0) and np.all(r.diagonal() >= 0)


@pytest.mark.parametrize("n", [1, 2, 32, 33, 64, 65, 128, 129, 257, 513, 700])
def test_eigh_size_classes(rt, n):
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, n))
    tol = 100 * np.sqrt(n) * EPS
    for A in (g + g.T, g[:, : max(1, n // 3)] @ g[:, : max(1, n // 3)].T, -np.outer(g[0], g[0])):
        A = 0.5 * (A + A.T)
        v, w, _ = factor(rt, "eigh", A)
        ref = np.linalg.eigvalsh(A)
        ref = ref[np.argsort(-np.abs(ref), kind="stable")]
        scale = np.abs(ref).max()
        assert np.abs(np.sort(w) - np.sort(ref)).max() <= tol * scale
        assert np.all(np.diff(np.abs(w)) <= 0)
        assert np.abs((v * w) @ v.T - A).max() <= np.sqrt(n) * tol * scale
        assert np.abs(v.T @ v - np.eye(n)).max() <= tol


@pytest.mark.parametrize("n", [20, 90, 150])
def test_degenerate_inputs(rt, n):
    rng = np.random.default_rng(n)
    tol = 100 * np.sqrt(n) * EPS
    low = rng.standard_normal((n, 5)) @ rng.standard_normal((5, n))
    for A in (np.zeros((n, n)), low, np.eye(n), 1e-200 * low, 1e200 * low, np.zeros((n, n + 3)), low[:, : n - 4]):
        u, s, v = factor(rt, "svd", A)
        big = np.abs(A).max() or 1.0
        assert np.linalg.norm((u * (s / big)) @ v - A / big) <= tol * n
        short = v if A.shape[0] >= A.shape[1] else u.T  # the accumulated side is orthonormal at any rank
        assert np.abs(short @ short.T - np.eye(len(short))).max() <= tol
    z, w, _ = factor(rt, "eigh", np.zeros((n, n)))
    assert np.all(w == 0) and np.abs(z.T @ z - np.eye(n)).max() <= tol
    q, _, r = factor(rt, "qr", np.zeros((n, n)))
    assert np.all(r == 0) and np.abs(q - np.eye(n)).max() == 0
    nan = rng.standard_normal((n, n))
    nan[1, 2] = np.nan
    factor(rt, "svd", nan)  # ends; what it returns is unspecified
    with pytest.raises(Exception):
        factor(rt, "eigh", nan + nan.T)
