"""SVD and eigh at both edges of every instantiation of the Jacobi kernels, and plans of
sectors that share a launch of a wider class.

Tolerances of tests/test_gpu_cluster_factor.py.
"""

import numpy as np
import pytest

from tests.test_gpu_cluster_factor import EPS, factor, graded, rt  # noqa: F401  (rt: the module's fixture)
from tests.test_gpu_few_columns import run

pytestmark = pytest.mark.gpu

RESIDENT = [16, 17, 48, 49, 96, 97, 112, 113, 128, 160, 161, 192, 193, 224, 225, 256, 288, 289, 320]


@pytest.mark.parametrize("n", RESIDENT + [321, 384, 385, 448, 449, 512, 608, 768, 769, 1024])
def test_svd(rt, n):  # noqa: F811
    tol = 100 * np.sqrt(n) * EPS
    A = graded(n, n, n) if n % 2 else np.random.default_rng(n).standard_normal((n, n))
    u, s, v = factor(rt, "svd", A)
    ref = np.linalg.svd(A, compute_uv=False)
    assert np.abs(s - ref).max() <= tol * ref[0] and np.all(np.diff(s) <= 0)
    assert np.linalg.norm((u * s) @ v - A) <= tol * np.linalg.norm(A)
    assert np.abs(u.T @ u - np.eye(n)).max() <= tol and np.abs(v @ v.T - np.eye(n)).max() <= tol


@pytest.mark.parametrize("n", RESIDENT + [321, 384, 385, 448, 449, 512, 513, 608, 609, 768, 1024])
def test_eigh(rt, n):  # noqa: F811
    g = np.random.default_rng(n).standard_normal((n, n))
    A = g + g.T if n % 2 else g[:, : n // 3] @ g[:, : n // 3].T
    A = 0.5 * (A + A.T)
    tol = 100 * np.sqrt(n) * EPS
    v, w, _ = factor(rt, "eigh", A)
    ref = np.linalg.eigvalsh(A)
    scale = np.abs(ref).max()
    assert np.abs(np.sort(w) - ref).max() <= tol * scale and np.all(np.diff(np.abs(w)) <= 0)
    assert np.abs((v * w) @ v.T - A).max() <= np.sqrt(n) * tol * scale
    assert np.abs(v.T @ v - np.eye(n)).max() <= tol


# narrower sectors join the clusters of the widest while these fit the device: idle CTAs, one
# column a block, columns padded to a larger class, square beside tall and wide ones
@pytest.mark.parametrize("shapes", [[(1, 1), (2, 2), (3, 3), (40, 40), (100, 100), (130, 130)],
                                    [(5, 9), (9, 5), (64, 64), (65, 65), (300, 300)], [(1, 200), (450, 330), (17, 17)],
                                    [(200, 200)] * 9 + [(100, 60)] * 30 + [(7, 3)] * 60])
@pytest.mark.parametrize("kind", ["svd", "qr"])
def test_plans_of_mixed_sectors(shapes, kind):
    rng = np.random.default_rng(len(shapes))
    for A, u, s, v in run(kind, shapes, [rng.standard_normal(x) for x in shapes]):
        k = min(A.shape)
        tol = 100 * np.sqrt(k) * EPS
        d = s if kind == "svd" else np.ones(k)
        assert np.linalg.norm((u * d) @ v - A) <= tol * np.linalg.norm(A)
        assert np.abs(u.T @ u - np.eye(k)).max() <= tol
        if kind == "svd":
            assert np.abs(v @ v.T - np.eye(k)).max() <= tol
            ref = np.linalg.svd(A, compute_uv=False)
            assert np.abs(s - ref).max() <= tol * ref[0]


@pytest.mark.parametrize("sizes", [[1, 2, 3, 40, 100, 130], [64, 65, 400, 5], [1, 460, 30]])
def test_eigh_of_mixed_sectors(sizes):
    import tenet_b200 as tb

    rule = tb.U1FusionRule()
    r = tb.Runtime(0)
    leg = [tb.GradedSpace(rule, [(q, n) for q, n in enumerate(sizes)])]
    space = r.space(rule, leg, leg)
    rng = np.random.default_rng(sum(sizes))
    host = np.empty(space.size)
    blocks = {}
    for _, n, _, off in space.sectors():
        g = rng.standard_normal((n, n))
        blocks[off] = g + g.T
        host[off: off + n * n] = blocks[off].ravel()
    d, v = tb.TensorMap.from_host(r, leg, leg, host).eigh_full()
    w, z = d.to_host(), v.to_host()
    for (_, n, _, off), (_, _, _, vo), (_, _, _, do) in zip(space.sectors(), v.space.sectors(), d.space.sectors()):
        V, W = z[vo: vo + n * n].reshape(n, n).T, w[do: do + n * n].reshape(n, n).diagonal()
        tol = 100 * np.sqrt(n) * EPS
        assert np.abs((V * W) @ V.T - blocks[off]).max() <= np.sqrt(n) * tol * np.abs(W).max()
        assert np.abs(V.T @ V - np.eye(n)).max() <= tol
