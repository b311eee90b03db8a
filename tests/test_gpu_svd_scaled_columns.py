"""Small singular values of sectors whose short side spans many decades.

A coupled sector's columns are uncoupled blocks side by side, each with its own
falling Schmidt weights.  A = B D with B of condition number 3 and D diagonal
determines every singular value to a relative error of 3 times the errors, column
by column, of the transformations (100 sqrt(k) eps, as for the factors of unscaled
sectors), whatever D.  Reference: one-sided Jacobi in extended precision.
"""

import numpy as np
import pytest

from tests.test_gpu_cluster_factor import EPS, factor, rt  # noqa: F401  (rt: the module's fixture)

pytestmark = pytest.mark.gpu


def jacobi_values(A):
    """Singular values of A (rows >= columns), descending: round robins of column pairs in extended precision."""
    W = A[:, np.argsort(-np.linalg.norm(A, axis=0))].astype(np.longdouble)
    n = W.shape[1]
    if n % 2:
        W = np.concatenate([W, np.zeros((len(W), 1), np.longdouble)], axis=1)
    order = np.arange(W.shape[1])
    h = len(order) // 2
    for _ in range(60):
        worst = 0.0
        for _ in range(len(order) - 1):
            p, q = order[:h], order[h:][::-1]
            x, y = W[:, p], W[:, q]
            al, be, ga = (x * x).sum(0), (y * y).sum(0), (x * y).sum(0)
            on = np.abs(ga) > 1e-18 * np.sqrt(al * be)
            worst = max(worst, float(np.max(np.abs(ga[on]) / np.sqrt(al * be)[on], initial=0)))
            z = (be - al) / np.where(on, 2 * ga, 1)
            t = np.where(on, np.where(z < 0, -1, 1) / (np.abs(z) + np.sqrt(1 + z * z)), 0)
            c = 1 / np.sqrt(1 + t * t)
            W[:, p], W[:, q] = c * (x - t * y), c * (t * x + y)
            order = np.concatenate([order[:1], order[-1:], order[1:-1]])
        if worst < 1e-17:
            break
    return np.sort(np.sqrt((W * W).sum(0)))[::-1][:n]


def test_reference_on_known_values():
    rng = np.random.default_rng(1)
    d = 10.0 ** -np.arange(13)
    q = np.linalg.qr(rng.standard_normal((13, 13)))[0]
    assert np.abs(jacobi_values(q * d) / d - 1).max() < 100 * EPS  # q is orthogonal to rounding


ORDERS = {
    "random": lambda k, rng: rng.permutation(np.linspace(0, -10, k)),
    "rising": lambda k, rng: np.linspace(-10, 0, k),
    "blocks": lambda k, rng: np.concatenate([np.linspace(0, -10, (k + 1) // 2), np.linspace(0, -10, k // 2)]),
}


# a ring in one CTA, on clusters, staged columns; square, tall and wide
@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("m,n", [(5, 3), (24, 24), (60, 24), (24, 60), (64, 64), (130, 130), (330, 330), (700, 33)])
def test_small_values_keep_their_relative_accuracy(rt, m, n, order):  # noqa: F811
    k = min(m, n)
    rng = np.random.default_rng(1000 * m + n)
    q = [np.linalg.qr(rng.standard_normal((x, k)))[0] for x in (max(m, n), k)]
    A = ((q[0] * np.linspace(1, 1 / 3, k)) @ q[1].T) * 10.0 ** ORDERS[order](k, rng)  # columns scaled
    ref = jacobi_values(A)
    u, s, v = factor(rt, "svd", A if m >= n else np.ascontiguousarray(A.T))
    assert np.abs(s / ref - 1).max() <= 3 * 100 * np.sqrt(k) * EPS
    short = v if m >= n else u.T
    assert np.abs(short @ short.T - np.eye(k)).max() <= 100 * np.sqrt(k) * EPS
