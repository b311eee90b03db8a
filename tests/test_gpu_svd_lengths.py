"""Lengths of the accumulated singular vectors, and the values with them.

The rounding of some 10 k rotations moves the length of every column they carry; it is
divided out at the end.  What is left on a squared length are the k reflections of the
QR pass, a rounding or two each, added like a random walk: 2 sqrt(k) eps; on a value,
relative to the largest, half of that.  (Left in, lengths were off by 30 to 95 eps.)
"""

import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_cluster_factor import EPS, factor, rt  # noqa: F401  (rt: the module's fixture)
from tests.test_gpu_svd_scaled_columns import jacobi_values

pytestmark = pytest.mark.gpu


# one CTA, clusters of four, wide clusters with the columns resident and staged
@pytest.mark.parametrize("n", [40, 64, 104, 300, 400])
@pytest.mark.parametrize("decades", [0, 3])
def test_accumulated_vectors_have_unit_length(rt, n, decades):  # noqa: F811
    rng = np.random.default_rng(n + decades)
    A = rng.standard_normal((n, n)) * 10.0 ** (-decades * np.arange(n) / n)
    u, s, v = factor(rt, "svd", A)
    length = (v.astype(np.longdouble) ** 2).sum(1)
    assert np.abs(length - 1).max() <= 2 * np.sqrt(n) * EPS
    if n <= 104:
        ref = jacobi_values(A)
        assert np.abs(s - ref).max() <= np.sqrt(n) * EPS * ref[0]


def test_two_by_two_rotations_over_all_angles(rt):  # noqa: F811
    """The tangent is found in single precision and its scale factor by one third-order
    step in FP64: an exact rotation to rounding, at every angle.  Two reflections and a
    handful of rotations, each a few roundings: 32 eps."""
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    rng = np.random.default_rng(3)
    count = 600
    angle = np.concatenate([rng.uniform(0, 2 * np.pi, 300), 10.0 ** -rng.uniform(0, 16, 300)])
    second = np.concatenate([np.linspace(0.5, 1, 300), 10.0 ** -rng.uniform(0, 8, 300)])
    rot = lambda a: np.stack([np.stack([np.cos(a), -np.sin(a)], -1), np.stack([np.sin(a), np.cos(a)], -1)], -2)
    A = rot(rng.uniform(0, 6, count)) @ (np.stack([np.ones(count), second], -1)[:, :, None] * rot(angle))
    rule = tb.U1FusionRule()
    leg = tb.GradedSpace(rule, [(q, 2) for q in range(count)])
    plan = rt.fplan(rt.space(rule, [leg], [leg]))
    a = torch.as_tensor(A.transpose(0, 2, 1).ravel().copy(), device="cuda")
    u, s, v = (torch.full((x,), np.nan, dtype=torch.float64, device="cuda") for x in (4 * count, 2 * count, 4 * count))
    p = lambda t: C.c_void_p(t.data_ptr())
    _lib.call("tnt_svd", rt._h, plan._h, p(a), p(u), p(s), p(v), rt.stream())
    m = lambda t: t.cpu().numpy().reshape(count, 2, 2).transpose(0, 2, 1).astype(np.longdouble)
    U, S, V = m(u), s.cpu().numpy().reshape(count, 2), m(v)
    eye = np.eye(2)
    assert np.abs(V @ V.transpose(0, 2, 1) - eye).max() <= 32 * EPS
    assert np.abs(U.transpose(0, 2, 1) @ U - eye).max() <= 32 * EPS
    assert np.abs((U * S[:, None, :]) @ V - A).max() <= 32 * EPS
