"""Factorisations whose output is written over their input."""

import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_cluster_factor import EPS

pytestmark = pytest.mark.gpu

# (rows, columns, output over the input): the whole of a is one factor
CASES = [("svd", 60, 60, "u"), ("svd", 60, 60, "vh"), ("svd", 200, 30, "u"), ("svd", 30, 200, "vh"), ("svd", 150, 150, "vh"),
         ("svd", 330, 330, "vh"), ("svd", 6, 6, "vh"), ("svd", 9, 1409, "vh"), ("qr", 90, 60, "u"), ("qr", 40, 300, "vh"),
         ("qr", 5, 5, "vh"), ("eigh", 40, 40, "u"), ("eigh", 150, 150, "u")]


@pytest.mark.parametrize("kind,m,n,over", CASES)
def test_output_over_input(kind, m, n, over):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    rt = tb.Runtime(0)
    rule, k = tb.U1FusionRule(), min(m, n)
    plan = rt.fplan(rt.space(rule, [tb.GradedSpace(rule, [(0, m)])], [tb.GradedSpace(rule, [(0, n)])]))
    A = np.random.default_rng(m + n).standard_normal((m, n))
    if kind == "eigh":
        A = A + A.T
    a = torch.as_tensor(A.T.ravel().copy(), device="cuda")
    new = lambda x: torch.full((x,), np.nan, dtype=torch.float64, device="cuda")
    u = a if over == "u" else new(m * k)
    v = a if over == "vh" else new(k * n)
    s = new(k)
    p = lambda t: C.c_void_p(t.data_ptr())
    args = {"svd": (u, s, v), "qr": (u, v), "eigh": (u, s, None)}[kind]
    _lib.call(f"tnt_{kind}", rt._h, plan._h, p(a), *(p(t) if t is not None else None for t in args), rt.stream())
    h = lambda t, r, c: t.cpu().numpy().reshape(c, r).T
    U = h(u, m, k)
    V = U.T if kind == "eigh" else h(v, k, n)
    S = np.ones(k) if kind == "qr" else s.cpu().numpy()
    tol = 100 * np.sqrt(k) * EPS
    assert np.linalg.norm((U * S) @ V - A) <= np.sqrt(k) * tol * np.linalg.norm(A)
    assert np.abs(U.T @ U - np.eye(k)).max() <= tol


def test_factors_in_one_arena_are_not_in_place():
    """All operands in one allocation (a serving arena): ranges that only neighbour are as apart."""
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    rt = tb.Runtime(0)
    rule = tb.U1FusionRule()
    leg = [tb.GradedSpace(rule, [(0, 90), (1, 40)])]
    plan = rt.fplan(rt.space(rule, leg, leg))
    sizes = [plan.u_size, plan.u_size, plan.s_size, plan.v_size]
    x = np.random.default_rng(2).standard_normal(sizes[0])
    arena = torch.zeros(sum(sizes), dtype=torch.float64, device="cuda")
    apart = [torch.zeros(n, dtype=torch.float64, device="cuda") for n in sizes]
    at = np.concatenate([[0], np.cumsum(sizes)])
    together = [arena[at[i]: at[i + 1]] for i in range(4)]
    for a, u, s, v in (together, apart):
        a.copy_(torch.as_tensor(x))
        p = lambda t: C.c_void_p(t.data_ptr())
        _lib.call("tnt_svd", rt._h, plan._h, p(a), p(u), p(s), p(v), rt.stream())
    assert all(torch.equal(x, y) for x, y in zip(together, apart))
