"""A sector's FP64 product is the same bits alone and in a plan with any others: thin plans
stream, others run as tensor-core tiles, and tile sizes follow from the whole plan, but every
output is one sum over rising k."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (3, 40, 2), (40, 3, 8), (300, 7, 5), (17, 90, 3), (2000, 2, 4), (9, 9, 7), (64, 64, 8), (65, 80, 6),
          (33, 47, 9), (100, 90, 64), (300, 200, 129), (20, 300, 50), (5, 6, 0), (128, 128, 1)]


@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.75, 0.5)])
@pytest.mark.parametrize("limit", [8, 10**6])
def test_bits_do_not_depend_on_the_plan(alpha, beta, limit):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib
    from tenet_b200._lib import arr, call, i64

    rt = tb.Runtime(0)
    rng = np.random.default_rng(4)
    p = lambda t: C.c_void_p(t.data_ptr())
    up = lambda x: torch.as_tensor(np.append(x, 0.0), device="cuda")

    def compose(jobs, a, b, c):
        h = C.c_void_p()
        call("tnt_cplan_from_jobs", len(jobs), arr(i64, [x for r in jobs for x in r]), len(a), len(b), len(c), C.byref(h))
        da, db, dc = up(a), up(b), up(c)
        call("tnt_compose", rt._h, h, 1, p(dc), len(c), p(da), len(a), p(db), len(b), alpha, beta, _lib.PREC_FP64, 0,
             rt.stream())
        out = dc.cpu().numpy()[:-1]
        _lib.lib().tnt_cplan_destroy(h)
        return out

    shapes = [s for s in SHAPES if s[2] <= limit]
    jobs, parts, ao, bo, co = [], [], 0, 0, 0
    for m, n, k in shapes:
        jobs.append((m, n, k, ao, bo, co, m, max(1, k), m))
        a, b, c = rng.standard_normal(m * k), rng.standard_normal(k * n), rng.standard_normal(m * n)
        parts.append((a, b, c, compose([(m, n, k, 0, 0, 0, m, max(1, k), m)], a, b, c)))
        ao, bo, co = ao + m * k, bo + k * n, co + m * n
    got = compose(jobs, *(np.concatenate([q[i] for q in parts]) for i in (0, 1, 2)))
    at = 0
    for (m, n, k), q in zip(shapes, parts):
        assert np.array_equal(got[at: at + m * n], q[3]), (m, n, k)
        at += m * n
