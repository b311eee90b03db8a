"""Sectors of every depth class in one split-precision plan, bit for bit as alone.

B is packed with its values in registers (two or four iterations) or, where some K is
beyond 1024, by a warp per column, beside a pass for K up to 512 if that has many columns.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEPTHS = [64, 1100, 512, 513, 1024, 1025, 3, 0, 2048, 70]  # few columns: one kernel for all


@pytest.mark.parametrize("depths,columns", [(DEPTHS, 11), (DEPTHS, 300), ([1100, 64, 500], 2000), ([2049, 1030], 40)])
@pytest.mark.parametrize("precision,slices", [("i8", 5), ("bf16", 3), ("bf16", 8)])
def test_mixed_depths_match_each_sector_alone(depths, columns, precision, slices, monkeypatch):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib
    from tenet_b200._lib import arr, call, i64

    monkeypatch.setenv("TNT_SPLIT_TILE_N", "64")
    rt = tb.Runtime(0)
    prec = _lib.PREC_INT8X if precision == "i8" else _lib.PREC_BF16X
    rng = np.random.default_rng(len(depths))
    p = lambda t: C.c_void_p(t.data_ptr())
    up = lambda x: torch.as_tensor(np.append(x, 0.0), device="cuda")  # a depth of 0 has no elements

    def compose(jobs, a, b, nc):
        h = C.c_void_p()
        call("tnt_cplan_from_jobs", len(jobs), arr(i64, [x for r in jobs for x in r]), len(a), len(b), nc, C.byref(h))
        da, db, dc = up(a), up(b), torch.full((nc,), np.nan, dtype=torch.float64, device="cuda")
        call("tnt_compose", rt._h, h, 1, p(dc), nc, p(da), len(a), p(db), len(b), 1.0, 0.0, prec, slices, rt.stream())
        out = dc.cpu().numpy()
        _lib.lib().tnt_cplan_destroy(h)
        return out

    jobs, parts, ao, bo, co = [], [], 0, 0, 0
    for i, k in enumerate(depths):
        m, n = 20 + 7 * i, 45 + columns * i
        jobs.append((m, n, k, ao, bo, co, m, max(1, k), m))
        a, b = rng.standard_normal(m * k), rng.standard_normal(k * n)
        parts.append((a, b, compose([(m, n, k, 0, 0, 0, m, max(1, k), m)], a, b, m * n)))
        ao, bo, co = ao + m * k, bo + k * n, co + m * n
    got = compose(jobs, *(np.concatenate([q[i] for q in parts]) for i in (0, 1)), co)
    assert np.array_equal(got, np.concatenate([q[2] for q in parts]))
