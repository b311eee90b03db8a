"""Strided block copies at the edges of their split over lanes, columns and row pieces."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows x columns: columns shared by a warp, warps per column, columns cut into pieces of rows
SHAPES = [(1, 1), (1, 700), (3, 130), (31, 2), (33, 5), (255, 1), (256, 1), (257, 2), (1000, 1), (4097, 3), (70000, 1),
          (300, 64), (300, 65), (640, 40), (5, 0), (0, 4)]


@pytest.mark.parametrize("scaled", [False, True])
def test_copies_match_numpy(scaled):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    rt = tb.Runtime(0)
    rng = np.random.default_rng(5)
    rows, so, do, ko = [], 3, 5, 2
    for r, c in SHAPES:
        rows.append([so, do, r, c, r + 2, r + 1, ko if scaled else -1])
        so, do, ko = so + (r + 2) * c, do + (r + 1) * c, ko + r
    src, dst, scales = rng.standard_normal(so + 1), rng.standard_normal(do + 1), rng.standard_normal(ko + 1)
    want = dst.copy()
    for s0, d0, r, c, ls, ld, k0 in rows:
        for j in range(c):
            col = src[s0 + j * ls: s0 + j * ls + r]
            want[d0 + j * ld: d0 + j * ld + r] = col * scales[k0: k0 + r] if scaled else col
    table = torch.tensor(rows, dtype=torch.int64, device="cuda")
    a, b, s = (torch.as_tensor(x, device="cuda") for x in (src, dst, scales))
    p = lambda t: C.c_void_p(t.data_ptr())
    _lib.call("tnt_copy_segments_async", rt._h, len(rows), p(table), p(a), p(b), p(s), rt.stream())
    assert np.array_equal(b.cpu().numpy(), want)
