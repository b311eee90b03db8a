"""Split-precision compose at the edges of its tiles, against numpy.

Extents around the 8-row copy groups, the 64-wide and 128-high tiles and the 32-
and 64-deep K blocks, padded leading dimensions and odd offsets.  With sigma and
tau the largest magnitudes of a row of A and a column of B (rounded up to powers
of two), an output's error is below K sigma tau times the dropped diagonals and
the rounding of the operands, (S + 1) base^-S up to a geometric tail below 1.01,
plus the FP64 rounding of the sum; BF16 slices add the FP32 accumulator of the
diagonals from 3 on (26 * 512 additions of terms 2^-21 below the result: 2^-31).
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    [(1, 1, 1), (7, 9, 31), (8, 8, 32), (9, 7, 33), (63, 65, 63), (64, 64, 64)],
    [(65, 63, 65), (127, 129, 95), (128, 128, 96), (129, 127, 97), (136, 200, 161), (5, 6, 0)],
    [(130, 256, 40), (255, 257, 600)],
    [(40, 33, 1100), (20, 40, 1025), (9, 65, 70), (5, 8, 2049), (3, 4, 0)],
    [(20 + i, 150 - i, 30 + i) for i in range(100)],
]


@pytest.mark.parametrize("shapes", SHAPES)
@pytest.mark.parametrize("precision,slices", [("i8", 1), ("i8", 2), ("i8", 3), ("i8", 4), ("i8", 5), ("i8", 6),
                                              ("bf16", 1), ("bf16", 3), ("bf16", 7), ("bf16", 8)])
@pytest.mark.parametrize("alpha,beta,nbatch", [(1.0, 0.0, 1), (-0.75, 0.5, 3)])
def test_split_edges_match_numpy(shapes, precision, slices, alpha, beta, nbatch):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib
    from tenet_b200._lib import arr, call, i64

    rt = tb.Runtime(0)
    rows, ao, bo, co = [], 1, 2, 3
    for m, n, k in shapes:
        lda, ldb, ldc = m + 1, max(1, k) + 2, m + 3
        rows.append((m, n, k, ao, bo, co, lda, ldb, ldc))
        ao, bo, co = ao + lda * k, bo + ldb * n, co + ldc * n
    na, nb, nc = ao + 1, bo + 1, co + 1
    h = C.c_void_p()
    call("tnt_cplan_from_jobs", len(rows), arr(i64, [x for r in rows for x in r]), na, nb, nc, C.byref(h))
    rng = np.random.default_rng(len(rows) * 13 + slices)
    a, b, c = (rng.standard_normal((nbatch, s)) for s in (na, nb, nc))
    if beta == 0.0:
        c[:] = np.nan
    da, db, dc = (torch.as_tensor(x, device="cuda") for x in (a, b, c))
    ptr = lambda t: C.c_void_p(t.data_ptr())
    call("tnt_compose", rt._h, h, nbatch, ptr(dc), nc, ptr(da), na, ptr(db), nb, alpha, beta,
         _lib.PREC_INT8X if precision == "i8" else _lib.PREC_BF16X, slices, rt.stream())
    got = dc.cpu().numpy()
    _lib.lib().tnt_cplan_destroy(h)
    if precision == "i8":
        unit = 1.01 * (slices + 1) * 2.0 ** (2 - 8 * slices) + 2.0 ** -50
    else:
        unit = 1.01 * (slices + 1) * 2.0 ** (-7 * slices) + 2.0 ** -31
    pow2 = lambda v: 2.0 ** np.ceil(np.log2(v) + 1e-9)
    for q in range(nbatch):
        for m, n, k, a0, b0, c0, lda, ldb, ldc in rows:
            blk = lambda x, off, r, cc, ld: np.lib.stride_tricks.as_strided(x[off:], (r, cc), (x.itemsize, x.itemsize * ld))
            A, B = blk(a[q], a0, m, k, lda), blk(b[q], b0, k, n, ldb)
            old = np.zeros((m, n)) if beta == 0.0 else beta * blk(c[q], c0, m, n, ldc)
            bound = 2.0 ** -51 * abs(old)
            if k:
                bound = bound + abs(alpha) * k * unit * np.outer(pow2(abs(A).max(1)), pow2(abs(B).max(0)))
            assert np.all(abs(blk(got[q], c0, m, n, ldc) - (alpha * (A @ B) + old)) <= bound)
        gaps = np.ones(nc, dtype=bool)  # nothing outside the blocks is written
        for m, n, k, a0, b0, c0, lda, ldb, ldc in rows:
            for j in range(n):
                gaps[c0 + j * ldc: c0 + j * ldc + m] = False
        assert np.array_equal(got[q][gaps], c[q][gaps], equal_nan=True)


# K per pass over B: two or four iterations in registers, one to three splits of a warp, and the two-pass kernel
@pytest.mark.parametrize("k", [40, 200, 300, 700, 1500])
@pytest.mark.parametrize("precision,slices", [("i8", 5), ("bf16", 5)])
def test_split_scales_over_the_exponent_range(k, precision, slices):
    """Rows and columns whose scales are at both ends of the exponent range, and zero ones:
    powers of two commute with the digits, so the bound is the unscaled product's."""
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib
    from tenet_b200._lib import arr, call, i64

    rt = tb.Runtime(0)
    e = np.array([0, -1015, -961, -959, -957, 1020, 1021, 1022, 3, 500] * 4)
    m = n = len(e)
    rng = np.random.default_rng(k)
    A, B = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, n))
    A[8::10], B[:, 8::10] = 0.0, 0.0
    As, Bs = np.ldexp(A, e[:, None]), np.ldexp(B, e[None, :])
    h = C.c_void_p()
    call("tnt_cplan_from_jobs", 1, arr(i64, [m, n, k, 0, 0, 0, m, k, m]), m * k, k * n, m * n, C.byref(h))
    da, db = (torch.as_tensor(np.ascontiguousarray(x.T).ravel(), device="cuda") for x in (As, Bs))
    dc = torch.empty(m * n, dtype=torch.float64, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    call("tnt_compose", rt._h, h, 1, ptr(dc), m * n, ptr(da), m * k, ptr(db), k * n, 1.0, 0.0,
         _lib.PREC_INT8X if precision == "i8" else _lib.PREC_BF16X, slices, rt.stream())
    got = dc.cpu().numpy().reshape(n, m).T
    _lib.lib().tnt_cplan_destroy(h)
    if precision == "i8":
        unit = 1.01 * (slices + 1) * 2.0 ** (2 - 8 * slices) + 2.0 ** -50
    else:
        unit = 1.01 * (slices + 1) * 2.0 ** (-7 * slices) + 2.0 ** -31
    s = e[:, None] + e[None, :]
    ok = abs(s) <= 900  # products that FP64 holds
    assert ok.sum() > m
    back = np.ldexp(np.where(ok, got, 0.0), np.where(ok, -s, 0))
    assert np.all(abs(back - np.where(ok, A @ B, 0.0)) <= k * unit)
