"""FP64 grouped compose at the edges of its tile partition, against numpy.

Extents around the 16-row blocks and the 32 .. 80 tile caps, K around the 16-deep
k-tiles and the three-deep ring, padded leading dimensions and odd offsets, in
plans of one tile, of a few and of many.  Each output is a dot product of K
terms: its error stays below 2 (K + 3) rounding errors of sum |a b|.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    [(1, 1, 9)],
    [(15, 17, 16), (16, 16, 17), (33, 31, 33), (1, 81, 47)],
    [(79, 80, 48), (80, 81, 15), (81, 161, 64), (96, 97, 49), (112, 240, 20)],
    [(437, 401, 100), (5, 300, 12), (300, 5, 200), (64, 64, 0)],
    [(200 + i, 230 - i, 40 + i) for i in range(60)],
]


@pytest.mark.parametrize("shapes", CASES)
@pytest.mark.parametrize("alpha,beta,nbatch", [(1.0, 0.0, 1), (-0.75, 0.5, 2)])
def test_f64_tiles_match_numpy(shapes, alpha, beta, nbatch):
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
    rng = np.random.default_rng(len(rows) * 11 + nbatch)
    a, b, c = (rng.standard_normal((nbatch, s)) for s in (na, nb, nc))
    if beta == 0.0:
        c[:] = np.nan
    da, db, dc = (torch.as_tensor(x, device="cuda") for x in (a, b, c))
    ptr = lambda t: C.c_void_p(t.data_ptr())
    call("tnt_compose", rt._h, h, nbatch, ptr(dc), nc, ptr(da), na, ptr(db), nb, alpha, beta, _lib.PREC_FP64, 0,
         rt.stream())
    got = dc.cpu().numpy()
    _lib.lib().tnt_cplan_destroy(h)
    for q in range(nbatch):
        seen = np.zeros(nc, dtype=bool)
        for m, n, k, a0, b0, c0, lda, ldb, ldc in rows:
            blk = lambda x, off, r, cc, ld: np.lib.stride_tricks.as_strided(x[off:], (r, cc), (x.itemsize, x.itemsize * ld))
            A, B = blk(a[q], a0, m, k, lda), blk(b[q], b0, k, n, ldb)
            old = np.zeros((m, n)) if beta == 0.0 else beta * blk(c[q], c0, m, n, ldc)
            bound = 2 * (k + 3) * 2.0 ** -53 * (abs(alpha) * (abs(A) @ abs(B)) + abs(old))
            assert np.all(abs(blk(got[q], c0, m, n, ldc) - (alpha * (A @ B) + old)) <= bound)
            blk(seen, c0, m, n, ldc)[:] = True
        left = got[q][~seen], c[q][~seen]  # what no job covers is left alone
        assert np.array_equal(left[0], left[1], equal_nan=True)


def test_tiles_of_a_small_plan_spread_over_the_gpu():
    """One square sector: the first compose of a plan too small to calibrate on uses the model's constants."""
    import torch

    import tenet_b200 as tb

    rt = tb.Runtime(0)
    rule = tb.U1FusionRule()
    V = tb.GradedSpace(rule, [(0, 304)])
    a, b = (tb.TensorMap(rt, rt.space(rule, [V], [V]), torch.randn(304 * 304, dtype=torch.float64, device="cuda"))
            for _ in range(2))
    x = lambda t: t.data.view(304, 304).t()
    got, want = x(a.compose(b)), x(a) @ x(b)
    assert float((got - want).abs().max()) <= 2 * 307 * 2.0 ** -53 * float((x(a).abs() @ x(b).abs()).max())
