"""The streaming FP64 compose of plans whose every K is at most 8, against numpy."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


# Rows around the wide/tall split (32) and the 512- and 2048-row tiles, columns around the
# 32-column tile and the 2048-element column range, K from 0 to the limit.
CASES = [
    [(1, 5000, 1)],
    [(31, 67, 8), (32, 33, 8), (33, 32, 7)],
    [(2047, 1, 1), (2049, 3, 3), (513, 31, 2), (1025, 65, 5), (4100, 8, 4)],
    [(3, 2049, 4), (40, 40, 0), (7, 9, 0), (200, 1, 8)],
]


@pytest.mark.parametrize("shapes", CASES)
@pytest.mark.parametrize("alpha,beta,nbatch", [(1.0, 0.0, 1), (-0.75, 0.5, 3)])
def test_thin_compose_matches_numpy(shapes, alpha, beta, nbatch):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib
    from tenet_b200._lib import arr, call, i64

    rt = tb.Runtime(0)
    rows, ao, bo, co = [], 1, 2, 3  # odd offsets and padded leading dimensions
    for m, n, k in shapes:
        lda, ldb, ldc = m + 1, max(1, k) + 2, m + 3
        rows.append((m, n, k, ao, bo, co, lda, ldb, ldc))
        ao, bo, co = ao + lda * k, bo + ldb * n, co + ldc * n
    na, nb, nc = ao + 1, bo + 1, co + 1
    h = C.c_void_p()
    call("tnt_cplan_from_jobs", len(rows), arr(i64, [x for r in rows for x in r]), na, nb, nc, C.byref(h))
    rng = np.random.default_rng(len(rows) * 7 + nbatch)
    a, b, c = (rng.standard_normal((nbatch, s)) for s in (na, nb, nc))
    if beta == 0.0:
        c[:] = np.nan  # beta = 0 must not read C
    da, db, dc = (torch.as_tensor(x, device="cuda") for x in (a, b, c))
    ptr = lambda t: C.c_void_p(t.data_ptr())
    call("tnt_compose", rt._h, h, nbatch, ptr(dc), nc, ptr(da), na, ptr(db), nb, alpha, beta, _lib.PREC_FP64, 0,
         rt.stream())
    got = dc.cpu().numpy()
    _lib.lib().tnt_cplan_destroy(h)
    want, bound = c.copy(), np.zeros_like(c)
    for m, n, k, a0, b0, c0, lda, ldb, ldc in rows:
        blk = lambda x, off, r, cc, ld: np.lib.stride_tricks.as_strided(x[off:], (r, cc), (8, 8 * ld))
        for q in range(nbatch):
            A, B = blk(a[q], a0, m, k, lda), blk(b[q], b0, k, n, ldb)
            Cq = blk(c[q], c0, m, n, ldc)
            old = np.zeros((m, n)) if beta == 0.0 else beta * Cq
            blk(want[q], c0, m, n, ldc)[:] = alpha * (A @ B) + old
            blk(bound[q], c0, m, n, ldc)[:] = 2 * (k + 3) * EPS * (abs(alpha) * (abs(A) @ abs(B)) + abs(old))
    same = np.isnan(want) & np.isnan(got)  # what no job covers is left alone
    assert np.all(same | (np.abs(got - want) <= bound))
