"""Transform plans over every layout of their blocks, against a replay of their tables.

The device runs a plan with neighbouring axes merged where all its blocks allow
it, and cuts transposing copies into tiles of planes.  Here blocks of rank 0 to
6 with extents of 1, small, odd and above a tile are laid out in random axis
orders, packed and padded, in groups of one block and of several: copies are
exact, a sum of n products is within n + 2 rounding errors of sum |u x|.  The
replay runs in extended precision, so that only the kernel rounds.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _replay(tables, src, dst_size):
    """(sum of u x, sum of |u x|) of every destination element."""
    groups, s_e, d_e, coef = tables
    out, mag = np.zeros(dst_size, dtype=np.longdouble), np.zeros(dst_size)
    for g in groups:
        nelem, nsrc, ndst, sf, df, co = (int(x) for x in g[:6])
        multi = np.unravel_index(np.arange(nelem), [int(x) for x in g[6:14]], order="F")
        pos = lambda e: e[0] + sum(multi[k].astype(np.int64) * e[1 + k] for k in range(8))
        at = [pos(s_e[sf + s]) for s in range(nsrc)]
        for d in range(ndst):
            to = pos(d_e[df + d])
            for s in range(nsrc):
                u = coef[co + d * nsrc + s]
                out[to] += np.longdouble(u) * src[at[s]]
                mag[to] += abs(u * src[at[s]])
    return out, mag


def _strides(rng, dims, order, pad):
    st, at = np.zeros(8, dtype=np.int64), 1
    for k in order:
        st[k] = at
        at *= dims[k]
        if pad and rng.random() < 0.4:
            at += int(rng.integers(1, 4))
    return st, at


def _plan(rng, rank, extents, ngroups, most):
    groups, src, dst, coef, ns, nd = [], [], [], [], 0, 0
    for _ in range(ngroups):
        dims = [int(rng.choice(extents)) for _ in range(rank)]
        while np.prod(dims, dtype=np.int64) > most:
            dims[int(rng.integers(rank))] = 1
        full = dims + [1] * (8 - rank)
        n = int(np.prod(full))
        a, b = ((1, 1), (1, 1), (2, 2), (3, 1), (0, 1), (5, 6))[int(rng.integers(6))]
        groups.append([n, a, b, len(src), len(dst), len(coef)] + full)
        coef += list(rng.standard_normal(a * b))
        # one axis order per group: as found, swapped halves, reversed or random
        order = [list(range(rank)), list(range(rank // 2, rank)) + list(range(rank // 2)), list(range(rank))[::-1],
                 list(rng.permutation(rank))][int(rng.integers(4))]
        pad = rng.random() < 0.5
        for _ in range(a):
            st, size = _strides(rng, full, order, pad)
            src.append([ns + int(rng.integers(2))] + list(st))
            ns += size + 1
        for _ in range(b):  # axis 0 runs with stride 1; extents of 1 may sit anywhere
            rest = list(rng.permutation(range(1, rank))) if rank > 1 and rng.random() < 0.5 else list(range(1, rank))
            st, _ = _strides(rng, full, ([0] if rank else []) + rest, False)
            dst.append([nd] + list(st))
            nd += n
    i = lambda x, w: np.asarray(x, dtype=np.int64).reshape(-1, w)
    return (i(groups, 14), i(src, 9), i(dst, 9), np.asarray(coef, dtype=np.float64)), ns + 1, nd


@pytest.mark.parametrize("rank,extents,ngroups,most,seed", [
    (0, [1], 3, 1, 0), (1, [1, 5, 70], 6, 70, 1), (2, [1, 4, 63, 64, 65, 130], 24, 20000, 2),
    (3, [1, 2, 3, 5, 33, 70], 40, 20000, 3), (4, [1, 2, 3, 4, 7, 12], 60, 20000, 4), (5, [1, 2, 3, 5], 60, 3000, 5),
    (6, [1, 2, 3], 60, 800, 6), (2, [700, 900, 1100], 4, 2000000, 7), (4, [24, 30, 37], 4, 2000000, 8),
    (4, [4, 5, 60], 12, 1000000, 9)])
def test_layouts_match_table_replay(rank, extents, ngroups, most, seed):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib
    from tenet_b200._lib import arr, call, i64
    from tenet_b200.typed import TransformPlan

    rt = tb.Runtime(0)
    rng = np.random.default_rng(seed)
    tables, ns, nd = _plan(rng, rank, extents, ngroups, most)
    plan = TransformPlan.from_tables(rank, *tables, ns, nd)
    x, y = rng.standard_normal(ns), rng.standard_normal(nd)
    want, mag = _replay(tables, x, nd)
    units = 2.0 ** -53 * (tables[0][:, 1].max() + 2)
    src = torch.as_tensor(x, device="cuda")
    for alpha, beta in ((1.0, 0.0), (-0.5, 2.0)):  # powers of two: exact
        out = torch.as_tensor(y if beta else np.full(nd, np.nan), device="cuda")
        _lib.call("tnt_transform", rt._h, plan._h, C.c_void_p(out.data_ptr()), C.c_void_p(src.data_ptr()), alpha, beta,
                  rt.stream())
        ref = alpha * want + (beta * y if beta else 0.0)
        assert np.all(abs(out.cpu().numpy() - ref) <= units * mag + 2.0 ** -53 * abs(ref))
    # joined plans keep their blocks apart
    h = C.c_void_p()
    call("tnt_xplan_concat", 2, (C.c_void_p * 2)(plan._h, plan._h), arr(i64, [0, ns]), arr(i64, [nd, 0]), C.byref(h))
    x2 = np.concatenate([x, rng.standard_normal(ns)])
    src, out = torch.as_tensor(x2, device="cuda"), torch.empty(2 * nd, dtype=torch.float64, device="cuda")
    _lib.call("tnt_transform", rt._h, h, C.c_void_p(out.data_ptr()), C.c_void_p(src.data_ptr()), 1.0, 0.0, rt.stream())
    got = out.cpu().numpy()
    _lib.lib().tnt_xplan_destroy(h)
    assert np.all(abs(got[nd:] - want) <= units * mag)
    want, mag = _replay(tables, x2[ns:], nd)
    assert np.all(abs(got[:nd] - want) <= units * mag)
