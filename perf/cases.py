"""Performance cases: the block-sparse tensor work a program has this package do.

Each case is one call sequence through the public entry points at one size.
``listed`` names fixed ones, ``draw`` gives more of the same ranges.  ``exact``
restates the result in 64-bit torch from the charges and degeneracies alone
(per coupled sector; abelian permutes on the dense tensor).

Inputs are N(0, 1) (the start of a simulation) or carry a decaying Schmidt
spectrum over ``decades`` powers of ten (a simulation under way).
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import tenet_b200 as tb
from tenet_b200 import _lib, heff, itebd

DEV = "cuda:0"
_rt = None


def _runtime():
    """One Runtime per process, as a user's program keeps it (plans are cached on it)."""
    global _rt
    if _rt is None:
        _rt = tb.Runtime(0)
    return _rt


def listed():
    return [
        # The smallest ordinary call: one U(1) compose and one permute of 36-dimensional legs (latency, launches).
        dict(name="u1_compose_permute", kind="u1_compose_permute", scale=1.0),
        # The bond matrix of a small chain of a simulation service (D = 32, spins 0..3): a truncated SVD, call by call.
        dict(name="svd_d32", kind="svd", profile="flat", D=32, policy="space", decades=3),
        # One whole two-site SU(2) iTEBD update (contract, gate, recouple, truncated SVD, factors), D = 224.
        dict(name="bond_update_d224", kind="bond", profile="bell", D=224, tau=0.05, policy="space", decades=3),
        # The bond matrix of the service's largest chain (D = 2048, sectors of 586 x 586).
        dict(name="svd_d2048", kind="svd", profile="flat", D=2048, policy="space", decades=0),
        # Canonical form of an MPS tensor: QR of a bond matrix whose sectors (293 x 293) exceed shared memory.
        dict(name="qr_d1024", kind="qr", profile="flat", D=1024),
        # Spectrum of a density matrix over (W x P), D = 224.
        dict(name="eigh_d224", kind="eigh", profile="bell", D=224, policy="full"),
        # Recoupling of the effective-Hamiltonian network's largest intermediate (6j, long rows, 0.5 GB moved).
        dict(name="permute_su2_heff_t1", kind="su2_permute", scale=1.0, step="t1"),
        # Swapping codomain and domain of a U(1) rank-4 tensor: a block transpose (0.6 GB moved).
        dict(name="permute_u1_transpose", kind="u1_permute", d=12, axes="23|01"),
        # The batched Hubbard contraction: 64 composes over 120 uneven coupled sectors, plain FP64.
        dict(name="hubbard_fp64", kind="hubbard", nsectors=60, mean=48.0, space_seed=0, batch=64, precision="fp64", slices=0),
        # The same batch in 8-bit digits on the tensor cores (five digits, about 4e-11).
        dict(name="hubbard_i8x5", kind="hubbard", nsectors=60, mean=48.0, space_seed=0, batch=64, precision="i8x", slices=5),
        # One effective-Hamiltonian matvec at full size, 8-bit digits with the constant operands packed once.
        dict(name="heff_i8x5", kind="heff", scale=1, precision="i8x", slices=5),
        # A whole ground-state solve of a small network: 30 Lanczos steps, FP64, vectors resident.
        dict(name="lanczos_fp64", kind="lanczos", scale=4, iterations=30, precision="fp64", slices=0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["u1_compose_permute", "svd", "svd", "bond", "qr", "eigh", "su2_permute", "u1_permute",
                       "hubbard", "hubbard", "heff", "lanczos"])
    prof = rng.choice(["flat", "bell"])
    policy = rng.choice(["space", "space", "rank", "tolerance", "full"])
    if kind == "u1_compose_permute":
        return dict(kind=kind, scale=round(_log(rng, 0.5, 5.0), 3))
    if kind == "svd":
        return dict(kind=kind, profile=prof, D=int(_log(rng, 32, 1400 if prof == "flat" else 900)), policy=policy,
                    decades=rng.choice([0, 3]))
    if kind == "bond":
        return dict(kind=kind, profile=prof, D=int(_log(rng, 32, 1000 if prof == "flat" else 600)),
                    tau=rng.choice([0.01, 0.05, 0.1]), policy="space", decades=rng.choice([0, 3]))
    if kind == "qr":
        return dict(kind=kind, profile=prof, D=int(_log(rng, 32, 2048 if prof == "flat" else 1200)))
    if kind == "eigh":
        return dict(kind=kind, profile=prof, D=int(_log(rng, 32, 1400 if prof == "flat" else 900)), policy="full")
    if kind == "su2_permute":
        return dict(kind=kind, scale=round(_log(rng, 1.0, 20.0), 3), step=rng.choice(["x", "t1", "t2"]))
    if kind == "u1_permute":
        return dict(kind=kind, d=rng.randint(3, 12), axes=rng.choice(["23|01", "01|32", "03|21", "2013|", "1|302"]))
    if kind == "hubbard":
        prec, sl = rng.choice([("fp64", 0), ("fp64", 0), ("i8x", 5), ("i8x", 6), ("i8x", 4), ("bf16x", 5), ("bf16x", 6)])
        return dict(kind=kind, nsectors=rng.randint(8, 60), mean=round(_log(rng, 6, 44), 2),
                    space_seed=rng.randrange(1000), batch=int(_log(rng, 1, 48)), precision=prec, slices=sl)
    if kind == "heff":
        prec, sl = rng.choice([("fp64", 0), ("i8x", 5), ("i8x", 6), ("bf16x", 5)])
        return dict(kind=kind, scale=int(_log(rng, 2 if prec != "i8x" else 1, 16)), precision=prec, slices=sl)
    prec, sl = rng.choice([("fp64", 0), ("i8x", 6)])
    return dict(kind=kind, scale=int(_log(rng, 4, 32)), iterations=rng.randint(8, 30), precision=prec, slices=sl)


# ---------------------------------------------------------------------------
# spaces of the cases: (label, degeneracy) lists
# ---------------------------------------------------------------------------


def _chain_leg(case):
    """The bond space W of a chain: D split evenly over spins 0..3, or a bell over spins 0..2."""
    D = case["D"]
    if case["profile"] == "flat":
        return [((t,), max(1, round(D / 7.0))) for t in range(7)]
    return [((t,), max(1, round(D * w / 224.0))) for t, w in zip(range(5), [40, 64, 64, 40, 16])]


def _u1_leg(degs):
    return [((q,), max(1, round(d))) for q, d in zip(range(-2, 3), degs)]


def _hubbard_legs(case):
    rng = np.random.default_rng(case["space_seed"])
    cand = [((tj % 2), q, tj) for q in range(-7, 8) for tj in range(0, 7)]
    pick = sorted(rng.choice(len(cand), size=case["nsectors"], replace=False))
    degs = np.clip(rng.geometric(1.0 / case["mean"], size=case["nsectors"]), 1, 256)
    return [(cand[i], int(d)) for i, d in zip(pick, degs)], [((0, 0, 0), 1), ((1, 1, 1), 1), ((0, 2, 0), 1)]


def _heff_legs(scale):
    w = [((t,), max(1, round(d / scale)))
         for t, d in zip(range(9), [256, 512, 768, 1024, 1024, 768, 512, 256, 128])]
    return w, [((0,), 2), ((2,), 1)], [((1,), 1)]


_SPIN_HALF = [((1,), 1)]
_MPO = dict(x=([0], [1, 2]), t1=([0, 3], [1, 2]), t2=([0, 3], [1, 2]))


# ---------------------------------------------------------------------------
# restatement helpers: coupled sectors and dense abelian tensors, from the charges alone
# ---------------------------------------------------------------------------


def _zigzag(q):
    return 2 * q if q >= 0 else -2 * q - 1


def _order(factors, label):
    """Storage order of a sector: the last factor is the most significant."""
    return tuple(_zigzag(v) if f == "U1" else v for f, v in zip(factors, label))[::-1]


def _fuse(factors, a, b):
    out = [()]
    for f, x, y in zip(factors, a, b):
        vals = [x + y] if f == "U1" else [(x + y) % 2] if f == "FZ2" else list(range(abs(x - y), x + y + 1, 2))
        out = [o + (v,) for o in out for v in vals]
    return out


def _coupled(factors, leg1, leg2):
    """[(sector, dimension)] of leg1 x leg2 in storage order."""
    dims = {}
    for a, da in leg1:
        for b, db in leg2:
            for c in _fuse(factors, a, b):
                dims[c] = dims.get(c, 0) + da * db
    return sorted(dims.items(), key=lambda kv: _order(factors, kv[0]))


def _square_sectors(factors, leg1, leg2):
    """[(offset, n)] of a tensor (leg1 x leg2) <- (leg2 x leg1) or <- (leg1 x leg2)."""
    out, off = [], 0
    for _, n in _coupled(factors, leg1, leg2):
        out.append((off, n))
        off += n * n
    return out


def _pairs(la, lb):
    """Block positions of a pair of U(1) legs per total charge: [(a, b)] first leg fastest."""
    out = {}
    for ib in range(len(lb)):
        for ia in range(len(la)):
            out.setdefault(la[ia][0] + lb[ib][0], []).append((ia, ib))
    return out


def _spans(leg):
    pos, out = 0, []
    for _, d in leg:
        out.append(slice(pos, pos + d))
        pos += d
    return out


def _trees(legs):
    """{total charge: [position tuple]} over any number of U(1) legs, first leg fastest."""
    tuples = [((), 0)]
    for leg in legs:
        tuples = [(t + (i,), q + leg[i][0]) for i in range(len(leg)) for t, q in tuples]
    out = {}
    for t, q in tuples:
        out.setdefault(q, []).append(t)
    return out


def _u1_blocks(cod, dom):
    """Yield (sector offset, rows, row offset, row shape, col offset, col shape, cod tuple, dom tuple)."""
    tc, td = _trees(cod), _trees(dom)
    off = 0
    for q in sorted(set(tc) & set(td), key=_zigzag):
        shape = lambda legs, t: [legs[k][i][1] for k, i in enumerate(t)]
        rows = sum(math.prod(shape(cod, t)) for t in tc[q])
        cols = sum(math.prod(shape(dom, t)) for t in td[q])
        co = 0
        for t2 in td[q]:
            ro = 0
            for t1 in tc[q]:
                yield off, rows, ro, shape(cod, t1), co, shape(dom, t2), t1, t2
                ro += math.prod(shape(cod, t1))
            co += math.prod(shape(dom, t2))
        off += rows * cols


def _u1_dense(data, cod, dom):
    legs = cod + dom
    out = torch.zeros([sum(d for _, d in l) for l in legs], dtype=torch.float64, device=data.device)
    sp = [_spans(l) for l in legs]
    for off, rows, ro, s1, co, s2, t1, t2 in _u1_blocks(cod, dom):
        n1, n2 = math.prod(s1), math.prod(s2)
        blk = data.as_strided((n2, n1), (rows, 1), off + co * rows + ro).reshape(s2[::-1] + s1[::-1])
        blk = blk.permute(list(range(len(legs)))[::-1])  # axis 0 .. rank-1, now dom axes come first reversed
        out[tuple(s[i] for s, i in zip(sp, t1 + t2))] = blk
    return out


def _u1_payload(dense, cod, dom):
    legs = cod + dom
    sp = [_spans(l) for l in legs]
    parts, cur, buf = [], None, None
    for off, rows, ro, s1, co, s2, t1, t2 in _u1_blocks(cod, dom):
        if off != cur:
            cols = sum(math.prod([dom[k][i][1] for k, i in enumerate(t)])
                       for t in _trees(dom)[sum(cod[k][i][0] for k, i in enumerate(t1))])
            buf = torch.empty((cols, rows), dtype=torch.float64, device=dense.device)
            parts.append(buf)
            cur = off
        n1, n2 = math.prod(s1), math.prod(s2)
        blk = dense[tuple(s[i] for s, i in zip(sp, t1 + t2))].permute(list(range(len(legs)))[::-1]).reshape(n2, n1)
        buf[co: co + n2, ro: ro + n1] = blk
    return torch.cat([p.reshape(-1) for p in parts])


def _u1_permuted(data, cod, dom, p1, p2):
    """The payload of permute(p1, p2): a leg that changes sides carries the negated charges."""
    legs, n1 = cod + dom, len(cod)
    dense = _u1_dense(data, cod, dom)
    new_c, new_d, axes = [], [], list(p1) + list(p2)
    for k, a in enumerate(axes):
        moved = (a < n1) != (k < len(p1))
        leg = legs[a]
        if moved:
            order = sorted(range(len(leg)), key=lambda i: _zigzag(-leg[i][0]))
            idx = torch.cat([torch.arange(s.start, s.stop) for s in (_spans(leg)[i] for i in order)]).to(dense.device)
            dense = dense.index_select(a, idx)
            leg = [(-leg[i][0], leg[i][1]) for i in order]
        (new_c if k < len(p1) else new_d).append(leg)
    return _u1_payload(dense.permute(axes), new_c, new_d)


def _plain_leg(leg):
    """(charge, degeneracy) in storage order."""
    return sorted([(s[0], d) for s, d in leg], key=lambda x: _zigzag(x[0]))


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------


def _space(rule, leg):
    return tb.GradedSpace(rule, [(s if rule.nfactors > 1 else s[0], d) for s, d in leg])


def _randn(gen, n):
    return torch.randn(n, dtype=torch.float64, device=DEV, generator=gen)


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _matrix_payload(case, gen):
    """Square sectors over (W x P): N(0, 1), or U diag(decay) V with a spectrum over `decades`."""
    out = []
    for _, n in _square_sectors(["SU2"], _chain_leg(case), _SPIN_HALF):
        g = _randn(gen, n * n).view(n, n)
        if case.get("decades", 0):
            dec = 10.0 ** (-case["decades"] * torch.arange(n, dtype=torch.float64, device=DEV) / n)
            g = (g * dec) @ _randn(gen, n * n).view(n, n) / math.sqrt(n)
        out.append(g.reshape(-1))
    return torch.cat(out)


def _symmetric_payload(case, gen):
    out = []
    for _, n in _square_sectors(["SU2"], _chain_leg(case), _SPIN_HALF):
        g = _randn(gen, n * n).view(n, n)
        h = g @ g.t() / n
        out.append((0.5 * (h + h.t())).reshape(-1))
    return torch.cat(out)


def _truncation(case, W):
    p = case["policy"]
    if p == "space":
        return tb.Truncation.space(W)
    if p == "rank":
        return tb.Truncation.rank(W.dim())
    if p == "tolerance":
        return tb.Truncation.tolerance(0.0, 1e-3)
    return tb.Truncation.full()


def _heff_tensors(rt, gen, legs):
    rule = tb.SU2FusionRule()
    W, M, P = (_space(rule, l) for l in legs)
    mk = lambda cod, dom: tb.TensorMap(rt, rt.space(rule, cod, dom), _randn(gen, rt.space(rule, cod, dom).size))
    return mk([W, P], [W]), mk([W, M], [W]), mk([M, P], [P, M]), mk([W, M.dual()], [W])


def _su2_permute_source(rt, case):
    """The source space of one permute of the effective-Hamiltonian network, and its axes."""
    rule = tb.SU2FusionRule()
    W, M, P = (_space(rule, l) for l in _heff_legs(case["scale"]))
    x = rt.space(rule, [W, P], [W])
    if case["step"] == "x":
        return x
    t1 = rt.space(rule, [W, M], [P.dual(), W])
    if case["step"] == "t1":
        return t1
    t1p = rt.xplan(t1, "permute", [0, 3], [1, 2]).dst
    op = rt.xplan(rt.space(rule, [M, P], [P, M]), "permute", [3, 2], [0, 1]).dst
    return rt.cplan(t1p, op).dst


def prepare(case, seed):
    rt, gen, kind = _runtime(), _generator(seed), case["kind"]
    st = dict(case=case, rt=rt)
    if kind in ("u1_compose_permute", "u1_permute"):
        rule = tb.U1FusionRule()
        V = _space(rule, _u1_case_leg(case))
        sp = rt.space(rule, [V, V], [V, V])
        st["A"] = tb.TensorMap(rt, sp, _randn(gen, sp.size))
        if kind == "u1_compose_permute":
            st["B"] = tb.TensorMap(rt, sp, _randn(gen, sp.size))
        else:
            st["axes"] = _axes(case)
    elif kind in ("svd", "qr", "eigh"):
        rule = tb.SU2FusionRule()
        W, P = _space(rule, _chain_leg(case)), _space(rule, _SPIN_HALF)
        sp = rt.space(rule, [W, P], [W, P])
        st["T"] = tb.TensorMap(rt, sp, _symmetric_payload(case, gen) if kind == "eigh" else _matrix_payload(case, gen))
        if kind != "qr":
            st["trunc"] = _truncation(case, W)
    elif kind == "bond":
        rule = tb.SU2FusionRule()
        W, P = _space(rule, _chain_leg(case)), _space(rule, _SPIN_HALF)
        sp = rt.space(rule, [W, P], [W])
        st["A"], st["B"] = (tb.TensorMap(rt, sp, _randn(gen, sp.size)) for _ in range(2))
        if case["decades"]:  # Schmidt values of the middle bond on A's domain
            for _, r, c, off in sp.sectors():
                dec = 10.0 ** (-case["decades"] * torch.arange(c, dtype=torch.float64, device=DEV) / c)
                st["A"].data[off: off + r * c].view(c, r).mul_(dec[:, None])
        st["G"] = itebd.heisenberg_gate(rt, rule, P, case["tau"])
        st["trunc"] = _truncation(case, W)
    elif kind == "su2_permute":
        sp = _su2_permute_source(rt, case)
        st["A"], st["axes"] = tb.TensorMap(rt, sp, _randn(gen, sp.size)), _MPO[case["step"]]
    elif kind == "hubbard":
        rule = tb.FusionRule(["FZ2", "U1", "SU2"])
        W, P = (_space(rule, l) for l in _hubbard_legs(case))
        a_sp, b_sp = rt.space(rule, [W, P], [P, W]), rt.space(rule, [P, W], [W, P])
        n = case["batch"]
        st["plan"] = rt.cplan(a_sp, b_sp)
        st["a"], st["b"] = _randn(gen, n * a_sp.size), _randn(gen, n * b_sp.size)
        st["c"] = torch.empty(n * st["plan"].dst.size, dtype=torch.float64, device=DEV)
        st["strides"] = (st["plan"].dst.size, a_sp.size, b_sp.size)
    else:  # heff, lanczos
        x, L, O, R = _heff_tensors(rt, gen, _heff_legs(case["scale"]))
        st["x"], st["H"] = x, heff.EffectiveHamiltonian(L, O, R)
    return st


def _u1_case_leg(case):
    if case["kind"] == "u1_permute":
        return _u1_leg([case["d"] * w for w in (1, 2, 4, 2, 1)])
    return _u1_leg([case["scale"] * d for d in (4, 8, 12, 8, 4)])


def _axes(case):
    a, b = case["axes"].split("|")
    return [int(x) for x in a], [int(x) for x in b]


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------


def _svd_outputs(res):
    u, s, vh = res.factors()
    return dict(u=u.data, s=[e.values for e in s], vh=vh.data, kept=np.asarray(res.kept), error=res.error)


def run(st):
    case, rt = st["case"], st["rt"]
    kind = case["kind"]
    if kind == "u1_compose_permute":
        c = st["A"].compose(st["B"])
        return dict(c=c.data, p=c.permute([0, 3], [2, 1]).data)
    if kind in ("u1_permute", "su2_permute"):
        return st["A"].permute(*st["axes"]).data
    if kind == "svd":
        return _svd_outputs(st["T"].svd_trunc(st["trunc"]))
    if kind == "bond":
        return _svd_outputs(itebd.bond_update(st["A"], st["B"], st["G"], st["trunc"]))
    if kind == "qr":
        q, r = st["T"].qr_compact()
        return dict(q=q.data, r=r.data)
    if kind == "eigh":
        res = st["T"].eigh_trunc(st["trunc"])
        d, v = res.factors()
        return dict(d=d.data, v=v.data, w=[e.values for e in res.eigenvalues])
    if kind == "hubbard":
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())
        prec = dict(fp64=_lib.PREC_FP64, i8x=_lib.PREC_INT8X, bf16x=_lib.PREC_BF16X)[case["precision"]]
        sc, sa, sb = st["strides"]
        _lib.call("tnt_compose", rt._h, st["plan"]._h, case["batch"], ptr(st["c"]), sc, ptr(st["a"]), sa,
                  ptr(st["b"]), sb, 1.0, 0.0, prec, case["slices"], rt.stream())
        return st["c"]
    if kind == "heff":
        return st["H"].apply(st["x"], case["precision"], case["slices"]).data
    e0, ritz, alphas, betas = heff.lanczos(st["H"], st["x"], case["iterations"], case["precision"], case["slices"])
    return dict(e0=e0, ritz=ritz.data, alphas=np.asarray(alphas), betas=np.asarray(betas))


# ---------------------------------------------------------------------------
# work: each input read once, each output written once; flops of the reduced blocks
# ---------------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind in ("u1_compose_permute", "u1_permute"):
        leg = _plain_leg(_u1_case_leg(case))
        ns = [sum(leg[a][1] * leg[b][1] for a, b in ps) for ps in _pairs(leg, leg).values()]
        el = sum(n * n for n in ns)
        if kind == "u1_permute":
            return dict(bytes=16 * el, flops=el)
        return dict(bytes=8 * 5 * el, flops=2 * sum(n ** 3 for n in ns))
    if kind in ("svd", "bond", "qr", "eigh"):
        ns = [n for _, n in _square_sectors(["SU2"], _chain_leg(case), _SPIN_HALF)]
        el, cube = sum(n * n for n in ns), sum(n ** 3 for n in ns)
        per = dict(svd=22, bond=22, qr=8.0 / 3, eigh=9)[kind]  # Golub-Van Loan counts of the dense factorisations
        return dict(bytes=8 * (2 if kind == "eigh" else 3) * el, flops=per * cube)
    if kind == "hubbard":
        ns = [n for _, n in _coupled(["FZ2", "U1", "SU2"], *_hubbard_legs(case))]
        return dict(bytes=case["batch"] * 8 * 3 * sum(n * n for n in ns),
                    flops=case["batch"] * 2 * sum(n ** 3 for n in ns))
    w, m, p = _heff_legs(case["scale"])
    dims = {c[0]: d for c, d in w}
    wp, wm = dict(_coupled(["SU2"], w, p)), dict(_coupled(["SU2"], w, m))
    x = sum(wp.get((j,), 0) * d for j, d in dims.items())
    env = sum(wm.get((j,), 0) * d for j, d in dims.items())
    if kind == "su2_permute":  # t1, t2: blocks (W x M) <- (P x W)
        el = x if case["step"] == "x" else sum(wm[c] * wp[c] for c in wp if c in wm)
        return dict(bytes=16 * el, flops=2 * el)
    flops = 2 * 2 * 2 * sum(wm.get((j,), 0) * d * wp.get((j,), 0) for j, d in dims.items())  # L, R, and the adjoints
    if kind == "heff":
        return dict(bytes=8 * (2 * x + 2 * env), flops=flops)
    k = case["iterations"]
    return dict(bytes=8 * (k * 2 * env + x * (2 * k + 2 * k * k)), flops=k * flops + 4 * k * k * x)


# ---------------------------------------------------------------------------
# exact
# ---------------------------------------------------------------------------


def _exact_svd(case, data):
    keep = dict((t[0], d) for t, d in _chain_leg(case))
    labels = [c for c, _ in _coupled(["SU2"], _chain_leg(case), _SPIN_HALF)]
    secs = _square_sectors(["SU2"], _chain_leg(case), _SPIN_HALF)
    us, ss, vs = [], [], []
    for off, n in secs:
        u, s, vh = torch.linalg.svd(data[off: off + n * n].view(n, n).t().cpu())
        sign = torch.where(u.gather(0, u.abs().argmax(0, keepdim=True)) < 0, -1.0, 1.0).to(torch.float64)
        us.append(u * sign)
        ss.append(s)
        vs.append(vh * sign.t())
    weight = [c[0] + 1 for c in labels]
    norm = math.sqrt(sum(w * float((s * s).sum()) for w, s in zip(weight, ss)))
    if case["policy"] == "space":
        kept = [min(keep.get(c[0], 0), n) for c, (_, n) in zip(labels, secs)]
    elif case["policy"] == "tolerance":
        kept = [int((s >= 1e-3 * norm).sum()) for s in ss]
    elif case["policy"] == "full":
        kept = [n for _, n in secs]
    else:
        budget = sum((j + 1) * d for j, d in keep.items())
        cand = sorted((-float(s[i]), j, i) for j, s in enumerate(ss) for i in range(len(s)))
        kept, total = [0] * len(ss), 0
        for _, j, i in cand:
            total += weight[j]
            if total > budget:
                break
            kept[j] += 1
    cut = math.sqrt(sum(w * float((s[k:] * s[k:]).sum()) for w, s, k in zip(weight, ss, kept)))
    live = [i for i, k in enumerate(kept) if k > 0]
    return dict(u=torch.cat([us[i][:, : kept[i]].t().reshape(-1) for i in live]),
                s=[ss[i][: kept[i]].numpy() for i in range(len(ss))],
                vh=torch.cat([vs[i][: kept[i]].t().reshape(-1) for i in live]),
                kept=np.asarray(kept), error=cut)


def exact(case, seed):
    kind, gen = case["kind"], _generator(seed)
    if kind in ("u1_compose_permute", "u1_permute"):
        leg = _plain_leg(_u1_case_leg(case))
        secs, off = [], 0
        for q, ps in sorted(_pairs(leg, leg).items(), key=lambda kv: _zigzag(kv[0])):
            n = sum(leg[a][1] * leg[b][1] for a, b in ps)
            secs.append((off, n))
            off += n * n
        a = _randn(gen, off)
        if kind == "u1_permute":
            return _u1_permuted(a, [leg, leg], [leg, leg], *_axes(case))
        b = _randn(gen, off)
        c = torch.cat([(b[o: o + n * n].view(n, n) @ a[o: o + n * n].view(n, n)).reshape(-1) for o, n in secs])
        return dict(c=c, p=_u1_permuted(c, [leg, leg], [leg, leg], [0, 3], [2, 1]))
    if kind == "svd":
        return _exact_svd(case, _matrix_payload(case, gen))
    if kind == "qr":
        data, qs, rs = _matrix_payload(case, gen), [], []
        for off, n in _square_sectors(["SU2"], _chain_leg(case), _SPIN_HALF):
            q, r = torch.linalg.qr(data[off: off + n * n].view(n, n).t().cpu())
            sign = torch.where(r.diagonal() < 0, -1.0, 1.0).to(torch.float64)
            qs.append((q * sign).t().reshape(-1))
            rs.append((r * sign[:, None]).t().reshape(-1))
        return dict(q=torch.cat(qs), r=torch.cat(rs))
    if kind == "eigh":
        data, ds, vs, ws = _symmetric_payload(case, gen), [], [], []
        for off, n in _square_sectors(["SU2"], _chain_leg(case), _SPIN_HALF):
            w, v = torch.linalg.eigh(data[off: off + n * n].view(n, n).cpu())
            w, v = w.flip(0), v.flip(1)
            v = v * torch.where(v.gather(0, v.abs().argmax(0, keepdim=True)) < 0, -1.0, 1.0).to(torch.float64)
            ds.append(torch.diag(w).reshape(-1))
            vs.append(v.t().reshape(-1))
            ws.append(w.numpy())
        return dict(d=torch.cat(ds), v=torch.cat(vs), w=ws)
    if kind == "hubbard":
        secs, n = _square_sectors(["FZ2", "U1", "SU2"], *_hubbard_legs(case)), case["batch"]
        size = secs[-1][0] + secs[-1][1] ** 2
        a, b = _randn(gen, n * size).view(n, size), _randn(gen, n * size).view(n, size)
        c = torch.empty_like(a)
        for off, d in secs:
            blk = lambda t: t[:, off: off + d * d].view(n, d, d)  # row-major view of a column-major block: transposed
            c[:, off: off + d * d] = torch.bmm(blk(b), blk(a)).reshape(n, d * d)
        return c.reshape(-1)
    return None  # SU(2) recoupling: no restatement without the 6j machinery
