"""The FP64 grouped GEMM's tiles and the rule that picks their size (host logic, no GPU)."""

import ctypes as C
import heapq
import time

import numpy as np
import pytest

from tenet_b200 import _lib

G, B, SMS = 0.67, 0.212, 148


def cplan(jobs):
    rows, a, b, c = [], 0, 0, 0
    for m, n, k in jobs:
        rows.append([m, n, k, a, b, c, m, max(1, k), m])
        a, b, c = a + m * k, b + k * n, c + m * n
    arr = np.asarray(rows, dtype=np.int64)
    h = C.c_void_p()
    _lib.call("tnt_cplan_from_jobs", len(jobs), arr.ctypes.data_as(C.POINTER(C.c_int64)), a, b, c, C.byref(h))
    return h


def tiles(jobs, nbatch=1, g=G, b=B, sms=SMS):
    h = cplan(jobs)
    cap, n = C.c_int32(), C.c_int64()
    try:
        _lib.call("tnt_cplan_f64_tiles", h, nbatch, g, b, sms, C.byref(cap), C.byref(n), 0, None)
        out = np.zeros((n.value, 6), dtype=np.int32)
        _lib.call("tnt_cplan_f64_tiles", h, nbatch, g, b, sms, C.byref(cap), C.byref(n), n.value,
                  out.ctypes.data_as(C.POINTER(C.c_int32)))
        return cap.value, out
    finally:
        _lib.lib().tnt_cplan_destroy(h)


RAGGED = [(1, 1, 1), (16, 16, 0), (17, 80, 33), (81, 96, 5), (437, 300, 64), (20, 300, 50), (300, 20, 50), (33, 33, 900)]


@pytest.mark.parametrize("nbatch", [1, 3, 40])
@pytest.mark.parametrize("sms", [1, 148])
def test_every_output_is_in_one_tile(nbatch, sms):
    cap, got = tiles(RAGGED, nbatch, sms=sms)
    assert 2 <= cap <= 5
    for q in range(nbatch):
        for j, (m, n, _) in enumerate(RAGGED):
            seen = np.zeros((m, n), dtype=int)
            for _, _, m0, n0, h, w in got[(got[:, 0] == j) & (got[:, 1] == q)]:
                assert h <= 16 * cap and w <= 16 * cap and m0 < m and n0 < n
                seen[m0: m0 + h, n0: n0 + w] += 1
            assert np.all(seen == 1)
    assert len(got) == len(np.unique(got[:, :4], axis=0))


def test_pieces_of_a_sector_are_even():
    _, got = tiles([(96, 96, 4000)] * 400)
    assert set(map(tuple, got[:, 4:])) == {(48, 48)}  # two pieces of three blocks, not five and one


def test_longest_tiles_come_first():
    jobs = RAGGED * 5
    _, got = tiles(jobs)
    steps = np.array([-(-jobs[j][2] // 16) + 1 for j in got[:, 0]])
    blocks = np.array([-(-m // 16) * -(-n // 16) for m, n, _ in (jobs[j] for j in got[:, 0])])
    small = blocks <= 4  # sectors of one tile at every cap
    cost = (steps * (G + B * blocks))[small]
    assert np.all(np.diff(cost) <= 1e-9)


def test_small_plans_take_small_tiles_and_large_batches_large_ones():
    assert tiles([(272, 272, 272)])[0] < 5  # one sector: the longest tile's chain is the time
    assert tiles([(272, 272, 272)] * 64)[0] == 5  # the SMs are full: fewest operand bytes per flop
    # a tile that costs no more whatever its size: as few as the SMs allow
    assert tiles([(160, 160, 64)] * 148, g=1.0, b=1e-6)[0] == 5


def test_the_choice_is_cheap_for_plans_of_many_sectors():
    # it runs on the first compose of every plan, and concatenated plans are made per step
    rng = np.random.default_rng(0)
    jobs = [tuple(int(x) for x in rng.integers(1, 200, 3)) for _ in range(60)]
    h = cplan(jobs)
    cap, n = C.c_int32(), C.c_int64()
    best = 1.0
    for _ in range(20):
        t = time.perf_counter()
        _lib.call("tnt_cplan_f64_tiles", h, 64, G, B, SMS, C.byref(cap), C.byref(n), 0, None)
        best = min(best, time.perf_counter() - t)
    _lib.lib().tnt_cplan_destroy(h)
    # these tiles are chosen and written in 0.2 ms; four candidate lists, sorted and dealt, took 10
    assert n.value > 10000 and best < 4e-3


def deal(jobs, nbatch, cap, g=G, b=B, sms=SMS):
    """Time of the cap's list, dealt longest first to the SMs."""
    def pieces(n):
        t = -(-n // cap)
        return [n // t + (i < n % t) for i in range(t)] if n else []

    rows = []
    for q in range(nbatch):
        for j, (m, n, k) in enumerate(jobs):
            h, w = pieces(-(-m // 16)), pieces(-(-n // 16))
            if h and w:
                ks = float(-(-k // 16) + 1)
                rows.append((-ks * (g + b * (h[0] * w[0])), q, j, ks, [x * y for x in h for y in w]))
    rows.sort(key=lambda r: r[:3])
    load, top, chain, total, count = [0.0] * sms, 0.0, 0.0, 0.0, 0
    for *_, ks, blocks in rows:
        for x in blocks:
            c = ks * (g + b * x)
            total, count, chain = total + c, count + 1, max(chain, ks * b * (6.0 + x))
            top = max(top, heapq.heapreplace(load, load[0] + c) + c)
    return max(top, chain) if count <= 20000 else total / sms


SU2_16 = [(s, s, s) for s in (768, 1024, 1536, 512, 256)]  # the SU(2) rank-4 map of 16-dimensional legs
CHOICES = [(SU2_16, 1), ([(768, 768, 768), (1024, 1024, 1024)], 2), (RAGGED, 7)]
for _seed in range(40):
    _r = np.random.default_rng(_seed)
    _n, _most = int(_r.integers(1, 40)), int(_r.choice([40, 200, 700]))
    CHOICES.append(([tuple(int(x) for x in _r.integers(1, _most, 3)) for _ in range(_n)], int(_r.integers(1, 9))))


@pytest.mark.parametrize("jobs,nbatch", CHOICES)
def test_the_choice_is_the_cap_whose_deal_ends_first(jobs, nbatch):
    times = [deal(jobs, nbatch, cap) for cap in (5, 4, 3, 2)]
    got = deal(jobs, nbatch, tiles(jobs, nbatch)[0])
    assert got <= min(times) * (1 + 1e-12)  # the sums' order
