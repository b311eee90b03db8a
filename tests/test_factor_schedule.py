"""How the factorisations group a plan's sectors, per device (host logic, no GPU).

A plan may be shared by threads on different devices, whose cluster widths differ:
each device's grouping is a value of its own, complete whatever the other threads ask.
"""

import ctypes as C
import threading

import pytest

import tenet_b200 as tb
from tenet_b200 import _lib, typed

U1 = tb.U1FusionRule()
# (rows, columns): general kernels on 16- and 8-CTA clusters and on one CTA, then the three Jacobi widths
SECTORS = [(1500, 1500), (1450, 20), (300, 300), (130, 200), (129, 129), (128, 128), (65, 70), (64, 64), (9, 5), (1, 1)]


def plan_of(sectors):
    rows = tb.GradedSpace(U1, [(q, m) for q, (m, _) in enumerate(sectors)])
    cols = tb.GradedSpace(U1, [(q, n) for q, (_, n) in enumerate(sectors)])
    return typed.FactorPlan(typed.HomSpace(U1, [rows], [cols]))


def schedule(plan, wide):
    counts, runs = (C.c_int32 * 6)(), (C.c_int32 * (2 * plan.nsectors))()
    _lib.call("tnt_fplan_schedule", plan._h, wide, counts, runs)
    return list(counts[:4]), [tuple(runs[2 * i: 2 * i + 2]) for i in range(counts[3])]


def test_grouping_follows_the_cluster_width():
    plan = plan_of(SECTORS)
    (old, clusters, wide, _), runs = schedule(plan, 16)
    assert (old, clusters, wide) == (2, 1, 1) and runs == [(8, 16)]  # 8 x 16 CTAs fit the SMs at once
    (old, clusters, wide, _), runs = schedule(plan, 0)
    assert (old, clusters, wide) == (2, 1, 0) and runs == [(8, 8)]
    many = plan_of([(200, 200)] * 20 + [(100, 100)] * 30 + [(3, 3)] * 150)
    assert schedule(many, 16)[1] == [(20, 16), (30, 4), (150, 1)]
    assert schedule(many, 0)[1] == [(20, 8), (30, 4), (150, 1)]


def test_threads_on_different_devices_share_a_plan():
    plan = plan_of(SECTORS + [(200, 200)] * 20)
    expect = {w: schedule(plan, w) for w in (0, 16)}
    assert expect[0] != expect[16]
    wrong, start = [], threading.Barrier(4)

    def use(w):
        start.wait()
        for _ in range(300):
            got = schedule(plan, w)
            if got != expect[w] or sum(n for n, _ in got[1]) + got[0][0] != plan.nsectors:
                wrong.append((w, got))

    threads = [threading.Thread(target=use, args=(w,)) for w in (0, 16, 0, 16)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("wide", [8, -1, 32])
def test_other_widths_are_refused(wide):
    with pytest.raises(_lib.TenetError):
        schedule(plan_of([(3, 3)]), wide)
