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


SVD, QR, EIGH = 0, 1, 2


def schedule(plan, wide, op=SVD):
    counts, runs = (C.c_int32 * 4)(), (C.c_int32 * (2 * plan.nsectors))()
    _lib.call("tnt_fplan_schedule", plan._h, op, wide, counts, runs)
    return list(counts), [tuple(runs[2 * i: 2 * i + 2]) for i in range(counts[3])]


def test_grouping_follows_the_sizes_and_the_cluster_width():
    plan = plan_of(SECTORS)
    (old, clusters, wide, _), runs = schedule(plan, 16)
    assert (old, clusters, wide) == (2, 1, 1) and runs == [(3, 320), (2, 128), (1, 64), (2, 0)]
    (old, clusters, wide, _), runs = schedule(plan, 0)
    assert (old, clusters, wide) == (2, 1, 0) and runs == [(3, 384), (2, 128), (1, 64), (2, 0)]
    assert schedule(plan, 16, QR)[1] == [(6, 640), (2, 0)]
    square = plan_of([(n, n) for n, _ in SECTORS])
    assert schedule(square, 16, EIGH)[1] == [(3, 448), (2, 128), (3, 64)]


@pytest.mark.parametrize("op", [SVD, QR, EIGH])
def test_a_sector_keeps_its_class_in_every_plan(op):
    sizes = [1, 4, 5, 8, 9, 64, 65, 128, 129, 320, 321, 385, 448, 449, 513, 609, 640, 641, 769, 1025, 1408]
    shapes = [(n, n) for n in sizes] + ([] if op == EIGH else [(2, 1408), (700, 8), (640, 8), (30, 641), (300, 900)])
    alone = []
    for s in shapes:
        (old, _, _, n), runs = schedule(plan_of([s]), 16, op)
        assert old == 0 and n == 1
        alone.append(runs[0][1])
    _, runs = schedule(plan_of(shapes), 16, op)
    # every class of the joint plan holds exactly the sectors that have it alone (an SVD splits a
    # class further by the panels of its QR passes)
    joint = {}
    for count, c in runs:
        joint[c] = joint.get(c, 0) + count
    assert joint == {c: alone.count(c) for c in set(alone)}


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
