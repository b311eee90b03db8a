"""Which sectors the SVD and the QR give to the one-CTA kernels (host logic)."""

import pytest

from tests.test_factor_schedule import QR, SVD, plan_of, schedule


def few(shape, op):
    # beside a larger sector: the rule looks at the sector alone
    return schedule(plan_of([shape, (100, 100)]), 16, op)[1][-1] == (1, 0)


@pytest.mark.parametrize("shape,svd,qr", [
    ((1, 1), True, True), ((4, 4), True, True), ((4, 1408), True, False), ((1408, 2), True, True),
    ((8, 8), True, True), ((9, 9), False, False), ((5, 640), True, False), ((641, 5), False, False),
    ((600, 5), True, True), ((601, 5), True, False), ((4, 625), True, True), ((4, 626), True, False),
])
def test_rule(shape, svd, qr):
    assert few(shape, SVD) == svd and few(shape, QR) == qr


def test_many_sectors_keep_it():
    assert schedule(plan_of([(8, 8)] * 300), 16)[1] == [(300, 0)]
