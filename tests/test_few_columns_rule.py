"""Which plans the SVD and the QR take in one launch of the one-CTA kernels (host logic)."""

import ctypes as C

import pytest

from tenet_b200 import _lib
from tests.test_factor_schedule import plan_of


def few(sectors):
    plan = plan_of(sectors)
    counts = (C.c_int32 * 6)()
    _lib.call("tnt_fplan_schedule", plan._h, 16, counts, None)
    return bool(counts[4]), bool(counts[5])


@pytest.mark.parametrize("sectors,svd,qr", [
    ([(1, 1)], True, True),
    ([(4, 4)] * 200, True, True),
    ([(4, 1408)], True, False),
    ([(1409, 2)], False, True),  # beyond the engine's rows the general kernels run as before
    ([(8, 8)] * 148, True, True),
    ([(8, 8)] * 149, False, True),
    ([(5, 640), (3, 3)], True, False),
    ([(641, 5)], False, False),
    ([(600, 5)], True, True),
    ([(9, 9)], False, False),
    ([(2, 2), (40, 40)], False, False),  # one launch per stage serves all: no further one for the small
    ([(4, 200), (200, 8)], True, True),
    ([(4, 600)] * 36, True, False),
    ([(4, 600)] * 37, True, True),
    ([(5, 600)] * 74, True, False),
    ([(5, 600)] * 75, True, True),
])
def test_rule(sectors, svd, qr):
    assert few(sectors) == (svd, qr)
