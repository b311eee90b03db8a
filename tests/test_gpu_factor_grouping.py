"""A sector's factors are the same bits alone and in a plan with any others.

A request runs alone, in a tick with others or on a lane of its own, and must publish the
same state; so nothing of a factorisation may depend on its neighbours: lanes per column,
blocks, panel widths, the order of a sum.
"""

import numpy as np
import pytest

from tests.test_gpu_few_columns import run

pytestmark = pytest.mark.gpu

# both edges of the classes, tall and wide sectors, few columns
SHAPES = [(1, 1), (3, 3), (4, 700), (8, 8), (9, 9), (17, 17), (33, 33), (64, 64), (65, 65), (97, 97), (128, 128), (130, 130),
          (161, 161), (300, 300), (330, 330), (400, 400), (620, 620), (650, 650), (20, 500), (500, 20), (60, 1000), (900, 100),
          (200, 641)]


@pytest.mark.parametrize("kind", ["svd", "qr", "eigh"])
@pytest.mark.parametrize("crowd", [0, 80])
def test_bits_do_not_depend_on_the_plan(kind, crowd):
    shapes = [s for s in SHAPES if kind != "eigh" or s[0] == s[1]]
    rng = np.random.default_rng(7)
    blocks = [rng.standard_normal(s) for s in shapes]
    more = [rng.standard_normal(s) for s in [(90, 90), (30, 30), (5, 5), (260, 260)] for _ in range(crowd // 4)]
    if kind == "eigh":
        blocks, more = [b + b.T for b in blocks], [b + b.T for b in more]
    together = {A.tobytes(): f for A, *f in run(kind, [b.shape for b in blocks + more], blocks + more)}
    for b in blocks:
        ((_, *alone),) = run(kind, [b.shape], [b])
        for x, y in zip(alone, together[b.tobytes()]):
            assert np.array_equal(x, y, equal_nan=True), b.shape
