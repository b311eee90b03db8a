"""The streaming FP64 compose at the edges of its row mappings, against numpy.

Rows around the flat mapping (9), the equal parts of at most 255 rows a thread each, and the
tall tiles (1024); columns around the groups, the 256 staged ones and the splits into
fewer columns per thread; plans of a few and of many tiles.
"""

import pytest

from tests.test_gpu_gemm_thin import test_thin_compose_matches_numpy as check

pytestmark = pytest.mark.gpu

ROWS = [8, 9, 10, 16, 31, 33, 64, 85, 86, 127, 128, 129, 255, 256, 257, 300, 511, 513, 1000, 1023, 1024, 1025]


@pytest.mark.parametrize("k", range(9))
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.75, 0.5)])
def test_row_mappings(k, alpha, beta):
    columns = [1, 3, 8, 9, 33, 65, 255, 256, 257, 300, 700]
    check([(m, columns[(i + k) % len(columns)], k) for i, m in enumerate(ROWS)], alpha, beta, 2)


# more tiles than resident CTAs: 32 columns per thread, 2048-row tiles
@pytest.mark.parametrize("shapes", [[(40, 70000, 5)], [(9, 60000, 8), (300, 3000, 3)], [(1500, 1300, 7)], [(3000, 2, 4)]])
def test_plans_that_fill_the_device(shapes):
    check(shapes, 1.0, 0.0, 1 if len(shapes[0]) and shapes[0][1] > 2 else 400)


def test_large_batch_of_middle_rows():
    check([(33, 40, 8), (100, 7, 2)], 0.5, 0.0, 300)


