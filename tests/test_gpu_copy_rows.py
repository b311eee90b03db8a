"""Plans made only of copies, around the sizes at which their rows and tiles change.

Plain copies of blocks with axis 0 shorter than a warp (rows that leave lanes idle
and rows that fill them), above and below 3 million elements, and transposing copies of
less than one wave of full tiles, between one and two, and more.  A copy is exact, and
scaling by powers of two is too.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("transposing", [False, True])
@pytest.mark.parametrize("dims,blocks", [
    ((20, 20, 20, 20), 18), ((20, 20, 20, 20), 19), ((17, 31, 5, 40), 40), ((32, 9, 32, 11), 31), ((1, 19, 3, 50), 1100),
    ((3, 90, 91, 4), 31), ((40, 37, 30, 7), 5), ((40, 37, 30, 7), 9), ((40, 37, 30, 7), 14)])
def test_copies_are_exact(dims, blocks, transposing):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib
    from tenet_b200.typed import TransformPlan

    rt = tb.Runtime(0)
    n = int(np.prod(dims))
    st = np.cumprod((1,) + dims[:-1])
    order = (2, 3, 0, 1) if transposing else (0, 1, 2, 3)  # axis order of the source
    inner = np.ones(4, dtype=np.int64)
    at = 1
    for k in order:
        inner[k], at = at, at * dims[k]
    groups = [[n, 1, 1, g, g, g, *dims, 1, 1, 1, 1] for g in range(blocks)]
    src = [[g * n, *inner, 0, 0, 0, 0] for g in range(blocks)]
    dst = [[(blocks - 1 - g) * n, *st, 0, 0, 0, 0] for g in range(blocks)]
    coef = 2.0 ** (np.arange(blocks) % 5)
    i = lambda x: np.asarray(x, dtype=np.int64)
    plan = TransformPlan.from_tables(4, i(groups), i(src), i(dst), coef, n * blocks, n * blocks)
    x = torch.randn(n * blocks, dtype=torch.float64, device="cuda")
    y = torch.randn_like(x)
    v = x.reshape(blocks, *[dims[k] for k in reversed(order)])
    back = [1 + [list(reversed(order)).index(k) for k in (3, 2, 1, 0)][j] for j in range(4)]
    want = (v.permute(0, *back) * torch.as_tensor(coef, device="cuda").reshape(-1, 1, 1, 1, 1)).flip(0).reshape(-1)
    for beta in (0.0, 0.5):
        out = y.clone() if beta else torch.full_like(x, float("nan"))
        _lib.call("tnt_transform", rt._h, plan._h, C.c_void_p(out.data_ptr()), C.c_void_p(x.data_ptr()), 1.0, beta,
                  rt.stream())
        assert torch.equal(out, want + beta * y if beta else want)
