"""SVD of a plan with a sector that is not finite."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("n", [20, 70, 150, 330])
def test_values_of_a_sector_that_is_not_finite(n, bad):
    """Every value is written, the ones that are not finite first; other sectors are as without it."""
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    rt = tb.Runtime(0)
    rule = tb.U1FusionRule()
    leg = [tb.GradedSpace(rule, [(0, n), (1, 25)])]
    space = rt.space(rule, leg, leg)
    plan = rt.fplan(space)
    x = np.random.default_rng(n).standard_normal(space.size)
    new = lambda c: torch.full((c,), -7.0, dtype=torch.float64, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    out = []
    for spoil in (False, True):
        y = x.copy()
        if spoil:
            y[next(off for _, m, _, off in space.sectors() if m == n) + n + 3] = bad
        a, u, s, v = torch.as_tensor(y, device="cuda"), new(plan.u_size), new(plan.s_size), new(plan.v_size)
        _lib.call("tnt_svd", rt._h, plan._h, p(a), p(u), p(s), p(v), rt.stream())
        s = s.cpu().numpy()
        out.append({r[2]: s[r[5]: r[5] + r[2]] for r in plan.records.tolist()})
    assert np.array_equal(out[0][25], out[1][25])
    finite = np.isfinite(out[1][n])
    assert not finite[0] and np.all(np.diff(finite.astype(int)) >= 0) and not np.any(out[1][n] == -7.0)
