"""A failed eigendecomposition leaves its outputs as they were."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# a bad sector beside good ones on every engine: one CTA, clusters, staged, the general SVD
@pytest.mark.parametrize("sizes,bad", [([20, 33], 0), ([20, 33], 1), ([70, 150, 20], 2), ([20, 460], 0), ([20, 460], 1),
                                       ([30, 1410], 0), ([30, 1410], 1)])
@pytest.mark.parametrize("how", ["asymmetric", "nan"])
def test_outputs_are_untouched(sizes, bad, how):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    rt = tb.Runtime(0)
    rule = tb.U1FusionRule()
    leg = tb.GradedSpace(rule, [(q, n) for q, n in enumerate(sizes)])
    space = rt.space(rule, [leg], [leg])
    plan = rt.fplan(space)
    rng = np.random.default_rng(sum(sizes))
    payload = np.empty(space.size)
    for i, (_, n, _, off) in enumerate(space.sectors()):
        g = rng.standard_normal((n, n))
        g = np.eye(n) + 1e-3 * (g + g.T) / n
        if n == sizes[bad]:
            g[1, 0] = 0.5 if how == "asymmetric" else np.nan
        payload[off: off + n * n] = g.ravel()
    a = torch.as_tensor(payload, device="cuda")
    outs = [torch.full((x,), 7.0, dtype=torch.float64, device="cuda") for x in (plan.u_size, plan.s_size, plan.s_size)]
    p = lambda t: C.c_void_p(t.data_ptr())
    with pytest.raises(_lib.TenetError, match="Hermitian"):
        _lib.call("tnt_eigh", rt._h, plan._h, p(a), *(p(t) for t in outs), rt.stream())
    torch.cuda.synchronize()
    assert all(bool((t == 7.0).all()) for t in outs)
