"""Plans give their device tables back when they are destroyed."""

import pytest

pytestmark = pytest.mark.gpu


def free_after(make, count):
    """Free device memory before and after `count` plans are made, used and destroyed."""
    import gc

    import torch

    make()
    torch.cuda.synchronize()
    gc.collect()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(count):
        make()
    torch.cuda.synchronize()
    gc.collect()
    torch.cuda.empty_cache()
    return before, torch.cuda.mem_get_info()[0]


# a transpose, a recoupled and an untransposed permute: every kind of transform tile
@pytest.mark.parametrize("kind", ["transposing", "recoupled", "plain"])
def test_transform_plans_leave_nothing(kind):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import typed

    rt = tb.Runtime(0)
    if kind == "recoupled":
        rule = tb.SU2FusionRule()
        leg = tb.GradedSpace(rule, [(0, 24), (1, 24), (2, 16)])
        space, axes = rt.space(rule, [leg, leg], [leg, leg]), ([0, 2], [1, 3])
    else:
        rule = tb.U1FusionRule()
        leg = tb.GradedSpace(rule, [(0, 1200), (1, 1200)])
        space = rt.space(rule, [leg], [leg])
        axes = ([1], [0]) if kind == "transposing" else ([0], [1])
    x = typed.TensorMap(rt, space, torch.randn(space.size, dtype=torch.float64, device="cuda"))

    def make():
        plan = typed.TransformPlan(space, "permute", *axes, (), 0)
        x._apply(plan)

    before, after = free_after(make, 150)
    # 150 leaked tables of 700 tiles and more would take 7 MB and more; an allocation of the
    # driver's own takes 2 MB at a time
    assert before - after <= 2 << 20
