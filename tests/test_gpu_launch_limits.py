"""Plans of different sizes launched by several host threads at once.

A kernel's limit on dynamic shared memory is one value per device: a small plan's
launch must not lower it under a large plan's that another thread is about to make.
Each thread has its own context and stream; no launch fails, and the results are those
of the same calls made alone.
"""

import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run_threads(work, count):
    errors, start = [], threading.Barrier(len(work))

    def loop(f):
        try:
            start.wait()
            for _ in range(count):
                f()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e))

    threads = [threading.Thread(target=loop, args=(f,)) for f in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def dense_space(rt, n):
    import tenet_b200 as tb

    rule = tb.U1FusionRule()
    leg = [tb.GradedSpace(rule, [(0, n)])]
    return rt.space(rule, leg, leg)


# one instantiation each: 54 and 70 KB in one CTA, 51 and 75 on clusters of four, 187 and 206 on wide ones
@pytest.mark.parametrize("sizes", [(49, 64), (65, 96), (289, 320)])
def test_jacobi_launches_of_different_sizes(sizes):
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    p = lambda t: C.c_void_p(t.data_ptr())
    new = lambda n: torch.empty(n, dtype=torch.float64, device="cuda")
    work, checks = [], []
    for n in sizes * 2:
        rt = tb.Runtime(0)
        plan = rt.fplan(dense_space(rt, n))
        stream = torch.cuda.Stream()
        a = torch.as_tensor(np.random.default_rng(n).standard_normal(n * n), device="cuda")
        u, s, v, ws, status = new(n * n), new(n), new(n * n), new(plan.work_elems), torch.zeros(2, dtype=torch.int32,
                                                                                                  device="cuda")
        args = (rt._h, plan._h, p(a), p(u), p(s), p(v), p(ws), p(status), C.c_void_p(stream.cuda_stream))
        _lib.call("tnt_svd_ws_async", *args)
        torch.cuda.synchronize()
        checks.append((s, s.clone(), (rt, plan, a, u, v, ws, status, stream)))
        work.append(lambda args=args: _lib.call("tnt_svd_ws_async", *args))
    for _ in range(10):
        run_threads(work, 150)
        torch.cuda.synchronize()
    assert all(torch.equal(s, want) for s, want, _ in checks)


def test_transposing_launches_of_different_sizes():
    import torch

    import tenet_b200 as tb
    from tenet_b200 import _lib

    p = lambda t: C.c_void_p(t.data_ptr())
    work, checks = [], []
    for n in (1550, 2000) * 2:  # staging of 2700 and 4096 doubles a buffer
        rt = tb.Runtime(0)
        space = dense_space(rt, n)
        plan = rt.xplan(space, "permute", [1], [0])
        stream = torch.cuda.Stream()
        x = torch.as_tensor(np.random.default_rng(n).standard_normal(n * n), device="cuda")
        out = torch.empty_like(x)
        args = (rt._h, plan._h, p(out), p(x), 1.0, 0.0, C.c_void_p(stream.cuda_stream))
        _lib.call("tnt_transform", *args)
        torch.cuda.synchronize()
        checks.append((out, out.clone(), (rt, plan, x, stream)))
        work.append(lambda args=args: _lib.call("tnt_transform", *args))
    for _ in range(10):
        run_threads(work, 800)
        torch.cuda.synchronize()
    assert all(torch.equal(out, want) for out, want, _ in checks)
