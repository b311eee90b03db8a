"""A factorisation plan's kept tables under several threads (host logic, no GPU)."""

import sys
import threading

import tenet_b200 as tb
from tenet_b200 import typed


class Table:
    device = "cpu"

    def record_stream(self, stream):
        pass


def test_threads_may_fill_and_drop_tables_at_once(monkeypatch):
    class Cuda:
        @staticmethod
        def current_stream(device):
            return None

    monkeypatch.setattr(typed, "_torch", type("Torch", (), {"cuda": Cuda}))
    rule = tb.U1FusionRule()
    leg = tb.GradedSpace(rule, [(0, 2)])
    plan = typed.FactorPlan(typed.HomSpace(rule, [leg], [leg]))
    errors, kept, interval = [], {}, sys.getswitchinterval()

    def use(seed):
        try:
            for i in range(20000):
                key = (seed * 7919 + i) % 1000
                assert plan._kept(kept, key, lambda: (Table(), key))[1] == key
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e))

    threads = [threading.Thread(target=use, args=(s,)) for s in range(8)]
    sys.setswitchinterval(1e-6)
    try:
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert not errors and len(kept) <= 64
