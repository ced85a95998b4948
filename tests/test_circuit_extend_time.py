"""Circuits built by many short Circuit.extend calls: time linear in their number."""
import time

import qmetal_gb300 as qm


def _seconds(calls):
    best = 1e9
    for _ in range(3):
        c = qm.Circuit(4)
        t0 = time.perf_counter()
        for _ in range(calls):
            c.extend([(qm.H, (0,), ())])
        best = min(best, time.perf_counter() - t0)
    assert len(c) == calls
    return best


def test_many_short_calls():
    # eight times the calls: 8 where every call costs the same, up to 64 where each copies all gates
    assert _seconds(40000) < 16 * _seconds(5000)
