"""Circuit.extend against Circuit.add, gate by gate: the same plan, and for a
gate that add refuses the same error with the same gates before it."""
import numpy as np
import pytest

import qmetal_gb300 as qm
from qmetal_gb300 import workloads as W

CIRCUITS = [W.hea(5, 2), W.qaoa_ring_seeded(6, 2), W.qft_swap(5), W.grover_proxy(5, 2), [],
            [(qm.U3, (1,), (0.1, 0.2, 0.3)), (W.CCX, (0, 1, 2), ()), (W.CP, (0, 2), (0.4,))],
            [(np.int64(W.RX), (np.int64(1),), (np.float32(0.5),)), (W.H, [0], [])]]
REFUSED = [[(W.X, (5,), ())], [(99, (0,), ())], [(W.X, (), ())], [(W.X, (0, 1, 2, 3), ())],
           [(W.H, (0,), ()), (W.RX, (1,), (0.2,)), (W.CX, (0, 7), ()), (W.H, (1,), ())],
           [(qm.U3, (0,), (0.1,))], [(W.RX, (0,), (0.1, 0.2, 0.3, 0.4))]]


def _one_at_a_time(c, gates):
    for k, qs, ps in gates:
        c.add(k, qs, ps)
    return c


@pytest.mark.parametrize("gates", CIRCUITS)
def test_extend(gates):
    a, b = qm.Circuit(6).extend(gates), _one_at_a_time(qm.Circuit(6), gates)
    assert len(a) == len(b) == len(gates)
    assert list(a.plan_export()) == list(b.plan_export())
    assert a.extend(gates) is a and len(a) == 2 * len(gates)


@pytest.mark.parametrize("gates", REFUSED)
def test_extend_refuses(gates):
    a, b = qm.Circuit(3), qm.Circuit(3)
    with pytest.raises(qm.QMetalError) as ea:
        a.extend(gates)
    with pytest.raises(qm.QMetalError) as eb:
        _one_at_a_time(b, gates)
    assert str(ea.value) == str(eb.value) and len(a) == len(b)
