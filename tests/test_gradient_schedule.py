"""The forward pass of gradients as it is launched, replayed in complex128 on the
CPU against the oracle's gate-by-gate run."""
import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm  # noqa: F401
from qmetal_gb300 import workloads as W
from test_schedules import Reader, apply_1q, gather, plan_op


def _replay(n, gates):
    c = W.to_circuit(n, gates)
    plan = np.array(c.plan_export())
    v = c.schedule_export("gradient")
    r, kinds = Reader(v), []
    st = np.zeros(1 << n, dtype=complex)
    st[0] = 1.0
    for _ in range(r.i()):
        kind = r.i()
        kinds.append(kind)
        assert kind in (0, 1, 2, 5)
        if kind == 1:
            cols, off = r.gather_map()
            for _ in range(r.i()):
                r.i()
            st = gather(st, n, cols, off)
            continue
        if kind != 0:
            st = oracle.run_plan(n, plan_op(plan, r.i()), init=st)
        if kind != 2:
            group = [(r.i(), r.mat()) for _ in range(r.i())]
            wires = [w for w, _ in group]
            assert wires == sorted(set(wires)) and wires
            if kind == 5:
                assert len(wires) <= 4 and wires[0] >= 13
            for w, m in group:
                st = apply_1q(st, n, w, m)
    assert r.p == len(v)
    return st, kinds


@pytest.mark.parametrize("n, folds", [(6, False), (13, False), (14, False), (18, True)])
def test_gradient_schedule(n, folds):
    seen = set()
    for gates in (W.qaoa_ring_seeded(n, 2), W.tfim_chain(n, 2), W.hea(n, 2), W.qft_swap(n)):
        got, kinds = _replay(n, gates)
        assert np.abs(got - oracle.run(n, gates)).max() <= 1e-12
        seen |= set(kinds)
    assert 1 in seen
    assert (5 in seen) == folds
