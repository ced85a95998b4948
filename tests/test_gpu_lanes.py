"""Batch lanes: one simulator per lane serves every width the lane meets,
widest first, in memory of its widest. Circuits with CX ladders (gathers into
a second buffer, state checkpoints), diagonal layers and samples, wide and
narrow mixed, against a simulator per request. A request's launches are the
same either way, so the numbers are equal to the bit.
"""
import numpy as np
import pytest

import qmetal_gb300 as qm
from qmetal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _requests():
    out = []
    for k, n in enumerate([9, 16, 13, 14, 3, 17, 14, 6, 16, 13]):
        gates = W.hea(n, 3, seed=k) if k % 2 else W.qaoa_ring_seeded(n, 2, seed=k)
        ham = W.to_hamiltonian(W.ring_tfim_hamiltonian(n, 0.7))
        out.append((W.to_circuit(n, gates), ham, (0, 200, 37)[k % 3], k))
    return out


@pytest.mark.parametrize("lanes", [1, 2, 3, 10, 16])
def test_lanes_equal_simulators(lanes):
    reqs = _requests()
    for _ in range(2):
        for (c, h, shots, seed), (e, g, s) in zip(reqs, qm.batch_serve(reqs, lanes=lanes)):
            (e1, g1, s1), = qm.batch_serve([(c, h, shots, seed)], mode=qm.BATCH_FUSED_LOOP)
            assert e == e1 and g == g1 and s == s1
            sim = qm.Simulator(c.num_qubits)
            assert sim.energy_and_gradient(c, h) == (e, list(g))
            if shots:
                sim.reset()
                sim.run_merged(c)
                assert s == sim.sample(shots, seed)


def test_failure_leaves_the_next_batch_whole():
    reqs = _requests()
    bad = W.to_circuit(12, [(W.RY, (0,), (0.1,)), (W.P, (1,), (0.2,))])   # P has no generator
    with pytest.raises(qm.QMetalError):
        qm.batch_serve(reqs + [(bad, reqs[0][1], 0, 0)], lanes=4)
    got = qm.batch_serve(reqs, lanes=4)
    assert np.isfinite([e for e, _, _ in got]).all()
