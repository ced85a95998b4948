"""Circuits of one to nine gates on up to 13 qubits, by themselves or in one
launch, against the oracle. The bound is that of test_gpu_small: eight roundings
of 2^-24 a gate."""
import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm
from qmetal_gb300 import workloads as W
from test_gpu_small import _gate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 4, 5, 9, 12, 13, 14])
def test_few(n):
    rng = np.random.default_rng(1500 + n)
    sim = qm.Simulator(n)
    cases = [[_gate(n, rng) for _ in range(k)] for k in (1, 2, 3, 4, 8, 9) for _ in range(6)]
    cases += [[], [(W.RY, (q,), (0.3 + q,)) for q in range(n)], [(W.CX, (q, q + 1), ()) for q in range(n - 1)],
              [(W.RZ, (q,), (0.3 + q,)) for q in range(n)], [(W.P, (0,), (0.4,))]]
    for gates in cases:
        psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        psi = (psi / np.linalg.norm(psi)).astype(np.complex64)
        want = oracle.run(n, gates, psi.astype(np.complex128))
        c = W.to_circuit(n, gates)
        for call in (sim.run, sim.run_merged, sim.run_cached, lambda c: sim.run(c, fuse=False)):
            sim.set_state(psi)
            call(c)
            assert np.abs(sim.get_state() - want).max() <= 8 * max(1, len(gates)) * 2.0 ** -24
