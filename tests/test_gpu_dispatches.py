"""dispatch_count up to 13 qubits: plan ops for run and its variants, the
launches themselves for run_merged and gradients, however many a circuit takes."""
import numpy as np
import pytest

import qmetal_gb300 as qm
from qmetal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _counted(sim, call, circuit):
    before = sim.dispatch_count
    call(circuit)
    return sim.dispatch_count - before


def test_counts():
    n = 12
    rng = np.random.default_rng(7)
    short = W.to_circuit(n, W.random_u3(n, 1))
    # 1500 groups of 20 words and 1500 CCX of 12: seven launches of 7936 words
    long = W.to_circuit(n, [(W.RY, (int(q),), (0.1,)) if k % 2 else (W.CCX, (0, 1, 2 + k % 10), ())
                            for k, q in enumerate(rng.integers(0, n, 3000))])
    layers = W.to_circuit(n, W.tfim_chain(n, 2))
    sim = qm.Simulator(n)
    for c in (short, long, layers):
        assert _counted(sim, sim.run, c) == c.plan_size()
    rx = W.to_circuit(n, [(W.RX, (q,), (0.2,)) for q in range(n)])
    assert _counted(sim, sim.run_merged, rx) <= 2          # by itself where that is a launch or two
    assert _counted(sim, sim.run_merged, W.to_circuit(n, W.hea(n, 2))) == 1
    for c in (short, layers):                              # the layers' tables, then the circuit
        assert _counted(sim, sim.run_merged, c) == 2
    assert _counted(sim, sim.run_merged, long) >= 6
    h = W.to_hamiltonian([(1.0, 1, 0, 0)])
    grad = lambda c: sim.energy_and_gradient(c, h)   # noqa: E731
    assert _counted(sim, grad, rx) == 2                    # the reset, then all of it
    many = W.to_circuit(n, [(W.RX, (k % n,), (0.01 * k,)) for k in range(1200)])
    assert _counted(sim, grad, many) >= 4
