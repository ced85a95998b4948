"""Fans of controlled phases with angles of many turns, against complex128: an
angle's phase is its own, to the state's precision, whatever its size.

Angles of both sides are the same doubles; cos and sin of a double are exact to
2^-53 there. The bound is the stages' own (test_gpu_stages): 3.1e-6 for ten.
"""
import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm
from qmetal_gb300 import workloads as W
from test_gpu_stages import TOL, _run, _state

pytestmark = pytest.mark.gpu


def _want(psi, n, stages):
    st = psi.astype(np.complex128)
    i = np.arange(1 << n)
    for w, m, phase, angles in stages:
        turn = np.ones(1 << n, dtype=complex)
        for v, a in enumerate(angles):   # a factor per angle: a sum of large ones would round
            turn = np.where((i >> w) & (i >> v) & 1, turn * np.exp(1j * a), turn)
        st = st * turn if phase == 2 else st
        st = np.einsum("ij,ajb->aib", m, st.reshape(-1, 2, 1 << w)).reshape(-1)
        st = st * turn if phase == 1 else st
    return st


@pytest.mark.parametrize("size", [1e3, 1e6, 1e9, 1e12, 1e15, 1e300])
@pytest.mark.parametrize("wires", [[13, 6, 9, 12, 7, 8, 11], [6, 13, 5, 0, 3]])
def test_large_angles(wires, size):
    n, rng = 14, np.random.default_rng(1200 + len(wires))
    had = np.array([[1, 1], [1, -1]]) * np.sqrt(0.5) + 0j
    stages = [(w, had, 1 + k % 2, list(rng.uniform(-size, size, n))) for k, w in enumerate(wires)]
    psi = _state(n, rng)
    rc, got = _run(n, psi, stages)
    assert rc == 0
    assert np.abs(got - _want(psi, n, stages)).max() <= TOL


@pytest.mark.parametrize("size", [1e8, 1e11, 1e14])
def test_circuit(size):
    n, rng = 14, np.random.default_rng(1230)
    gates = []
    for w in reversed(range(n)):
        gates.append((W.H, (w,), ()))
        gates += [(W.CP, (v, w), (float(rng.uniform(-size, size)),)) for v in range(w)]
    psi = _state(n, rng)
    want = oracle.run(n, gates, psi.astype(np.complex128))
    sim = qm.Simulator(n)
    sim.set_state(psi)
    sim.run(W.to_circuit(n, gates))
    assert np.abs(sim.get_state() - want).max() <= TOL * n / 10


def test_a_sum_that_overflows_is_taken():
    """Two angles of a pair of wires whose sum is infinite: no phase, and no error."""
    n = 14
    gates = [(W.H, (13,), ()), (W.CP, (2, 13), (1.5e308,)), (W.CP, (2, 13), (1.5e308,)),
             (W.H, (12,), ()), (W.CP, (2, 12), (0.5,)), (W.CP, (3, 12), (0.5,)), (W.H, (11,), ())]
    sim = qm.Simulator(n)
    sim.run(W.to_circuit(n, gates))
    st = sim.get_state()
    assert np.isfinite(st[np.arange(1 << n) & 1 << 13 == 0]).all()
