"""Gradients of circuits whose CX and SWAP runs do not stand one to one against
the runs that the backward sweep undoes: windows of angles zero leave the plan,
so that the runs around them become one there, and runs before the first
rotation are never undone.

Both states carry the gates' roundings (at most eight of 2^-24 each), forward
and back, and H's norm: 32 gates 2^-24 sum |c|.
"""
import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm
from qmetal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _brick(n):
    return [(W.CX, (q, q + 1), ()) for q in range(0, n - 1, 2)]


def _ladder(n):
    return [(W.CX, (q, q + 1), ()) for q in range(n - 1)]


def _swaps(n):
    return [(W.SWAP, (q, n - 1 - q), ()) for q in range(n // 2)]


def _wall(n, angle=None):
    return [(W.H, (q,), ()) if angle is None else (W.RY, (q,), (angle * (q + 1),)) for q in range(n)]


def _circuits(n):
    """As many runs in the plan as in the sweep, each map its partner's inverse,
    but of other gates; and the same with runs that differ in number or map."""
    out = []
    for run in (_brick(n), _swaps(n), _ladder(n)):
        out.append(_wall(n) + run + _wall(n) + run + _wall(n, 0.3) + run + _wall(n, 0.0) + run
                   + _wall(n, 0.0) + run)
        out.append(_wall(n, 0.2) + run + _wall(n, 0.0) + run + _wall(n, 0.1) + run)
        out.append(run + _wall(n, 0.0) + run + _wall(n, 0.4) + run + _wall(n, 0.0))
    return out


@pytest.mark.parametrize("n", [4, 7, 12, 13, 14])
def test_gradient(n):
    terms = W.ring_tfim_hamiltonian(n, 0.7)
    h = W.to_hamiltonian(terms)
    reqs, want = [], []
    for gates in _circuits(n):
        e0, g0 = oracle.energy_and_gradient(n, gates, terms)
        want.append((e0, g0, 32 * len(gates) * 2.0 ** -24 * sum(abs(t[0]) for t in terms)))
        reqs.append((W.to_circuit(n, gates), h, 0, 0))
    sim = qm.Simulator(n)
    got = [sim.energy_and_gradient(c, h) for c, *_ in reqs]
    for mode in (qm.BATCH_LANES, qm.BATCH_GRAPH):
        got += [r[:2] for r in qm.batch_serve(reqs, mode=mode)]
    for k, (e, g) in enumerate(got):
        e0, g0, tol = want[k % len(want)]
        assert abs(e - e0) <= tol
        assert np.abs(np.array(g) - g0).max() <= tol, (k % len(want), k // len(want))
