"""Circuits on states of up to 13 qubits, which run in one launch, against the
oracle: every op kind, circuits that outgrow one launch's arguments, and more
diagonal layers than one launch tabulates.

An op leaves an amplitude (at most 1) with at most eight FP32 roundings of
2^-24, so a circuit of g gates is held to 8 g 2^-24.
"""
import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm
from qmetal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _gate(n, rng):
    kind = int(rng.integers(0, 18))
    arity = 1 if kind < 12 else 3 if kind == W.CCX else 2
    if arity > n:
        return _gate(n, rng)
    qubits = tuple(int(q) for q in rng.choice(n, arity, replace=False))
    return kind, qubits, ((float(rng.uniform(-3, 3)),) if kind in (W.RX, W.RY, W.RZ, W.P, W.CP)
                          else ())


def _check(n, gates, rng):
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64)
    want = oracle.run(n, gates, psi.astype(np.complex128))
    c = W.to_circuit(n, gates)
    tol = 8 * len(gates) * 2.0 ** -24
    for how in ("run", "unfused", "merged", "cached", "blocked"):
        sim = qm.Simulator(n)
        sim.set_state(psi)
        if how == "run":
            sim.run(c)
        elif how == "unfused":
            sim.run(c, fuse=False)
        elif how == "merged":
            sim.run_merged(c)
        elif how == "cached":
            sim.run_cached(c)
            sim.set_state(psi)
            sim.run_cached(c)
        elif n >= 2:
            sim.run_options(c, block_bits=min(n, 10))
        else:
            continue
        assert np.abs(sim.get_state() - want).max() <= tol, how


@pytest.mark.parametrize("n", range(1, 15))
def test_every_gate(n):
    rng = np.random.default_rng(300 + n)
    _check(n, [_gate(n, rng) for _ in range(120)], rng)


@pytest.mark.parametrize("n", [2, 6, 9, 13])
def test_long(n):
    rng = np.random.default_rng(330 + n)
    _check(n, [_gate(n, rng) for _ in range(2500)], rng)          # more than one launch's ops
    layers = []
    for _ in range(40):                                            # ... and phase tables
        layers += [(W.P, (q,), (float(rng.uniform(-3, 3)),)) for q in range(n)]
        layers += [(W.H, (0,), ())]
    _check(n, layers, rng)
    wide = []
    for _ in range(12):                                            # ... and terms
        wide += [(W.CP, (a, b), (float(rng.uniform(-3, 3)),)) for a in range(n) for b in range(a)]
        wide += [(W.CP, (a, b), (0.2,)) for a in range(n) for b in range(n) if a != b]
        wide += [(W.RY, (q,), (0.4,)) for q in range(n)]
    _check(n, wide, rng)


def test_norm_and_layers_repeat():
    n = 12
    gates = W.tfim_chain(n, 20)
    sim = qm.Simulator(n)
    sim.run(W.to_circuit(n, gates))
    want = oracle.run(n, gates)
    assert np.abs(sim.get_state() - want).max() <= 8 * len(gates) * 2.0 ** -24
