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


def _terms(n, rng):
    full = (1 << n) - 1
    out = [(0.5, 0, 0, 0), (-1.0, 0, 0, 1), (0.7, 1 << (n - 1), 0, 0), (0.3, 0, 1, 0)]
    for _ in range(6):
        x = int(rng.integers(0, full + 1))
        y = int(rng.integers(0, full + 1)) & ~x
        z = int(rng.integers(0, full + 1)) & ~(x | y)
        out.append((float(rng.uniform(-1, 1)), x, y, z))
    return out


def _check_gradient(n, gates, terms):
    e0, g0 = oracle.energy_and_gradient(n, gates, terms)
    c, h = W.to_circuit(n, gates), W.to_hamiltonian(terms)
    # both states carry the gates' roundings, forward and back, and H's norm
    tol = 4 * 8 * max(1, len(gates)) * 2.0 ** -24 * sum(abs(t[0]) for t in terms)
    sim = qm.Simulator(n)
    for _ in range(2):
        e, g = sim.energy_and_gradient(c, h)
        assert abs(e - e0) <= tol
        assert len(g) == len(gates) and np.abs(np.array(g) - g0).max(initial=0.0) <= tol
    (eb, gb, sb), = qm.batch_serve([(c, h, 50, 3)], lanes=1)
    assert abs(eb - e0) <= tol and np.abs(np.array(gb) - g0).max(initial=0.0) <= tol
    ref = qm.Simulator(n)
    ref.run_merged(c)
    assert sb == ref.sample(50, seed=3)


@pytest.mark.parametrize("n", range(1, 15))
def test_gradient(n):
    rng = np.random.default_rng(360 + n)
    terms = _terms(n, rng)
    rotations = [(int(k), (int(q),), (float(rng.uniform(-3, 3)),))
                 for k, q in zip(rng.choice([W.RX, W.RY, W.RZ], 60), rng.integers(0, n, 60))]
    _check_gradient(n, rotations, terms)
    _check_gradient(n, [(W.RX, (0,), (0.1 * k,)) for k in range(40)], terms)
    if n == 1:
        return
    free = [g for g in (_gate(n, rng) for _ in range(150)) if g[0] not in (W.P, W.CP)]
    _check_gradient(n, free, terms)
    _check_gradient(n, W.hea(n, 4), W.ring_tfim_hamiltonian(n, 0.7) if n > 2 else terms)
    if n > 2:
        _check_gradient(n, W.qaoa_ring_seeded(n, 3), W.maxcut_hamiltonian(
            [(i, (i + 1) % n) for i in range(n)]))
        _check_gradient(n, W.tfim_chain(n, 4), W.ring_tfim_hamiltonian(n, 0.7))
        coupled = []
        for _ in range(2):   # more couplings than one step's sums
            for a in range(n):
                for b in range(a):
                    coupled += [(W.CX, (a, b), ()), (W.RZ, (b,), (0.2 + a,)), (W.CX, (a, b), ())]
            coupled += [(W.RX, (q,), (0.5,)) for q in range(n)]
        _check_gradient(n, coupled, terms)


@pytest.mark.parametrize("n, depth", [(4, 40), (10, 20), (13, 12)])
def test_gradient_long(n, depth):
    _check_gradient(n, W.hea(n, depth), W.ring_tfim_hamiltonian(n, 0.7))   # several launches
