"""Diagonal layers on the routes that skip amplitudes: one term as a masked
phase, and layers whose masks all hold one wire (that wire's clear half is not
touched), against the oracle on random states.

An amplitude is multiplied by at most four FP32 complex factors of modulus 1
(three in the phase, one for the product), each within 3 * 2^-24 of exact:
12 * 2^-24 = 7.2e-7 of an amplitude of at most 1, so 1e-6.
"""
import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm
from qmetal_gb300 import workloads as W

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _random_state(n, rng):
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    return (psi / np.linalg.norm(psi)).astype(np.complex64)


def _check(n, gates, rng):
    psi = _random_state(n, rng)
    want = oracle.run(n, gates, psi.astype(np.complex128))
    for fuse in (True, False):
        sim = qm.Simulator(n)
        sim.set_state(psi)
        sim.run(W.to_circuit(n, gates), fuse=fuse)
        assert np.abs(sim.get_state() - want).max() <= TOL, (n, gates[:2], fuse)


@pytest.mark.parametrize("n", [1, 2, 3, 6, 7, 13, 14, 17])
def test_one_term(n):
    rng = np.random.default_rng(600 + n)
    for q in {0, n // 2, n - 1}:
        _check(n, [(W.P, (q,), (0.8,))], rng)
        for r in {0, 1, n - 1} - {q}:
            if r < n:
                _check(n, [(W.CP, (q, r), (-2.3,))], rng)


@pytest.mark.parametrize("n", [3, 6, 7, 13, 14, 16])
def test_common_wire(n):
    rng = np.random.default_rng(700 + n)
    for j in sorted({0, 1, 2, 5, 6, n - 2, n - 1}):
        if j < n:
            _check(n, [(W.CP, (k, j), (float(rng.uniform(-3, 3)),)) for k in range(n) if k != j], rng)
            _check(n, [(W.P, (j,), (0.4,)), (W.CP, (j, (j + 1) % n), (1.1,))], rng)
