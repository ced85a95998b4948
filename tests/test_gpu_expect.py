"""Expectation values of many strings against the oracle: every kernel that
serves them, at the widths where their tiles begin and end.

Up to 14 qubits a block takes each string; above, Z strings go 32 a read, X
terms up to seven wires >= 6 with wires 0..5 a read, and the rest by flip
mask. A value is a sum of products whose magnitudes add up to at most 1, in
FP32 runs of at most ten additions on three roundings each and FP64 from
there: 13 * 2^-24 = 7.8e-7, so 1e-6.
"""
import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _terms(n, rng):
    """(x, y, z) masks: Z strings of every weight (more than one read takes),
    each X twice, every Y, and mixed strings with wires 0 and n - 1 flipped."""
    full = (1 << n) - 1
    out = [(0, 0, 0), (0, 0, full)]
    out += [(0, 0, 1 << q) for q in range(n)]
    out += [(0, 0, int(rng.integers(0, full + 1))) for _ in range(33)]
    out += [(1 << q, 0, 0) for q in range(n)]
    out += [(1 << q, 0, 0) for q in reversed(range(n))]
    out += [(0, 1 << q, 0) for q in range(n)]
    for flip in {1, 1 << (n - 1), full, int(rng.integers(1, full + 1))}:
        for _ in range(9):
            y = int(rng.integers(0, full + 1)) & flip
            out.append((flip ^ y, y, int(rng.integers(0, full + 1)) & ~flip))
    return out


@pytest.mark.parametrize("n", [1, 2, 5, 9, 10, 13, 14, 15, 16, 17, 18, 20])
def test_terms_against_the_oracle(n):
    rng = np.random.default_rng(500 + n)
    psi = (rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)) * rng.uniform(0, 1, 1 << n)
    psi[: 1 << (n // 2)] *= 20   # uneven, so that strings have values of their own
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64)
    terms = _terms(n, rng)
    ham = qm.Hamiltonian()
    for x, y, z in terms:
        ham.add(1.0, x, y, z)
    sim = qm.Simulator(n)
    sim.set_state(psi)
    got = np.array(sim.expectation_terms(ham))
    st = psi.astype(np.complex128)
    want = np.array([oracle.expectation(n, st, *t) for t in terms])
    assert np.abs(got - want).max() <= TOL, terms[int(np.abs(got - want).argmax())]
    # a few wires of one read, and one Z string alone
    few = qm.Hamiltonian()
    for q in {0, n // 2, n - 1}:
        few.add(1.0, 1 << q)
    few.add(1.0, 0, 0, 1 << (n - 1))
    got = np.array(sim.expectation_terms(few))
    want = np.array([oracle.expectation(n, st, *t[1:]) for t in few.terms])
    assert np.abs(got - want).max() <= TOL
