"""How far values that are read from a state may be off: no further than the
FP32 rounding of each amplitude's or pair's product makes them.

Random amplitudes of about one size, whose squares q_i are small. A product has
two roundings and a sum of two amplitudes (four products) one or two more, each
of at most 2^-24 / sqrt 3 rms of its value: variances of 2/3 q^2 and, with both
amplitudes', 2 q^2 an amplitude in units of 2^-48. Z strings, the norm and the
doubled X terms (q a pair, half as many) all stay under 2^-24 sqrt(2 sum q^2)
rms; the rms over forty values or more may be a half above that. In FP32 sums
of 16 and 128 such products (strings that add all of them with one sign) would
be off by 3 to 7 times 2^-24 sqrt(sum q^2).
"""
import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm

pytestmark = pytest.mark.gpu


def _state(n, rng):
    """Amplitudes of much the same phase, so that X terms add up too."""
    psi = rng.uniform(0.8, 1.2, 1 << n) * np.exp(1j * rng.uniform(-0.3, 0.3, 1 << n))
    return (psi / np.linalg.norm(psi)).astype(np.complex64)


@pytest.mark.parametrize("n", [9, 10, 12, 14, 15, 16, 18, 20, 21])
def test_values(n):
    rng = np.random.default_rng(1400 + n)
    seeds = max(2, 60 // n)
    z, x, mixed, norms = [], [], [], []
    for _ in range(seeds):
        psi = _state(n, rng)
        st = psi.astype(np.complex128)
        unit = 2.0 ** -24 * np.sqrt(2 * (np.abs(st) ** 4).sum())
        # Z on the highest wire of all but a few amplitudes' sign; the identity; X
        terms = [(0, 0, 0)] + [(0, 0, 1 << q) for q in range(n)] + [(1 << q, 0, 0) for q in range(n)]
        flips = [int(f) for f in rng.integers(1, 1 << n, 6)] + [(1 << n) - 1]
        terms += [(f, 0, 0) for f in flips] + [(f, 0, ~f & 1 << q) for q, f in enumerate(flips)]
        h = qm.Hamiltonian()
        for t in terms:
            h.add(1.0, *t)
        sim = qm.Simulator(n)
        sim.set_state(psi)
        got = np.array(sim.expectation_terms(h))
        want = np.array([oracle.expectation(n, st, *t) for t in terms])
        off = (got - want) / unit
        z += list(off[:n + 1])
        x += list(off[n + 1:2 * n + 1])
        mixed += list(off[2 * n + 1:])
        norms.append((sim.norm() ** 2 - (np.abs(st) ** 2).sum()) / unit)
    for name, e in (("Z", z), ("X", x), ("mixed", mixed)):
        assert np.sqrt(np.mean(np.square(e))) <= 1.5, name
    assert np.abs(norms).max() <= 6    # of a few values, six times the rms


def test_unnormalised():
    """Sums of values near FP32's limits, and infinite ones."""
    n = 16
    h = qm.Hamiltonian()
    for q in (0, 7, 15):
        h.add(1.0, 0, 0, 1 << q)
        h.add(1.0, 1 << q)
    sim = qm.Simulator(n)
    for amplitude in (1e-18, 1e16):
        psi = np.zeros(1 << n, dtype=np.complex64)
        psi[:64] = amplitude
        sim.set_state(psi)
        got = np.array(sim.expectation_terms(h))
        total = 64 * float(np.float32(amplitude)) ** 2
        want = np.array([0, total, total, 0, total, 0])
        assert np.abs(got - want).max() <= 4 * 2.0 ** -24 * total
    psi[3] = np.inf
    sim.set_state(psi)
    got = sim.expectation_terms(h)
    assert got[2] == got[4] == np.inf and got[0] == -np.inf
