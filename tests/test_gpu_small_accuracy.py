"""Accuracy of circuits and gradients in one launch: 2x2s that were narrowed to
FP32 alone would fail here.

Narrowing cos and sin to FP32 changes a rotation's norm by up to 4e-8, the same
at every wire and layer that has the angle, so that it adds up; the angles here
are picked for it. With the low parts there are roundings alone, of 2^-24 / sqrt 3
rms each: two per 2x2 (of 80 to 240), three per layer's phases and one, the same in
every layer, of their table, eight layers. States: sqrt(240 * 2 + 24) + 8 = 31 of
them, 1.1e-6 of the norm. Gradients: both states forward and back, four times that
at most of |lambda|; against gradients of a thirtieth of it a random error of the 1024
amplitudes counts by 30 / sqrt 1024: 4.2e-6.
"""
import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm
from qmetal_gb300 import workloads as W

N, LAYERS = 10, 8
STATE_TOL, GRAD_TOL = 1.1e-6, 4.2e-6
PAULI = {W.RX: np.array([[0, 1], [1, 0]]), W.RY: np.array([[0, -1j], [1j, 0]]),
         W.RZ: np.array([[1, 0], [0, -1]])}


def _rot(kind, t):
    return np.cos(t / 2) * np.eye(2) - 1j * np.sin(t / 2) * PAULI[kind]


def _narrowed(m):
    return m.astype(np.complex64).astype(np.complex128)


def _growth(m):
    """Relative change of the norm of what the narrowed 2x2 is applied to, on average."""
    return np.linalg.norm(_narrowed(m)) ** 2 / np.linalg.norm(m) ** 2 - 1


def _angles(kinds, seed):
    """The candidates whose narrowed product and rotations grow a state most."""
    rng = np.random.default_rng(seed)
    best = None
    for _ in range(4000):
        ts = rng.uniform(0.2, 1.2, len(kinds))
        m, each = np.eye(2), []
        for k, t in zip(kinds, ts):
            m = _rot(k, t) @ m
            each.append(_growth(_rot(k, -t)))
        score = min([_growth(m)] + each)
        if best is None or score > best[0]:
            best = (score, [float(t) for t in ts])
    return best[1]


def _circuit(name):
    kinds = {"trotter": [W.RX], "hea": [W.RY, W.RZ], "mixed": [W.RX, W.RY, W.RZ]}[name]
    ts = _angles(kinds, len(kinds))
    gates = [] if name == "hea" else [(W.RY, (q,), (0.5 + 0.1 * q,)) for q in range(N)]
    for _ in range(LAYERS):
        if name != "hea":
            for q in range(N):
                gates += [(W.CX, (q, (q + 1) % N), ()), (W.RZ, ((q + 1) % N,), (0.3,)),
                          (W.CX, (q, (q + 1) % N), ())]
        gates += [(k, (q,), (t,)) for q in range(N) for k, t in zip(kinds, ts)]
        if name == "hea":
            gates += [(W.CX, (q, q + 1), ()) for q in range(N - 1)]
    return gates


def _on(st, q, m):
    return np.einsum("ij,ajb->aib", m, st.reshape(-1, 2, 1 << q)).reshape(-1)


def _cx(st, c, t):
    i = np.arange(st.size)
    return st[i ^ (((i >> c) & 1) << t)]


def _one_part(gates, terms):
    """State and gradient with every rotation narrowed and no other rounding; a
    wire's rotations of a layer narrowed as their product going forward."""
    st = np.zeros(1 << N, dtype=complex)
    st[0] = 1.0
    held = {}

    def flush():
        nonlocal st
        for q, m in held.items():
            st = _on(st, q, _narrowed(m))
        held.clear()

    for k, (kind, qs, ps) in enumerate(gates):
        if kind == W.CX:
            flush()
            st = _cx(st, *qs)
        elif k and kind == W.RZ and gates[k - 1][0] == W.CX:   # a coupling: tabulated in FP64
            st = _on(st, qs[0], _rot(kind, ps[0]))
        else:
            held[qs[0]] = _rot(kind, ps[0]) @ held.get(qs[0], np.eye(2))
    flush()
    psi, grad = st.copy(), np.zeros(len(gates))
    lam, i = np.zeros_like(st), np.arange(st.size)
    for c, x, y, z in terms:
        assert y == 0
        sign = 1 - 2 * (np.array([bin(v & z).count("1") for v in range(st.size)]) & 1)
        lam += c * (sign * st)[i ^ x] if z == 0 else c * sign * st
    for k in reversed(range(len(gates))):
        kind, qs, ps = gates[k]
        if kind == W.CX:
            psi, lam = _cx(psi, *qs), _cx(lam, *qs)
            continue
        grad[k] = np.imag(np.vdot(lam, _on(psi, qs[0], PAULI[kind])))
        m = _rot(kind, -ps[0])
        if not (kind == W.RZ and gates[k - 1][0] == W.CX):
            m = _narrowed(m)
        psi, lam = _on(psi, qs[0], m), _on(lam, qs[0], m)
    return st, grad


def _off(got, want):
    return np.linalg.norm(np.asarray(got) - want) / np.linalg.norm(want)


@pytest.mark.parametrize("name", ["trotter", "hea", "mixed"])
def test_the_bounds_tell(name):
    gates, terms = _circuit(name), W.ring_tfim_hamiltonian(N, 0.7)
    st, grad = _one_part(gates, terms)
    assert _off(st, oracle.run(N, gates)) > 1.2 * STATE_TOL
    e0, g0 = oracle.energy_and_gradient(N, gates, terms)
    assert _off(grad, g0) > 1.5 * GRAD_TOL


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["trotter", "hea", "mixed"])
def test_accuracy(name):
    gates, terms = _circuit(name), W.ring_tfim_hamiltonian(N, 0.7)
    c = W.to_circuit(N, gates)
    sim = qm.Simulator(N)
    sim.run(c)
    assert _off(sim.get_state(), oracle.run(N, gates)) <= STATE_TOL
    e, g = sim.energy_and_gradient(c, W.to_hamiltonian(terms))
    e0, g0 = oracle.energy_and_gradient(N, gates, terms)
    lam2 = sum(abs(t[0]) for t in terms)
    assert abs(e - e0) <= 2 * STATE_TOL * lam2
    assert _off(g, g0) <= GRAD_TOL
