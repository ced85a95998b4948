"""The schedules of Simulator.run, replayed in complex128 on the CPU against
the oracle's gate-by-gate run, with the limits their kernels rely on. In place:
a pass with moves holds any of wires 0..5 and up to four wires >= 6, or up to
seven wires >= 6, and exists from 13 qubits. In one launch (up to 13 qubits):
groups of up to three ascending wires, gathers without an offset."""
import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm  # noqa: F401
from qmetal_gb300 import workloads as W
from test_schedules import Reader, apply_1q, decode_forward, gather, plan_op

CX, CZ, SWAP, CP = W.CX, W.CZ, W.SWAP, W.CP


def _steps(c):
    n = c.num_qubits
    v = c.schedule_export("inplace")
    r, out = Reader(v), []
    for _ in range(r.i()):
        kind = r.i()
        assert kind in (0, 2, 3, 4, 5)
        op = r.i() if kind == 5 else None
        if kind == 4:
            out.append(("stages", [(r.i(), r.i(), r.mat(), r.i(), [r.f() for _ in range(n)])
                                   for _ in range(r.i())]))
            continue
        if kind == 2:
            out.append(("op", r.i()))
            continue
        mats = [(r.i(), r.mat()) for _ in range(r.i())]
        moves = [(r.i(), r.i(), r.i()) for _ in range(r.i())] if kind == 3 else []
        out.append(({0: "group", 3: "moves", 5: "diag"}[kind], mats, moves, op))
    assert r.p == len(v)
    return out


def _move(st, swap, a, b):
    i = np.arange(st.size)
    d = ((i >> a) ^ (i >> b)) & 1 if swap else (i >> a) & 1
    out = np.empty_like(st)
    out[i ^ (d << b) ^ ((d << a) if swap else 0)] = st
    return out


def _fan(n, wire, angles):
    i = np.arange(1 << n)
    f = sum(a * ((i >> w) & 1) for w, a in enumerate(angles))
    return np.where((i >> wire) & 1, np.exp(1j * f), 1.0)


def _inverse_qft(n):
    return [(k, q, tuple(-x for x in ps)) for k, q, ps in reversed(W.qft(n))]


def _fans(n, rng, count=30):
    """Single gates and controlled phases from random wires, as many stages' passes meet them."""
    gates = []
    for _ in range(count):
        w = int(rng.integers(n))
        gates.append((int(rng.choice([W.H, W.RY, W.RX])), (w,), ()) if rng.integers(2) else (W.H, (w,), ()))
        if gates[-1][0] != W.H:
            gates[-1] = (gates[-1][0], (w,), (float(rng.uniform(-3, 3)),))
        c = w if rng.integers(4) else int(rng.integers(n))
        others = [int(q) for q in rng.choice(n, int(rng.integers(1, 6)), replace=False) if q != c]
        gates += [(CP, (q, c), (float(rng.uniform(-3, 3)),)) for q in others]
        if rng.integers(3) == 0:
            gates.append((W.P, (c,), (0.4,)))
    return gates


def _replay(n, gates):
    c = W.to_circuit(n, gates)
    plan = np.array(c.plan_export())
    st = np.zeros(1 << n, dtype=complex)
    st[0] = 1.0
    steps = _steps(c)
    for s in steps:
        if s[0] == "op":
            st = oracle.run_plan(n, plan_op(plan, s[1]), init=st)
            continue
        if s[0] == "stages":
            wires = [x[0] for x in s[1]]
            high = [w for w in wires if w >= 6]
            assert n >= 13 and len(set(wires)) == len(wires) >= 2
            assert wires[:len(high)] == high
            assert len(high) <= (7 if len(high) == len(wires) else 4)
            for w, has, m, phase, angles in s[1]:
                turn = _fan(n, w, angles)
                st = st * turn if phase == 2 else st
                st = apply_1q(st, n, w, m) if has else st
                st = st * turn if phase == 1 else st
            continue
        wires = [w for w, _ in s[1]]
        assert wires == sorted(set(wires))
        if s[0] == "diag":
            assert 1 <= len(wires) <= 4 and wires[0] >= 13
            st = oracle.run_plan(n, plan_op(plan, s[3]), init=st)
        for w, m in s[1]:
            st = apply_1q(st, n, w, m)
        if s[0] == "moves":
            assert n >= 13 and s[2]
            held = set(wires) | {q for _, a, b in s[2] for q in (a, b)}
            assert sum(q >= 6 for q in held) <= (4 if min(held) < 6 else 7)
            for swap, a, b in s[2]:
                assert a != b
                st = _move(st, swap, a, b)
    return st, steps


def _random(n, count, rng):
    gates = []
    for _ in range(count):
        a, b = (int(q) for q in rng.choice(n, 2, replace=False))
        kind = int(rng.choice([CX, CX, CX, SWAP, CZ, CP, W.RY, W.RZ, W.H]))
        if kind == CP:
            gates.append((kind, (a, b), (0.4,)))
        elif kind in (CX, SWAP, CZ):
            gates.append((kind, (a, b), ()))
        else:
            gates.append((kind, (a,), (0.7,) if kind in (W.RY, W.RZ) else ()))
    return gates


@pytest.mark.parametrize("n", [5, 11, 12, 13, 14, 18])
def test_inplace_schedule(n):
    rng = np.random.default_rng(40 + n)
    reverse = [(CX, (q + 1, q), ()) for q in reversed(range(n - 1))]
    swaps = [(SWAP, (q, n - 1 - q), ()) for q in range(n // 2)]
    layer = [(W.RY, (q,), (0.1 + q,)) for q in range(n)]
    for gates in (W.ghz(n), W.hea(n, 2), W.qft_swap(n), W.tfim_chain(n, 2), W.random_u3(n, 2),
                  W.qaoa_ring_seeded(n, 2), layer + reverse + layer + swaps, layer + swaps + reverse,
                  _random(n, 60, rng), _random(n, 60, rng), W.qft(n) + _inverse_qft(n),
                  _fans(n, rng), _fans(n, rng)):
        got, _ = _replay(n, gates)
        assert np.abs(got - oracle.run(n, gates)).max() <= 1e-12


@pytest.mark.parametrize("n, passes", [(28, 4), (30, 5), (13, 2)])
def test_hea_layer_passes(n, passes):
    steps = _steps(W.to_circuit(n, W.hea(n, 1)))
    assert len(steps) == passes
    assert sum(len(s[2]) for s in steps) == n - 1
    assert sorted(w for s in steps for w, _ in s[1]) == list(range(n))


@pytest.mark.parametrize("n", [1, 2, 3, 6, 9, 13])
def test_small_schedule(n):
    rng = np.random.default_rng(70 + n)
    circuits = [[(W.RY, (q,), (0.3 + q,)) for q in range(n)] * 2]
    if n > 1:
        circuits += [W.hea(n, 2), W.random_u3(n, 2), _random(n, 80, rng)]
    if n > 2:
        circuits += [W.ghz(n), W.qft_swap(n), W.qaoa_ring_seeded(n, 2),
                     [(W.CCX, (0, 1, 2), ()), (W.CY, (2, 0), ())] * 2]
    for gates in circuits:
        c = W.to_circuit(n, gates)
        plan = np.array(c.plan_export())
        st = np.zeros(1 << n, dtype=complex)
        st[0] = 1.0
        for s in decode_forward(c.schedule_export("small")):
            if s[0] == "group":
                wires = [w for w, _ in s[1]]
                assert wires == sorted(set(wires)) and 1 <= len(wires) <= 3
                for w, m in s[1]:
                    st = apply_1q(st, n, w, m)
            elif s[0] == "permute":
                assert s[2] == 0
                st = gather(st, n, s[1], s[2])
            else:
                st = oracle.run_plan(n, plan_op(plan, s[1]), init=st)
        assert np.abs(st - oracle.run(n, gates)).max() <= 1e-12


@pytest.mark.parametrize("n, passes", [(13, 2), (20, 3), (28, 4), (31, 4), (33, 5)])
def test_qft_passes(n, passes):
    steps = _steps(W.to_circuit(n, W.qft(n)))
    assert [s[0] for s in steps] == ["stages"] * passes
    # the inverse meets wires 0..5 first, and may end on a stage of its own
    steps = _steps(W.to_circuit(n, _inverse_qft(n)))
    assert sum(s[0] == "stages" for s in steps) >= 1 + (n - 6) // 7
    assert len(steps) <= 1 + (n - 6) // 7 + 2


@pytest.mark.parametrize("n, passes", [(14, 3), (18, 3), (21, 3), (25, 4), (28, 4), (30, 5)])
def test_layer_passes(n, passes):
    steps = _steps(W.to_circuit(n, W.tfim_chain(n, 1)))
    assert len(steps) == passes
    assert sorted(w for s in steps if s[0] != "op" for w, _ in s[1]) == list(range(n))


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_angles_without_a_value_stay_diagonal_layers(bad):
    gates = [(k, q, (bad,) if q == (3, 9) else ps) for k, q, ps in W.qft(14)]
    steps = _steps(W.to_circuit(14, gates))
    assert any(s[0] == "op" for s in steps)
    for s in steps:
        if s[0] == "stages":
            assert np.isfinite([a for x in s[1] for a in x[4]]).all()
