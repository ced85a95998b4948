"""qmk_apply_stages through the C ABI: 2x2s and fans of controlled phases, one
after another in one pass, on the block tile (up to seven wires >= 6) and the
warp tile (up to four, then any of wires 0..5), against the same stages one at
a time in complex128. Stages outside both are refused without a launch.

A random state of n >= 13 qubits has no amplitude above 0.1. Of ten stages each
leaves it with at most six roundings of its 2x2 and fifteen complex products of
its phase, 51 roundings of 2^-24: 10 * 51 * 2^-24 * 0.1 = 3.1e-6.
"""
import ctypes
from ctypes import POINTER, Structure, c_double, c_float, c_int, c_uint32, c_void_p

import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm
from qmetal_gb300 import workloads as W
from test_gpu_group_routes import _unitary
from test_inplace_schedule import _fan, _fans, _inverse_qft

pytestmark = pytest.mark.gpu
TOL = 3.1e-6


class _Stage(Structure):
    _fields_ = [("wire", c_uint32), ("has_matrix", c_uint32), ("phase", c_uint32),
                ("m", c_float * 8), ("m_lo", c_float), ("angles", POINTER(c_double))]


def _run(n, psi, stages):
    import torch
    L = ctypes.CDLL(qm.library_path())
    f = L.qmk_apply_stages
    f.restype = c_int
    f.argtypes = [c_void_p, c_uint32, c_uint32, c_void_p, c_void_p]
    items, keep = (_Stage * max(1, len(stages)))(), []
    for o, (w, m, phase, angles) in zip(items, stages):
        o.wire, o.has_matrix, o.phase = w, m is not None, phase
        if m is not None:
            o.m = (c_float * 8)(*[x for z in np.asarray(m).reshape(-1) for x in (z.real, z.imag)])
            o.m_lo = float(np.real(m[0, 0])) - o.m[0]
        if angles is not None:
            keep.append((c_double * n)(*angles))
            o.angles = keep[-1]
    st = torch.tensor(psi, device="cuda")
    torch.cuda.synchronize()
    rc = f(st.data_ptr(), n, len(stages), items, None)
    torch.cuda.synchronize()
    return rc, st.cpu().numpy()


def _want(psi, n, stages):
    st = psi.astype(np.complex128)
    for w, m, phase, angles in stages:
        turn = _fan(n, w, angles) if phase else None
        st = st * turn if phase == 2 else st
        if m is not None:
            st = np.einsum("ij,ajb->aib", m, st.reshape(-1, 2, 1 << w)).reshape(-1)
        st = st * turn if phase == 1 else st
    return st


def _state(n, rng):
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    return (psi / np.linalg.norm(psi)).astype(np.complex64)


def _stages(wires, n, rng, cls):
    out = []
    for w in wires:
        t = rng.uniform(-3, 3)
        m = {"hadamard": np.array([[1, 1], [1, -1]]) * np.sqrt(0.5) + 0j,
             "real": np.array([[np.cos(t), -np.sin(t)], [np.sin(t), np.cos(t)]]) + 0j,
             "general": _unitary(rng)}[cls]
        phase = int(rng.integers(3))
        out.append((w, m if rng.integers(4) or not phase else None, phase,
                    list(rng.uniform(-8, 8, n) * rng.integers(0, 2, n)) if phase else None))
    return out


@pytest.mark.parametrize("cls", ["hadamard", "real", "general"])
@pytest.mark.parametrize("n", [13, 14, 17, 20])
def test_stages(n, cls):
    rng = np.random.default_rng(950 + n)
    top, low = list(range(6, n)), list(range(6))
    sets = [top[::-1][:7], top[:7], top[:1], [n - 1, 6], low[::-1], low, [0], [5],
            top[:4] + low[::-1], top[::-1][:4] + [0, 3, 1], top[:2] + [4]]
    sets += [[int(q) for q in rng.permutation(top)[:k]] for k in (3, 5, 7)]
    sets += [[int(q) for q in rng.permutation(top)[:k]] + [int(q) for q in rng.permutation(low)]
             for k in (1, 4)]
    for wires in sets:
        stages = _stages(wires, n, rng, cls)
        psi = _state(n, rng)
        rc, got = _run(n, psi, stages)
        assert rc == 0
        assert np.abs(got - _want(psi, n, stages)).max() <= TOL, wires


def test_refused():
    rng = np.random.default_rng(5)
    psi, m = _state(14, rng), np.eye(2)
    ok = [0.1] * 14
    for n, stages in ((12, [(0, m, 0, None)]), (14, []), (14, [(14, m, 0, None)]),
                      (14, [(3, m, 0, None)] * 2), (14, [(0, m, 0, None), (6, m, 0, None)]),
                      (14, [(w, m, 0, None) for w in range(6, 14)]),
                      (14, [(w, m, 0, None) for w in (6, 7, 8, 9, 10, 0)]),
                      (14, [(2, m, 3, ok)]), (14, [(2, m, 1, None)]),
                      (14, [(2, m, 1, ok[:13] + [float("inf")])])):
        rc, got = _run(n, psi, stages)
        assert rc == -1
        assert np.array_equal(got, psi)


@pytest.mark.parametrize("n", [13, 15, 19])
def test_circuits(n):
    rng = np.random.default_rng(980 + n)
    for gates in (W.qft_swap(n), _inverse_qft(n), _fans(n, rng), _fans(n, rng)):
        psi = _state(n, rng)
        sim = qm.Simulator(n)
        sim.set_state(psi)
        sim.run(W.to_circuit(n, gates))
        want = oracle.run(n, gates, psi.astype(np.complex128))
        assert np.abs(sim.get_state() - want).max() <= TOL * max(1.0, n / 10)
