"""qmk_apply_diagonal_group through the C ABI against qmk_apply_diagonal and
qmk_apply_group in turn. The arithmetic is theirs in the same order, so the
states are equal up to the compiler's choice of fused multiply-adds: four 2x2s
and a phase, 36 roundings of 2^-24 on amplitudes of at most 0.1, 2.2e-7. Wires
below 13 and other calls it does not take are refused without a launch.
"""
import ctypes
from ctypes import c_double, c_int, c_size_t, c_uint32, c_uint64, c_void_p

import numpy as np
import pytest

import qmetal_gb300 as qm
from test_gpu_group_routes import _unitary

pytestmark = pytest.mark.gpu
TOL = 2.2e-7


def _lib():
    L = ctypes.CDLL(qm.library_path())
    L.qmk_workspace_bytes.restype = c_size_t
    L.qmk_apply_diagonal.argtypes = [c_void_p, c_uint32, c_uint32, c_void_p, c_void_p, c_double,
                                     c_void_p, c_size_t, c_void_p]
    L.qmk_apply_group.argtypes = [c_void_p, c_uint32, c_uint32, c_void_p, c_void_p, c_void_p]
    L.qmk_apply_diagonal_group.argtypes = [c_void_p, c_uint32, c_uint32, c_void_p, c_void_p,
                                           c_double, c_uint32, c_void_p, c_void_p, c_void_p,
                                           c_size_t, c_void_p]
    return L


def _matrix(rng, cls):
    t = rng.uniform(-3, 3)
    c, s = np.cos(t / 2), np.sin(t / 2)
    return {"real": np.array([[c, -s], [s, c]], dtype=complex),
            "rx": np.array([[c, -1j * s], [-1j * s, c]]), "general": _unitary(rng)}[cls]


def _call(n, psi, terms, wires, mats, together):
    import torch
    L = _lib()
    st = torch.tensor(psi, device="cuda")
    ws = torch.zeros(L.qmk_workspace_bytes(c_uint32(n)), dtype=torch.uint8, device="cuda")
    masks, angles, gp = terms
    mm, aa = (c_uint64 * max(1, len(masks)))(*masks), (c_double * max(1, len(masks)))(*angles)
    w = (c_uint32 * max(1, len(wires)))(*wires)
    f = np.array([[(z.real, z.imag) for z in np.asarray(m).reshape(-1)] for m in mats],
                 dtype=np.float32).reshape(-1)
    torch.cuda.synchronize()
    if together:
        rc = L.qmk_apply_diagonal_group(st.data_ptr(), n, len(masks), mm, aa, gp, len(wires), w,
                                        f.ctypes.data, ws.data_ptr(), ws.numel(), None)
    else:
        rc = L.qmk_apply_diagonal(st.data_ptr(), n, len(masks), mm, aa, gp, ws.data_ptr(),
                                  ws.numel(), None)
        rc = rc or L.qmk_apply_group(st.data_ptr(), n, len(wires), w, f.ctypes.data, None)
    torch.cuda.synchronize()
    return rc, st.cpu().numpy()


def _state(n, rng):
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    return (psi / np.linalg.norm(psi)).astype(np.complex64)


@pytest.mark.parametrize("cls", ["real", "rx", "general"])
@pytest.mark.parametrize("n", [14, 15, 17, 20, 22])
def test_layer_and_wires(n, cls):
    rng = np.random.default_rng(700 + n)
    pairs = [(1 << int(a)) | (1 << int(b)) for a, b in
             (rng.choice(n, 2, replace=False) for _ in range(40))]
    terms = (pairs + [1 << q for q in range(n)] + [0],
             list(rng.uniform(-4, 4, len(pairs) + n + 1)), 0.9)
    top = list(range(13, n))
    sets = [top[:k] for k in (1, 2, 3, 4)] + [top[-k:] for k in (1, 2, 3, 4)]
    sets += [sorted(int(q) for q in rng.choice(top, min(len(top), k), replace=False)) for k in (2, 3, 4)]
    for wires in {tuple(s) for s in sets}:
        mats = [_matrix(rng, cls) for _ in wires]
        psi = _state(n, rng)
        rc, got = _call(n, psi, terms, wires, mats, True)
        rc2, want = _call(n, psi, terms, wires, mats, False)
        assert rc == rc2 == 0
        assert np.abs(got - want).max() <= TOL, wires


def test_refused():
    rng = np.random.default_rng(5)
    psi, m = _state(16, rng), [np.eye(2)] * 5
    ok = ([3, 5], [0.1, 0.2], 0.0)
    for n, terms, wires in ((13, ok, [12]), (16, ok, [12]), (16, ok, [14, 13]), (16, ok, [13, 13]),
                            (16, ok, [16]), (16, ok, []), (16, ([7, 1], [0.1, 0.2], 0.0), [13]),
                            (16, ([1 << 16, 1], [0.1, 0.2], 0.0), [13])):
        rc, got = _call(n, psi, terms, wires, m[:len(wires)], True)
        assert rc == -1
        assert np.array_equal(got, psi)
