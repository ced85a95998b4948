"""qmk_apply_group_moves through the C ABI: 2x2s, then CX and SWAP gates among
the pass's wires, on the warp tile (any of wires 0..5, up to four wires >= 6)
and the block tile (up to seven wires >= 6), against the same ops one at a time
in complex128. Wire sets outside both are refused without a launch.

A random state of n >= 13 qubits has no amplitude above 0.1. Ten 2x2s are at
most 60 dependent FP32 roundings of 2^-24 on that: 3.6e-7, so 5e-7; a pass
without 2x2s moves amplitudes unchanged.
"""
import ctypes
from ctypes import c_int, c_uint32, c_void_p

import numpy as np
import pytest

import qmetal_gb300 as qm
from test_gpu_group_routes import _apply_ref, _unitary

pytestmark = pytest.mark.gpu
TOL = 5e-7


def _matrix(rng, cls):
    t = rng.uniform(-3, 3)
    c, s = np.cos(t / 2), np.sin(t / 2)
    return {"real": np.array([[c, -s], [s, c]], dtype=complex),
            "rx": np.array([[c, -1j * s], [-1j * s, c]]), "general": _unitary(rng)}[cls]


def _move(st, swap, a, b):
    i = np.arange(st.size)
    d = ((i >> a) ^ (i >> b)) & 1 if swap else (i >> a) & 1
    out = np.empty_like(st)
    out[i ^ (d << b) ^ ((d << a) if swap else 0)] = st
    return out


def _run(n, psi, wires, mats, moves):
    import torch
    L = ctypes.CDLL(qm.library_path())
    f = L.qmk_apply_group_moves
    f.restype = c_int
    f.argtypes = [c_void_p, c_uint32, c_uint32, c_void_p, c_void_p, c_uint32, c_void_p, c_void_p]
    st = torch.tensor(psi, device="cuda")
    w = (c_uint32 * max(1, len(wires)))(*wires)
    m = np.array([[(z.real, z.imag) for z in np.asarray(x).reshape(-1)] for x in mats],
                 dtype=np.float32).reshape(-1)
    g = (c_uint32 * max(1, 3 * len(moves)))(*[int(x) for mv in moves for x in mv])
    torch.cuda.synchronize()
    rc = f(st.data_ptr(), n, len(wires), w, m.ctypes.data, len(moves), g, None)
    torch.cuda.synchronize()
    return rc, st.cpu().numpy()


def _state(n, rng):
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    return (psi / np.linalg.norm(psi)).astype(np.complex64)


def _random_moves(wires, count, rng):
    return [(int(rng.integers(2)), *(int(q) for q in rng.choice(wires, 2, replace=False)))
            for _ in range(count)]


@pytest.mark.parametrize("cls", ["real", "rx", "general"])
@pytest.mark.parametrize("n", [13, 14, 17, 20])
def test_moves(n, cls):
    rng = np.random.default_rng(900 + n)
    low, top = list(range(6)), list(range(6, n))
    sets = [low + top[-4:], low + top[:4], [0, n - 1], [3, 5] + top[1:3], low]
    sets += [top[-k:] for k in (2, 5, 6, 7)] + [top[:7], sorted(rng.choice(top, 7, replace=False))]
    for tile in sets:
        tile = [int(q) for q in tile]
        ladder = [(0, a, b) for a, b in zip(tile, tile[1:])]
        rows = [q for q in tile if q] or tile
        kept = _random_moves(rows, 9, rng) if len(rows) > 1 else ladder   # wire 0 as it is
        for moves in (ladder, ladder[::-1], _random_moves(tile, 12, rng), kept,
                      [(0, 0, tile[-1])] + kept if 0 in tile else kept[::-1]):
            for wires in ([], tile[:1], tile[1:], tile):
                psi = _state(n, rng)
                mats = [_matrix(rng, cls) for _ in wires]
                rc, got = _run(n, psi, wires, mats, moves)
                assert rc == 0
                want = _apply_ref(psi.astype(np.complex128), n, wires, mats)
                for mv in moves:
                    want = _move(want, *mv)
                err = np.abs(got - want).max()
                assert err <= (TOL if wires else 0.0), (wires, moves)


def test_refused():
    rng = np.random.default_rng(5)
    psi = _state(14, rng)
    m = [_unitary(rng)] * 8
    for n, wires, moves in ((12, [0], [(0, 0, 1)]), (14, list(range(6, 14)), [(0, 6, 7)]),
                            (14, [0] + list(range(6, 11)), [(0, 6, 7)]), (14, [14], [(0, 6, 7)]),
                            (14, [3, 3], [(0, 6, 7)]), (14, [], [(0, 2, 2)]),
                            (14, [], [(1, 2, 14)]), (14, [], [(2, 2, 3)]), (14, [2], [])):
        rc, got = _run(n, psi, wires, m[:len(wires)], moves)
        assert rc == -1
        assert np.array_equal(got, psi)
