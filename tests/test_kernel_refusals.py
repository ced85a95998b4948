"""What the kernel layer's narrow-state and expectation calls refuse: -1 from the
host's checks, before a launch and without a device."""
import ctypes
from ctypes import POINTER, Structure, c_double, c_float, c_int, c_size_t, c_uint32, c_uint64, c_void_p

import pytest

import qmetal_gb300 as qm

L = ctypes.CDLL(qm.library_path())
STATE = 1 << 20        # an address, never read
WS_BYTES = 1 << 30


class Layer(Structure):
    _fields_ = [("num_terms", c_uint32), ("masks", POINTER(c_uint64)),
                ("angles", POINTER(c_double)), ("global_phase", c_double)]


class Op(Structure):
    _fields_ = [("kind", c_uint32), ("count", c_uint32), ("q", c_uint32 * 3), ("both", c_uint32),
                ("conj", c_uint32), ("save", c_uint32), ("mats", POINTER(c_float)),
                ("mats_lo", POINTER(c_float)), ("mask", c_uint64), ("phase", c_double * 2),
                ("cols", POINTER(c_uint64)), ("layer", Layer), ("num_items", c_uint32),
                ("items", POINTER(c_uint32))]


class Adjoint(Structure):
    _fields_ = [("costate", c_void_p), ("grad", c_void_p), ("num_grad", c_size_t),
                ("energy", c_void_p)]


GROUP, PHASE, CONTROLLED, MAP, LAYER, WINDOW, COSTATE, DIAG_GRAD = range(8)
MATS = (c_float * 256)()


def u32(*v):
    return (c_uint32 * len(v))(*v)


def u64(*v):
    return (c_uint64 * len(v))(*v)


def op(kind, **kw):
    o = Op(kind=kind)
    for k, v in kw.items():
        if k == "q":
            o.q = (c_uint32 * 3)(*v)
        elif k in ("masks", "angles", "num_terms"):
            setattr(o.layer, k, v)
        else:
            setattr(o, k, v)
    return o


def run_small(n, ops, adjoint=None, state=STATE, ws=STATE, ws_bytes=WS_BYTES):
    f = L.qmk_run_small
    f.restype = c_int
    f.argtypes = [c_void_p, c_uint32, c_size_t, POINTER(Op), POINTER(Adjoint), c_void_p, c_size_t,
                  c_void_p]
    arr = (Op * max(1, len(ops)))(*ops)
    return f(state, n, len(ops), arr, ctypes.byref(adjoint) if adjoint else None, ws, ws_bytes, None)


ADJ = Adjoint(STATE, STATE, 4, STATE)

BAD = [
    op(GROUP, count=0, mats=MATS), op(GROUP, count=4, mats=MATS), op(GROUP, count=1),
    op(GROUP, count=1, q=(6, 0, 0), mats=MATS), op(GROUP, count=2, q=(1, 1, 0), mats=MATS),
    op(GROUP, count=2, q=(2, 1, 0), mats=MATS),
    op(PHASE), op(PHASE, mask=64),
    op(CONTROLLED, mask=1), op(CONTROLLED, mask=1, mats=MATS), op(CONTROLLED, mask=64, mats=MATS),
    op(CONTROLLED, mask=1, q=(6, 0, 0), mats=MATS),
    op(MAP), op(MAP, cols=u64(1, 2, 4, 8, 16, 64)), op(MAP, cols=u64(1, 2, 4, 8, 16, 32), save=33),
    op(LAYER, num_terms=1), op(LAYER, num_terms=3001, masks=u64(1), angles=(c_double * 1)()),
    op(LAYER, num_terms=1, masks=u64(64), angles=(c_double * 1)()), op(8),
]
BAD_ADJOINT = [
    op(WINDOW, count=1, num_items=0, items=u32(0, 1, 0), mats=MATS),
    op(WINDOW, count=1, num_items=25, items=u32(*[0] * 75), mats=MATS),
    op(WINDOW, count=1, num_items=13, items=u32(*[0, 1, 0] * 13), mats=MATS),
    op(WINDOW, count=1, num_items=1, items=u32(1, 1, 0), mats=MATS),
    op(WINDOW, count=1, num_items=1, items=u32(0, 4, 0), mats=MATS),
    op(WINDOW, count=1, num_items=1, items=u32(0, 1, 4), mats=MATS),
    op(WINDOW, count=1, num_items=1, items=u32(0, 1, 0)),
    op(WINDOW, count=1, q=(6, 0, 0), num_items=1, items=u32(0, 1, 0), mats=MATS),
    op(COSTATE, num_items=1), op(COSTATE, num_items=1, items=u32(64, 0, 0), mats=MATS),
    op(COSTATE, num_items=1, items=u32(0, 64, 0), mats=MATS), op(COSTATE, num_terms=1),
    op(DIAG_GRAD, num_items=1), op(DIAG_GRAD, num_items=1, items=u32(64, 0)),
    op(DIAG_GRAD, num_items=1, items=u32(1, 4)),
]


@pytest.mark.parametrize("k", range(len(BAD)))
def test_run_small_op(k):
    assert run_small(6, [BAD[k]]) == -1
    assert run_small(6, [BAD[k]], ADJ) == -1


@pytest.mark.parametrize("k", range(len(BAD_ADJOINT)))
def test_run_small_adjoint_op(k):
    assert run_small(6, [BAD_ADJOINT[k]], ADJ) == -1
    assert run_small(6, [BAD_ADJOINT[k]]) == -1


def test_run_small_arguments():
    good = op(PHASE, mask=1)
    for kw in (dict(n=0), dict(n=14), dict(state=None), dict(ws=None), dict(ws_bytes=1024),
               dict(n=13, adjoint=ADJ), dict(adjoint=Adjoint(None, STATE, 4, STATE)),
               dict(adjoint=Adjoint(STATE, None, 4, STATE)), dict(adjoint=Adjoint(STATE, STATE, 4, None))):
        assert run_small(**{"n": 6, "ops": [good], **kw}) == -1, kw
    # both states and kept states without a co-state; a good op before a bad one
    assert run_small(6, [op(PHASE, mask=1, both=1)]) == -1
    assert run_small(6, [op(MAP, cols=u64(1, 2, 4, 8, 16, 32), save=1)]) == -1
    assert run_small(6, [good, BAD[0]]) == -1


def test_z_expect():
    f = L.qmk_z_expect
    f.restype = c_int
    f.argtypes = [c_void_p, c_uint32, c_uint32, POINTER(c_uint64), c_void_p, c_void_p, c_size_t, c_void_p]
    good = dict(state=STATE, n=14, nt=1, masks=u64(1), out=STATE, ws=STATE, size=WS_BYTES)
    for kw in (dict(state=None), dict(state=STATE + 8), dict(n=9), dict(n=41), dict(nt=0),
               dict(nt=33, masks=u64(*[1] * 33)), dict(masks=None), dict(masks=u64(1 << 14)),
               dict(out=None), dict(ws=None), dict(size=16)):
        a = {**good, **kw}
        assert f(a["state"], a["n"], a["nt"], a["masks"], a["out"], a["ws"], a["size"], None) == -1, kw


def test_x_expect():
    f = L.qmk_x_expect
    f.restype = c_int
    f.argtypes = [c_void_p, c_uint32, c_uint32, POINTER(c_uint32), c_void_p, c_void_p, c_size_t, c_void_p]
    good = dict(state=STATE, n=14, nw=1, wires=u32(1), out=STATE, ws=STATE, size=WS_BYTES)
    for kw in (dict(state=None), dict(state=STATE + 8), dict(n=9), dict(n=41), dict(nw=0),
               dict(nw=14, wires=u32(*range(14))), dict(wires=None), dict(wires=u32(14)),
               dict(nw=2, wires=u32(3, 3)), dict(nw=8, wires=u32(*range(6, 14))),
               dict(out=None), dict(ws=None), dict(size=16)):
        a = {**good, **kw}
        assert f(a["state"], a["n"], a["nw"], a["wires"], a["out"], a["ws"], a["size"], None) == -1, kw


def test_expect_small():
    f = L.qmk_expect_small
    f.restype = c_int
    f.argtypes = [c_void_p, c_uint32, c_uint32, POINTER(c_uint64), POINTER(c_uint64),
                  POINTER(c_uint32), c_void_p, c_void_p]
    good = dict(state=STATE, n=6, nt=1, flips=u64(1), signs=u64(1), ny=u32(0), out=STATE)
    for kw in (dict(state=None), dict(n=0), dict(n=15), dict(nt=0), dict(nt=65), dict(flips=None),
               dict(flips=u64(64)), dict(signs=None), dict(ny=None), dict(out=None)):
        a = {**good, **kw}
        assert f(a["state"], a["n"], a["nt"], a["flips"], a["signs"], a["ny"], a["out"], None) == -1, kw
