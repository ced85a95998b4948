"""qmk_pauli_expect on a state whose address is a multiple of 8 bytes only: with
a flip it takes it, as it takes one on 16 bytes; without one it is refused.

The bound is that of test_gpu_expect: products that add up to at most 1, thirteen
roundings of 2^-24.
"""
import ctypes
from ctypes import c_double, c_int, c_size_t, c_uint32, c_uint64, c_void_p

import numpy as np
import pytest

import oracle
import qmetal_gb300 as qm

pytestmark = pytest.mark.gpu
TOL = 1e-6


@pytest.mark.parametrize("n", [1, 2, 3, 9, 14, 17])
def test_with_a_flip(n):
    import torch
    L = ctypes.CDLL(qm.library_path())
    L.qmk_workspace_bytes.restype, L.qmk_workspace_bytes.argtypes = c_size_t, [c_uint32]
    L.qmk_workspace_init.restype = c_int
    L.qmk_workspace_init.argtypes = [c_void_p, c_size_t, c_void_p]
    f = L.qmk_pauli_expect
    f.restype = c_int
    f.argtypes = [c_void_p, c_uint32, c_uint64, c_uint32, ctypes.POINTER(c_uint64),
                  ctypes.POINTER(c_uint32), c_void_p, c_void_p, c_size_t, c_void_p]
    rng = np.random.default_rng(1300 + n)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64)
    wide = torch.zeros((1 << n) + 1, dtype=torch.complex64, device="cuda")
    wide[1:] = torch.tensor(psi, device="cuda")
    size = L.qmk_workspace_bytes(n)
    ws = torch.zeros(size, dtype=torch.uint8, device="cuda")
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert L.qmk_workspace_init(ws.data_ptr(), size, None) == 0
    full = (1 << n) - 1
    for flip in {0, 1, 1 << (n - 1), full, int(rng.integers(1, full + 1))}:
        y = int(rng.integers(0, full + 1)) & flip
        z = int(rng.integers(0, full + 1)) & ~flip & full
        strings = [(flip, 0, 0), (flip ^ y, y, z)]
        signs = (c_uint64 * 2)(*[b | c for _, b, c in strings])
        nys = (c_uint32 * 2)(*[bin(b).count("1") for _, b, _ in strings])
        rc = f(wide.data_ptr() + 8, n, flip, 2, signs, nys, out.data_ptr(), ws.data_ptr(), size, None)
        torch.cuda.synchronize()
        if flip == 0:
            assert rc == -1
            continue
        assert rc == 0
        # each pair of amplitudes once: half the value, up to the sign of i^ny
        got = 2 * np.abs(out.cpu().numpy())
        want = [abs(oracle.expectation(n, psi.astype(np.complex128), *s)) for s in strings]
        assert np.abs(got - want).max() <= TOL
