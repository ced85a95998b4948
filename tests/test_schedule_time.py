"""The host time of Simulator.run's schedule grows with a circuit, not with its square."""
import time

import numpy as np

import qmetal_gb300 as qm  # noqa: F401
from qmetal_gb300 import workloads as W
from test_inplace_schedule import _replay

import oracle


def _moves(n, count, seed):
    rng = np.random.default_rng(seed)
    a = rng.integers(0, n, count)
    b = (a + rng.integers(1, n, count)) % n
    return [(W.SWAP if k % 5 == 0 else W.CX, (int(x), int(y)), ()) for k, (x, y) in enumerate(zip(a, b))]


def _seconds(n, count):
    c = W.to_circuit(n, _moves(n, count, count))
    best = 1e9
    for _ in range(3):
        t0 = time.perf_counter()
        c.schedule_export("inplace")
        best = min(best, time.perf_counter() - t0)
    return best


def test_long_runs_of_moves():
    # four times the gates: 4 where it is linear, 16 where it is quadratic
    assert _seconds(28, 16000) < 8 * _seconds(28, 4000)


def test_runs_longer_than_a_piece():
    n = 13
    layer = [(W.RY, (q,), (0.1 + q,)) for q in range(n)]
    for count in (511, 512, 513, 1300):
        gates = layer + _moves(n, count, count) + layer + _moves(n, 20, 1)
        got, _ = _replay(n, gates)
        assert np.abs(got - oracle.run(n, gates)).max() <= 1e-12
