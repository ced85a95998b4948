"""The bench's byte counts of a served request follow the schedules it is served by."""
import pytest

import qmetal_gb300 as qm  # noqa: F401
from qmetal_gb300 import workloads as W
from test_bench_sets import _bench


@pytest.mark.parametrize("n", [8, 12, 14, 18, 20])
def test_request_bytes(n):
    S = 8.0 * (1 << n)
    gates = W.qaoa_ring_seeded(n, 3)
    terms = W.maxcut_hamiltonian([(i, (i + 1) % n) for i in range(n)])
    args = (n, gates, W.to_circuit(n, gates), W.to_hamiltonian(terms))
    got, sampled = (_bench().request_bytes(*args, shots, 6) for shots in (0, 100))
    if n <= 12:   # one launch: the state in, both states out
        assert got == 4 * S and sampled == 8 * S
        return
    assert sampled == got + S
    passes = W.to_circuit(n, gates).schedule_export("gradient")[0]
    merged = W.to_circuit(n, gates).schedule_export("forward")[0]
    assert passes < merged if n == 18 else passes <= merged
    # reset, forward passes of 2 S, Z strings 2 S, and the sweep's passes of at most 4 S
    assert S * (1 + 2 * passes + 2) < got <= S * (1 + 2 * passes + 2 + 4 * 3 * (1 + -(-n // 6) + 1))
