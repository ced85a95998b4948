"""The work that a user of this simulator has it do, as cases that can be timed and compared.

A case names an entry point (`kind`), a workload family of `qmetal_gb300.workloads` and its sizes:

    run       Simulator.run / run(fuse=False) / run_merged on a circuit, then the read-out of the result
    expect    expectation values of a Hamiltonian on a state that is there already
    sample    draws from a state that is there already
    grad      Simulator.energy_and_gradient, or the torch step of `qmetal_gb300.autograd`
    batch     batch_serve on MaxCut requests of mixed widths

Small states are read out whole (`Simulator.get_state`), large ones through expectation values: nobody moves
gigabytes of amplitudes to the host. Amplitudes are complex64, and what is summed from them (expectation values,
energies, gradients) is as accurate as that type allows, so those are handed on as float32.
"""
import math

import numpy as np
import torch

import qmetal_gb300 as qm
from qmetal_gb300 import workloads as W
from qmetal_gb300.autograd import Template, energy

READ_ALL = 22  # the widest state that is read out amplitude by amplitude


def listed():
    return [
        # A circuit of a few qubits, as teaching, testing and small studies run by the thousand: launches count.
        dict(name="run_u3_9", kind="run", family="u3", n=9, depth=10, how="fused"),
        # The plain gate-by-gate QFT on a random state, one launch per gate (231 controlled phases among them).
        dict(name="run_qft_gates_22", kind="run", family="qft", n=22, depth=1, how="gates"),
        # Trotterised time evolution and the terms of its energy after it, at an odd width.
        dict(name="run_tfim_25", kind="run", family="tfim", n=25, depth=20, how="fused"),
        # A fused circuit on an 8 GiB state, and every term of its Hamiltonian.
        dict(name="run_hea_30", kind="run", family="hea", n=30, depth=3, how="fused"),
        # A QAOA layer stack through the merged executor, with the couplings' values.
        dict(name="merged_qaoa_28", kind="run", family="qaoa", n=28, depth=6, how="merged"),
        # Measuring a state on its own: its norm, each term of couplings and a transverse field, a few longer strings.
        dict(name="expect_tfim_27", kind="expect", n=27, strings=4),
        # The draws of one request from a 2 GiB state.
        dict(name="sample_28", kind="sample", n=28, shots=4096),
        # One step of a small variational loop in torch: new angles, energy, backward pass.
        dict(name="vqe_step_10", kind="grad", family="hea", n=10, depth=4, how="torch"),
        # Adjoint gradients: a hardware-efficient ansatz in cache, QAOA at an odd width, and the ansatz on 2 GiB states.
        dict(name="grad_hea_20", kind="grad", family="hea", n=20, depth=8, how="call"),
        dict(name="grad_qaoa_25", kind="grad", family="qaoa", n=25, depth=4, how="call"),
        dict(name="grad_hea_28", kind="grad", family="hea", n=28, depth=8, how="call"),
        # A sweep's worth of MaxCut instances of mixed widths: energies and gradients for an optimiser.
        dict(name="batch_maxcut_24", kind="batch", count=24, n=22, depth=8),
    ]


def draw(rng):
    kind = rng.choice(["run", "run", "run", "expect", "sample", "grad", "grad", "grad", "batch"])
    if kind == "run":
        family = rng.choice(["u3", "qft", "tfim", "hea", "qaoa"])
        how = rng.choice(["fused", "fused", "merged", "gates"])
        depth = {"u3": rng.randint(2, 10), "qft": 1, "tfim": rng.randint(2, 20), "hea": rng.randint(1, 6),
                 "qaoa": rng.randint(1, 6)}[family]
        return dict(kind=kind, family=family, n=rng.randint(6, 24 if how == "gates" else 28), depth=depth, how=how)
    if kind == "expect":
        return dict(kind=kind, n=rng.randint(8, 28), strings=rng.randint(0, 12))
    if kind == "sample":
        return dict(kind=kind, n=rng.randint(8, 28), shots=int(2 ** rng.uniform(6, 13)))
    if kind == "grad":
        family = rng.choice(["hea", "qaoa", "tfim"])
        how = rng.choice(["call", "call", "torch"])
        return dict(kind=kind, family=family, n=rng.randint(6, 27), depth=rng.randint(1, 8), how=how)
    return dict(kind=kind, count=rng.randint(4, 32), n=2 * rng.randint(7, 11), depth=rng.randint(2, 8))


# --- inputs -------------------------------------------------------------------


def gates_of(case, seed):
    """The gate stream of a run or gradient, its angles (or couplings and step) from the seed."""
    n, d, family = case["n"], case["depth"], case["family"]
    rng = np.random.default_rng([seed, 11])
    if family == "u3":
        return W.random_u3(n, d, seed=seed)
    if family == "qft":
        return W.qft_swap(n)
    if family == "tfim":
        return W.tfim_chain(n, d, J=rng.uniform(0.8, 1.2), h=rng.uniform(0.5, 0.9), dt=rng.uniform(0.03, 0.07))
    if family == "hea":
        return W.hea(n, d, seed=seed)
    return W.qaoa_ring_seeded(n, d, seed=seed)


def terms_of(case):
    """The Hamiltonian that goes with the family, as (coefficient, x, y, z) terms; `strings` longer ones for `expect`."""
    n = case["n"]
    if case.get("family") == "qaoa":
        return W.maxcut_hamiltonian([(i, (i + 1) % n) for i in range(n)])
    terms = W.ring_tfim_hamiltonian(n, 0.7)
    rng = np.random.default_rng([n, 14])
    for _ in range(case.get("strings", 0)):
        masks = [0, 0, 0]
        for q in rng.choice(n, int(rng.integers(2, 5)), replace=False):
            masks[rng.integers(3)] |= 1 << int(q)
        terms.append((0.25, *masks))
    return terms


def requests_of(case, seed):
    """[(n, gates, terms)] of a batch: even widths from 12 to n and 1 to `depth` layers, which are the batch's own;
    random 3-regular graphs and angles from the seed."""
    sizes = np.random.default_rng([case["count"], case["n"], case["depth"]])
    rng = np.random.default_rng([seed, 12])
    out = []
    for _ in range(case["count"]):
        n = 2 * int(sizes.integers(6, case["n"] // 2 + 1))
        p = int(sizes.integers(1, case["depth"] + 1))
        edges = W.random_3regular(n, rng)
        gates = W.maxcut_qaoa(n, edges, rng.uniform(0, math.pi, p), rng.uniform(0, math.pi, p))
        out.append((n, gates, W.maxcut_hamiltonian(edges)))
    return out


def random_state(n, seed, spread):
    """A normalised complex64 state on the GPU: a product of one-qubit states, each amplitude turned by a random
    angle in [0, spread)."""
    rng = np.random.default_rng([seed, 13])
    psi = torch.ones(1, dtype=torch.complex64, device="cuda")
    for _ in range(n):
        a, b = rng.uniform(0.3, math.pi - 0.3), rng.uniform(-math.pi, math.pi)
        q = torch.tensor([math.cos(a / 2), complex(math.cos(b), math.sin(b)) * math.sin(a / 2)], dtype=torch.complex64,
                         device="cuda")
        psi = torch.outer(q, psi).reshape(-1)
    g = torch.Generator(device="cuda").manual_seed(seed)
    turn = torch.rand(1 << n, generator=g, device="cuda") * spread
    psi = psi * torch.polar(torch.ones_like(turn), turn)
    norm = math.sqrt(sum(float(part.to(torch.complex128).abs().square().sum()) for part in psi.chunk(8)))
    return psi / norm


def initial_state(case, seed):
    """The state that a pass starts from, where it is not |0...0>."""
    if case["kind"] in ("expect", "sample"):
        return random_state(case["n"], seed, 1.5)
    if case["kind"] == "run" and case["family"] == "qft":
        return random_state(case["n"], seed, 2 * math.pi)
    return None


def prepare(case, seed):
    if case["kind"] == "batch":
        reqs = [(W.to_circuit(n, gates), W.to_hamiltonian(terms), 0, 0) for n, gates, terms in requests_of(case, seed)]
        return dict(case=case, requests=reqs)
    state = dict(case=case, sim=qm.Simulator(case["n"]))
    psi = initial_state(case, seed)
    if psi is not None:
        state["sim"].set_state(psi.cpu().numpy())
        del psi
        torch.cuda.empty_cache()
    if case["kind"] in ("run", "grad"):
        gates = gates_of(case, seed)
        state["circuit"] = W.to_circuit(case["n"], gates)
    if case["kind"] != "sample":
        state["ham"] = W.to_hamiltonian(terms_of(case))
    if case.get("how") == "torch":
        state["template"] = Template(case["n"], gates)
        state["angles"] = torch.tensor(state["template"].angles(), dtype=torch.float64, requires_grad=True)
    return state


# --- a pass -------------------------------------------------------------------


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        return [torch.tensor([e, *g]) for e, g, _ in qm.batch_serve(state["requests"])]
    sim = state["sim"]
    if case["kind"] == "sample":
        return torch.tensor(sim.sample(case["shots"], seed=7))
    if case["kind"] == "expect":
        return dict(norm=sim.norm(), terms=torch.tensor(sim.expectation_terms(state["ham"])))
    if case["kind"] == "grad":
        if case["how"] == "torch":
            angles = state["angles"]
            angles.grad = None
            e = energy(angles, state["template"], state["ham"], sim)
            e.backward()
            return torch.cat([e.detach().reshape(1), angles.grad]).float()
        e, g = sim.energy_and_gradient(state["circuit"], state["ham"])
        return torch.tensor([e, *g])
    if case["family"] != "qft":  # the transform goes on from the state that is there
        sim.reset()
    if case["how"] == "merged":
        sim.run_merged(state["circuit"])
    else:
        sim.run(state["circuit"], fuse=case["how"] == "fused")
    if case["n"] <= READ_ALL:
        return sim.get_state()
    return torch.tensor(sim.expectation_terms(state["ham"]))


def gate_flops(gates):
    """Operations per amplitude of a gate stream: a one-qubit gate's two complex products and sum, a phase's product."""
    total = 0
    for kind, qubits, _ in gates:
        if kind in (W.RZ, W.P, W.Z, W.S, W.SDG, W.T, W.TDG, W.CZ, W.CP):
            total += 6
        elif len(qubits) == 1:
            total += 14
    return total


def work(case):
    """A state is read or written once for each time that it has to be: written by a circuit, read by what is asked of
    it, and for a gradient the co-state as well."""
    if case["kind"] == "batch":
        reqs = requests_of(case, 1)
        return {"bytes": sum(2 * 8 * 2.0 ** n for n, _, _ in reqs),
                "flops": sum(3 * gate_flops(g) * 2.0 ** n for n, g, _ in reqs)}
    dim = 2.0 ** case["n"]
    if case["kind"] == "expect":
        return {"bytes": 8 * dim, "flops": 2 * 4 * len(terms_of(case)) * dim}
    if case["kind"] == "sample":
        return {"bytes": 8 * dim, "flops": 4 * dim}
    flops = gate_flops(gates_of(case, 1)) * dim
    if case["kind"] == "grad":
        return {"bytes": 2 * 8 * dim, "flops": 3 * flops}
    return {"bytes": 2 * 8 * dim, "flops": flops}


# --- the same in 64 bits, by torch alone -------------------------------------------


def matrix(kind, params):
    """The 2x2 of a one-qubit gate."""
    t = params[0] if params else 0.0
    c, s = math.cos(t / 2), math.sin(t / 2)
    r = math.sqrt(0.5)
    return np.array({
        W.X: [[0, 1], [1, 0]], W.Y: [[0, -1j], [1j, 0]], W.Z: [[1, 0], [0, -1]], W.H: [[r, r], [r, -r]],
        W.RX: [[c, -1j * s], [-1j * s, c]], W.RY: [[c, -s], [s, c]],
        W.RZ: [[complex(c, -s), 0], [0, complex(c, s)]],
    }[kind], dtype=np.complex128)


def axis(psi, q):
    """`psi` with qubit q as the middle one of three axes."""
    return psi.view(-1, 2, 1 << q)


def apply_matrix(psi, q, m):
    v = axis(psi, q)
    a, b = v[:, 0], v[:, 1]
    if m[0, 1] == 0 and m[1, 0] == 0:
        a.mul_(complex(m[0, 0]))
        b.mul_(complex(m[1, 1]))
        return
    old = a.clone()
    a.mul_(complex(m[0, 0])).add_(b, alpha=complex(m[0, 1]))
    b.mul_(complex(m[1, 1])).add_(old, alpha=complex(m[1, 0]))


def quarter(psi, q, r):
    """Views of psi by the bits of the two qubits: [bit q][bit r]."""
    lo, hi = min(q, r), max(q, r)
    v = psi.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)
    return [[v[:, j, :, i] if lo == q else v[:, i, :, j] for j in (0, 1)] for i in (0, 1)]


def apply_pair(psi, kind, qubits, params):
    v = quarter(psi, *qubits)
    if kind in (W.CZ, W.CP):
        t = math.pi if kind == W.CZ else params[0]
        v[1][1].mul_(complex(math.cos(t), math.sin(t)))
        return
    x, y = (v[1][0], v[1][1]) if kind == W.CX else (v[0][1], v[1][0])
    old = x.clone()
    x.copy_(y)
    y.copy_(old)


def apply_gates(psi, gates):
    """Every gate in turn, the one-qubit gates that follow one another on a wire as one."""
    held = {}
    for kind, qubits, params in gates:
        if len(qubits) == 1:
            q = qubits[0]
            held[q] = matrix(kind, params) @ held.get(q, np.eye(2))
            continue
        for q in qubits:
            if q in held:
                apply_matrix(psi, q, held.pop(q))
        apply_pair(psi, kind, qubits, params)
    for q, m in held.items():
        apply_matrix(psi, q, m)


def zero_state(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1
    return psi


def inner(a, b):
    return sum(complex(torch.vdot(x.reshape(-1), y.reshape(-1))) for x, y in zip(a.chunk(4), b.chunk(4)))


def parity_sign(index, mask):
    """+1 or -1 (float64) by the parity of the index bits in mask."""
    odd = torch.zeros_like(index)
    for q in range(64):
        if mask >> q & 1:
            odd ^= index >> q
    return (1 - 2 * (odd & 1)).double()


def exact_terms(psi, terms):
    """<P> for each Pauli string, in parts that a large state's temporaries fit beside."""
    out, part = [], min(psi.numel(), 1 << 27)
    for _, x, y, z in terms:
        total, turn = 0.0, 1j ** (bin(y).count("1") % 4)
        for at in range(0, psi.numel(), part):
            index = torch.arange(at, at + part, device=psi.device)
            here = psi[at:at + part]
            there = psi[index ^ (x | y)] if x | y else here
            sign = parity_sign(index, y | z)
            total += (turn * complex(torch.dot((there.conj() * here).real, sign), torch.dot((there.conj() * here).imag, sign))).real
        out.append(total)
    return torch.tensor(out, dtype=torch.float64)


def apply_terms(psi, terms):
    out = torch.zeros_like(psi)
    for c, x, y, z in terms:
        if x:
            out.view(-1, 2, x).add_(psi.view(-1, 2, x).flip(1), alpha=c)
            continue
        bits = [q for q in range(64) if z >> q & 1]
        if not bits:
            out.add_(psi, alpha=c)
            continue
        v, w = quarter(out, *bits), quarter(psi, *bits)
        for i in (0, 1):
            for j in (0, 1):
                v[i][j].add_(w[i][j], alpha=c * (-1) ** (i + j))
    return out


def exact_gradient(n, gates, terms):
    """[energy, one entry per gate] by the adjoint method."""
    psi = zero_state(n)
    apply_gates(psi, gates)
    lam = apply_terms(psi, terms)
    e, g = inner(psi, lam).real, [0.0] * len(gates)
    for k in range(len(gates) - 1, -1, -1):
        kind, qubits, params = gates[k]
        if len(qubits) > 1:
            for s in (psi, lam):
                apply_pair(s, kind, qubits, [-t for t in params])
            continue
        a, b = axis(lam, qubits[0]), axis(psi, qubits[0])
        if kind == W.RZ:
            g[k] = (complex((a[:, 0].conj() * b[:, 0]).sum()) - complex((a[:, 1].conj() * b[:, 1]).sum())).imag
        elif kind in (W.RX, W.RY):
            up, down = complex((a[:, 0].conj() * b[:, 1]).sum()), complex((a[:, 1].conj() * b[:, 0]).sum())
            g[k] = (up + down).imag if kind == W.RX else (-1j * up + 1j * down).imag
        for s in (psi, lam):
            apply_matrix(s, qubits[0], matrix(kind, params).conj().T)
    return torch.tensor([e, *g], dtype=torch.float64)


def exact(case, seed):
    if case["kind"] == "batch":
        return [exact_gradient(*r) for r in requests_of(case, seed)]
    n = case["n"]
    if case["kind"] == "sample":
        return None
    if case["kind"] == "expect":
        psi = random_state(n, seed, 1.5).to(torch.complex128)
        return dict(norm=math.sqrt(inner(psi, psi).real), terms=exact_terms(psi, terms_of(case)))
    gates = gates_of(case, seed)
    if case["kind"] == "grad":
        if n > 22 and 2.0 ** n * len(gates) > 2.0 ** 35:
            return None
        out = exact_gradient(n, gates, terms_of(case))
        if case["how"] == "torch":  # one entry per angle, not per gate
            out = out[[0] + [1 + k for k, g in enumerate(gates) if g[2]]]
        return out
    psi = initial_state(case, seed)
    psi = zero_state(n) if psi is None else psi.to(torch.complex128)
    if 2.0 ** n * len(gates) > 2.0 ** 39:
        return None
    apply_gates(psi, gates)
    if n <= READ_ALL:
        return psi.cpu().numpy()
    return exact_terms(psi, terms_of(case))
