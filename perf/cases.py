"""Performance cases: the work users of this framework give it, through its
public entry points, with the same results in plain 64-bit torch beside them.

Kinds (field ``kind`` of a case):

``layers``   Circuit.run from |0..0>: random one-qubit unitaries on every
             qubit, then CZ on a random matching, per layer (the circuit
             family of the repository's benchmark).
``gops``     Circuit.run of the gate-throughput circuit of
             quantumflow_gb300/benchmark.py (H everywhere, then X, T, CNOT).
``qft``      Circuit.run of the Fourier transform on a state in hand.
``qaoa``     QAOAMaxCut.expectation_and_grad: one optimiser step's work on
             one graph.
``batch``    QAOABatch.set_angles + evaluate: one optimiser step's work on
             many graphs of uneven size and depth.
``noise``    Circuit.evolve of a density matrix: gates, with a noise channel
             on every qubit after each layer.
``readout``  the read-outs of a state in hand: probabilities, the expectation
             of a diagonal observable, the norm, and sampled counts.
"""
import math
import random

import numpy as np
import torch

import quantumflow_gb300 as qf
from quantumflow_gb300 import qaoa
from quantumflow_gb300.batched import QAOABatch

_BYTES = {"complex64": 8, "complex128": 16}
_REAL = {"complex64": torch.float32, "complex128": torch.float64}


def listed():
    return [
        # a small circuit in a loop (variational inner loop, teaching,
        # tests): launches and host work count
        {"name": "layers_n10_c128", "kind": "layers", "n": 10, "layers": 4, "dtype": "complex128"},
        # the gate-throughput benchmark at its default size
        {"name": "gops_n16_c128", "kind": "gops", "n": 16, "gates": 100, "dtype": "complex128"},
        # an ordinary simulation that fits the last-level cache, odd size
        {"name": "layers_n21_c128", "kind": "layers", "n": 21, "layers": 10, "dtype": "complex128"},
        # the headline: a state of 4 GiB, the largest case
        {"name": "layers_n28_c128", "kind": "layers", "n": 28, "layers": 8, "dtype": "complex128"},
        # the same family in single precision
        {"name": "layers_n26_c64", "kind": "layers", "n": 26, "layers": 10, "dtype": "complex64"},
        # the circuit library's diagonal-heavy circuit, odd size
        {"name": "qft_n23_c128", "kind": "qft", "n": 23, "dtype": "complex128"},
        # one gradient step of the QAOA example on a small graph
        {"name": "qaoa_n12_c128", "kind": "qaoa", "n": 12, "p": 5, "graph": "gnp", "dtype": "complex128"},
        # ... on graphs whose states are large, in both precisions
        {"name": "qaoa_n22_c128", "kind": "qaoa", "n": 22, "p": 8, "graph": "regular", "dtype": "complex128"},
        {"name": "qaoa_n24_c64", "kind": "qaoa", "n": 24, "p": 6, "graph": "gnp", "dtype": "complex64"},
        # a training set's worth of uneven graphs, one evaluation
        {"name": "batch_200_c64", "kind": "batch", "count": 200, "nmin": 8, "nmax": 18, "pmax": 6,
         "dtype": "complex64"},
        # noisy evolution of a density matrix (2 * 11 axes)
        {"name": "noise_n11_c128", "kind": "noise", "n": 11, "layers": 2, "dtype": "complex128"},
        # the read-outs after a run
        {"name": "readout_n22_c128", "kind": "readout", "n": 22, "trials": 1000, "dtype": "complex128"},
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["layers", "layers", "layers", "gops", "qft", "qaoa", "qaoa", "qaoa", "batch", "noise",
                       "readout"])
    dtype = rng.choice(["complex128", "complex128", "complex64"])
    # sizes of a state go by its number of qubits, the logarithm of its size
    if kind == "layers":
        return {"kind": kind, "n": rng.randint(6, 27), "layers": _log(rng, 2, 14), "dtype": dtype}
    if kind == "gops":
        return {"kind": kind, "n": rng.randint(8, 24), "gates": _log(rng, 40, 400), "dtype": dtype}
    if kind == "qft":
        return {"kind": kind, "n": rng.randint(6, 25), "dtype": dtype}
    if kind == "qaoa":
        return {"kind": kind, "n": rng.randint(6, 24), "p": rng.randint(1, 8),
                "graph": rng.choice(["gnp", "regular"]), "dtype": dtype}
    if kind == "batch":
        nmin = rng.randint(6, 12)
        return {"kind": kind, "count": _log(rng, 8, 300), "nmin": nmin, "nmax": rng.randint(nmin, 18),
                "pmax": rng.randint(1, 6), "dtype": dtype}
    if kind == "noise":
        return {"kind": kind, "n": rng.randint(3, 12), "layers": rng.randint(1, 4), "dtype": dtype}
    return {"kind": kind, "n": rng.randint(8, 25), "trials": _log(rng, 1, 100000), "dtype": dtype}


# ------------------------------------------------------------------ inputs --
def _unitary(rng, count):
    """Haar-random 2x2 unitaries: the QR of complex Gaussian matrices, its
    phases fixed by R's diagonal."""
    z = rng.normal(size=(count, 2, 2)) + 1j * rng.normal(size=(count, 2, 2))
    q, r = np.linalg.qr(z)
    d = np.diagonal(r, axis1=1, axis2=2)
    return q * (d / np.abs(d))[:, None, :]


def _layer_ops(n, layers, seed):
    """(qubits, matrix) per gate; None stands for CZ."""
    rng = np.random.default_rng(seed)
    ops = []
    for _ in range(layers):
        for q, u in enumerate(_unitary(rng, n)):
            ops.append(((q,), u))
        perm = rng.permutation(n)
        for a in range(0, n - 1, 2):
            ops.append(((int(perm[a]), int(perm[a + 1])), None))
    return ops


def _circuit(ops):
    return qf.Circuit([qf.CZ(*qs) if u is None else qf.Gate(u, qubits=qs) for qs, u in ops])


def _gops_ops(n, gates, seed):
    """(gate name, qubits): H on every qubit, then rounds of X on a random
    qubit, T on another and CNOT between them."""
    rng = random.Random(seed)
    ops = [("H", (q,)) for q in range(n)]
    for _ in range((gates - n) // 3):
        q0, q1 = rng.sample(range(n), 2)
        ops += [("X", (q0,)), ("T", (q1,)), ("CNOT", (q0, q1))]
    return ops


def _noise_ops(n, layers, seed):
    """(kind, qubits, value) per element: gates, then one channel per qubit."""
    rng = np.random.default_rng(seed)
    ops = []
    for _ in range(layers):
        ops += [("gate", qs, u) for qs, u in _layer_ops(n, 1, int(rng.integers(1 << 30)))]
        for q in range(n):
            name = ("depolarizing", "damping", "dephasing")[int(rng.integers(3))]
            ops.append((name, (q,), float(rng.uniform(0.001, 0.1))))
    return ops


def _noise_circuit(ops):
    chan = {"depolarizing": qf.Depolarizing, "damping": qf.Damping, "dephasing": qf.Dephasing}
    elems = []
    for kind, qs, v in ops:
        if kind != "gate":
            elems.append(chan[kind](v, qs[0]))
        else:
            elems.append(qf.CZ(*qs) if v is None else qf.Gate(v, qubits=qs))
    return qf.Circuit(elems)


def _random_ket(n, dtype, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.randn(2 ** n, 2, dtype=_REAL[dtype], device="cuda", generator=gen)
    t /= t.norm()
    return torch.view_as_complex(t)


def _graph(n, kind, rng):
    """A graph with at least one edge: 3-regular where n allows it, else
    (or asked) G(n, 1/2)."""
    seed = int(rng.integers(1 << 30))
    if kind == "regular" and n % 2 == 0 and n > 3:
        return qaoa.random_regular_graph(3, n, seed=seed)
    g = qaoa.gnp_random_graph(n, 0.5, seed=seed)
    if not g.edges():
        g.add_edge(0, n - 1)
    return g


def _angles(p, rng):
    """Angles on an optimiser's way: the linear ramp, moved at random."""
    b, g = qaoa.linear_ramp_angles(p)
    return b + 0.1 * rng.normal(size=p), g + 0.1 * rng.normal(size=p)


def _qaoa_inputs(case, seed):
    rng = np.random.default_rng(seed)
    return (_graph(case["n"], case["graph"], rng), *_angles(case["p"], rng))


def _batch_inputs(case, seed):
    """The sizes and depths are the case's, the graphs and angles the seed's."""
    sizes, rng = random.Random(case["count"]), np.random.default_rng(seed)
    graphs, betas, gammas = [], [], []
    for i in range(case["count"]):
        n, p = sizes.randint(case["nmin"], case["nmax"]), sizes.randint(1, case["pmax"])
        graphs.append(_graph(n, "gnp" if i % 2 else "regular", rng))
        b, g = _angles(p, rng)
        betas.append(b)
        gammas.append(g)
    return graphs, betas, gammas


def _diagonal(n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    return torch.rand(2 ** n, dtype=torch.float64, device="cuda", generator=gen)


def prepare(case, seed):
    kind, n, dtype = case["kind"], case.get("n"), case["dtype"]
    s = {"kind": kind, "n": n, "dtype": dtype}
    if kind == "layers":
        s["circuit"] = _circuit(_layer_ops(n, case["layers"], seed))
    elif kind == "gops":
        gate = {"H": qf.H, "X": qf.X, "T": qf.T, "CNOT": qf.CNOT}
        s["circuit"] = qf.Circuit([gate[name](*qs) for name, qs in _gops_ops(n, case["gates"], seed)])
    elif kind == "qft":
        s["circuit"] = qf.qft_circuit(range(n))
        s["ket"] = qf.State(_random_ket(n, dtype, seed))
    elif kind == "qaoa":
        graph, s["beta"], s["gamma"] = _qaoa_inputs(case, seed)
        s["problem"] = qf.QAOAMaxCut(graph, case["p"], dtype=dtype)
    elif kind == "batch":
        graphs, s["betas"], s["gammas"] = _batch_inputs(case, seed)
        s["batch"] = QAOABatch(graphs, [len(b) for b in s["betas"]], dtype=dtype)
    elif kind == "noise":
        s["circuit"] = _noise_circuit(_noise_ops(n, case["layers"], seed))
        s["rho"] = qf.State(_random_ket(n, dtype, seed)).asdensity()
    else:
        s["ket"] = qf.State(_random_ket(n, dtype, seed))
        s["diagonal"] = _diagonal(n, seed)
        s["trials"], s["seed"] = case["trials"], seed
    return s


def run(state):
    kind = state["kind"]
    if kind in ("layers", "gops"):
        return state["circuit"].run(qf.zero_state(state["n"], dtype=state["dtype"])).tensor
    if kind == "qft":
        return state["circuit"].run(state["ket"]).tensor
    if kind == "qaoa":
        return state["problem"].expectation_and_grad(state["beta"], state["gamma"])
    if kind == "batch":
        state["batch"].set_angles(state["betas"], state["gammas"])
        e, db, dg = state["batch"].evaluate()
        return e, np.concatenate(db), np.concatenate(dg)
    if kind == "noise":
        return state["circuit"].evolve(state["rho"]).tensor
    ket = state["ket"]
    return {"probabilities": ket.probabilities(), "expectation": ket.expectation(state["diagonal"]),
            "norm": ket.norm(), "counts": ket.sample(state["trials"], seed=state["seed"])}


# -------------------------------------------------------------------- work --
def work(case):
    """State bytes in and out once, tables read once; the arithmetic of the
    gates on each amplitude (14 for a 2x2 matrix, 6 for a phase, 0 for a sign
    or a permutation)."""
    kind, dtype = case["kind"], case["dtype"]
    S = _BYTES[dtype]
    if kind == "layers":
        n = case["n"]
        return {"bytes": S * 2 ** n, "flops": 14 * n * case["layers"] * 2 ** n}
    if kind == "gops":
        n = case["n"]
        # H on every qubit (4 adds or scalings a part pair) and the T phases
        return {"bytes": S * 2 ** n, "flops": (4 * n + 3 * max(0, (case["gates"] - n) // 3)) * 2 ** n}
    if kind == "qft":
        n = case["n"]
        return {"bytes": 2 * S * 2 ** n, "flops": (4 * n + 6 * n * (n - 1) / 8) * 2 ** n}
    if kind == "qaoa":
        # forward once, backward on two vectors: a phase (6) per layer and
        # RX (6 an amplitude) and a gradient term (4) per qubit and layer
        n, p = case["n"], case["p"]
        return {"bytes": 2 * 2 ** n, "flops": p * (3 * (6 + 6 * n) + 4 * n) * 2 ** n}
    if kind == "batch":
        lo, hi, p = case["nmin"], case["nmax"], (1 + case["pmax"]) / 2
        sizes = range(lo, hi + 1)
        flops = sum(p * (3 * (6 + 6 * n) + 4 * n) * 2 ** n for n in sizes) / len(sizes)
        return {"bytes": case["count"] * sum(2 * 2 ** n for n in sizes) / len(sizes),
                "flops": case["count"] * flops}
    if kind == "noise":
        n = case["n"]
        # 2x2 matrices on ket and bra axes, and a channel's five terms
        return {"bytes": 2 * S * 4 ** n, "flops": case["layers"] * n * (2 * 14 + 6) * 4 ** n}
    n = case["n"]
    return {"bytes": (S + 8 + 8 + 8) * 2 ** n, "flops": 7 * 2 ** n}


# ------------------------------------------------------ plain 64-bit values --
def _apply(t, u, axis, n):
    """A 2x2 matrix on one axis of a flat 2^n tensor."""
    v = t.reshape(2 ** axis, 2, -1)
    u = [[complex(x) for x in row] for row in np.asarray(u).reshape(2, 2)]
    return torch.stack([v[:, 0] * u[0][0] + v[:, 1] * u[0][1], v[:, 0] * u[1][0] + v[:, 1] * u[1][1]],
                       dim=1).reshape(-1)


def _phase_(t, axes, n, factor):
    """In place: `factor` where all the given axes are 1."""
    v, at, last = t, [], -1
    shape = []
    for a in sorted(axes):
        shape += [2 ** (a - last - 1), 2]
        at += [slice(None), 1]
        last = a
    v = t.reshape(shape + [-1])
    v[tuple(at)] *= factor
    return t


def _cnot(t, control, target, n):
    v = t.reshape([2] * n).movedim((control, target), (0, 1))
    out = torch.stack([v[0], v[1].flip(0)])
    return out.movedim((0, 1), (control, target)).reshape(-1)


_H = np.array([[1, 1], [1, -1]]) / math.sqrt(2)


def _zero(n):
    t = torch.zeros(2 ** n, dtype=torch.complex128, device="cuda")
    t[0] = 1
    return t


def _bits(n):
    x = torch.arange(2 ** n, device="cuda")
    return [(x >> (n - 1 - a)) & 1 for a in range(n)]


def _cuts(graph, n):
    b = _bits(n)
    c = torch.zeros(2 ** n, dtype=torch.float64, device="cuda")
    for u, v in graph.edges():
        c += b[u] ^ b[v]
    return c


def _flip(t, axis):
    return t.reshape(2 ** axis, 2, -1).flip(1).reshape(-1)


def _rx(t, theta, axis, n):
    return t * math.cos(theta / 2) + _flip(t, axis) * (-1j * math.sin(theta / 2))


def _qaoa_exact(graph, n, beta, gamma):
    cuts = _cuts(graph, n)
    edges = len(graph.edges())
    psi = torch.full((2 ** n,), 2 ** (-n / 2), dtype=torch.complex128, device="cuda")
    for b, g in zip(beta, gamma):
        psi = psi * torch.exp(1j * g * (edges / 2 - cuts))
        for a in range(n):
            psi = _rx(psi, b, a, n)
    e = (cuts * (psi.real ** 2 + psi.imag ** 2)).sum()
    lam = cuts * psi
    gb, gg = np.zeros(len(beta)), np.zeros(len(gamma))
    for l in reversed(range(len(beta))):
        # d/dbeta of prod_j RX_j(beta) = -i/2 sum_j X_j
        gb[l] = float(sum(torch.vdot(lam, _flip(psi, a)).imag for a in range(n)))
        for a in range(n):
            psi, lam = _rx(psi, -beta[l], a, n), _rx(lam, -beta[l], a, n)
        # d/dgamma of exp(i gamma (E/2 - C)) = i (E/2 - C)
        gg[l] = -2 * float(torch.vdot(lam, (edges / 2 - cuts) * psi).imag)
        back = torch.exp(-1j * gamma[l] * (edges / 2 - cuts))
        psi, lam = psi * back, lam * back
    return float(e), gb, gg


def _noise_exact(case, seed):
    n = case["n"]
    ket = _random_ket(n, case["dtype"], seed).to(torch.complex128)
    rho = torch.outer(ket, ket.conj()).reshape(-1)
    x, y, z = np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), np.diag([1, -1])
    for kind, qs, v in _noise_ops(n, case["layers"], seed):
        if kind == "gate":
            if v is None:
                rho = _phase_(_phase_(rho, qs, 2 * n, -1), [n + q for q in qs], 2 * n, -1)
                continue
            kraus = [v]
        elif kind == "depolarizing":
            kraus = [math.sqrt(1 - v) * np.eye(2)] + [math.sqrt(v / 3) * m for m in (x, y, z)]
        elif kind == "damping":
            kraus = [np.diag([1, math.sqrt(1 - v)]), np.array([[0, math.sqrt(v)], [0, 0]])]
        else:
            kraus = [math.sqrt(1 - v / 2) * np.eye(2), math.sqrt(v / 2) * z]
        rho = sum(_apply(_apply(rho, k, qs[0], 2 * n), np.conj(k), n + qs[0], 2 * n) for k in kraus)
    return rho.reshape([2] * (2 * n))


def exact(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind == "layers":
        t = _zero(n)
        for qs, u in _layer_ops(n, case["layers"], seed):
            t = _phase_(t, qs, n, -1) if u is None else _apply(t, u, qs[0], n)
        return t.reshape([2] * n)
    if kind == "gops":
        t = _zero(n)
        for name, qs in _gops_ops(n, case["gates"], seed):
            if name == "H":
                t = _apply(t, _H, qs[0], n)
            elif name == "X":
                t = _flip(t, qs[0])
            elif name == "T":
                t = _phase_(t.clone(), qs, n, complex(math.cos(math.pi / 4), math.sin(math.pi / 4)))
            else:
                t = _cnot(t, qs[0], qs[1], n)
        return t.reshape([2] * n)
    if kind == "qft":
        # the transform is the inverse DFT, unitary
        t = torch.fft.ifft(_random_ket(n, case["dtype"], seed).to(torch.complex128), norm="ortho")
        return t.reshape([2] * n)
    if kind == "qaoa":
        graph, beta, gamma = _qaoa_inputs(case, seed)
        return _qaoa_exact(graph, n, beta, gamma)
    if kind == "batch":
        if case["count"] * (case["nmin"] + case["nmax"]) * case["pmax"] > 40000:
            return None  # too many small launches to finish in time
        es, db, dg = [], [], []
        for graph, beta, gamma in zip(*_batch_inputs(case, seed)):
            e, gb, gg = _qaoa_exact(graph, len(graph), beta, gamma)
            es.append(e)
            db.append(gb)
            dg.append(gg)
        return np.array(es), np.concatenate(db), np.concatenate(dg)
    if kind == "noise":
        return _noise_exact(case, seed)
    ket = _random_ket(n, case["dtype"], seed).to(torch.complex128)
    p = ket.real ** 2 + ket.imag ** 2
    return {"probabilities": p.reshape([2] * n), "expectation": float((p * _diagonal(n, seed)).sum()),
            "norm": float(p.sum()), "counts": None}
