"""Complex64 passes on wide tiles against the oracle (complex128 values of the
same circuit): gates on every register position, low and high qubits,
overlapping stages, signs before, between and after, in place and out of
place, one tile per CTA and several."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _kinds(circ, n):
    from quantumflow_gb300 import _native as nat
    op_k, op_axes, op_mats, nops = circ.packed(tuple(range(n)))
    stats = (nat.ctypes.c_int32 * (8 * 4096))()
    nb = nat.ctypes.c_int(0)
    nat.call("qf_plan_circuit", n, nat.LAYOUT_C64, nops, op_k.ctypes.data_as(nat._ip),
             op_axes.ctypes.data_as(nat._ip), op_mats.ctypes.data_as(nat._dp), 0, stats, 4096,
             nat.ctypes.byref(nb))
    return [stats[8 * b + 7] for b in range(nb.value)]


def _check(circ, n, seed):
    import quantumflow_gb300 as qf
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.randn(2 ** n, 2, dtype=torch.float32, device="cuda", generator=gen)
    t = torch.view_as_complex(t / t.norm())
    want = circ.run(qf.State(t.to(torch.complex128))).tensor
    got = circ.run(qf.State(t.clone())).tensor
    # each gate rounds like a dot product of 8 terms: 8 u of the amplitudes it
    # mixes, and errors of unitary gates add up
    tol = 8 * len(circ.elements) * 2.0 ** -24
    assert float((got - want).abs().square().sum().sqrt()) <= tol
    # in place
    got = circ.run(qf.zero_state(n, dtype="complex64")).tensor
    want = circ.run(qf.zero_state(n)).tensor
    assert float((got - want).abs().square().sum().sqrt()) <= tol


@pytest.mark.parametrize("n", [15, 16, 20, 21, 23])
@pytest.mark.parametrize("layers", [2, 5])
def test_random_layers(n, layers):
    import quantumflow_gb300 as qf
    rng = np.random.default_rng(n)
    circ = qf.Circuit()
    for _ in range(layers):
        for q in range(n):
            circ += qf.random_gate([q], random_state=rng)
        perm = rng.permutation(n)
        for a in range(0, n - 1, 2):
            circ += qf.CZ(int(perm[a]), int(perm[a + 1]))
    assert 7 in _kinds(circ, n)
    _check(circ, n, 1)


@pytest.mark.parametrize("n", [15, 20, 22])
@pytest.mark.parametrize("where", ["low", "high", "both", "any"])
def test_pairs_of_bits(n, where):
    import quantumflow_gb300 as qf
    rng = np.random.default_rng(n)
    pool = {"low": range(n - 5, n), "high": range(5), "both": [0, 1, 2, n - 3, n - 2, n - 1], "any": range(n)}[where]
    pool = list(pool)
    circ = qf.Circuit()
    for _ in range(40):
        r = rng.random()
        a, b = (int(x) for x in rng.choice(pool, 2, replace=False))
        if r < 0.35:
            circ += qf.random_gate([a, b], random_state=rng)
        elif r < 0.6:
            circ += qf.random_gate([a], random_state=rng)
        elif r < 0.8:
            circ += qf.CZ(a, int(rng.choice([q for q in range(n) if q != a])))
        else:
            circ += qf.Gate(np.diag([1, 1, 1, 1, 1, 1, 1, -1]), qubits=[a, b, next(q for q in range(n) if q not in (a, b))])
    _check(circ, n, 2)


def test_other_gates_end_a_run():
    import quantumflow_gb300 as qf
    n = 20
    rng = np.random.default_rng(1)
    circ = qf.Circuit()
    for k in range(60):
        a, b, c = (int(x) for x in rng.choice(n, 3, replace=False))
        circ += qf.random_gate([a, b], random_state=rng)
        if k % 12 == 5:
            circ += qf.CPHASE(0.3, a, c)
        if k % 20 == 9:
            circ += qf.CCNOT(a, b, c)
        if k % 7 == 0:
            for q in range(0, n - 1, 2):
                circ += qf.CZ(q, (q + a) % n if (q + a) % n != q else (q + 1) % n)
    kinds = _kinds(circ, n)
    assert 7 in kinds and len(set(kinds)) > 1
    _check(circ, n, 3)
