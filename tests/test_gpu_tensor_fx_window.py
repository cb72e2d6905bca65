"""The pass unitary of a window of many gates: outputs bit for bit those of the
integer model whose U is the gates' exact product, rounded once to 2^-62.
Gates with entries down to 2^-40, permutations, diagonals and signs among
them; the host's product carries 2^-91."""
from fractions import Fraction

import numpy as np
import pytest

import txarith as tx

pytestmark = pytest.mark.gpu

N = 11
WINDOW = (0, 1, 2, 3)  # qubits; window index bit j is qubit 3 - j


def _gates(kind, count):
    rng = np.random.default_rng(count)
    # all four bits from the second gate on (one pass), and never a pair twice
    # running (two gates on one pair are multiplied in FP64 before)
    pairs = [(0, 1), (2, 3), (1, 2)]
    out = []
    for i in range(count):
        q = pairs[i % 3]
        if kind == "small":  # off-diagonal entries from 2^-6 down to 2^-40
            eps = 2.0 ** -rng.integers(6, 40)
            h = rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4))
            u = np.linalg.qr(np.eye(4) + eps * h)[0]
        else:
            u = np.linalg.qr(rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4)))[0]
        if kind == "mixed" and i > 1 and i % 4 == 1:
            u = np.eye(4)[rng.permutation(4)] * np.exp(1j * rng.uniform(0, 6, 4))[:, None]
        elif kind == "mixed" and i % 4 == 2:
            u = np.diag(np.exp(1j * rng.uniform(0, 6, 4)))
        elif kind == "mixed" and i % 4 == 3:
            u = np.diag([1.0, 1, 1, -1])
        out.append((np.asarray(u, complex), q))
    return out


def _plan(circ):
    from quantumflow_gb300 import _native as nat
    op_k, op_axes, op_mats, nops = circ.packed(tuple(range(N)))
    stats = (nat.ctypes.c_int32 * (8 * 64))()
    nb = nat.ctypes.c_int(0)
    nat.call("qf_plan_circuit", N, nat.LAYOUT_FX, nops, op_k.ctypes.data_as(nat._ip),
             op_axes.ctypes.data_as(nat._ip), op_mats.ctypes.data_as(nat._dp), 0, stats, 64, nat.ctypes.byref(nb))
    return [(stats[8 * b + 7], stats[8 * b]) for b in range(nb.value)]


def _product(gates):
    """16 x 16 exact product: object arrays of Fractions (re, im)."""
    re = np.array([[Fraction(int(r == c)) for c in range(16)] for r in range(16)], object)
    im = np.array([[Fraction(0)] * 16 for _ in range(16)], object)
    for m, (a, b) in gates:
        bits = (3 - a, 3 - b)  # window bits, matrix MSB first
        local = lambda r: (((r >> bits[0]) & 1) << 1) | ((r >> bits[1]) & 1)
        keep = 15 & ~(1 << bits[0]) & ~(1 << bits[1])
        nr, ni = re.copy(), im.copy()
        for r in range(16):
            tr, ti = 0, 0
            for k in range(16):
                if (k & keep) != (r & keep):
                    continue
                v = m[local(r), local(k)]
                vr, vi = Fraction(float(v.real)), Fraction(float(v.imag))
                tr = tr + vr * re[k] - vi * im[k]
                ti = ti + vr * im[k] + vi * re[k]
            nr[r], ni[r] = tr, ti
        re, im = nr, ni
    return re, im


@pytest.mark.parametrize("kind", ["haar", "small", "mixed"])
@pytest.mark.parametrize("count", [2, 5, 30])
def test_product_is_rounded_once(kind, count):
    import quantumflow_gb300 as qf
    gates = _gates(kind, count)
    rng = np.random.default_rng(1)
    psi = rng.normal(size=2 ** N) + 1j * rng.normal(size=2 ** N)
    psi /= np.linalg.norm(psi)
    circ = qf.Circuit([qf.Gate(m, qubits=list(q)) for m, q in gates])
    assert _plan(circ) == [(6, count)]
    got = circ.run(qf.State(psi.reshape((2,) * N))).asarray().reshape(16, -1)
    re, im = _product(gates)
    g = np.zeros((16, 16, 2), object)
    for r in range(16):
        for c in range(16):
            g[r][c][0] = tx._round_half_away(re[r, c] * 2 ** 62)
            g[r][c][1] = tx._round_half_away(im[r, c] * 2 ** 62)
    gd = tx.gate_digits(g)
    rows = psi.reshape(16, -1)
    want = np.stack([tx.pass_row(g, rows[:, x], gd) for x in range(rows.shape[1])], axis=1)
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64)), float(np.max(np.abs(got - want)))
