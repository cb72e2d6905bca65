"""Noise channels taken into the gate passes of a density's circuit: every
channel, weak and strong, alone and two to a window (a window of norm above
one is held halved), after one- and two-qubit gates, on 6 to 9 qubits, and the
gates that are not unitary but channel-like on a state vector."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# a pass errs by 2^-55 of its row's largest part (at most 1, twice that where
# the window is held halved) and one rounding; fewer than 60 passes
TOL = 60 * 2.0 ** -52


def _ref(rho, n, ops):
    """Kraus sums in complex128; rho as 2n axes, kets first."""
    for ks, qs in ops:
        k = len(qs)
        out = 0
        for op in ks:
            m = op.reshape((2,) * 2 * k)
            t = np.tensordot(m, rho, (list(range(k, 2 * k)), list(qs)))
            t = np.moveaxis(t, range(k), qs)
            t = np.tensordot(m.conj(), t, (list(range(k, 2 * k)), [n + q for q in qs]))
            out = out + np.moveaxis(t, range(k), [n + q for q in qs])
        rho = out
    return rho


def _haar(rng, d):
    q, r = np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def _kinds(ops, n):
    from quantumflow_gb300 import _native as nat
    k = np.array([len(q) for _, q in ops], np.int32)
    axes = np.array([a for _, q in ops for a in q], np.int32)
    mats = np.concatenate([np.ascontiguousarray(m, complex).view(float).reshape(-1) for m, _ in ops])
    stats = (nat.ctypes.c_int32 * (8 * 512))()
    nb = nat.ctypes.c_int(0)
    nat.call("qf_plan_circuit", n, nat.LAYOUT_FX, len(k), k.ctypes.data_as(nat._ip), axes.ctypes.data_as(nat._ip),
             mats.ctypes.data_as(nat._dp), 0, stats, 512, nat.ctypes.byref(nb))
    return [stats[8 * b + 7] for b in range(nb.value)]


def _superop(ks):
    return sum(np.kron(k, k.conj()) for k in ks)


@pytest.mark.parametrize("n", [6, 7, 9])
@pytest.mark.parametrize("strength", [1e-12, 0.05, 0.3, 0.6, 1.0])
def test_channels_with_gates(n, strength):
    import quantumflow_gb300 as qf
    rng = np.random.default_rng(int(100 * strength) + n)
    elems, ref = [], []
    for layer in range(3):
        for q in range(n):
            u = _haar(rng, 2)
            elems.append(qf.Gate(u, qubits=[q]))
            ref.append(([u], (q,)))
        perm = rng.permutation(n)
        for a in range(0, n - 1, 2):
            i, j = int(perm[a]), int(perm[a + 1])
            u = _haar(rng, 4) if layer else np.diag([1, 1, 1, -1]).astype(complex)
            elems.append(qf.Gate(u, qubits=[i, j]))
            ref.append(([u], (i, j)))
        for q in range(n):
            for cls in [(qf.Depolarizing,), (qf.Damping,), (qf.Dephasing,), (qf.Damping, qf.Dephasing)][(q + layer) % 4]:
                c = cls(strength, q)
                elems.append(c)
                ref.append(([np.asarray(k.asoperator()) * np.sqrt(w) for k, w in zip(c.operators, c.weights)], (q,)))
    rho = qf.random_density(n) if n < 8 else qf.random_state(n).asdensity()
    start = np.asarray(rho.asarray()).reshape((2,) * 2 * n).copy()
    got = qf.Circuit(elems).evolve(rho)
    want = _ref(start, n, ref)
    assert np.max(np.abs(np.asarray(got.asarray()).reshape(want.shape) - want)) < TOL
    assert np.array_equal(np.asarray(rho.asarray()).reshape(start.shape), start)


def test_channel_routes():
    """Weak channels run inside gate passes; strong ones, projections and
    channels without a gate on their bits keep passes of their own."""
    rng = np.random.default_rng(3)
    u, n = _haar(rng, 4), 6
    gates = [(u, (0, 1)), (u.conj(), (n, n + 1))]
    damp = lambda p: _superop([np.diag([1, np.sqrt(1 - p)]), np.array([[0, np.sqrt(p)], [0, 0]])])
    assert _kinds(gates + [(damp(0.1), (0, n)), (damp(0.1), (1, n + 1))], 2 * n) == [6]
    assert _kinds(gates + [(damp(0.9), (0, n))], 2 * n) == [6, 5]
    assert _kinds(gates + [(np.diag([1.0, 0, 0, 0]), (0, n))], 2 * n) == [6, 5]
    assert _kinds(gates + [(damp(0.1), (2, n + 2))], 2 * n) == [6, 5]
    assert _kinds([(damp(0.1), (0, n))], 2 * n) == [5]


@pytest.mark.parametrize("n", [11, 12, 16])
@pytest.mark.parametrize("scale", [0.6, 1.0, 1.9])
def test_nonunitary_gates_on_a_state(n, scale):
    import quantumflow_gb300 as qf
    rng = np.random.default_rng(n)
    ket = qf.random_state(n)
    psi = ket.asarray().reshape((2,) * n).copy()
    elems, ops = [], []
    for q in range(0, n, 2):
        for m, qs in ((_haar(rng, 4), (q, (q + 1) % n)), (np.diag([scale, 0.75]).astype(complex), (q,)),
                      (np.array([[0.9, 0.2j], [0.1, 0.95]]), ((q + 1) % n,))):
            elems.append(qf.Gate(m, qubits=list(qs)))
            ops.append((m, qs))
    for m, qs in ops:
        k = len(qs)
        psi = np.moveaxis(np.tensordot(m.reshape((2,) * 2 * k), psi, (list(range(k, 2 * k)), list(qs))), range(k), qs)
    got = qf.Circuit(elems).run(ket).asarray().reshape(psi.shape)
    assert np.max(np.abs(got - psi)) < TOL * max(1.0, np.max(np.abs(psi)))
