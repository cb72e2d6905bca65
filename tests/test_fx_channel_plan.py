"""Host-side routing of gates that are not unitary (noise channels and the
like) into tensor-core passes, read through qf_plan_circuit on the CPU: which
entries the 2^62 integers of a pass can hold."""
import numpy as np
import pytest

N = 12


def _plan(ops, n=N):
    """(kernel kind, number of ops) of every planned pass."""
    from quantumflow_gb300 import _native as nat
    k = np.array([len(q) for _, q in ops], np.int32)
    axes = np.array([a for _, q in ops for a in q], np.int32)
    mats = np.concatenate([np.ascontiguousarray(m, complex).view(float).reshape(-1) for m, _ in ops])
    stats = (nat.ctypes.c_int32 * (8 * 4096))()
    nb = nat.ctypes.c_int(0)
    nat.call("qf_plan_circuit", n, nat.LAYOUT_FX, len(k), k.ctypes.data_as(nat._ip), axes.ctypes.data_as(nat._ip),
             mats.ctypes.data_as(nat._dp), 0, stats, 4096, nat.ctypes.byref(nb))
    return [(stats[8 * b + 7], stats[8 * b]) for b in range(nb.value)]


def _haar(rng, d):
    q, r = np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


@pytest.mark.parametrize("value", [2.0, -2.0, 2.0j, -2.0j])
def test_entries_of_two_stay_in_fp64(value):
    """2 * 2^62 does not fit 64 bits: such gates run in native FP64 (kind 5),
    the next smaller ones inside the gate's pass (kind 6)."""
    gate = (_haar(np.random.default_rng(1), 4), (0, 1))
    below = value * (1 - 2.0 ** -52)
    for make in (lambda v: (np.diag([v, 1.0]), (0,)), lambda v: (np.diag([1.0, 1.0, v, 1.0]), (0, 1))):
        assert [kind for kind, _ in _plan([gate, make(value)])].count(5) == 1
        assert [kind for kind, _ in _plan([gate, make(below)])] == [6]


def _window_gates(count, scale):
    rng = np.random.default_rng(5)
    return [(_haar(rng, 4) * scale, ([0, 1], [1, 2], [2, 3])[i % 3]) for i in range(count)]


@pytest.mark.parametrize("extra", [0, 300])
def test_long_runs_on_one_window_are_cut(extra):
    """A gate may be off unitarity by 1e-9, and the integers of a pass leave
    1 + 2^-20 for its norm: a pass takes at most 256 gates, the diagonals that
    wait for it included, whatever the length of the run."""
    diags = [(np.diag(np.exp(1j * np.arange(4) * (i + 1))), (i % 4, (i + 1) % 4)) for i in range(extra)]
    plan = _plan(diags + _window_gates(3000, 1 + 4e-10))
    assert max(ops for kind, ops in plan if kind == 6) <= 256
    assert sum(ops for kind, ops in plan if kind == 6) >= 2500


@pytest.mark.gpu
def test_long_runs_off_unitarity():
    """3000 gates, each 4e-10 above unit norm, and the result grown by all of
    them: once refused by the pass after earlier ones had run."""
    import quantumflow_gb300 as qf
    n, growth = 11, 4e-10
    ops = _window_gates(3000, 1 + growth)
    got = qf.Circuit([qf.Gate(m, qubits=list(q)) for m, q in ops]).run(qf.zero_state(n)).asarray().reshape(-1)
    psi = np.zeros((2,) * 4, np.clongdouble)
    psi[0, 0, 0, 0] = 1
    for m, q in ops:
        t = np.moveaxis(psi, q, (0, 1)).reshape(4, 4)
        t = (m.astype(np.clongdouble)[:, :, None] * t[None]).sum(axis=1)
        psi = np.moveaxis(t.reshape((2,) * 4), (0, 1), q)
    want = np.zeros(2 ** n, complex)
    want[:: 2 ** (n - 4)] = psi.reshape(-1)
    assert abs(np.linalg.norm(want) - (1 + growth) ** 3000) < 1e-9
    # a pass errs by 2^-55 of its row's largest part and one rounding, at most
    # 3000 / 32 of them
    assert np.max(np.abs(got - want)) < 94 * 2.0 ** -52


def test_waiting_diagonals_are_bounded():
    """Diagonals that no later gate touches do not pile up while a long circuit
    is planned: a phase pass of them every few hundred."""
    rng = np.random.default_rng(4)
    ops = []
    for _ in range(6000):
        a, b = (int(x) for x in rng.choice(6, 2, replace=False))
        ops.append((np.diag(np.exp(1j * rng.uniform(0, 6, 4))), (a, b)) if rng.random() < 0.5
                   else (_haar(rng, 4), (6 + a, 6 + b)))
    plan = _plan(ops)
    waiting = [count for kind, count in plan if kind == 0]
    assert max(waiting) <= 256 + 128 and len(waiting) >= 4
    assert sum(count for kind, count in plan if kind in (0, 6)) > 4000
