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
