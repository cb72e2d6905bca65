"""Window bits of the complex128 phase passes, read through qf_plan_circuit
(CPU): every pass has two at least while there are bits that no two-qubit
diagonal touches."""
import numpy as np
import pytest

N = 16


def _plan(circ, n=N):
    """(kernel kind, window bits from bit 5 up) of every planned pass."""
    from quantumflow_gb300 import _native as nat
    op_k, op_axes, op_mats, nops = circ.packed(tuple(range(n)))
    stats = (nat.ctypes.c_int32 * (8 * 64))()
    nb = nat.ctypes.c_int(0)
    nat.call("qf_plan_circuit", n, nat.LAYOUT_FX, nops, op_k.ctypes.data_as(nat._ip),
             op_axes.ctypes.data_as(nat._ip), op_mats.ctypes.data_as(nat._dp), 0, stats, 64, nat.ctypes.byref(nb))
    return [(stats[8 * b + 7], stats[8 * b + 6]) for b in range(nb.value)]


@pytest.mark.parametrize("make", ["RZ", "T", "Z", "CZ", "CPHASE", "ZZ", "layer"])
def test_lone_diagonals_get_a_window(make):
    import quantumflow_gb300 as qf
    gates = {"RZ": [qf.RZ(0.3, 4)], "T": [qf.T(2)], "Z": [qf.Z(0)], "CZ": [qf.CZ(1, 7)],
             "CPHASE": [qf.CPHASE(0.2, 0, 3)], "ZZ": [qf.ZZ(0.2, 1, 2)],
             "layer": [qf.RZ(0.1 * q + 0.1, q) for q in range(N)]}[make]
    assert _plan(qf.Circuit(gates)) == [(0, 2)]


def test_shared_bits_stay_outside():
    """Every bit is in a two-qubit diagonal with bit 0: one window bit."""
    import quantumflow_gb300 as qf
    star = qf.Circuit([qf.CPHASE(0.1 * q, 0, q) for q in range(1, N)])
    assert _plan(star) == [(0, 1)]
