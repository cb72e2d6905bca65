"""Circuit.run's choice of route after the public packing of the same gates
(CPU: the launches are recorded, not made)."""
import numpy as np


class _Ket:
    """A stand-in for a state: counts how the circuit runs."""

    def __init__(self, n):
        self.qubits = tuple(range(n))


def _routes(circ, n, monkeypatch):
    from quantumflow_gb300 import _native as nat
    from quantumflow_gb300.ops import Gate
    seen = []
    monkeypatch.setattr(Gate, "run", lambda gate, ket: seen.append(("alone", gate.qubit_nb)) or ket)

    class Launched(Exception):
        pass

    def launch(name, *args):
        seen.append((name, args[4] if len(args) > 4 else None))
        raise Launched

    ket = _Ket(n)

    class Buf:
        data, n, layout, device = None, len(ket.qubits), 0, None

        def compute(self):
            return self

        def empty_like(self):
            return self

    ket.buffer, ket._memory = Buf(), {}
    monkeypatch.setattr(nat, "call", launch)
    monkeypatch.setattr(nat, "ptr", lambda t: None)
    monkeypatch.setattr(nat, "stream_handle", lambda d=None: None)
    monkeypatch.setattr("quantumflow_gb300.circuits.gate_layout", lambda b: 0)
    try:
        circ.run(ket, 0)
    except Launched:
        pass
    return seen


def test_wide_gate_after_the_public_packing(monkeypatch):
    import quantumflow_gb300 as qf
    n = 6
    circ = qf.Circuit([qf.X(0)])
    assert [name for name, _ in _routes(circ, n, monkeypatch)] == ["qf_run_circuit"]
    wide = qf.Gate(np.eye(2 ** 6), qubits=range(6))
    circ.elements[0] = wide
    assert circ.packed(tuple(range(n)))[0].tolist() == [6]
    # a gate above the fused launch's width runs on its own, packed or not
    assert _routes(circ, n, monkeypatch) == [("alone", 6)]
    circ.elements[0] = qf.X(1)
    circ.packed(tuple(range(n)))
    assert [name for name, _ in _routes(circ, n, monkeypatch)] == ["qf_run_circuit"]
