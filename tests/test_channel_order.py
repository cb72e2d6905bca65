"""Channels that join a circuit's launch: only those whose superoperator is laid
out as the launch takes it."""
import numpy as np
import pytest


def _reordered():
    import quantumflow_gb300 as qf

    class Reordered(qf.Kraus):
        """Kraus operators given on (3, 1); the channel keeps that order."""

        def aschannel(self):
            return self.operators[0].aschannel()

    u = qf.random_gate([3, 1], random_state=np.random.default_rng(2))
    return Reordered([u])


def test_a_channel_in_its_own_order_keeps_its_pass():
    import quantumflow_gb300 as qf
    from quantumflow_gb300.channels import narrow_superop
    chan = _reordered()
    assert chan.qubits == (1, 3) and chan.aschannel().qubits == (3, 1)
    assert narrow_superop(chan) is None
    damp = qf.Damping(0.1, 0)
    assert narrow_superop(damp) is not None
    damp.evolve = lambda rho: rho  # the object's own way
    assert narrow_superop(damp) is None


def test_a_channel_alone_runs_by_itself(monkeypatch):
    """Which launches a circuit of gates and channels makes (recorded, not
    made): one for every run of two or more, a lone channel through its own
    entry point."""
    import quantumflow_gb300 as qf
    from quantumflow_gb300 import channels, densities
    seen = []

    class Rho:
        dtype = "complex128"

    monkeypatch.setattr(densities, "evolve_gates", lambda rho, ops: seen.append(len(ops)) or rho)
    monkeypatch.setattr(channels, "evolve_superop", lambda rho, *a: seen.append("alone") or rho)
    damp = lambda q: qf.Damping(0.1, q)
    wide = qf.join_channels(*(damp(q).aschannel() for q in range(3)))  # three qubits: always by itself
    for elems, want in (([damp(0)], ["alone"]), ([damp(0), damp(1)], [2]), ([qf.X(0), damp(0)], [2]),
                        ([damp(0), qf.X(0)], [2]), ([qf.X(0)], [1]),
                        ([damp(0), wide, damp(1)], ["alone"] * 3), ([qf.X(0), wide, damp(1), damp(2)], [1, "alone", 2]),
                        ([], [])):
        seen.clear()
        qf.Circuit(elems).evolve(Rho())
        assert seen == want


@pytest.mark.gpu
def test_evolution_with_a_channel_in_its_own_order():
    import quantumflow_gb300 as qf
    n = 4
    rho = qf.random_density(n)
    chan = _reordered()
    u = chan.operators[0]
    got = qf.Circuit([qf.H(0), chan, qf.X(2)]).evolve(rho).asarray()
    want = qf.X(2).evolve(u.evolve(qf.H(0).evolve(rho))).asarray()
    # five passes at most, each within a few units of the largest entry
    assert np.max(np.abs(got - want)) < 40 * 2.0 ** -53
