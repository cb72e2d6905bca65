"""Host-side paths that carry many small gates: the superoperator of a channel
and the circuit's gate packing (CPU), and noisy circuits whose channels run
inside one launch (GPU) against the elements applied one by one."""
import numpy as np
import pytest


def test_superoperator_equals_the_composition():
    import quantumflow_gb300 as qf
    from quantumflow_gb300.channels import gate_aschannel, narrow_superop
    rng = np.random.default_rng(3)
    k2 = [qf.random_gate([4, 1], random_state=rng) for _ in range(3)]
    for kraus in (qf.Depolarizing(0.07, 2), qf.Damping(0.3, 0), qf.Dephasing(0.2, 5),
                  qf.Kraus([qf.P0(3), qf.P1(3)]), qf.UnitaryMixture(k2, [0.2, 0.5, 0.3])):
        want = sum(gate_aschannel(op).permute(kraus.qubits).tensor * w
                   for op, w in zip(kraus.operators, kraus.weights))
        got = kraus.aschannel()
        assert got.qubits == kraus.qubits
        # the same products, summed in the same order
        assert np.max(np.abs(got.tensor - want)) <= 4 * 2.0 ** -53
        d = 4 ** len(kraus.qubits)
        assert np.array_equal(narrow_superop(kraus), got.tensor.reshape(d, d))
    assert narrow_superop(qf.X(0)) is None
    assert narrow_superop(qf.join_channels(*(qf.Damping(0.1, q).aschannel() for q in range(3)))) is None

    class Own(qf.Damping):
        def evolve(self, rho):
            return rho

    assert narrow_superop(Own(0.1, 0)) is None


def test_replaced_gates_are_packed_again():
    import quantumflow_gb300 as qf
    circ = qf.Circuit([qf.X(0), qf.H(1)])
    first = circ.packed((0, 1))
    assert circ.packed((0, 1)) is first
    for _ in range(50):  # a new gate may take a freed one's address
        circ.elements[0] = qf.RX(0.3, 0)
        circ.elements[0] = qf.RX(0.7, 0)
        mats = circ.packed((0, 1))[2]
        assert np.array_equal(mats[:8], qf.RX(0.7, 0).matrix_doubles())
    assert circ.packed((1, 0))[1].tolist() == [1, 0]
    circ.extend(qf.Z(0))
    assert circ.packed((0, 1))[3] == 3


@pytest.mark.gpu
@pytest.mark.parametrize("n,dtype", [(2, "complex128"), (5, "complex128"), (6, "complex128"), (7, "complex128"),
                                     (4, "complex64"), (7, "complex64")])
def test_noisy_circuits_in_one_launch(n, dtype):
    import quantumflow_gb300 as qf
    rng = np.random.default_rng(n)
    elems = []
    for _ in range(3):
        for q in range(n):
            elems.append(qf.random_gate([q], random_state=rng))
        perm = rng.permutation(n)
        for a in range(0, n - 1, 2):
            elems.append(qf.CZ(int(perm[a]), int(perm[a + 1])))
        for q in range(n):
            elems.append([qf.Depolarizing, qf.Damping, qf.Dephasing][int(rng.integers(3))](0.05, q))
        elems.append(qf.Kraus([qf.P0(0), qf.P1(0)]))
        if n > 2:
            elems.append(qf.join_channels(qf.Damping(0.2, 1).aschannel(), qf.Depolarizing(0.1, 2).aschannel()))
            elems.append(qf.join_channels(*(qf.Damping(0.1, q).aschannel() for q in (0, 1, 2))))
        elems.append(qf.Gate(rng.normal(size=(2, 2)), qubits=[n - 1]))  # not unitary
    rho = qf.random_density(n, dtype=dtype)
    before = rho.asarray().copy()
    got = qf.Circuit(elems).evolve(rho).asarray()
    assert np.array_equal(rho.asarray(), before)
    want = qf.Density(before.astype(np.complex128), range(n))
    for e in elems:
        want = e.evolve(want)
    want = want.asarray()
    # about 20 n passes, each within a few units of the largest entry
    tol = 40 * n * (2.0 ** -53 if dtype == "complex128" else 2.0 ** -24)
    assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))
