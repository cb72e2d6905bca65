"""Complex128 phase passes and qubit-exchange passes against the oracle:
every window width, window bits low and high, diagonals inside, across and
outside the windows, signs, and table sizes around each eight bits of the
compact index (n = 11 .. 21)."""
import numpy as np
import pytest
import torch

from oracle import qf_oracle as orc

pytestmark = pytest.mark.gpu

# a pass errs by 2^-55 of a row's largest part plus one rounding; 400 gates
# of unit norm stay far below
TOL = 400 * 2.0 ** -53


def _ket(n, seed):
    import quantumflow_gb300 as qf
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.randn(2 ** n, 2, dtype=torch.float64, device="cuda", generator=gen)
    return qf.State(torch.view_as_complex(t / t.norm()))


def _check(circ, n, seed, fusion_k=None):
    ket = _ket(n, seed)
    before = ket.asarray().copy()
    got = circ.run(ket, fusion_k).asarray().reshape(-1)
    ops = [(g.asoperator(), tuple(g.qubits)) for g in circ]
    ref = orc.run_ops(before, ops).reshape(-1)
    assert np.array_equal(ket.asarray(), before)  # out of place
    assert np.max(np.abs(got - ref)) < TOL


def _unit(rng, size):
    return np.exp(2j * np.pi * rng.random(size))


def _diag(rng, qubits):
    import quantumflow_gb300 as qf
    return qf.Gate(np.diag(_unit(rng, 2 ** len(qubits))), qubits=qubits)


@pytest.mark.parametrize("n", [11, 12, 13, 16, 20])
@pytest.mark.parametrize("kind", ["one", "star", "pairs", "signs"])
def test_runs_of_diagonal_gates(n, kind):
    import quantumflow_gb300 as qf
    rng = np.random.default_rng(n)
    circ = qf.Circuit()
    if kind == "one":  # no window at all, then one bit
        for q in range(n):
            circ += _diag(rng, [q])
        _check(circ, n, 1)
        circ += qf.ZZ(0.37, 0, n - 1)
    elif kind == "star":  # every pair shares qubit 3, or the lowest bits
        for q in range(n):
            if q != 3:
                circ += qf.CPHASE(0.1 * q + 0.2, q, 3)
        for q in range(n - 1):
            circ += _diag(rng, [n - 1, q])
    elif kind == "pairs":  # a window of four does not cover them
        for a in range(n):
            for b in range(a + 1, n):
                if rng.random() < 0.4:
                    circ += _diag(rng, [a, b] if rng.random() < 0.5 else [b, a])
    else:
        for _ in range(60):  # more signs than one pass takes, and phases between
            a, b = (int(x) for x in rng.choice(n, 2, replace=False))
            circ += qf.CZ(a, b)
        circ += qf.RZ(0.3, 2)
        circ += _diag(rng, [0, 5])
    _check(circ, n, 2)


@pytest.mark.parametrize("n", [11, 14, 17, 19, 21])
@pytest.mark.parametrize("fusion_k", [None, 1, 2, 3])
def test_diagonals_between_dense_gates(n, fusion_k):
    import quantumflow_gb300 as qf
    rng = np.random.default_rng(10 * n)
    circ = qf.Circuit()
    for _ in range(100):
        r = rng.random()
        a, b = (int(x) for x in rng.choice(n, 2, replace=False))
        if r < 0.3:
            circ += qf.random_gate([a], random_state=rng)
        elif r < 0.4:
            circ += qf.random_gate([a, b], random_state=rng)
        elif r < 0.75:
            circ += _diag(rng, [a, b])
        elif r < 0.85:
            circ += _diag(rng, [a])
        elif r < 0.95:
            circ += qf.CZ(a, b)
        else:
            circ += qf.SWAP(a, b)
    circ += qf.CCNOT(0, 5, 9)
    circ += _diag(rng, [1, 4, n - 1])
    circ += qf.CPHASE(0.4, 1, n - 2)
    _check(circ, n, 3, fusion_k)


@pytest.mark.parametrize("n", [11, 12, 15, 18])
def test_runs_of_swaps(n):
    import quantumflow_gb300 as qf
    rng = np.random.default_rng(n)
    for pairs in (3, n // 2):  # partly fixed bits; the whole register
        perm = rng.permutation(n)
        _check(qf.Circuit([qf.SWAP(int(perm[2 * i]), int(perm[2 * i + 1])) for i in range(pairs)]), n, 4)
    # a qubit exchanged twice ends the run; in place from |0..0> too
    circ = qf.Circuit([qf.H(0), qf.T(1)] + [qf.SWAP(i, i + 1) for i in range(n - 1)] + [qf.RX(0.2, 3)])
    _check(circ, n, 5)
    circ = qf.Circuit([qf.RX(0.1 * q + 0.1, q) for q in range(n)]) + qf.reversal_circuit(range(n))
    got = circ.run(qf.zero_state(n)).asarray().reshape(-1)
    ops = [(g.asoperator(), tuple(g.qubits)) for g in circ]
    assert np.max(np.abs(got - orc.run_ops(orc.zero_state(n), ops).reshape(-1))) < TOL


@pytest.mark.parametrize("n", [11, 12, 16, 21])
def test_fourier_transform(n):
    import quantumflow_gb300 as qf
    ket = _ket(n, 6)
    got = qf.qft_circuit(range(n)).run(ket).tensor.reshape(-1)
    ref = np.fft.ifft(ket.asarray().reshape(-1), norm="ortho")
    assert np.max(np.abs(got.cpu().numpy() - ref)) < TOL
    back = qf.qft_circuit(range(n)).H.run(qf.State(got)).asarray().reshape(-1)
    assert np.max(np.abs(back - ket.asarray().reshape(-1))) < TOL
