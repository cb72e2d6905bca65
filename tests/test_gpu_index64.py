"""States of 2^32 amplitudes, where indices no longer fit 32 bits: the phase
passes, the sparse 4x4 sweep and the qubit exchange, against the exact values at
sampled indices (128 GiB of device memory)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N = 32


def _cases(bit):
    import quantumflow_gb300 as qf
    one = np.ones((), np.clongdouble)
    ops, want = [], one
    for a, b, t in ((0, N - 1, 0.3), (0, 5, 0.7), (1, 29, 0.2), (30, 2, 0.9), (4, 9, 0.4)):
        ops.append(qf.CPHASE(t, a, b))
        want = want * np.exp(1j * np.longdouble(t) * (bit(a) & bit(b)))
    for q in range(N):
        ops.append(qf.PHASE(0.01 * q, q))
        want = want * np.exp(1j * np.longdouble(0.01 * q) * bit(q))
    for a, b in ((0, 1), (N - 1, 3)):
        ops.append(qf.CZ(a, b))
        want = want * (1 - 2 * (bit(a) & bit(b)))
    yield ops, want
    yield [qf.CZ(0, N - 1), qf.Z(2)], one * (1 - 2 * (bit(0) & bit(N - 1))) * (1 - 2 * bit(2))
    m = np.zeros((4, 4))  # real, at most two entries a row: row sums 1, 2, -1, 0.5
    m[0, 0], m[0, 3], m[1, 2], m[2, 1], m[3, 3] = 0.9, 0.1, 2, -1, 0.5
    yield [qf.Gate(m, qubits=[N - 2, 1])], one * np.array([1.0, 2, -1, 0.5])[2 * bit(N - 2) + bit(1)]
    yield ([qf.PHASE(0.3, 0), qf.SWAP(0, N - 1), qf.SWAP(1, N - 2), qf.SWAP(3, 17)],
           one * np.exp(1j * np.longdouble(0.3) * bit(N - 1)))


def test_index_forms_beyond_32_bits():
    import quantumflow_gb300 as qf
    if torch.cuda.mem_get_info()[0] < 140 << 30:
        pytest.skip("not enough device memory")
    rng = np.random.default_rng(0)
    idx = np.unique(np.concatenate([rng.integers(0, 2 ** N, 100000), [0, 2 ** N - 1, 2 ** 31, 2 ** 31 - 1]]))
    at = torch.from_numpy(idx.astype(np.int64)).cuda()
    bit = lambda q: (idx >> (N - 1 - q)) & 1
    for ops, want in _cases(bit):
        got = qf.Circuit(ops).run(qf.uniform_state(N)).tensor.reshape(-1)[at].cpu().numpy()
        torch.cuda.empty_cache()
        # three passes at most, each 2^-55 of an amplitude and one rounding; a
        # factor of the reference is rounded once
        assert np.max(np.abs(got * 2.0 ** (N // 2) - want)) <= 12 * 2.0 ** -53
