"""Read-out kernels at the edges of their launch shapes: FP64 reductions of
complex128 states (unrolled loop and remainder), and sampling (scan blocks of
1024 amplitudes, 32 blocks per warp, chunks of 1024 block totals)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _ket(n, dtype, seed):
    import quantumflow_gb300 as qf
    gen = torch.Generator(device="cuda").manual_seed(seed)
    real = torch.float32 if dtype == "complex64" else torch.float64
    t = torch.randn(2 ** n, 2, dtype=real, device="cuda", generator=gen)
    return qf.State(torch.view_as_complex(t / t.norm()))


@pytest.mark.parametrize("n", [1, 2, 9, 10, 17, 19, 21])
def test_fp64_reductions(n):
    import quantumflow_gb300 as qf
    from quantumflow_gb300.states import _reduce
    from quantumflow_gb300 import _native as nat
    a, b = _ket(n, "complex128", n), _ket(n, "complex128", n + 100)
    va, vb = a.asarray().reshape(-1), b.asarray().reshape(-1)
    p = np.abs(va.astype(np.clongdouble)) ** 2
    diag = torch.randn(2 ** n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    cuts = torch.randint(0, 60000, (2 ** n,), device="cuda").to(torch.uint16)
    # a sum in any order errs by at most (depth + 3) u of the sum of
    # magnitudes; depth: up to 2^n / 2^18 terms per thread, then 8 + 11 levels
    depth = max(1, 2 ** n // 2 ** 18) * 4 + 40
    for got, terms in ((a.norm(), p), (a.expectation(diag), p * diag.cpu().numpy()),
                       (_reduce("qf_expectation_cuts", a.buffer, 1, extra=(nat.ptr(cuts),))[0],
                        p * cuts.cpu().numpy().astype(np.float64))):
        assert abs(got - float(terms.sum())) <= depth * U * float(np.abs(terms).sum())
    bit = _reduce("qf_qubit_probabilities", a.buffer, 2, extra=(0,))
    half = p.reshape(2, -1).sum(axis=1)
    assert np.all(np.abs(np.array(bit) - half.astype(np.float64)) <= depth * U * float(p.sum()))
    ip = qf.inner(a, b)
    ref = (va.conj().astype(np.clongdouble) * vb).sum()
    mag = float((np.abs(va) * np.abs(vb)).sum())
    assert abs(ip - complex(ref)) <= 2 * depth * U * mag


def _mix64(z):
    z = (z + np.uint64(0x9E3779B97F4A7C15))
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


@pytest.mark.parametrize("n,dtype", [(1, "complex128"), (3, "complex64"), (10, "complex128"), (11, "complex128"),
                                     (15, "complex64"), (16, "complex128"), (20, "complex128"), (21, "complex64"),
                                     (22, "complex128")])
def test_draws_follow_the_distribution(n, dtype):
    ket = _ket(n, dtype, 7 * n)
    trials = 3000
    draws = ket._draws(trials, seed=99)
    with np.errstate(over="ignore"):
        r = _mix64(np.uint64(99) ^ _mix64(np.arange(trials, dtype=np.uint64)))
    cdf = np.cumsum(ket.probabilities().cpu().numpy().reshape(-1).astype(np.longdouble))
    u = (r >> np.uint64(11)).astype(np.longdouble) * np.longdouble(2.0 ** -53) * cdf[-1]
    # the device sums 1024 amplitudes in order from an offset that is itself a
    # scan: at most 1024 + 4 + 8 + 10 + chunks additions deep
    eps = (1024 + 30 + 2 ** max(0, n - 20)) * U * float(cdf[-1])
    assert np.all(draws >= 0) and np.all(draws < 2 ** n)
    assert np.all(cdf[draws] + eps > u)
    assert np.all(np.where(draws > 0, cdf[np.maximum(draws, 1) - 1], 0) <= u + eps)


@pytest.mark.parametrize("n", [1, 4, 12, 16, 21])
def test_counts_are_the_histogram_of_the_draws(n):
    import quantumflow_gb300 as qf
    from quantumflow_gb300 import _native as nat
    ket = _ket(n, "complex128", n)
    for trials in (0, 1, 5000):
        counts = torch.full((2 ** n,), -1, dtype=torch.int64, device="cuda")
        nbytes = nat.lib.qf_sample_workspace_bytes(n)
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        nat.call("qf_sample", nat.ptr(ket.buffer.data), n, ket.buffer.layout, trials, 42, nat.ptr(counts), nat.ptr(ws),
                 nbytes, nat.stream_handle())
        hist = np.bincount(ket._draws(trials, seed=42), minlength=2 ** n)
        assert np.array_equal(counts.cpu().numpy(), hist)
        assert np.array_equal(ket.sample(trials, seed=42).reshape(-1), hist)
    with pytest.raises(nat.NativeError):
        ket.sample(-1)
    assert qf.zero_state(n).measure(seed=3).tolist() == [0] * n
