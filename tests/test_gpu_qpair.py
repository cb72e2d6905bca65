"""Complex64 QAOA two register groups a pass: the same FP32 operations in the
same order as the warp-tile kernels, so states are equal bit for bit and
gradients to the rounding of their FP64 sums; every remainder of the groups,
odd and even numbers of them, one to three layers."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pair(n, p, kind):
    import quantumflow_gb300 as qf
    seed = 31 * n + p

    def graph():
        if kind == "regular" and n % 2 == 0:
            return qf.qaoa.random_regular_graph(3, n, seed=seed)
        return qf.qaoa.gnp_random_graph(n, 0.5, seed=seed)

    g = graph()
    g.add_node(0, weight=0.0)  # a node phase of exactly 1 keeps the warp-tile kernels
    return qf.QAOAMaxCut(graph(), p, dtype="complex64"), qf.QAOAMaxCut(g, p, dtype="complex64")


@pytest.mark.parametrize("n", [13, 14, 15, 16, 17, 18, 19, 20, 21, 22, 24])
@pytest.mark.parametrize("p,kind", [(1, "gnp"), (2, "regular"), (3, "gnp")])
def test_same_as_warp_tiles(n, p, kind):
    import quantumflow_gb300 as qf
    new, old = _pair(n, p, kind)
    rng = np.random.default_rng(n)
    beta, gamma = rng.uniform(-3, 3, p), rng.uniform(-1.5, 1.5, p)
    a, b = new.state(beta, gamma).tensor, old.state(beta, gamma).tensor
    assert torch.equal(a, b)
    del a, b
    ga, gb = new.expectation_and_grad(beta, gamma), old.expectation_and_grad(beta, gamma)
    # psi, taken back to |+>^n by the adjoint sweep
    assert torch.equal(qf.State(new._grad_bufs[1]).tensor, qf.State(old._grad_bufs[1]).tensor)
    # the same FP32 partial sums, added up in another order: 48-bit
    # accumulators, then FP64; each term is at most 2 E |psi| |X psi|
    edges = len(new.edges)
    assert abs(ga[0] - gb[0]) <= 2.0 ** -44 * edges
    assert np.max(np.abs(ga[1] - gb[1])) <= 2.0 ** -42 * edges * n
    assert np.max(np.abs(ga[2] - gb[2])) <= 2.0 ** -42 * edges * edges


@pytest.mark.parametrize("dtype,sizes", [("complex64", (9, 12, 13, 13, 14, 16, 17, 18, 19, 20)),
                                         ("complex128", (7, 10, 11, 12, 13, 15, 18, 19))])
@pytest.mark.parametrize("tile_bits", [8, None])
def test_batches(dtype, sizes, tile_bits):
    """Instances on either side of a two-group tile in one batch, against the
    single-instance sweep: the same FP32 (or 48-bit) operations in complex64;
    <C> sums its FP32 terms per thread there."""
    import quantumflow_gb300 as qf
    rng = np.random.default_rng(7)
    graphs = [qf.qaoa.gnp_random_graph(n, 0.5, seed=5 * n + i) for i, n in enumerate(sizes)]
    ps = [1 + i % 3 for i in range(len(sizes))]
    betas = [rng.uniform(-2, 2, p) for p in ps]
    gammas = [rng.uniform(-1, 1, p) for p in ps]
    batch = qf.batched.QAOABatch(graphs, ps, dtype=dtype, tile_bits=tile_bits)
    batch.set_angles(betas, gammas)
    first = batch.evaluate()
    again = batch.evaluate()
    for i, n in enumerate(sizes):
        e, db, dg = qf.QAOAMaxCut(graphs[i], ps[i], dtype=dtype).expectation_and_grad(betas[i], gammas[i])
        edges = len(graphs[i].edges())
        u = 2.0 ** -20 if dtype == "complex64" else 2.0 ** -41
        assert abs(first[0][i] - e) <= u * edges
        grad = u * ps[i] * edges * max(n, edges)
        assert np.max(np.abs(first[1][i] - db)) <= grad and np.max(np.abs(first[2][i] - dg)) <= grad
        for a, b in zip(first, again):
            assert np.array_equal(a[i], b[i])
    # a skipped instance keeps its outputs
    if batch.nwave:
        batch._wave_skip[0] = 1
        batch._skip_on = True
        which = int(batch._wave_idx[0])
        batch.set_angles([b + 0.3 for b in betas], gammas)
        batch.launch()
        batch._skip_on = False
        out = batch.expectations().cpu().numpy()
        assert out[which] == first[0][which]
        assert sum(out[i] != first[0][i] for i in range(len(sizes))) == len(sizes) - 1
