"""QAOA on wide tiles against the warp-tile kernels and the oracle: every tile
width, one, two and three groups of qubits, ragged last groups, both forms of
the rotation, one to three layers, the smallest workspace."""
import numpy as np
import pytest
import torch

from oracle import qf_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture
def modes():
    from quantumflow_gb300 import _native as nat
    yield lambda m: nat.call("qf_set_tile_kernel", m)
    nat.call("qf_set_tile_kernel", 0)


def _angles(p, seed, wide):
    rng = np.random.default_rng(seed)
    # |tan(beta / 2)| on both sides of 1, zero and large angles
    beta = rng.uniform(-4, 4, p) if wide else rng.uniform(0.1, 0.7, p)
    return beta, rng.uniform(-1.5, 1.5, p)


def _tols(n, p, dtype):
    """Forward and backward: 2 n + 4 roundings an amplitude and layer, each of
    2^-47 (float-float) or 2^-23 relative; unit norm states."""
    u = 2.0 ** -47 if dtype == "complex128" else 2.0 ** -23
    return u * (2 * n + 4) * p


SIZES = [("complex128", n) for n in (8, 9, 10, 12, 15, 16, 18, 19, 22, 23, 24)] + [("complex64", n) for n in (9, 17)]


@pytest.mark.parametrize("dtype,n", SIZES)
@pytest.mark.parametrize("p,wide", [(1, True), (2, False), (3, True)])
def test_against_warp_tiles(modes, dtype, n, p, wide):
    import quantumflow_gb300 as qf
    g = qf.qaoa.gnp_random_graph(n, 0.5, seed=n)
    prob = qf.QAOAMaxCut(g, p, dtype=dtype)
    beta, gamma = _angles(p, 100 * n + p, wide)
    e, db, dg = prob.expectation_and_grad(beta, gamma)
    # psi is left at |+>^n
    psi = qf.State(prob._grad_bufs[1]).tensor.reshape(-1)
    tol = _tols(n, p, dtype)
    amp = 2.0 ** (-n / 2)
    assert float((psi - amp).abs().square().sum().sqrt()) <= 2 * tol
    del psi
    st = prob.state(beta, gamma).tensor.reshape(-1)
    modes(3)
    e0, db0, dg0 = prob.expectation_and_grad(beta, gamma)
    st0 = prob.state(beta, gamma).tensor.reshape(-1)
    assert float((st - st0).abs().square().sum().sqrt()) <= 2 * tol
    edges = len(g.edges())
    # |<lambda| H |psi>| <= |lambda| |H| with |lambda| <= E, |H| <= n or E
    assert abs(e - e0) <= 4 * tol * edges
    assert np.max(np.abs(db - db0)) <= 4 * tol * edges * n
    assert np.max(np.abs(dg - dg0)) <= 4 * tol * edges * edges


@pytest.mark.parametrize("dtype,n", [("complex128", 8), ("complex128", 11), ("complex64", 10)])
def test_against_oracle(dtype, n):
    import quantumflow_gb300 as qf
    g = qf.qaoa.gnp_random_graph(n, 0.5, seed=3 * n)
    p = 2
    beta, gamma = _angles(p, n, True)
    prob = qf.QAOAMaxCut(g, p, dtype=dtype)
    st = prob.state(beta, gamma).asarray().reshape(-1)
    ref = orc.run_ops(orc.zero_state(n), orc.qubo_ops(n, g.edges(), p, beta, gamma)).reshape(-1)
    assert np.linalg.norm(st - ref) <= 2 * _tols(n, p, dtype) + 1e-14
    e, db, dg = prob.expectation_and_grad(beta, gamma)
    cuts = orc.graph_cuts(n, g.edges())

    def energy(b, c):
        s = orc.run_ops(orc.zero_state(n), orc.qubo_ops(n, g.edges(), p, b, c)).reshape(-1)
        return orc.expectation(s, cuts)

    h = 1e-5  # central differences: h^2 / 6 of a third derivative below (2 E)^3, and rounding / h
    edges = len(g.edges())
    tol = h * h / 6 * (2 * edges) ** 2 * edges + 1e-13 * edges / h + 4 * _tols(n, p, dtype) * edges * edges
    for l in range(p):
        d = np.eye(p)[l] * h
        assert abs(db[l] - (energy(beta + d, gamma) - energy(beta - d, gamma)) / (2 * h)) <= tol
        assert abs(dg[l] - (energy(beta, gamma + d) - energy(beta, gamma - d)) / (2 * h)) <= tol


@pytest.mark.parametrize("dtype,n", [("complex128", 12), ("complex64", 16)])
def test_smaller_workspace_and_node_weights(modes, dtype, n):
    """A workspace sized for the warp-tile sweep is still accepted; graphs
    with node weights keep that sweep."""
    import quantumflow_gb300 as qf
    from quantumflow_gb300 import _native as nat
    from quantumflow_gb300.qaoa import compute_layout
    p, layout = 2, compute_layout(dtype)
    g = qf.qaoa.gnp_random_graph(n, 0.5, seed=n)
    prob = qf.QAOAMaxCut(g, p, dtype=dtype)
    beta, gamma = _angles(p, 5, True)
    want = prob.expectation_and_grad(beta, gamma)
    amps = 2 ** n * (8 if dtype == "complex64" else 16)
    full = nat.lib.qf_qaoa_grad_workspace_bytes(n, p, layout)
    rows_min = 4 if dtype == "complex128" else 32
    small = amps + rows_min * (2 * p + 1) * 8 + 512
    assert small <= full
    for nbytes in (small, full):
        psi = torch.empty(amps, dtype=torch.uint8, device="cuda")
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        out = torch.empty(2 * p + 1, dtype=torch.float64, device="cuda")
        nat.call("qf_qaoa_expectation_grad", nat.ptr(psi), n, layout, nat.ptr(prob.cuts16), len(prob.edges), p,
                 nat.double_array(beta), nat.double_array(gamma), None, 0, nat.ptr(out), nat.ptr(ws), nbytes,
                 nat.stream_handle())
        o = out.cpu().numpy()
        tol = 8 * _tols(n, p, dtype) * len(prob.edges) ** 2
        assert abs(o[2 * p] - want[0]) <= tol and np.max(np.abs(o[p:2 * p] - want[1])) <= tol
    g.add_node(2, weight=0.4)
    weighted = qf.QAOAMaxCut(g, p, dtype=dtype)
    a = weighted.expectation_and_grad(beta, gamma)
    modes(3)
    b = weighted.expectation_and_grad(beta, gamma)
    assert abs(a[0] - b[0]) <= 4 * _tols(n, p, dtype) * len(prob.edges)
