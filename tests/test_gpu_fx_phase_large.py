"""Phase passes on states of 2^19 to 2^24 amplitudes, on both sides of the
size from which three CTAs share an SM, for every window width, against
element-wise products in complex128."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("side", [-1, 0, 1])
def test_phase_passes_by_size(width, side):
    import quantumflow_gb300 as qf
    n = 19 + width + side
    rng = np.random.default_rng(10 * width + side + 1)
    gen = torch.Generator(device="cuda").manual_seed(width)
    t = torch.randn(2 ** n, 2, dtype=torch.float64, device="cuda", generator=gen)
    psi = torch.view_as_complex(t / t.norm())
    hubs = [int(q) for q in rng.permutation(n)[:width]]
    circ, ref = qf.Circuit([]), psi.clone()
    for a in hubs or [None]:
        for b in [int(q) for q in rng.permutation(n)[:8]]:
            angle = float(rng.uniform(0.1, 3.0))
            if b in hubs:
                continue
            # exp(i angle) where the qubits are 1
            f = complex(np.exp(1j * angle))
            axes = sorted([b] if a is None else [a, b])
            circ += qf.PHASE(angle, b) if a is None else qf.CPHASE(angle, a, b)
            shape, last = [], -1
            for x in axes:
                shape += [2 ** (x - last - 1), 2]
                last = x
            ref.reshape(shape + [-1])[tuple(v for _ in axes for v in (slice(None), 1))] *= f
    got = circ.run(qf.State(psi)).buffer.complex()
    ngates = len(list(circ))
    # a gate of the reference rounds twice and its factor once; the pass errs by
    # 2^-55 of an amplitude and one rounding
    tol = (4 * ngates + 4) * 2.0 ** -53 * float(psi.abs().max())
    assert float((got.reshape(-1) - ref).abs().max()) < tol
