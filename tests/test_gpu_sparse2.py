"""Two-qubit complex128 gates with a real matrix of at most two nonzeros a row
(noise channels, projectors) and real diagonals in native FP64: equal, bit for
bit, to the same sums on the host; every pair of bit positions that matters,
zero rows, in place."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _matrix(kind, rng):
    m = np.zeros((4, 4))
    if kind == "channel":  # depolarizing form
        m[0, 0] = m[3, 3] = 0.93
        m[0, 3] = m[3, 0] = 0.07
        m[1, 1] = m[2, 2] = 0.86
    elif kind == "zero_rows":
        m[1, 2], m[1, 3] = rng.normal(size=2)
        m[3, 0] = rng.normal()
    else:
        for r in range(4):
            for c in rng.choice(4, size=2, replace=False):
                m[r, c] = rng.normal()
    return m


@pytest.mark.parametrize("n", [2, 3, 5, 12, 18])
@pytest.mark.parametrize("kind", ["channel", "zero_rows", "random"])
def test_sparse_real_gates(n, kind):
    from quantumflow_gb300 import _native as nat
    rng = np.random.default_rng(n)
    st = rng.normal(size=2 ** n) + 1j * rng.normal(size=2 ** n)
    for axes in {(0, 1), (1, 0), (n - 1, 0), (n - 2, n - 1), (n // 2, 0 if n > 3 else n - 1)}:
        if axes[0] == axes[1]:
            continue
        m = _matrix(kind, rng)
        v = np.moveaxis(st.reshape([2] * n), axes, (0, 1)).reshape(4, -1)
        want = np.zeros_like(v)
        for r in range(4):  # one fused multiply-add per term: exact in extended precision, then one rounding
            for part in ("real", "imag"):
                acc = np.zeros(v.shape[1])
                for c in np.nonzero(m[r])[0]:
                    x = getattr(v[c], part)
                    acc = (np.longdouble(m[r, c]) * x + acc).astype(np.float64)
                if part == "real":
                    want[r] += acc
                else:
                    want[r] += 1j * acc
        want = np.moveaxis(want.reshape([2] * n), (0, 1), axes).reshape(-1)
        flat = np.ascontiguousarray(m.astype(np.complex128)).view(np.float64).reshape(-1)
        for layout in (nat.LAYOUT_FX, nat.LAYOUT_C128):
            buf = torch.from_numpy(st).cuda()
            nat.call("qf_apply_gate", nat.ptr(buf), nat.ptr(buf), n, layout, 2, nat.int_array(axes),
                     flat.ctypes.data_as(nat._dp), nat.stream_handle())
            # the host's extended product may round twice: one unit in the last place
            assert np.max(np.abs(buf.cpu().numpy() - want)) <= 2.0 ** -52 * np.max(np.abs(want))


@pytest.mark.parametrize("n", [1, 2, 9, 17])
def test_real_and_complex_diagonals(n):
    from quantumflow_gb300 import _native as nat
    rng = np.random.default_rng(n)
    st = rng.normal(size=2 ** n) + 1j * rng.normal(size=2 ** n)
    for k in (1, 2):
        if k > n:
            continue
        for d in (rng.normal(size=2 ** k) + 0j, rng.normal(size=2 ** k) + 1j * rng.normal(size=2 ** k)):
            flat = np.ascontiguousarray(np.diag(d)).view(np.float64).reshape(-1)
            axes = list(range(n - 1, n - 1 - k, -1))
            buf = torch.from_numpy(st).cuda()
            nat.call("qf_apply_gate", nat.ptr(buf), nat.ptr(buf), n, nat.LAYOUT_C128, k, nat.int_array(axes),
                     flat.ctypes.data_as(nat._dp), nat.stream_handle())
            idx = np.arange(2 ** n)
            row = sum(((idx >> (n - 1 - a)) & 1) << (k - 1 - j) for j, a in enumerate(axes))
            want = d[row] * st
            assert np.max(np.abs(buf.cpu().numpy() - want)) <= 2 * 2.0 ** -52 * np.max(np.abs(want))
