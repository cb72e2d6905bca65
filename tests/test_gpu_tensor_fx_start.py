"""The accumulators' start values of the tensor-core pass: outputs bit for bit
those of the integer model where the digits are extreme (all bytes 0x80, 0x7f,
0x00, 0xff), of one sign, sparse or zero, against gates with equal, sparse and
generic entries."""
import numpy as np
import pytest

from test_gpu_tensor_fx import _apply, _model, tensor_cores  # noqa: F401

pytestmark = pytest.mark.gpu

N = 11


def _state(kind):
    rng = np.random.default_rng(1)
    mant = {"ones": 0xFFFFFFFFFFFFF, "80": 0x8080808080808, "7f": 0xF7F7F7F7F7F7F, "00": 0}.get(kind)
    if mant is not None:
        v = np.full(2 ** N, (1022 << 52) | mant, np.uint64).view(np.float64)
        return v * rng.choice([1, -1], 2 ** N) + 1j * v
    if kind == "same":
        return np.full(2 ** N, 2.0 ** -5 * (1 - 1j))
    st = np.zeros(2 ** N, complex)
    if kind == "one":
        st[[3, 700, 2047]] = 1e-30j, -1.0, 0.1
    return st


def _gate(kind):
    h = np.array([[1, 1], [1, -1]]) / np.sqrt(2)
    if kind == "equal":
        return np.kron(h, h)
    if kind == "dft":
        return np.exp(0.5j * np.pi * np.outer(range(4), range(4))) / 2
    if kind == "swap":
        return np.eye(4)[[0, 2, 1, 3]]
    if kind == "minus":
        return -1j * np.kron(h, np.eye(2))
    rng = np.random.default_rng(2)
    return np.linalg.qr(rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4)))[0]


@pytest.mark.parametrize("state", ["ones", "80", "7f", "00", "same", "one", "zero"])
@pytest.mark.parametrize("gate", ["equal", "dft", "swap", "minus", "haar"])
def test_extreme_digits_bit_exact(tensor_cores, state, gate):  # noqa: F811
    st, u, axes = _state(state), np.asarray(_gate(gate), complex), [1, 8]
    got, want = _apply(st, u, axes), _model(st, u, axes)
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64)), float(np.max(np.abs(got - want)))
