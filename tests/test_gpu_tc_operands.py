"""The tensor-core 512-point transform's fixed-point operands: rows scaled by
their own maximum, cut into signed bytes. A power of two moves only the row
exponents, so it moves the outputs alone and exactly; a sequence's outputs do
not depend on its neighbours or on how full the engine's chunk is; an infinity
or a NaN has no digits and makes its whole sequence NaN and no other."""
import numpy as np
import pytest

import oceanlib_b200 as ob
from oceanlib_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _device(cuda_device):
    yield


def tensor_dft(x):
    import torch

    count, n = x.shape
    dev_in = torch.from_numpy(np.ascontiguousarray(x).view(np.float32).reshape(-1)).cuda()
    dev_out = torch.empty_like(dev_in)
    st = ob.lib().ocean_dft_batch(n, count, abi.OCEAN_FFT_TENSOR, dev_in.data_ptr(), dev_out.data_ptr(), None)
    assert st == abi.OCEAN_OK, ob.status_string(st)
    return dev_out.cpu().numpy().view(np.complex64).reshape(count, n)


def sequences(count):
    rng = np.random.default_rng(512 + count)
    x = (rng.standard_normal((count, 512)) + 1j * rng.standard_normal((count, 512))).astype(np.complex64)
    x[0, ::2] *= np.float32(2.0 ** -20)  # rows whose digits span the fixed point
    return x


@pytest.mark.parametrize("count", [1, 3, 4, 5, 8, 9, 2369])
def test_sequences_stand_alone(count):
    x = sequences(count)
    got = tensor_dft(x)
    ref = np.fft.ifft(x.astype(np.complex128), axis=1) * 512
    # 2e-6 of a sequence's RMS is the form's own bar (ocean_fft_form).
    rms = np.sqrt(np.mean(np.abs(ref) ** 2, axis=1, keepdims=True))
    assert (np.abs(got - ref) / rms).max() <= 2e-6
    for i in {0, count // 2, count - 1}:
        assert np.array_equal(tensor_dft(x[i : i + 1])[0].view(np.uint32), got[i].view(np.uint32))


@pytest.mark.parametrize("power", [-60, -1, 1, 60])
def test_powers_of_two_are_exact(power):
    x = sequences(9)
    scale = np.float32(2.0) ** power
    assert np.array_equal((tensor_dft(x) * scale).view(np.uint32), tensor_dft(x * scale).view(np.uint32))


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("where", [0, 31, 32, 511])
def test_non_finite_values_stay_in_their_sequence(bad, where):
    x = sequences(9)
    want = tensor_dft(x)
    x[4, where] = np.complex64(complex(1.0, bad))
    got = tensor_dft(x)
    assert np.isnan(got[4].real).all() and np.isnan(got[4].imag).all()
    keep = [i for i in range(9) if i != 4]
    assert np.array_equal(got[keep].view(np.uint32), want[keep].view(np.uint32))


def test_zeros_give_zeros():
    assert not tensor_dft(np.zeros((3, 512), np.complex64)).any()
