"""A batch on a device that has room for it but not for the larger intermediate
ring of the register-resident frames: it is created all the same and runs on a
ring of three, with the same bits."""
import numpy as np
import pytest
import torch

import oceanlib_b200 as ob
from oceanlib_b200 import abi

pytestmark = pytest.mark.gpu

# Of the memory that a batch takes with its full ring, what is kept from it. The
# ring's slots past the least that the batch can run on take 45 to 63 MB below.
SHORT = 24 << 20


@pytest.fixture(autouse=True)
def _device(cuda_device):
    ob.force_simd_level(None)
    yield


def _frames(descs, form, foam):
    batch = ob.OceanBatch(descs, form=form, foam=ob.FoamDesc() if foam else None)
    n = descs[0].size
    out = []
    for t in (2.0, 7.25):
        batch.update(t, 1.0 / 60.0 if foam else 0.0)
    batch.synchronize()
    for i in (0, len(descs) // 2, len(descs) - 1):
        b = batch.device_buffers(i)
        for ptr, width in ((b.displacement, 4), (b.normal, 4)) + (((b.foam, 1),) if foam else ()):
            a = np.empty((n * n, width), np.float32)
            assert ob.lib().ocean_copy_to_host(a.ctypes.data, ptr, a.nbytes) == 0
            out.append(a.view(np.uint32))
    used = torch.cuda.mem_get_info()[0]
    batch.close()
    return out, used


@pytest.mark.parametrize("n,count,velocity,foam,form", [
    (512, 16, True, False, abi.OCEAN_FFT_EXACT), (512, 16, True, True, abi.OCEAN_FFT_FAST),
    (512, 16, True, False, abi.OCEAN_FFT_PRECISE), (1024, 8, True, False, abi.OCEAN_FFT_EXACT),
    (256, 40, True, False, abi.OCEAN_FFT_EXACT), (64, 500, True, False, abi.OCEAN_FFT_EXACT)])
def test_a_batch_without_room_for_its_ring(n, count, velocity, foam, form):
    descs = [ob.OceanDesc(size=n, patch_length=1.3 * n, wind_speed=8.0 + k % 7, choppiness=1.1, seed=300 + k,
                          compute_velocity=velocity) for k in range(count)]
    _frames(descs, form, foam)  # kernels loaded
    before = torch.cuda.mem_get_info()[0]
    roomy, left = _frames(descs, form, foam)
    need = before - left
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - need + SHORT, dtype=torch.uint8, device="cuda")
    short, _ = _frames(descs, form, foam)
    del fill
    torch.cuda.empty_cache()
    for a, b in zip(roomy, short):
        assert np.array_equal(a, b)
