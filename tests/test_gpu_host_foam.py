"""update_host's copies with persistent foam: every output is the frame's own,
with no, one and several foam substeps, in batches of several chunks and above
1024^2, where the foam comes after every ocean's frame."""
import numpy as np
import pytest

import oceanlib_b200 as ob

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


@pytest.fixture(autouse=True)
def _device(cuda_device):
    ob.force_simd_level(None)
    yield


@pytest.mark.parametrize("n,count,chunk", [(128, 7, 3), (512, 5, 0), (2048, 3, 1), (2048, 2, 2)])
def test_host_outputs_are_the_frames(n, count, chunk):
    descs = [ob.OceanDesc(size=n, patch_length=1.2 * n, wind_speed=9.0 + k, choppiness=1.4, seed=20 + k,
                          compute_velocity=True) for k in range(count)]
    host = ob.OceanBatch(descs, foam=ob.FoamDesc(), chunk=chunk)
    dev = ob.OceanBatch(descs, foam=ob.FoamDesc(), chunk=chunk)
    cells = n * n
    for f, dt in enumerate((0.0, DT, 2.01 * DT, DT, 3.01 * DT)):
        out = [np.full((count, cells, w), -7.0, np.float32) for w in (4, 4, 4, 1)]
        host.update_host([1.0 + 0.3 * f], dt, *out)
        dev.update(1.0 + 0.3 * f, foam_dt=dt)
        dev.synchronize()
        assert host.last_foam_substeps == dev.last_foam_substeps
        for i in range(count):
            b = dev.device_buffers(i)
            for got, ptr in zip(out, (b.displacement, b.normal, b.velocity, b.foam)):
                want = np.empty_like(got[i])
                assert ob.lib().ocean_copy_to_host(want.ctypes.data, ptr, want.nbytes) == 0
                assert np.array_equal(got[i].view(np.uint32), want.view(np.uint32)), (f, i)
        # Without a plane for the foam the rest is copied all the same.
        if f == 3:
            some = [np.zeros((count, cells, 4), np.float32) for _ in range(2)]
            host.update_host([2.5], DT, *some)
            dev.update(2.5, foam_dt=DT)
            dev.synchronize()
            b = dev.device_buffers(count - 1)
            want = np.empty_like(some[1][count - 1])
            assert ob.lib().ocean_copy_to_host(want.ctypes.data, b.normal, want.nbytes) == 0
            assert np.array_equal(some[1][count - 1].view(np.uint32), want.view(np.uint32))
    host.close()
    dev.close()
