"""The host mirror of an ocean's outputs, on both sides of the size from which
a copy engine moves it (768 KiB: 128^2 with velocity is the last below), and
the single queries, which read and write pinned memory, against many at once."""
import numpy as np
import pytest

import oceanlib_b200 as ob

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _device(cuda_device):
    yield


def device_plane(ptr, n):
    a = np.empty((n * n, 4), np.float32)
    assert ob.lib().ocean_copy_to_host(a.ctypes.data, ptr, a.nbytes) == 0
    return a


@pytest.mark.parametrize("velocity", [False, True])
@pytest.mark.parametrize("n", [16, 64, 128, 256])
def test_mirror_holds_the_device_outputs(n, velocity):
    o = ob.Ocean(ob.OceanDesc(size=n, patch_length=90.0, wind_speed=11.0, seed=5, compute_velocity=velocity))
    for t in (0.25, 7.5):  # the second update overwrites the first's mirror
        o.update(t)
        got, dev = o.buffers(), o.device_buffers()
        for name in ("displacement", "normal") + (("velocity",) if velocity else ()):
            want = device_plane(getattr(dev, name), n)
            assert want.any() and np.array_equal(got[name].view(np.uint32), want.view(np.uint32)), name
    xz = np.array([[3.5, -17.25], [1e3, 2.0], [-0.0, 44.9]], np.float32)
    many = o.sample_many(xz)
    for i, (x, z) in enumerate(xz.tolist()):
        one = np.array(list(o.sample_at(x, z).values()), np.float32)
        assert np.array_equal(one.view(np.uint32), many[i].view(np.uint32))
    o.close()
