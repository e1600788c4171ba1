"""What the ensemble's autotuner says of the one launch is what that launch does:
register-resident tasks have one ring depth, so none is named for them."""
import numpy as np
import pytest

import oceanlib_b200 as ob
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _device(cuda_device):
    ob.force_simd_level(None)
    yield


def _descs(sizes, velocity):
    return [ob.OceanDesc(size=n, patch_length=1.5 * n, wind_speed=8.0 + i % 9, choppiness=1.0, seed=70 + i,
                         compute_velocity=velocity) for i, n in enumerate(sizes)]


def test_no_ring_depth_is_named_for_register_resident_tasks():
    # Sizes from 64 on with several hundred row tasks; three oceans of a size and more,
    # so that a batch has a shallower ring. Ensembles whose one launch is often
    # the fastest schedule.
    for sizes, velocity in (([128] * 20 + [256] * 3 + [512], True),
                            ([64] * 3 + [128] * 3 + [256] * 3 + [512] * 3 + [1024] * 3, False)):
        for _ in range(10):
            ens = ob.OceanEnsemble(_descs(sizes, velocity), autotune=True)
            assert "one persistent launch at" not in ens.schedule
            ens.close()
    descs = _descs([64] * 4 + [256] * 4 + [512] * 4, False)
    ens = ob.OceanEnsemble(descs, autotune=True)
    ens.update(3.25)
    ens.synchronize()
    for i in (0, 5, 11):
        d, n = ens.read(i)
        od, on, _ = O.update(descs[i], 3.25)
        assert np.array_equal(np.ascontiguousarray(d).view(np.uint32), np.ascontiguousarray(od).view(np.uint32))
        assert np.array_equal(np.ascontiguousarray(n).view(np.uint32), np.ascontiguousarray(on).view(np.uint32))
    ens.close()
