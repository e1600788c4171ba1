"""Batches on both sides of the counts where the register-resident frame takes
over, by form, field count and foam: an ocean's bits do not depend on the side.
The FP32 forms against the oracle, the precise form against a batch of its own,
foam (also a frame without a foam step) against a batch of one."""
import numpy as np
import pytest

import oceanlib_b200 as ob
import oracle as O
from oceanlib_b200 import abi

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.fixture(autouse=True)
def _device(cuda_device):
    ob.force_simd_level(None)
    yield


def _descs(n, count, velocity):
    return [ob.OceanDesc(size=n, patch_length=0.9 * n + 11.0, wind_speed=9.0 + k % 6, wind_direction=0.3 * k,
                         choppiness=1.2, seed=900 + k, compute_velocity=velocity) for k in range(count)]


def _read(batch, n, i, velocity, foam=False):
    b = batch.device_buffers(i)
    ptrs = [b.displacement, b.normal] + ([b.velocity] if velocity else [])
    out = [np.empty((n * n, 4), np.float32) for _ in ptrs]
    if foam:
        ptrs.append(b.foam)
        out.append(np.empty(n * n, np.float32))
    for dst, ptr in zip(out, ptrs):
        assert ob.lib().ocean_copy_to_host(dst.ctypes.data, ptr, dst.nbytes) == 0
    return out


@pytest.mark.parametrize("n,velocity,counts", [(64, True, (6, 7)), (64, False, (3, 4)), (256, False, (2, 3)),
                                               (256, True, (3, 4)), (512, True, (1, 2))])
def test_fp32_forms(n, velocity, counts):
    for count in counts:
        ds = _descs(n, count, velocity)
        batch = ob.OceanBatch(ds)
        for t in (2.0, 7.25):
            batch.update(t)
        batch.synchronize()
        for i in {0, count // 2, count - 1}:
            for got, want in zip(_read(batch, n, i, velocity), O.update(ds[i], 7.25)):
                assert np.array_equal(bits(got), bits(want)), (count, i)
        batch.close()


@pytest.mark.parametrize("n,velocity,counts", [(32, True, (3, 4)), (64, False, (6, 7)), (64, True, (6, 7)),
                                               (128, True, (9, 10)), (256, True, (6, 7)), (512, False, (1, 2)),
                                               (512, True, (15, 16))])
def test_precise_form(n, velocity, counts):
    for count in counts:
        ds = _descs(n, count, velocity)
        batch = ob.OceanBatch(ds, form=abi.OCEAN_FFT_PRECISE)
        for t in (2.0, 7.25):
            batch.update(t)
        batch.synchronize()
        for i in (0, count - 1):
            one = ob.OceanBatch(ds[i:i + 1], form=abi.OCEAN_FFT_PRECISE, schedule=abi.OCEAN_SCHEDULE_CHUNKED)
            one.update(7.25)
            one.synchronize()
            for got, want in zip(_read(batch, n, i, velocity), _read(one, n, 0, velocity)):
                assert np.array_equal(bits(got), bits(want)), (count, i)
            one.close()
        batch.close()


@pytest.mark.parametrize("form", [abi.OCEAN_FFT_EXACT, abi.OCEAN_FFT_FAST], ids=["exact", "fast"])
@pytest.mark.parametrize("n,counts", [(64, (6, 7)), (1024, (1, 2))])
def test_foam_and_frames_between_its_steps(n, counts, form):
    def frames(descs, schedule):
        b = ob.OceanBatch(descs, foam=ob.FoamDesc(), form=form, schedule=schedule)
        for t, dt in ((1.0, 1 / 60), (1.5, 0.0), (2.0, 1 / 60), (2.5, 1 / 60)):
            b.update(t, foam_dt=dt)
        b.synchronize()
        return b

    for count in counts:
        ds = _descs(n, count, True)
        for d in ds:
            d.foam_threshold = 0.98  # foam nearly everywhere
        batch = frames(ds, abi.OCEAN_SCHEDULE_PERSISTENT)
        for i in (0, count - 1):
            one = frames(ds[i:i + 1], abi.OCEAN_SCHEDULE_CHUNKED)
            for got, want in zip(_read(batch, n, i, True, True), _read(one, n, 0, True, True)):
                assert np.array_equal(bits(got), bits(want)), (count, i)
            assert got.max() > 0.0
            one.close()
        batch.close()
