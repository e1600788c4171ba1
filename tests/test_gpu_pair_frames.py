"""Batches around the counts where the register-resident frame takes over, at
every size it has: oceans of different patches, both field counts, foam, both
ring depths and publish timings, and more oceans than the rows run ahead, all
with the oracle's bits; the precise form gives an ocean the same bits alone and
in a batch, and a server's sessions of one size equal the oracle."""
import numpy as np
import pytest

import oceanlib_b200 as ob
import oracle as O
from oceanlib_b200 import abi
from oceanlib_b200.serve import OceanServer

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.fixture(autouse=True)
def _device(cuda_device):
    ob.force_simd_level(None)
    yield


def descs(n, count, velocity, same_patch=False):
    return [ob.OceanDesc(size=n, patch_length=0.7 * n + (0.0 if same_patch else 3.0 * (k % 3)), wind_speed=11.0 + k % 5,
                         wind_direction=0.2 * k, choppiness=1.3, seed=500 + k, compute_velocity=velocity)
            for k in range(count)]


def frame(batch, n, count, velocity, t, dt=0.0, foam=False):
    out = [np.empty((count * n * n, 4), np.float32) for _ in range(3 if velocity else 2)]
    fo = np.empty(count * n * n, np.float32) if foam else None
    batch.update(t, foam_dt=dt)
    batch.synchronize()
    for i in range(count):
        b = batch.device_buffers(i)
        sl = slice(i * n * n, (i + 1) * n * n)
        for dst, ptr in zip(out, (b.displacement, b.normal, b.velocity)):
            assert ob.lib().ocean_copy_to_host(dst[sl].ctypes.data, ptr, dst[sl].nbytes) == 0
        if foam:
            assert ob.lib().ocean_copy_to_host(fo[sl].ctypes.data, b.foam, fo[sl].nbytes) == 0
    return out, fo


# (size, counts): below, at and above the change of kernel, and past a ring.
SIZES = [(16, (3, 4, 70)), (32, (3, 4, 50)), (64, (3, 4, 33)), (128, (3, 4, 19)), (256, (3, 4, 31)), (512, (1, 2, 11)),
         (1024, (1, 6))]


@pytest.mark.parametrize("velocity", [False, True])
@pytest.mark.parametrize("n,counts", SIZES)
def test_counts_match_the_oracle(n, counts, velocity):
    for count in counts:
        ds = descs(n, count, velocity)
        batch = ob.OceanBatch(ds)
        for t in (4.25, 9.5):
            got, _ = frame(batch, n, count, velocity, t)
        for i in {0, 1 % count, count // 2, count - 1}:
            for g, want in zip(got, O.update(ds[i], 9.5)):
                assert np.array_equal(bits(g[i * n * n:(i + 1) * n * n]), bits(want)), (count, i)
        batch.close()


@pytest.mark.parametrize("n,count", [(32, 9), (128, 6), (512, 3), (512, 12), (1024, 2)])
def test_foam_and_queue_settings_do_not_change_the_bits(n, count):
    # Three frames of foam under every ring depth and publish timing; an ocean
    # of the batch equals the same ocean in a batch of its own.
    ds = descs(n, count, True, same_patch=True)
    alone = [frame(b, n, 1, True, t, 1 / 60, True) for b in [ob.OceanBatch(ds[-1:], foam=ob.FoamDesc())]
             for t in (1.0, 1.5, 2.0)][-1]
    for slots in sorted({min(count, 3), 2}):
        for defer in (False, True):
            batch = ob.OceanBatch(ds, foam=ob.FoamDesc())
            batch.set_ring_slots(slots)
            batch.set_deferred_publish(defer)
            for t in (1.0, 1.5, 2.0):
                got, fo = frame(batch, n, count, True, t, 1 / 60, True)
            sl = slice((count - 1) * n * n, count * n * n)
            for g, a in zip(got, alone[0]):
                assert np.array_equal(bits(g[sl]), bits(a)), (slots, defer)
            assert np.array_equal(bits(fo[sl]), bits(alone[1])), (slots, defer)
            batch.close()


@pytest.mark.parametrize("n,count", [(16, 8), (32, 8), (64, 8), (128, 12), (256, 8), (512, 2), (1024, 2)])
def test_precise_rounds_at_the_same_blocks_in_a_batch(n, count):
    ds = descs(n, count, True)
    batch = ob.OceanBatch(ds, form=abi.OCEAN_FFT_PRECISE)
    got, _ = frame(batch, n, count, True, 3.75)
    for i in (0, count - 1):
        one = ob.OceanBatch(ds[i:i + 1], form=abi.OCEAN_FFT_PRECISE, schedule=abi.OCEAN_SCHEDULE_CHUNKED)
        want, _ = frame(one, n, 1, True, 3.75)
        for g, w in zip(got, want):
            assert np.array_equal(bits(g[i * n * n:(i + 1) * n * n]), bits(w)), i
        one.close()
    batch.close()


def test_sessions_of_one_size():
    n, count = 64, 24
    ds = descs(n, count, False)
    with OceanServer(hbm_budget=1e9) as srv:
        ids = [srv.open_session(d) for d in ds]
        for t in (1.0, 2.5):
            for s in ids:
                srv.submit_update(s, t, 0.0)
            srv.drain()
        for i in range(0, count, 5):
            disp, normal, _ = srv.read_session(ids[i], n)
            od, on, _ = O.update(ds[i], 2.5)
            assert np.array_equal(bits(disp.reshape(-1, 4)), bits(od)) and np.array_equal(bits(normal.reshape(-1, 4)), bits(on))
