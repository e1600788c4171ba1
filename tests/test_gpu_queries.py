"""World queries run as pairs of lanes: point counts around a warp's 16 points
and a block's 128, points far outside the patch and exactly on cell edges, and
early-stopping inversions in mixed company all equal the CPU oracle's bits."""
import numpy as np
import pytest

import oceanlib_b200 as ob
import oracle as O

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.fixture(autouse=True)
def _device(cuda_device):
    ob.force_simd_level(None)
    yield


def points(count, length, n):
    rng = np.random.default_rng(count)
    xz = rng.uniform(-3.0 * length, 3.0 * length, (count, 2)).astype(np.float32)
    edge = np.float32(length / n) * np.array([[0, 0], [n, n], [-1, n - 1], [n // 2, -n]], np.float32)
    far = np.array([[3.0e9, -3.0e9], [-1.0e12, 1.0e12]], np.float32)
    xz[: min(count, 4)] = edge[:count]
    xz[4:6] = far[: max(0, min(count, 6) - 4)]
    return xz


def unit(v):
    return v * (np.float32(1.0) / np.sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]))


def corner_record(n, disp, nrm, vel, p):
    """The record of a point past the range of int, where the oracle's
    conversion is undefined in C. The device's saturates (a coordinate of that
    size has no fraction), so it is the last or first texel's."""
    x, z = (n - 1 if v > 0 else 0 for v in p)
    k = z * n + x
    v = vel[k, :3] if vel is not None else np.zeros(3, np.float32)
    return np.array([disp[k, 1], disp[k, 0], disp[k, 2], *unit(nrm[k, :3]), disp[k, 3], *v], np.float32)


@pytest.mark.parametrize("velocity", [False, True])
@pytest.mark.parametrize("count", [1, 2, 15, 16, 17, 127, 128, 129, 1000])
def test_counts_and_edges(count, velocity):
    d = ob.OceanDesc(size=32, patch_length=40.0, wind_speed=14.0, choppiness=1.7, seed=9, compute_velocity=velocity)
    ocean = ob.Ocean(d)
    ocean.update(3.25)
    xz = points(count, d.patch_length, d.size)
    disp, nrm, vel = O.update(d, 3.25)
    want = O.sample_many(d.size, d.patch_length, disp, nrm, vel, xz)
    for i in np.flatnonzero(np.abs(xz).max(axis=1) > 2.0e9):
        want[i] = corner_record(d.size, disp, nrm, vel, xz[i])
    assert np.array_equal(bits(ocean.sample_many(xz)), bits(want))


@pytest.mark.parametrize("iterations,tolerance", [(4, 0.0), (0, 0.0), (1, 0.0), (12, 1e-3), (12, 0.3)])
def test_cascade_stopping_rules(iterations, tolerance):
    ds = [ob.OceanDesc(size=n, patch_length=length, wind_speed=14.0, depth=30.0, choppiness=1.3, seed=k,
                       compute_velocity=True) for k, (n, length) in enumerate(((64, 300.0), (16, 20.0), (32, 55.0)))]
    stack = ob.CascadeStack(ds)
    stack.update(7.5)
    xz = points(333, 300.0, 64)
    frames = [O.update(d, 7.5) for d in ds]
    want = O.cascade_sample_many(ds, frames, xz, iterations, tolerance)
    for i in np.flatnonzero(np.abs(xz).max(axis=1) > 2.0e9):
        # Level by level: only some put the point past the range of int. (A
        # coordinate of this size does not move, whatever the step count.)
        r = np.zeros(10, np.float32)
        clear = np.float32(1.0)
        for d, f in zip(ds, frames):
            past = np.abs(xz[i]).min() * d.size / d.patch_length >= 2.0**31
            s = corner_record(d.size, *f, xz[i]) if past else O.sample_many(d.size, d.patch_length, *f, xz[i:i + 1])[0]
            r += s
            clear *= np.float32(1.0) - s[6]
        r[3:6] = unit(r[3:6])
        r[6] = np.float32(1.0) - clear
        want[i] = r
    assert np.array_equal(bits(stack.sample_many(xz, iterations=iterations, tolerance=tolerance)), bits(want))
