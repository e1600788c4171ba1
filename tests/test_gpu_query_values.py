"""World queries at points that are no numbers: a coordinate that is NaN or an
infinity makes that point's surface NaN and its normal straight up, as the
reference's arithmetic does, and leaves its neighbours in the warp alone."""
import numpy as np
import pytest

import oceanlib_b200 as ob
import oracle as O

pytestmark = pytest.mark.gpu

INF, NAN = np.float32(np.inf), np.float32(np.nan)
BAD = [(NAN, 1.0), (2.0, NAN), (NAN, NAN), (INF, 3.0), (4.0, -INF), (-INF, INF), (INF, NAN)]


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def _points(length):
    xz = np.random.default_rng(5).uniform(-2 * length, 2 * length, (61, 2)).astype(np.float32)
    at = np.arange(len(BAD)) * 8 + 3  # among others, in both halves of a warp's points
    xz[at] = BAD
    return xz, at


def _check(got, want, at, velocity):
    good = np.setdiff1d(np.arange(len(got)), at)
    assert np.array_equal(bits(got[good]), bits(want[good]))
    bad = got[at]
    assert np.isnan(bad[:, [0, 1, 2, 6]]).all()
    assert np.array_equal(bad[:, 3:6], np.tile(np.float32([0, 1, 0]), (len(at), 1)))
    assert np.isnan(bad[:, 7:]).all() if velocity else (bad[:, 7:] == 0).all()


@pytest.mark.parametrize("velocity", [False, True])
def test_one_ocean(cuda_device, velocity):
    ob.force_simd_level(None)
    d = ob.OceanDesc(size=64, patch_length=50.0, wind_speed=13.0, choppiness=1.6, seed=21, compute_velocity=velocity)
    ocean = ob.Ocean(d)
    ocean.update(4.5)
    xz, at = _points(d.patch_length)
    fine = xz.copy()
    fine[at] = 0.0
    disp, nrm, vel = O.update(d, 4.5)
    _check(ocean.sample_many(xz), O.sample_many(d.size, d.patch_length, disp, nrm, vel, fine), at, velocity)
    assert np.isnan(ocean.height_at(float("nan"), 1.0)) and np.isnan(ocean.height_at(1.0, float("inf")))
    ocean.close()


@pytest.mark.parametrize("iterations,tolerance", [(4, 0.0), (12, 1e-3)])
def test_cascade(cuda_device, iterations, tolerance):
    ob.force_simd_level(None)
    ds = [ob.OceanDesc(size=n, patch_length=length, wind_speed=13.0, choppiness=1.2, seed=k, compute_velocity=True)
          for k, (n, length) in enumerate(((64, 210.0), (32, 37.0)))]
    stack = ob.CascadeStack(ds)
    stack.update(2.75)
    xz, at = _points(210.0)
    fine = xz.copy()
    fine[at] = 0.0
    want = O.cascade_sample_many(ds, [O.update(d, 2.75) for d in ds], fine, iterations, tolerance)
    _check(stack.sample_many(xz, iterations=iterations, tolerance=tolerance), want, at, True)
    stack.close()
