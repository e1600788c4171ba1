"""A server's larger intermediate rings: batches of many sessions of a size use
one where the budget has room beside the sessions, do without where it has not,
and give it back to a session that needs the room; the same bits either way."""
import time

import numpy as np
import pytest

import oceanlib_b200 as ob
from oceanlib_b200 import abi
from oceanlib_b200.serve import OceanServer, session_bytes

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _device(cuda_device):
    ob.force_simd_level(None)
    yield


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def _descs(sizes, velocity):
    return [ob.OceanDesc(size=n, patch_length=20.0 + 0.5 * n, wind_speed=7.0 + i % 9, choppiness=0.8 + 0.02 * i,
                         seed=40 + i, compute_velocity=velocity) for i, n in enumerate(sizes)]


def _round(b):
    return (b + 255) // 256 * 256


def _kind_bytes(n, velocity):
    return _round(3 * n * n * (6 if velocity else 4) * 8) + _round((n - 1) * 8)


def _bytes(descs):
    kinds = {(d.size, bool(d.compute_velocity)) for d in descs}
    return sum(session_bytes(d) for d in descs) + sum(_kind_bytes(n, v) for n, v in kinds)


def _tick(srv, sids, t):
    for s in sids:
        srv.submit_update(s, t, 0.0)
    srv.drain()


def _run(descs, budget, form, want_ring):
    """Ticks until a batch was large enough for a ring (several are gathered
    while one runs), at least 20; the last frame of every session."""
    srv = OceanServer(hbm_budget=budget, max_inflight=1, form=form)
    base = srv.stats()["bytes_staging"]
    sids = [srv.open_session(d) for d in descs]
    for k in range(200):
        _tick(srv, sids, 1.0 + 0.1 * k)
        if k >= 20 and (not want_ring or srv.stats()["bytes_staging"] > base):
            break
    _tick(srv, sids, 33.5)
    out = [srv.read_session(s, d.size, 0)[:2] for s, d in zip(sids, descs)]
    st = srv.stats()
    srv.close()
    assert st["requests_failed"] == 0
    return out, st["bytes_staging"] - base


SIZES = {
    "512": ([512] * 12, True),
    "512_plain": ([512] * 12, False),
    "1024": ([1024] * 7, False),
    "64": ([64] * 40, True),
    "mixed_velocity": ([64] * 20 + [256] * 8 + [512] * 9, True),
    "mixed": ([128] * 12 + [512] * 6 + [1024] * 6, False),
}
# The precise form's 1024^2, its 512^2 with velocity below 16 oceans and its one
# launch of several sizes have three slots.
CASES = [(n, f) for n in SIZES for f in (abi.OCEAN_FFT_EXACT, abi.OCEAN_FFT_FAST)] + \
    [("512_plain", abi.OCEAN_FFT_PRECISE), ("64", abi.OCEAN_FFT_PRECISE)]


@pytest.mark.parametrize("name,form", CASES)
def test_sessions_are_the_same_with_and_without_room_for_a_ring(name, form):
    descs = _descs(*SIZES[name])
    roomy, ring = _run(descs, 8_000_000_000, form, True)
    assert ring > 0
    tight, none = _run(descs, _bytes(descs), form, False)
    assert none == 0
    for i, d in enumerate(descs):
        for a, b in zip(roomy[i], tight[i]):
            assert np.array_equal(bits(a), bits(b)), (d.size, i)
    for i in (0, len(descs) // 2, len(descs) - 1):
        d = descs[i]
        alone = ob.OceanBatch([d], form=form)
        want = [np.empty((d.size * d.size, 4), np.float32) for _ in range(2)]
        alone.update_host([33.5], 0.0, *want)
        alone.close()
        for a, w in zip(roomy[i], want):
            assert np.array_equal(bits(a), bits(w.reshape(a.shape))), (d.size, i)


def test_a_ring_makes_way_for_a_session():
    descs = _descs([256] * 16, True)
    late = _descs([512], True)
    # Room for the sixteen and the late one, or for the sixteen and a ring.
    budget = _bytes(descs + late)
    srv = OceanServer(hbm_budget=budget, max_inflight=1)
    base = srv.stats()["bytes_staging"]
    sids = [srv.open_session(d) for d in descs]
    k = 0
    while srv.stats()["bytes_staging"] == base and k < 200:
        _tick(srv, sids, 1.0 + 0.1 * k)
        k += 1
    st = srv.stats()
    ring = st["bytes_staging"] - base
    assert ring > 0 and st["bytes_in_use"] + ring <= budget
    assert st["bytes_in_use"] + ring + session_bytes(late[0]) + _kind_bytes(512, True) > budget
    sid = srv.open_session(late[0])
    deadline = time.time() + 20
    while srv.state(sid) != abi.OCEAN_SESSION_ACTIVE and time.time() < deadline:
        time.sleep(0.01)
    assert srv.state(sid) == abi.OCEAN_SESSION_ACTIVE
    for k in range(20):
        _tick(srv, sids + [sid], 5.0 + 0.1 * k)
    st = srv.stats()
    assert st["bytes_in_use"] <= budget and st["bytes_staging"] == base
    for s, d in ((sids[7], descs[7]), (sid, late[0])):
        got = srv.read_session(s, d.size, 0)[:2]
        alone = ob.OceanBatch([d])
        want = [np.empty((d.size * d.size, 4), np.float32) for _ in range(2)]
        alone.update_host([5.0 + 0.1 * 19], 0.0, *want)
        alone.close()
        for a, w in zip(got, want):
            assert np.array_equal(bits(a), bits(w.reshape(a.shape))), d.size
    srv.close()
