"""A server on a device that is almost full: no session is refused for want of
device memory while a larger intermediate ring holds some, and the sessions that
were there go on with the same bits."""
import time

import numpy as np
import pytest
import torch

import oceanlib_b200 as ob
from oceanlib_b200 import abi
from oceanlib_b200.serve import OceanServer

pytestmark = pytest.mark.gpu

LEFT = 300 << 20  # device memory left to the server besides what it has


@pytest.fixture(autouse=True)
def _device(cuda_device):
    ob.force_simd_level(None)
    yield


def _descs(n, count, velocity):
    return [ob.OceanDesc(size=n, patch_length=20.0 + 0.5 * n, wind_speed=7.0 + i % 9, choppiness=0.9, seed=60 + i,
                         compute_velocity=velocity) for i in range(count)]


def _tick(srv, sids, t):
    for s in sids:
        srv.submit_update(s, t, 0.0)
    srv.drain()


def test_rings_make_way_before_a_session_is_refused():
    early, late = _descs(256, 16, True), _descs(1024, 40, False)
    srv = OceanServer(hbm_budget=170e9, max_inflight=1)
    base = srv.stats()["bytes_staging"]
    sids = [srv.open_session(d) for d in early]
    late_sids = [srv.open_session(late[0])]  # brings its size's tables
    k = 0
    while srv.stats()["bytes_staging"] == base and k < 200:
        _tick(srv, sids, 1.0 + 0.1 * k)
        k += 1
    assert srv.stats()["bytes_staging"] > base
    free = torch.cuda.mem_get_info()[0]
    fill = torch.empty(max(0, free - LEFT), dtype=torch.uint8, device="cuda")
    refused = False
    for d in late[1:]:
        sid = srv.open_session(d)
        deadline = time.time() + 20
        while srv.state(sid) not in (abi.OCEAN_SESSION_ACTIVE, abi.OCEAN_SESSION_CLOSED) and time.time() < deadline:
            time.sleep(0.002)
        if srv.state(sid) == abi.OCEAN_SESSION_CLOSED:
            refused = True
            break
        assert srv.state(sid) == abi.OCEAN_SESSION_ACTIVE
        late_sids.append(sid)
    assert refused
    assert srv.stats()["bytes_staging"] == base
    _tick(srv, sids + late_sids, 33.5)
    got = [(early[7], srv.read_session(sids[7], 256, 0)[:2])]
    got += [(late[i], srv.read_session(late_sids[i], 1024, 0)[:2]) for i in (0, len(late_sids) - 1)]
    srv.close()
    del fill
    torch.cuda.empty_cache()
    for d, planes in got:
        alone = ob.OceanBatch([d])
        want = [np.empty((d.size * d.size, 4), np.float32) for _ in range(2)]
        alone.update_host([33.5], 0.0, *want)
        alone.close()
        for a, w in zip(planes, want):
            assert np.array_equal(a.view(np.uint32), w.reshape(a.shape).view(np.uint32)), d.size
