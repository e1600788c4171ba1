"""Every size of an ensemble in one launch of register-resident tasks: both field
counts, the exact and the fast form, and more oceans of a size than its ring
holds, so that slots are taken again (ring: 444 oceans of 64^2, 112 of 128^2, 28
of 256^2, 8 of 512^2, 4 of 1024^2). And the schedules that replay a graph, frame
after frame."""
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


def _descs(counts, velocity):
    return [ob.OceanDesc(size=n, patch_length=0.8 * n + 15.0, wind_speed=8.0 + k % 7, wind_direction=0.17 * k,
                         choppiness=1.1, seed=3 * n + k, compute_velocity=velocity)
            for n, count in counts.items() for k in range(count)]


def _read(owner, i, d):
    b = owner.device_buffers(i)
    out = []
    for ptr in [b.displacement, b.normal] + ([b.velocity] if d.compute_velocity else []):
        a = np.empty((d.size * d.size, 4), np.float32)
        assert ob.lib().ocean_copy_to_host(a.ctypes.data, ptr, a.nbytes) == 0
        out.append(a)
    return out


def _want(d, t, form):
    if form == abi.OCEAN_FFT_EXACT:
        return O.update(d, t)
    one = ob.OceanBatch([d], form=form, schedule=abi.OCEAN_SCHEDULE_CHUNKED)
    one.update(t)
    one.synchronize()
    out = _read(one, 0, d)
    one.close()
    return out


@pytest.mark.parametrize("form", [abi.OCEAN_FFT_EXACT, abi.OCEAN_FFT_FAST], ids=["exact", "fast"])
@pytest.mark.parametrize("velocity", [False, True])
@pytest.mark.parametrize("counts", [{64: 450, 512: 11}, {128: 115, 256: 31, 1024: 6}, {1024: 1, 64: 5, 256: 4, 512: 1}],
                         ids=["64_512", "128_256_1024", "few"])
def test_one_launch_past_the_rings(counts, velocity, form):
    descs = _descs(counts, velocity)
    ens = ob.OceanEnsemble(descs, autotune=False, form=form)
    ens.set_schedule(ob.OceanEnsemble.ONE_LAUNCH)
    for t in (1.5, 8.0, 21.25):
        ens.update(t)
    ens.synchronize()
    first = 0
    for n, count in counts.items():
        for i in {0, count // 2, count - 1}:
            d = descs[first + i]
            for got, want in zip(_read(ens, first + i, d), _want(d, 21.25, form)):
                assert np.array_equal(bits(got), bits(want)), (n, i)
        first += count
    ens.close()


@pytest.mark.parametrize("schedule", [ob.OceanEnsemble.SEQUENTIAL, ob.OceanEnsemble.CONCURRENT])
def test_graph_replay_and_calls_in_turn(schedule):
    # A replay's launches have queue words of their own; calls take turns with
    # theirs. Both in alternation, twice.
    counts = {64: 5, 256: 5, 512: 3}
    descs = _descs(counts, True)
    ens = ob.OceanEnsemble(descs, autotune=False)
    ens.set_schedule(schedule)
    t = 1.0
    for graph in (True, False, True, False):
        ens.set_graph(graph)
        for _ in range(3):
            t += 0.75
            ens.update(t)
        ens.synchronize()
        for i in (0, 4, 7, 12):
            for got, want in zip(_read(ens, i, descs[i]), O.update(descs[i], t)):
                assert np.array_equal(bits(got), bits(want)), (graph, i)
    ens.close()
