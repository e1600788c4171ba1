"""The ensemble's autotuner also times the concurrent schedule with the sizes'
default plans, replayed as use replays it, and whatever it keeps runs with the
same bits."""
import numpy as np
import pytest

import oceanlib_b200 as ob
import oracle as O
from oceanlib_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _device(cuda_device):
    ob.force_simd_level(None)
    yield


def _descs(sizes, velocity):
    return [ob.OceanDesc(size=n, patch_length=1.5 * n, wind_speed=8.0 + i % 9, choppiness=1.0, seed=70 + i,
                         compute_velocity=velocity) for i, n in enumerate(sizes)]


@pytest.mark.parametrize("sizes,velocity,form", [
    ([64] * 8 + [256] * 8 + [512] * 4, False, abi.OCEAN_FFT_PRECISE),
    ([128] * 6 + [256] * 3, False, abi.OCEAN_FFT_EXACT),
    ([32] * 3 + [512, 1024], True, abi.OCEAN_FFT_EXACT)])
def test_default_plans_are_a_candidate(sizes, velocity, form):
    descs = _descs(sizes, velocity)
    for _ in range(3):
        ens = ob.OceanEnsemble(descs, autotune=True, form=form)
        assert "default plans" in ens.schedule
        # As the pick they are the concurrent schedule, with no plans of the sizes' own to name.
        if "default plans (" in ens.schedule:
            assert ens.schedule_kind == ob.OceanEnsemble.CONCURRENT and "task plans" not in ens.schedule
        else:
            assert "task plans" in ens.schedule
        for t in (1.0, 3.25):
            ens.update(t)
        ens.synchronize()
        for i in (0, len(sizes) // 2, len(sizes) - 1):
            got = ens.read(i)
            if form == abi.OCEAN_FFT_EXACT:
                want = O.update(descs[i], 3.25)
            else:
                alone = ob.OceanBatch([descs[i]], form=form)
                want = [np.empty((sizes[i] * sizes[i], 4), np.float32) for _ in range(2)]
                alone.update_host([3.25], 0.0, *want)
                alone.close()
            for a, w in zip(got, want):
                a = np.ascontiguousarray(a).view(np.uint32).reshape(-1)
                assert np.array_equal(a, np.ascontiguousarray(w).view(np.uint32).reshape(-1)), i
        ens.close()
