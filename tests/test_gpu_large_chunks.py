"""Sizes above 1024 walk one wave of CTAs over the tasks of a whole chunk:
oceans of different patches in one chunk (the wavenumber table changes between
tasks), a last chunk that is not full, both field counts, and the precise form,
whose sequences go one after the other."""
import numpy as np
import pytest

import oceanlib_b200 as ob
import oracle as O
from oceanlib_b200 import abi

pytestmark = pytest.mark.gpu
N = 2048


def frame(descs, form, chunk, velocity, t):
    cells = N * N
    out = [np.empty((len(descs) * cells, 4), np.float32) for _ in range(3 if velocity else 2)]
    batch = ob.OceanBatch(descs, form=form, chunk=chunk)
    batch.update_host([t], 0.0, *out)
    batch.close()
    return out


def oceans(velocity):
    return [ob.OceanDesc(size=N, patch_length=length, wind_speed=14.0, wind_direction=0.3 * i, choppiness=1.2,
                         seed=90 + i, compute_velocity=velocity) for i, length in enumerate((600.0, 410.0, 600.0))]


@pytest.mark.parametrize("velocity", [False, True])
def test_chunks_of_mixed_patches_match_the_oracle(cuda_device, velocity):
    ob.force_simd_level(None)
    descs = oceans(velocity)
    got = frame(descs, abi.OCEAN_FFT_EXACT, 2, velocity, 6.75)
    for i, d in enumerate(descs):
        for g, want in zip(got, O.update(d, 6.75)):
            assert np.array_equal(g[i * N * N:(i + 1) * N * N].view(np.uint32), want.view(np.uint32)), (i, velocity)


@pytest.mark.parametrize("form", [abi.OCEAN_FFT_PRECISE, abi.OCEAN_FFT_FAST])
def test_chunking_does_not_change_a_form(cuda_device, form):
    descs = oceans(True)
    whole = frame(descs, form, 3, True, 6.75)
    for i, d in enumerate(descs):
        for g, alone in zip(whole, frame([d], form, 1, True, 6.75)):
            assert np.array_equal(g[i * N * N:(i + 1) * N * N].view(np.uint32), alone.view(np.uint32)), i
