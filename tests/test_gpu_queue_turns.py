"""The persistent launches' queue words take turns (each launch zeroes the next
one's) and a captured launch has words of its own: frames in plain streams,
graph replays in a row and frames after them, one time for all oceans and a
time per ocean, all give the oracle's bits."""
import numpy as np
import pytest

import oceanlib_b200 as ob
import oracle as O

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def read(buffers, n):
    out = []
    for ptr in (buffers.displacement, buffers.normal):
        a = np.empty((n * n, 4), np.float32)
        assert ob.lib().ocean_copy_to_host(a.ctypes.data, ptr, a.nbytes) == 0
        out.append(a)
    return out


def check(get, descs, times):
    for i, (d, t) in enumerate(zip(descs, times)):
        for got, want in zip(read(get(i), d.size), O.update(d, t)):
            assert np.array_equal(bits(got), bits(want)), (i, t)


@pytest.mark.parametrize("count", [1, 5])
@pytest.mark.parametrize("kind", ["batch", "ensemble"])
def test_turns_and_replays(cuda_device, kind, count):
    torch = pytest.importorskip("torch")
    ob.force_simd_level(None)
    sizes = [32, 64, 32, 128, 64] if kind == "ensemble" else [64] * 5
    descs = [ob.OceanDesc(size=sizes[i], patch_length=90.0 + i, wind_speed=13.0, seed=i) for i in range(count)]
    if kind == "batch":
        obj = ob.OceanBatch(descs)
    else:
        obj = ob.OceanEnsemble(descs, autotune=False)
        obj.set_schedule(obj.ONE_LAUNCH)
    stream = torch.cuda.Stream()
    for k in range(3):
        obj.update(1.0 + k, stream=stream.cuda_stream)
    torch.cuda.synchronize()
    check(obj.device_buffers, descs, [3.0] * count)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        obj.update(4.5, stream=torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    check(obj.device_buffers, descs, [4.5] * count)
    obj.update(5.25)
    obj.synchronize()
    check(obj.device_buffers, descs, [5.25] * count)
    graph.replay()
    torch.cuda.synchronize()
    check(obj.device_buffers, descs, [4.5] * count)
    if kind == "batch" and count > 1:
        times = [0.5 * i for i in range(count)]
        obj.update(times)
        obj.update(times)
        obj.synchronize()
        check(obj.device_buffers, descs, times)
    del graph
