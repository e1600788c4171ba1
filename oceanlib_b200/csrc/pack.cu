// oceanlib-b200: RGBA16F packing of the RGBA32F outputs on the device.
//
// The reference's viewer narrows every output to half floats before the
// upload, and substitutes the persistent foam for the displacement's alpha
// during the same pass (examples/viewer/half.hpp:58-125,
// examples/viewer/ocean_view.cpp:830-862). Here the same conversion runs on
// the GPU, so a host that wants half floats copies half the bytes.
// Rounding: IEEE round-to-nearest-even, overflow to infinity, NaN kept as a
// quiet NaN (sign | 0x7E00) - the reference's float_to_half, bit for bit.
#include <cuda_fp16.h>
#include <cstdint>

#include "spectrum.h"

namespace ocean_b200 {
namespace {

__device__ __forceinline__ uint16_t to_half(float v)
{
    if (isnan(v)) return static_cast<uint16_t>(((__float_as_uint(v) >> 16) & 0x8000u) | 0x7E00u);
    return __half_as_ushort(__float2half_rn(v));
}

// One texel per thread: RGB from src, A from alpha (or src's own A).
__global__ void pack_rgba16_kernel(const float4* __restrict__ src, const float* __restrict__ alpha,
                                   uint64_t cells, ushort4* __restrict__ dst)
{
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= cells) return;
    const float4 v = __ldcs(&src[i]);
    const float a = alpha != nullptr ? __ldcs(&alpha[i]) : v.w;
    __stcs(&dst[i], make_ushort4(to_half(v.x), to_half(v.y), to_half(v.z), to_half(a)));
}

// One output texel per thread and step, from the L2 to pinned host memory over
// PCIe. What bounds it is PCIe (51 GB/s of writes); what it saves is the hand-
// over to a copy engine and back.
__global__ void mirror_kernel(const float4* __restrict__ src, size_t n, float4* __restrict__ dst)
{
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x)
        __stcs(&dst[i], __ldcg(&src[i]));
}

}  // namespace

// Up to 768 KiB the kernel's stores are in host memory before a copy engine's
// are (one ocean's update with its mirror, with velocity: 16^2 28.9 -> 21.2 us,
// 64^2 30.6 -> 27.0, 128^2 40.3 -> 39.7); beyond, the engine's 55 GB/s win (256^2
// without velocity, 2 MiB: 63.4 us against 65.3). A field's one plane stays with
// the engine: 64^2 48.2 us against 49.5, 256^2 66.5 against 68.4.
cudaError_t launch_mirror(const float4* src, size_t n, float4* pinned, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (n * sizeof(float4) > (768u << 10))
        return cudaMemcpyAsync(pinned, src, n * sizeof(float4), cudaMemcpyDeviceToHost, st);
    const size_t blocks = (n + 255) / 256;
    mirror_kernel<<<static_cast<unsigned>(blocks < 592 ? blocks : 592), 256, 0, st>>>(src, n, pinned);
    return cudaGetLastError();
}

cudaError_t launch_pack_rgba16(const float4* src, const float* alpha, uint64_t cells, ushort4* dst,
                               cudaStream_t st)
{
    if (cells == 0) return cudaSuccess;
    const unsigned blocks = static_cast<unsigned>((cells + 255) / 256);
    pack_rgba16_kernel<<<blocks, 256, 0, st>>>(src, alpha, cells, dst);
    return cudaGetLastError();
}

}  // namespace ocean_b200
