// oceanlib-b200: world queries of one ocean and of a cascade
// (src/ocean.cpp:322-452, src/cascade.cpp:82-153): one launch for any number
// of points, a pair of lanes a point (query_device.cuh).
#include "query_device.cuh"
#include "spectrum.h"

namespace ocean_b200 {
namespace {

constexpr int kThreads = 256;
constexpr int kPointsPerBlock = kThreads / qdev::kQueryLanes;

// This lane's point (the last one for the lanes past the end, which work
// along so that the warp's shuffles are whole) and whether it is its own.
__device__ __forceinline__ bool my_point(uint64_t count, uint64_t& i)
{
    i = static_cast<uint64_t>(blockIdx.x) * kPointsPerBlock + threadIdx.x / qdev::kQueryLanes;
    const bool mine = i < count;
    if (!mine) i = count - 1;
    return mine;
}

__global__ void __launch_bounds__(kThreads)
sample_kernel(int n, float inv_cell, const float4* __restrict__ disp, const float4* __restrict__ normal,
              const float4* __restrict__ vel, const float2* __restrict__ xz, uint64_t count,
              SurfaceEx* __restrict__ out)
{
    uint64_t i;
    const bool mine = my_point(count, i);
    const uint32_t odd = threadIdx.x & 1u;
    const qdev::PairSurface s = qdev::sample_pair(static_cast<uint32_t>(n), inv_cell, disp, normal, vel, xz[i], 4, 0.0f,
                                                  odd);
    if (mine) qdev::store_surface(out + i, s, odd);
}

// Summed surface of several cascade levels (src/cascade.cpp:82-153): height,
// offsets and velocity add exactly; normals add then renormalise; foam
// combines as 1 - prod(1 - foam_i). Levels are visited in order, so the float
// sums round as the reference's loop does.
__global__ void __launch_bounds__(kThreads)
cascade_sample_kernel(const __grid_constant__ CascadeLevels lv, const float2* __restrict__ xz, uint64_t count,
                      SurfaceEx* __restrict__ out, int iters, float tol)
{
    uint64_t i;
    const bool mine = my_point(count, i);
    const uint32_t odd = threadIdx.x & 1u;
    const float2 p = xz[i];
    qdev::PairSurface o{};
    float transparency = 1.0f;
    for (int l = 0; l < lv.count; ++l) {
        const LevelView& L = lv.level[l];
        const qdev::PairSurface s = qdev::sample_pair(static_cast<uint32_t>(L.n), L.inv_cell, L.disp, L.normal,
                                                      L.velocity, p, iters, tol, odd);
        o.v[0] += s.v[0];
        o.v[1] += s.v[1];
        o.v[2] += s.v[2];
        if (odd)
            o.v[3] += s.v[3];
        else
            transparency *= (1.0f - s.v[3]);
        o.v[4] += s.v[4];
    }
    if (odd) {
        const float nx = o.v[0], ny = o.v[1], nz = o.v[2];
        const float len2 = nx * nx + ny * ny + nz * nz;
        if (len2 > 0.0f) {
            const float inv = 1.0f / sqrtf(len2);
            o.v[0] = nx * inv;
            o.v[1] = ny * inv;
            o.v[2] = nz * inv;
        } else {
            o.v[0] = 0.0f;
            o.v[1] = 1.0f;
            o.v[2] = 0.0f;
        }
    } else {
        o.v[3] = 1.0f - transparency;
    }
    if (mine) qdev::store_surface(out + i, o, odd);
}

unsigned blocks_for(uint64_t count) { return static_cast<unsigned>((count + kPointsPerBlock - 1) / kPointsPerBlock); }

}  // namespace

cudaError_t launch_cascade_sample(const CascadeLevels& levels, const float2* xz, uint64_t count, SurfaceEx* out,
                                  int iters, float tol, cudaStream_t stream)
{
    if (count == 0) return cudaSuccess;
    cascade_sample_kernel<<<blocks_for(count), kThreads, 0, stream>>>(levels, xz, count, out, iters, tol);
    return cudaGetLastError();
}

cudaError_t launch_sample(int n, float inv_cell, const float4* disp, const float4* normal, const float4* velocity,
                          const float2* xz, uint64_t count, SurfaceEx* out, cudaStream_t stream)
{
    if (count == 0) return cudaSuccess;
    sample_kernel<<<blocks_for(count), kThreads, 0, stream>>>(n, inv_cell, disp, normal, velocity, xz, count, out);
    return cudaGetLastError();
}

}  // namespace ocean_b200
