// oceanlib-b200: device-side surface queries shared by the query kernels.
//
//   sample_pair       - one ocean's surface at a world position: the
//                       fixed-point displacement inversion and the final
//                       periodic bilinear taps (src/ocean.cpp:322-452);
//   interaction_tap   - the interaction field's (eta, d/dx, d/dz, d/dt) at a
//                       world position, bilinear, zero outside the grid
//                       (src/interaction.cpp:729-770).
// Compiled with -fmad=false like every other kernel, so each product and sum
// rounds as the reference's does.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "spectrum.h"

namespace ocean_b200 {
namespace qdev {

// A query is worked by a pair of neighbouring lanes, 2k and 2k + 1: lane
// parity p loads the two texels (rows z0 and z1) of column x0 + p of the
// bilinear tap and multiplies them by its weights, and the products are
// exchanged by shuffles.
//
// What bounds these kernels is the L1's tag lookups: queries land anywhere,
// so every lane of a 16-byte texel load touches a cache line of its own, and
// the SM looks up about one line a cycle (a million queries of three levels
// are 84 million texel loads: 0.30 ms over 148 SMs; one lane a query measured
// 0.265 ms). A tap's two columns are neighbours in memory, so a pair's two
// loads share a line, which halves the lookups. A tap in the cell of the
// previous inversion step keeps the texels it has (the steps contract, so
// the later ones mostly stay in one cell). A million points, three 256^2
// levels: 266 -> 110 us.
//
// Every sum keeps the reference's order: ((i00 + i10) + i01) + i11.
constexpr int kQueryLanes = 2;

__device__ __forceinline__ float pair_xchg(float v) { return __shfl_xor_sync(0xffffffffu, v, 1); }

// One lane's share of a bilinear tap: its two texels and their weights.
struct PairTap {
    uint32_t i0, i1;  // rows z0 and z1 of the lane's column
    float w0, w1;
};

// Periodic: n is a power of two, so masking wraps negative indices too.
__device__ __forceinline__ PairTap make_tap(float u, float v, uint32_t n, float inv_cell, uint32_t odd)
{
    const float gu = u * inv_cell;
    const float gv = v * inv_cell;
    const float fu = floorf(gu);
    const float fv = floorf(gv);
    const uint32_t x = (static_cast<uint32_t>(__float2int_rz(fu)) + odd) & (n - 1u);
    const uint32_t z0 = static_cast<uint32_t>(__float2int_rz(fv)) & (n - 1u);
    const uint32_t z1 = (z0 + 1u) & (n - 1u);
    const float tu = gu - fu;
    const float tv = gv - fv;
    const float wx = odd ? tu : 1.0f - tu;
    PairTap t;
    t.i0 = z0 * n + x;
    t.i1 = z1 * n + x;
    t.w0 = wx * (1.0f - tv);
    t.w1 = wx * tv;
    return t;
}

// ((even0 + odd0) + even1) + odd1 of the pair's products, in both lanes.
__device__ __forceinline__ float pair_sum(float m0, float m1, uint32_t odd)
{
    const float o0 = pair_xchg(m0), o1 = pair_xchg(m1);
    return ((m0 + o0) + (odd ? o1 : m1)) + (odd ? m1 : o1);
}

// Two of the pair's sums at once: the even lane gets the sum of the `even`
// products, the odd lane that of the `odd_` products.
__device__ __forceinline__ float pair_sum_split(float even0, float even1, float odd0, float odd1, uint32_t odd)
{
    const float o0 = pair_xchg(odd ? even0 : odd0), o1 = pair_xchg(odd ? even1 : odd1);
    const float m0 = odd ? odd0 : even0, m1 = odd ? odd1 : even1;
    return ((m0 + o0) + (odd ? o1 : m1)) + (odd ? m1 : o1);
}

// Where the water of world point p rests: `iters` fixed-point steps of the
// displacement inversion (the reference takes 4, src/ocean.cpp:366), a query
// stopping early once both parameter coordinates move by <= tol (tol = 0:
// never). Leaves the final tap and its displacement texels. Every lane of
// the warp takes part.
struct Inverted {
    PairTap t;
    float4 d0, d1;
};

__device__ __forceinline__ Inverted invert(uint32_t n, float inv_cell, const float4* __restrict__ disp, float2 p,
                                           int iters, float tol, uint32_t odd)
{
    float u = p.x, v = p.y;
    bool done = false;
    Inverted r;
    r.t = make_tap(u, v, n, inv_cell, odd);
    r.d0 = __ldg(&disp[r.t.i0]);
    r.d1 = __ldg(&disp[r.t.i1]);
    for (int it = 0; it < iters; ++it) {
        const float un = p.x - pair_sum(r.d0.x * r.t.w0, r.d1.x * r.t.w1, odd);
        const float vn = p.y - pair_sum(r.d0.z * r.t.w0, r.d1.z * r.t.w1, odd);
        if (!done) {
            done = tol > 0.0f && fabsf(un - u) <= tol && fabsf(vn - v) <= tol;
            u = un;
            v = vn;
            const uint32_t had = r.t.i0;
            r.t = make_tap(u, v, n, inv_cell, odd);
            if (r.t.i0 != had) {
                r.d0 = __ldg(&disp[r.t.i0]);
                r.d1 = __ldg(&disp[r.t.i1]);
            }
        }
        if (tol > 0.0f && __all_sync(0xffffffffu, done)) break;
    }
    return r;
}

// One ocean's surface at world point p (src/ocean.cpp:370-452): the final
// bilinear taps and the renormalised normal. The even lane holds (height,
// offset x, offset z, foam, velocity x), the odd lane (normal x, y, z,
// velocity y, z).
struct PairSurface {
    float v[5];
};

__device__ __forceinline__ PairSurface sample_pair(uint32_t n, float inv_cell, const float4* __restrict__ disp,
                                                   const float4* __restrict__ normal, const float4* __restrict__ vel,
                                                   float2 p, int iters, float tol, uint32_t odd)
{
    const Inverted r = invert(n, inv_cell, disp, p, iters, tol, odd);
    const float w0 = r.t.w0, w1 = r.t.w1;
    const float4 n0 = __ldg(&normal[r.t.i0]), n1 = __ldg(&normal[r.t.i1]);
    float4 v0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v1 = v0;
    if (vel != nullptr) {
        v0 = __ldg(&vel[r.t.i0]);
        v1 = __ldg(&vel[r.t.i1]);
    }
    PairSurface s;
    s.v[0] = pair_sum_split(r.d0.y * w0, r.d1.y * w1, n0.x * w0, n1.x * w1, odd);
    s.v[1] = pair_sum_split(r.d0.x * w0, r.d1.x * w1, n0.y * w0, n1.y * w1, odd);
    s.v[2] = pair_sum_split(r.d0.z * w0, r.d1.z * w1, n0.z * w0, n1.z * w1, odd);
    s.v[3] = pair_sum_split(r.d0.w * w0, r.d1.w * w1, v0.y * w0, v1.y * w1, odd);
    s.v[4] = pair_sum_split(v0.x * w0, v1.x * w1, v0.z * w0, v1.z * w1, odd);
    if (odd) {
        float nx = s.v[0], ny = s.v[1], nz = s.v[2];
        const float len2 = nx * nx + ny * ny + nz * nz;
        if (len2 > 0.0f) {
            const float inv = 1.0f / sqrtf(len2);
            nx *= inv;
            ny *= inv;
            nz *= inv;
        } else {
            nx = 0.0f;
            ny = 1.0f;
            nz = 0.0f;
        }
        s.v[0] = nx;
        s.v[1] = ny;
        s.v[2] = nz;
    }
    if (vel == nullptr) {
        if (odd) s.v[3] = 0.0f;
        s.v[4] = 0.0f;
    }
    return s;
}

// A pair's record (SurfaceEx: height, offset x, z, normal x, y, z, foam,
// velocity x, y, z), each lane its own five floats.
__device__ __forceinline__ void store_surface(SurfaceEx* out, const PairSurface& s, uint32_t odd)
{
    static_assert(sizeof(SurfaceEx) == 10 * sizeof(float), "a record is ten floats");
    float* o = reinterpret_cast<float*>(out) + (odd ? 3 : 0);
    o[0] = s.v[0];
    o[1] = s.v[1];
    o[2] = s.v[2];
    float* q = reinterpret_cast<float*>(out) + (odd ? 8 : 6);
    q[0] = s.v[3];
    q[1] = s.v[4];
}

// Bilinear, zero outside the grid (src/interaction.cpp:729-770).
__device__ __forceinline__ float4 interaction_tap(const float4* __restrict__ out, int n, float cell,
                                                  float origin_x, float origin_z, float wx, float wz,
                                                  bool& inside)
{
    const float gx = (wx - origin_x) / cell - 0.5f;
    const float gz = (wz - origin_z) / cell - 0.5f;
    inside = !(gx < 0.0f || gz < 0.0f || gx >= static_cast<float>(n - 1) ||
               gz >= static_cast<float>(n - 1));
    if (!inside) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int x0 = static_cast<int>(gx);
    const int z0 = static_cast<int>(gz);
    const float tx = gx - static_cast<float>(x0);
    const float tz = gz - static_cast<float>(z0);
    const size_t i00 = static_cast<size_t>(z0) * n + x0;
    const float4 a = out[i00], b = out[i00 + 1], c = out[i00 + n], d = out[i00 + n + 1];
    const float w00 = (1.0f - tx) * (1.0f - tz);
    const float w10 = tx * (1.0f - tz);
    const float w01 = (1.0f - tx) * tz;
    const float w11 = tx * tz;
    return make_float4(a.x * w00 + b.x * w10 + c.x * w01 + d.x * w11,
                       a.y * w00 + b.y * w10 + c.y * w01 + d.y * w11,
                       a.z * w00 + b.z * w10 + c.z * w01 + d.z * w11,
                       a.w * w00 + b.w * w10 + c.w * w01 + d.w * w11);
}

}  // namespace qdev
}  // namespace ocean_b200
