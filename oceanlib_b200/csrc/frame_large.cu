// oceanlib-b200: the frame at N = 2048 and 4096.
//
// The persistent frame kernel (frame.cu) keeps every field of a row pair, or
// of a strip of columns, in one CTA's shared memory. Above N = 1024 that no
// longer fits: six 4096-point sequences alone are 209 KB. These sizes (the
// reference accepts N up to 4096, src/ocean.cpp:28-59) run two passes per
// chunk of oceans instead, through an intermediate that crosses HBM once each
// way (800 MB at 4096 with velocity, beyond the L2):
//
//   rows      two neighbouring rows per task: evolve the rows' cells once
//             (src/core/evolve.cpp:28-184), then field pair by field pair
//             transform the rows and write them to the intermediate;
//   columns   two neighbouring columns per task: field pair by field pair
//             read and transform the columns, then finalize every cell
//             (src/core/evolve.cpp:186-327) into the RGBA32F outputs.
//
// Persistent foam runs every substep as its own launch at these sizes: a
// column strip's foam taps are scattered four-byte reads (4096^2 with velocity
// and foam: 1448 us fused, 1151 us apart).
//
// What bounds a pass is shared memory (capacity and wavefronts) and the phases
// between barriers, so values stay in registers wherever a thread needs them
// again:
//   * A sequence pair (fields 2q and 2q+1, packed f32x2 arithmetic) spans
//     N / 16 lanes of 16 indices each: 4-stage register blocks, and only the
//     two exchanges between the three blocks go through shared memory, real
//     and imaginary parts one after the other in the same 8 bytes per index.
//     The first block takes its values straight from evolve or from global
//     memory (index c + j N/16 in lane c), and the last leaves the same
//     indices in the same lane, straight for the intermediate or finalize.
//   * The evolved amplitudes (rows) and the transformed first field pair
//     (columns) wait for the later pairs in their own thread's slots of
//     shared memory. The velocity pair goes first: nothing of it is needed
//     afterwards.
// The intermediate is inter[ocean][x / 2][pair][y][x & 1], 16 bytes (a.re,
// b.re, a.im, b.im) a cell and pair: a column task's pair is one contiguous
// run, which a bulk prefetch brings into the L2 while the pair before it is
// transformed. Threads 2c and 2c + 1 are lane c of the task's two rows
// (columns), so a warp's stores to the intermediate are 64-byte runs and those
// to the outputs whole 32-byte sectors.
//
// Measured, one ocean with velocity: 4096^2 1618 -> 960 us, 2048^2 376 -> 260 us
// a frame against rows, columns and finalize as three passes that each moved
// every field through HBM; without velocity 1081 -> 667 and 253 -> 190 us;
// the precise form at 4096^2 with velocity 2524 -> 1590 us. What is left at
// 4096^2: FP32 pipe time of about 23k of a task's 63k cycles, exchanges 14k
// (16 warps in one phase), loads from the L2 and stores 12k each. Without the
// output stores 837 us, without the prefetches 1055 us. Keeping the second
// exchange inside a warp by regrouping the lanes (no CTA barrier) was slower
// (978 -> 1063 us): it halves the runs that the rows store.
//
// Evolve, butterflies, twiddles and finalize are the persistent kernel's own
// functions (frame_cells.cuh, ocean_device.cuh), so these sizes match the
// reference bit for bit too.
#include "frame_cells.cuh"
#include "ocean_device.cuh"
#include "spectrum.h"

#include <type_traits>

namespace ocean_b200 {
namespace {

template <int LOG_N>
struct Large {
    static constexpr int N = 1 << LOG_N;
    static constexpr int G = N / 16;                // lanes per sequence pair
    static constexpr int THREADS = 2 * G;           // two rows (columns) per task
    static constexpr int CTAS = 512 / THREADS;      // resident per SM: 128 registers a thread
    static constexpr int TASKS = N / 2;             // per ocean and pass
    static constexpr int SEQ = seq_stride_bytes(N, 16, 2) / 8;  // exchange stride (f32x2)
    static constexpr int HELD = 15;                 // of a thread's 16 cells, those the column stash holds
    static constexpr int BUF = 2 * SEQ;
    static constexpr size_t EXCHANGE = sizeof(f32x2) * BUF;
    static constexpr size_t TWIDDLES = sizeof(float2) * N;
    static constexpr size_t ROW_SMEM = EXCHANGE + TWIDDLES + (sizeof(float2) + sizeof(float)) * 16 * THREADS + sizeof(float) * N;
    static constexpr size_t COL_SMEM = EXCHANGE + TWIDDLES + sizeof(float4) * HELD * THREADS;
    static_assert((COL_SMEM + 1024) * CTAS <= 228 * 1024 && COL_SMEM <= 227 * 1024, "the column CTAs fit on an SM");
    static_assert((ROW_SMEM + 1024) * CTAS <= 228 * 1024 && ROW_SMEM <= 227 * 1024, "the row CTAs fit on an SM");
};

// A thread's place: row (column) r of the task's two, lane c of its pair, and
// that row's exchange buffer.
template <int LOG_N>
struct Place {
    int r, c;
    f32x2* buf;

    __device__ __forceinline__ explicit Place(void* smem)
        : r(threadIdx.x & 1), c(threadIdx.x >> 1), buf(static_cast<f32x2*>(smem) + r * Large<LOG_N>::SEQ)
    {
    }
};

// Brings `bytes` (a multiple of 16 KB) at `p` into the L2: threads
// [first, first + bytes / 16 KB) of the CTA take a piece each.
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned bytes, int first)
{
    constexpr unsigned kPiece = 16384;
    const unsigned k = threadIdx.x - first;
    if (k < bytes / kPiece)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(static_cast<const char*>(p) + k * kPiece),
                     "r"(kPiece)
                     : "memory");
}

template <int LOG_N>
__device__ __forceinline__ void load_twiddles(float2* tws, const float2* __restrict__ src)
{
    for (int i = threadIdx.x; i < Large<LOG_N>::N - 1; i += Large<LOG_N>::THREADS) tws[i] = __ldg(&src[i]);
}

template <int LOG_N, int NF, int AR>
__global__ void __launch_bounds__(Large<LOG_N>::THREADS, Large<LOG_N>::CTAS) large_row_kernel(FrameArgs a)
{
    using S = Large<LOG_N>;
    using Fft = RegFft<LOG_N, 16, AR>;
    constexpr int N = S::N, G = S::G, Q = NF / 2, NT = S::THREADS;
    extern __shared__ float4 smem4[];
    const int tid = threadIdx.x;
    const Place<LOG_N> p(smem4);
    float2* tws = reinterpret_cast<float2*>(smem4) + S::BUF;
    float* kv = reinterpret_cast<float*>(tws + N);
    float2* held_h = reinterpret_cast<float2*>(kv + N) + tid;                   // (hr, hi) of cell j at [j * NT]
    float* held_k = reinterpret_cast<float*>(held_h - tid + 16 * NT) + tid;     // its 1/|k|
    load_twiddles<LOG_N>(tws, a.twiddles);

    const size_t cells = static_cast<size_t>(N) * N;
    const int tasks = S::TASKS * a.chunk;
    // Task t's rows are y and y + 1. Rows 2k, 2k + 1 and the rows with their
    // mirrors are neighbouring tasks, which share what the L2 fetched.
    auto first_row = [](int t) { return 2 * ((t & 1) ? S::TASKS - 1 - (t >> 1) : (t >> 1)); };
    int kv_of = -1;
#pragma unroll 1
    for (int task = blockIdx.x; task < tasks; task += gridDim.x) {
        const int o = task / S::TASKS;
        const int y = first_row(task % S::TASKS) + p.r;
        const int ocean = a.ocean_base + o;
        const int geom_of = a.consts[ocean].geom;
        const float2* h0 = a.h0 + static_cast<size_t>(ocean) * cells;
        const float2* h0_row = h0 + static_cast<size_t>(y) * N;
        const float2* h0_mirror = h0 + static_cast<size_t>((N - y) & (N - 1)) * N;
        const float2* geom = a.omega_kinv + static_cast<size_t>(geom_of) * cells + static_cast<size_t>(y) * N;
        if (geom_of != kv_of) {
            __syncthreads();  // the table's last readers are done
            for (int i = tid; i < N; i += NT) kv[i] = __ldg(&a.kvec[static_cast<size_t>(geom_of) * N + i]);
            __syncthreads();
            kv_of = geom_of;
        }
        const float kz = kv[y];
        const double top = frame_time(a, ocean);
        ulonglong2* out = reinterpret_cast<ulonglong2*>(a.inter + static_cast<size_t>(o) * NF * cells) + 2 * y;
#pragma unroll 1
        for (int k = 0; k < Q; ++k) {
            const int q = Q == 3 ? (k + 2) % 3 : k;  // the velocity pair first
            f32x2 re[16], im[16];
            if (k == 0) {
                // Every cell's loads before the first is evolved: 96 registers
                // that the fields then take over.
                float2 av[16], bm[16], wks[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int x = p.c + G * j;
                    av[j] = load_now(&h0_row[x]);
                    bm[j] = load_now(&h0_mirror[(N - x) & (N - 1)]);
                    wks[j] = load_now(&geom[x]);
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int x = p.c + G * j;
                    const float2 wk = wks[j];
                    const Amplitude e = evolve_amplitude(av[j], bm[j], wk.x, top);
                    held_h[j * NT] = make_float2(e.hr, e.hi);
                    held_k[j * NT] = wk.y;
                    float2 pa, pb;
                    if constexpr (Q == 3) {
                        evolve_pair2(e.dr, e.di, wk.x, wk.y, kv[x], kz, pa, pb);
                    } else {
                        evolve_pair0(e.hr, e.hi, wk.y, kv[x], kz, pa, pb);
                    }
                    re[j] = px_pack(pa.x, pb.x);
                    im[j] = px_pack(pa.y, pb.y);
                }
                // The next task's rows while this one's are transformed.
                if (task + static_cast<int>(gridDim.x) < tasks) {
                    const int next = task + gridDim.x, no = a.ocean_base + next / S::TASKS;
                    const int ny = first_row(next % S::TASKS);
                    const float2* nh = a.h0 + static_cast<size_t>(no) * cells;
                    const float2* ng = a.omega_kinv + static_cast<size_t>(a.consts[no].geom) * cells;
                    constexpr unsigned kRows = 2u * N * sizeof(float2);
                    prefetch_l2(nh + static_cast<size_t>(ny) * N, kRows, 0);
                    prefetch_l2(ng + static_cast<size_t>(ny) * N, kRows, 32);
                    // Rows N - y - 1 and N - y; row N - 1 alone for y = 0.
                    prefetch_l2(nh + static_cast<size_t>(N - ny - 1) * N, ny == 0 ? kRows / 2 : kRows, 64);
                }
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float kx = kv[p.c + G * j];
                    const float2 h = held_h[j * NT];
                    const float ki = held_k[j * NT];
                    float2 pa, pb;
                    if (Q == 3 && q == 0) {
                        evolve_pair0(h.x, h.y, ki, kx, kz, pa, pb);
                    } else {
                        evolve_pair1(h.x, h.y, ki, kx, kz, pa, pb);
                    }
                    re[j] = px_pack(pa.x, pb.x);
                    im[j] = px_pack(pa.y, pb.y);
                }
            }
            Fft::run(re, im, p.buf, tws, p.c);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int x = Fft::index(j, p.c);
                out[(static_cast<size_t>(x >> 1) * Q + q) * 2 * N + (x & 1)] = make_ulonglong2(re[j], im[j]);
            }
        }
    }
}

template <int LOG_N, int NF, int AR>
__global__ void __launch_bounds__(Large<LOG_N>::THREADS, Large<LOG_N>::CTAS) large_col_kernel(FrameArgs a)
{
    using S = Large<LOG_N>;
    using Fft = RegFft<LOG_N, 16, AR>;
    constexpr int N = S::N, Q = NF / 2, NT = S::THREADS;
    constexpr unsigned kPairBytes = 2u * N * sizeof(float4);  // a task's pair
    extern __shared__ float4 smem4[];
    const int tid = threadIdx.x;
    const Place<LOG_N> p(smem4);
    float2* tws = reinterpret_cast<float2*>(smem4) + S::BUF;
    ulonglong2* held = reinterpret_cast<ulonglong2*>(tws + N) + tid;  // pair 0 of cell j at [j * NT]
    load_twiddles<LOG_N>(tws, a.twiddles);
    __syncthreads();

    const size_t cells = static_cast<size_t>(N) * N;
    const int tasks = S::TASKS * a.chunk;
    // Pair q of a task's two columns; the chunk's oceans follow each other.
    auto pair_at = [&](int task, int q) {
        return reinterpret_cast<const float4*>(a.inter) + (static_cast<size_t>(task) * Q + q) * 2 * N;
    };
#pragma unroll 1
    for (int task = blockIdx.x; task < tasks; task += gridDim.x) {
        ulonglong2 last;  // pair 0 of the 16th cell
#pragma unroll 1
        for (int k = 0; k < Q; ++k) {
            // The velocity pair first, the pair that completes the cell last.
            const int q = Q == 3 ? (k + 2) % 3 : k;
            if (k + 1 < Q) {
                prefetch_l2(pair_at(task, Q == 3 ? k : k + 1), kPairBytes, 0);
            } else if (task + static_cast<int>(gridDim.x) < tasks) {
                prefetch_l2(pair_at(task + gridDim.x, Q == 3 ? 2 : 0), kPairBytes, 0);
            }
            const float4* src = pair_at(task, q) + tid;
            f32x2 re[16], im[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float4 v = __ldcs(src + NT * j);
                re[j] = px_pack(v.x, v.y);
                im[j] = px_pack(v.z, v.w);
            }
            Fft::run(re, im, p.buf, tws, p.c);
            const int ocean = a.ocean_base + task / S::TASKS;
            const size_t base = static_cast<size_t>(ocean) * cells + 2 * (task % S::TASKS) + p.r;
            if (Q == 3 && q == 2) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float ux, uz, uy, zero;
                    px_unpack(re[j], ux, uz);
                    px_unpack(im[j], uy, zero);
                    __stcs(&a.velocity[base + static_cast<size_t>(Fft::index(j, p.c)) * N], make_float4(ux, uy, uz, 0.0f));
                }
            } else if (q == 0) {
#pragma unroll
                for (int j = 0; j < S::HELD; ++j) held[j * NT] = make_ulonglong2(re[j], im[j]);
                last = make_ulonglong2(re[15], im[15]);
            } else {
                const OceanConsts cst = a.consts[ocean];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const ulonglong2 h = j < S::HELD ? held[j * NT] : last;
                    float2 f0, f1, f2, f3;
                    px_unpack(h.x, f0.x, f1.x);
                    px_unpack(h.y, f0.y, f1.y);
                    px_unpack(re[j], f2.x, f3.x);
                    px_unpack(im[j], f2.y, f3.y);
                    const CellOut c = finalize_cell(f0, f1, f2, f3, cst.lambda, cst.foam_threshold, cst.inv_threshold);
                    const size_t idx = base + static_cast<size_t>(Fft::index(j, p.c)) * N;
                    __stcs(&a.disp[idx], c.disp);
                    __stcs(&a.normal[idx], c.normal);
                }
            }
        }
    }
}

template <typename Kernel>
cudaError_t launch(Kernel k, int tasks, int threads, int ctas, size_t smem, const FrameArgs& a, cudaStream_t st)
{
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    int dev = 0, sms = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // One wave of CTAs, each walking over tasks: a twiddle table load serves them all.
    const int grid = tasks < sms * ctas ? tasks : sms * ctas;
    k<<<grid, threads, smem, st>>>(a);
    return cudaGetLastError();
}

template <int LOG_N, int NF, int AR>
cudaError_t rows_launch(const FrameArgs& a, cudaStream_t st)
{
    using S = Large<LOG_N>;
    return launch(large_row_kernel<LOG_N, NF, AR>, S::TASKS * a.chunk, S::THREADS, S::CTAS, S::ROW_SMEM, a, st);
}

template <int LOG_N, int NF, int AR>
cudaError_t cols_launch(const FrameArgs& a, cudaStream_t st)
{
    using S = Large<LOG_N>;
    return launch(large_col_kernel<LOG_N, NF, AR>, S::TASKS * a.chunk, S::THREADS, S::CTAS, S::COL_SMEM, a, st);
}

// The arithmetic `ar` (kArExact, kArFast, kArPrecise) as a compile-time
// constant for `fn`.
template <typename Fn>
cudaError_t with_arith(int ar, Fn&& fn)
{
    if (ar == kArFast) return fn(std::integral_constant<int, kArFast>{});
    if (ar == kArPrecise) return fn(std::integral_constant<int, kArPrecise>{});
    return fn(std::integral_constant<int, kArExact>{});
}

template <int LOG_N>
cudaError_t rows_n(int nf, int ar, const FrameArgs& a, cudaStream_t st)
{
    return with_arith(ar, [&](auto A) {
        constexpr int AR = decltype(A)::value;
        return nf == 4 ? rows_launch<LOG_N, 4, AR>(a, st) : rows_launch<LOG_N, 6, AR>(a, st);
    });
}

template <int LOG_N>
cudaError_t cols_n(int nf, int ar, const FrameArgs& a, cudaStream_t st)
{
    return with_arith(ar, [&](auto A) {
        constexpr int AR = decltype(A)::value;
        return nf == 4 ? cols_launch<LOG_N, 4, AR>(a, st) : cols_launch<LOG_N, 6, AR>(a, st);
    });
}

}  // namespace

cudaError_t launch_large_rows(int log_n, int nf, int ar, const FrameArgs& a, cudaStream_t st)
{
    if (nf != 4 && nf != 6) return cudaErrorInvalidValue;
    switch (log_n) {
        case 11: return rows_n<11>(nf, ar, a, st);
        case 12: return rows_n<12>(nf, ar, a, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_large_cols(int log_n, int nf, int ar, const FrameArgs& a, cudaStream_t st)
{
    if (nf != 4 && nf != 6) return cudaErrorInvalidValue;
    switch (log_n) {
        case 11: return cols_n<11>(nf, ar, a, st);
        case 12: return cols_n<12>(nf, ar, a, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ocean_b200
