// oceanlib-b200: the persistent frame with its transforms in registers.
//
// The same frame, queue protocol and arithmetic as frame_kernel (frame.cu), for
// the batches where it is the faster one (pair_frame_ok). There, a task's every
// field sat in shared memory and each step of the frame - evolve, three stage
// blocks, the store - read and wrote all of it: the shared-memory pipe was the
// frame's busiest unit (71% of 64 x 512^2 with velocity and foam). Here a task
// takes ROWS neighbouring rows (columns) through the field pairs one after the
// other, E indices of a pair a lane, and a value passes through shared memory
// only between two stage blocks:
//
//   rows     evolve straight into the first block's registers; the last block's
//            registers go to the intermediate. The evolved amplitudes and 1/|k|
//            wait in the thread's own shared memory for the later pairs; the
//            velocity pair, which needs more of the cell, goes first.
//   columns  the first block reads the intermediate; the last block's registers
//            are finalized and stored. The first pair waits in the thread's own
//            shared memory until the second completes the cell; the velocity
//            pair goes last, with the foam step, which needs the cell's foam
//            source (kept in the same place) and velocity.
//
// Neighbouring threads are the same lane of the task's ROWS rows (columns), and
// the intermediate is inter[x / ROWS][pair][y][x % ROWS], 16 bytes (a.re, b.re,
// a.im, b.im) a cell and pair: a warp reads it in whole 512-byte runs, writes it
// in runs of ROWS^2 x 16 bytes and writes the outputs in runs of ROWS x 16.
//
// A resident wave of CTAs holds several oceans' worth of tasks (3.5 at 512^2, 222
// at 64^2). So that a column task does not wait for rows still in flight, nor a
// row task for its ring slot, the queue runs the rows `ahead` oceans before the
// columns, R(0) .. R(ahead - 1) | R(ahead) C(0) | R(ahead + 1) C(1) | .. |
// C(count - 1), with ahead = that many oceans and a ring of twice as many slots.
// (frame_kernel's ring of three keeps a large batch of small oceans to a few
// CTAs.) Every awaited task holds an earlier ticket, as in frame_kernel, since
// the ring has more slots than rows run ahead. 64 x 512^2 with velocity, us a
// frame by (ahead, ring): (2, 4) 983, (2, 5) 810, (3, 6) 740, (3, 7) 715,
// (4, 8) 672, (5, 10) 664.
#include "frame_cells.cuh"
#include "ocean_device.cuh"
#include "queue_device.cuh"
#include "spectrum.h"

#include <type_traits>

namespace ocean_b200 {
namespace {

// E indices of a pair a lane, ROWS rows (columns) a task.
template <int LOG_N_, int E_, int ROWS_>
struct RegPlan {
    static constexpr int LOG_N = LOG_N_, N = 1 << LOG_N, E = E_, ROWS = ROWS_;
    static constexpr int G = N / E;             // lanes per pair
    static constexpr int T = ROWS * G;          // threads
    static constexpr int CTAS = (E == 16 ? 512 : 768) / T;  // resident per SM: 128 or 80 registers a thread
    static constexpr int TASKS = N / ROWS;      // per ocean, rows and columns alike
    static constexpr int SEQ = seq_stride_bytes(N, E, ROWS);
    // Shared memory, in bytes from the start: exchange buffers, twiddles, the
    // threads' own values (16 bytes a cell in a column task).
    static constexpr size_t TW = ROWS * SEQ;
    static constexpr size_t HELD = TW + sizeof(float2) * N;
    static constexpr size_t SMEM = HELD + sizeof(float4) * E * T;
    // Oceans that the rows run ahead of the columns and slots of the ring, at
    // q.slots = slots (see above). From a B200's 148 SMs: on a part of one the
    // rows run further ahead than its wave, with the same results.
    static constexpr int WAVE = (148 * CTAS + TASKS - 1) / TASKS;  // oceans' worth of tasks on the GPU
    static constexpr int IN_FLIGHT = WAVE > 2 ? WAVE : 2;
    __host__ __device__ static constexpr unsigned ahead(unsigned slots)
    {
        return slots >= 3 ? IN_FLIGHT : (IN_FLIGHT + 1) / 2;
    }
    __host__ __device__ static constexpr unsigned ring(unsigned slots) { return 2 * ahead(slots) + (slots >= 3 ? 0 : 1); }
    static_assert(E * T == ROWS * N && TW % 16 == 0 && HELD % 16 == 0, "a thread holds E cells");
    static_assert(CTAS * (SMEM + 1280) <= 228 * 1024, "the resident CTAs fit on an SM");
};
// Eight indices a lane (80 registers); a task takes as many rows as 128 threads
// hold, but at least two (1024^2), and four with foam at 512^2: two columns' foam
// is 8 bytes a row (64 oceans: 829 us against 745; without foam four rows cost
// 670 against 651). The precise form rounds where a stage block ends, so it
// keeps the blocks it always had: 3 + 3 + .. stages at N = 32, 64 and 512, 4 + 3
// and 4 + 4 (16 indices a lane) at 128 and 256, and at 1024, whose blocks of
// five would take 32 indices a lane, and 16, one block of four, frame_kernel.
template <int LOG_N, int AR, bool FOAM>
struct PairPlanOf {
    static constexpr int E = AR == kArPrecise && (LOG_N == 7 || LOG_N == 8) ? 16 : 8;
    static constexpr int T = LOG_N == 4 ? 32 : (LOG_N == 10 || (LOG_N == 9 && FOAM) ? 256 : 128);
    using type = RegPlan<LOG_N, E, T * E / (1 << LOG_N)>;
};
template <int LOG_N, int AR, bool FOAM>
using PairPlan = typename PairPlanOf<LOG_N, AR, FOAM>::type;

// A task's areas of shared memory: exchange buffers, the size's twiddles, the
// threads' own values (16 bytes a cell in a column task).
struct Shared {
    unsigned char* exchange;
    const float2* tw;
    unsigned char* held;
};

// Adds this CTA's finished row task (pub[0]) or its own column task (pub[1]).
__device__ __forceinline__ void publish(unsigned* counter, int tid)
{
    if (tid == 0 && counter != nullptr) red_release_add(counter, 1u);
}

template <class P, int NF, int AR>
__device__ __forceinline__ void pair_row_task(const FrameArgs& a, int ocean, int task, float2* inter_slot,
                                              const Shared& sh, int tid, unsigned* const* pub)
{
    using Fft = RegFft<P::LOG_N, P::E, AR>;
    constexpr int N = P::N, G = P::G, E = P::E, ROWS = P::ROWS, T = P::T, Q = NF / 2;
    const int r = tid % ROWS, c = tid / ROWS;
    void* buf = sh.exchange + r * P::SEQ;
    float2* held_h = reinterpret_cast<float2*>(sh.held) + tid;                         // (hr, hi) of cell j at [j * T]
    float* held_k = reinterpret_cast<float*>(sh.held + sizeof(float2) * E * T) + tid;  // its 1/|k|

    // Rows and the rows with their mirrors are neighbouring tasks: the second
    // read of h0 finds it in the L2.
    const int y = ROWS * ((task & 1) ? P::TASKS - 1 - (task >> 1) : (task >> 1)) + r;
    const float2 *geom, *h0;
    const float* kvec;
    if (a.table != nullptr) {
        const OceanSlot& s = a.table[ocean];
        geom = s.omega_kinv;
        kvec = s.kvec;
        h0 = s.h0;
    } else {
        const int g = a.consts[ocean].geom;
        geom = a.omega_kinv + static_cast<size_t>(g) * N * N;
        kvec = a.kvec + static_cast<size_t>(g) * N;
        h0 = a.h0 + static_cast<size_t>(ocean) * N * N;
    }
    const double top = frame_time(a, ocean);
    const float kz = __ldg(&kvec[y]);
    const float2* h0_row = h0 + y * N;
    const float2* h0_mirror = h0 + ((N - y) & (N - 1)) * N;
    geom += y * N;
    ulonglong2* out = reinterpret_cast<ulonglong2*>(inter_slot) + y * ROWS;
#pragma unroll 1
    for (int k = 0; k < Q; ++k) {
        const int q = Q == 3 ? (k + 2) % 3 : k;  // the velocity pair first
        f32x2 re[E], im[E];
        if (k == 0) {
            float2 av[E], bm[E], wk[E];
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int x = c + G * j;
                av[j] = load_now(&h0_row[x]);
                bm[j] = load_now(&h0_mirror[(N - x) & (N - 1)]);
                wk[j] = load_now(&geom[x]);
            }
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const float kx = __ldg(&kvec[c + G * j]);
                const Amplitude e = evolve_amplitude(av[j], bm[j], wk[j].x, top);
                held_h[j * T] = make_float2(e.hr, e.hi);
                held_k[j * T] = wk[j].y;
                float2 pa, pb;
                if constexpr (Q == 3) {
                    evolve_pair2(e.dr, e.di, wk[j].x, wk[j].y, kx, kz, pa, pb);
                } else {
                    evolve_pair0(e.hr, e.hi, wk[j].y, kx, kz, pa, pb);
                }
                re[j] = px_pack(pa.x, pb.x);
                im[j] = px_pack(pa.y, pb.y);
            }
        } else {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const float kx = __ldg(&kvec[c + G * j]);
                const float2 h = held_h[j * T];
                const float ki = held_k[j * T];
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
        Fft::run(re, im, buf, sh.tw, c);
        if (k == 0) publish(pub[0], tid);  // the CTA's previous row task, whose stores have drained by now
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const int x = Fft::index(j, c);
            out[((x / ROWS) * Q + q) * N * ROWS + x % ROWS] = make_ulonglong2(re[j], im[j]);
        }
    }
}

template <class P, int NF, int AR, bool FOAM>
__device__ __forceinline__ void pair_col_task(const FrameArgs& a, int ocean, int strip, const float2* inter_slot,
                                              const Shared& sh, int tid, unsigned* const* pub)
{
    using Fft = RegFft<P::LOG_N, P::E, AR>;
    constexpr int N = P::N, E = P::E, ROWS = P::ROWS, T = P::T, Q = NF / 2;
    const int w = tid % ROWS, c = tid / ROWS;
    void* buf = sh.exchange + w * P::SEQ;
    ulonglong2* held = reinterpret_cast<ulonglong2*>(sh.held) + tid;  // pair 0 of cell j at [j * T]
    float* src = reinterpret_cast<float*>(held);                      // later its foam source, at [4 T j]
    const int x0 = strip * ROWS;
    const size_t base = static_cast<size_t>(ocean) * N * N;
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
        const float4* in = reinterpret_cast<const float4*>(inter_slot) + (strip * Q + q) * N * ROWS + tid;
        f32x2 re[E], im[E];
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const float4 v = __ldcg(in + T * j);
            re[j] = px_pack(v.x, v.y);
            im[j] = px_pack(v.z, v.w);
        }
        Fft::run(re, im, buf, sh.tw, c);
        if (q == 0) publish(pub[0], tid);
        // Every thread's values of the last pair were in registers before the
        // transform's first barrier: the slot is free.
        if (q == Q - 1) publish(pub[1], tid);
        float4 *out_disp, *out_normal, *out_vel;
        OceanConsts cst;
        if (a.table != nullptr) {
            const OceanSlot& s = a.table[ocean];
            out_disp = s.disp;
            out_normal = s.normal;
            out_vel = s.velocity;
            cst = s.cst;
        } else {
            out_disp = a.disp + base;
            out_normal = a.normal + base;
            out_vel = a.velocity + base;
            cst = a.consts[ocean];
        }
        if (q == 0) {
#pragma unroll
            for (int j = 0; j < E; ++j) held[j * T] = make_ulonglong2(re[j], im[j]);
        } else if (q == 1) {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const ulonglong2 h = held[j * T];
                float2 f0, f1, f2, f3;
                px_unpack(h.x, f0.x, f1.x);
                px_unpack(h.y, f0.y, f1.y);
                px_unpack(re[j], f2.x, f3.x);
                px_unpack(im[j], f2.y, f3.y);
                const CellOut o = finalize_cell(f0, f1, f2, f3, cst.lambda, cst.foam_threshold, cst.inv_threshold);
                const int idx = Fft::index(j, c) * N + x0 + w;
                __stcs(&out_disp[idx], o.disp);
                __stcs(&out_normal[idx], o.normal);
                if constexpr (FOAM) src[4 * T * j] = o.disp.w;
            }
        } else {
            // The foam step's taps, within a cell or so of the strip, straight
            // from memory: staging the strip's surroundings in shared memory,
            // four bytes a copy, cost more than the loads (921 us against 881
            // for 64 x 512^2).
            const float* cur = a.foam_cur + base;
            auto foam_get = [&](int zz, int xx) { return __ldg(&cur[zz * N + xx]); };
#pragma unroll
            for (int j = 0; j < E; ++j) {
                float ux, uz, uy, zero;
                px_unpack(re[j], ux, uz);
                px_unpack(im[j], uy, zero);
                const int y = Fft::index(j, c);
                const int idx = y * N + x0 + w;
                __stcs(&out_vel[idx], make_float4(ux, uy, uz, 0.0f));
                if constexpr (FOAM) {
                    const FoamTaps t = foam_taps(N, x0 + w, y, ux, uz, a.foam_dt, a.foam_scale, a.foam_drift_x,
                                                 a.foam_drift_z, a.foam_inv_cell, foam_get);
                    __stcs(&a.foam_next[base + idx],
                           foam_finish(t, src[4 * T * j], a.foam_decay, a.foam_gain));
                }
            }
        }
    }
}

// Ticket -> (row?, ocean, task index) for the queue order above: `tasks` tickets
// each of R(0 .. ahead - 1), then R(ahead + i) and C(i) in turn, then the last C's.
__device__ __forceinline__ void decode(unsigned t, unsigned tasks, unsigned ahead, unsigned count, bool& row,
                                       unsigned& ocean, unsigned& idx)
{
    idx = t % tasks;
    unsigned b = t / tasks;
    if (b < ahead) {
        row = true, ocean = b;
        return;
    }
    b -= ahead;
    const unsigned pairs = count - ahead;
    row = b < 2u * pairs && (b & 1u) == 0u;
    ocean = b < 2u * pairs ? (b >> 1) + (row ? ahead : 0u) : b - pairs;
}

template <class P, int NF, int AR, bool FOAM>
__global__ void __launch_bounds__(P::T, P::CTAS) pair_frame_kernel(FrameArgs a, QueueArgs q)
{
    constexpr int N = P::N;
    constexpr unsigned TASKS = P::TASKS;
    extern __shared__ float4 smem4[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(smem4);
    // Thread 0's queue state between tasks, as in frame_kernel.
    __shared__ unsigned s_ticket;
    __shared__ int s_ok;
    __shared__ unsigned* s_publish;
    __shared__ unsigned* s_pub[2];
    unsigned r_next = 0;  // thread 0: the ticket drawn one task ahead
    int r_have_next = 0;

    const int tid = threadIdx.x;
    clear_words(q.clear, q.clear_words, tid, P::T);
    float2* tws = reinterpret_cast<float2*>(smem + P::TW);
    for (int i = tid; i < N - 1; i += P::T) tws[i] = a.twiddles[i];
    const Shared sh{smem, tws, smem + P::HELD};

    const unsigned count = static_cast<unsigned>(q.count);
    const unsigned slots = static_cast<unsigned>(q.slots);
    const unsigned ring = min(P::ring(slots), count);
    const unsigned ahead = min(P::ahead(slots), count);
    const unsigned total = 2u * count * TASKS;
    if (tid == 0) {
        s_publish = nullptr;
        r_next = atomicAdd(q.ticket, 1u);
        r_have_next = 1;
    }
    // frame_kernel's protocol: a ticket drawn one task ahead far from the end,
    // the finished row task published by the next task unless that has to wait.
    while (true) {
        __syncthreads();  // previous task's writes issued; shared memory free
        if (tid == 0) {
            unsigned* prev = s_publish;
            const unsigned t = r_have_next ? r_next : atomicAdd(q.ticket, 1u);
            r_have_next = 0;
            int ok = 1;
            unsigned* pub = nullptr;
            unsigned* self = nullptr;
            const unsigned* dep = nullptr;
            if (t < total) {
                if (t + 2u * gridDim.x < total) {
                    r_next = atomicAdd(q.ticket, 1u);
                    r_have_next = 1;
                }
                bool row;
                unsigned ocean, idx;
                decode(t, TASKS, ahead, count, row, ocean, idx);
                if (row) {
                    if (ocean >= ring) dep = q.cols_done + (ocean - ring);
                    pub = q.rows_done + ocean;
                } else {
                    dep = q.rows_done + ocean;
                    self = q.cols_done + ocean;
                }
            }
            if (t >= total || !q.defer || (dep != nullptr && ld_acquire(dep) < TASKS)) {
                if (prev != nullptr) red_release_add(prev, 1u);
                prev = nullptr;
                if (dep != nullptr) ok = wait_at_least(dep, TASKS, q.error, q.wait_ns);
            }
            s_pub[0] = prev;
            s_pub[1] = self;
            s_publish = pub;
            s_ticket = t;
            s_ok = ok;
        }
        __syncthreads();
        const unsigned t = s_ticket;
        if (t >= total || !s_ok) break;
        bool row;
        unsigned ocean, idx;
        decode(t, TASKS, ahead, count, row, ocean, idx);
        float2* inter = a.inter + static_cast<size_t>(ocean % ring) * N * N * NF;
        const int abs_ocean = a.ocean_base + static_cast<int>(ocean);
        if (row) {
            pair_row_task<P, NF, AR>(a, abs_ocean, static_cast<int>(idx), inter, sh, tid, s_pub);
        } else {
            pair_col_task<P, NF, AR, FOAM>(a, abs_ocean, static_cast<int>(idx), inter, sh, tid, s_pub);
        }
    }
}

// ---------------------------------------------------------------------------
// Several sizes in one launch (N = 64 to 1024, one field count, FP32 forms): the
// tickets of group after group, each in the order above with its own counters,
// ring and rows ahead. Every size's tasks take 256 threads, which 1024^2 needs
// (the sizes below are 5 to 30 % faster alone with 128). Each size's twiddles
// stay in shared memory. 64 oceans of 64^2 to 1024^2: 826 -> 531 us a frame, with
// velocity 1209 -> 760; 5 oceans 110 -> 91. With fewer row tasks than SMs
// (3 oceans up to 256^2 with velocity: 33 us there, 57 here) frame.cu's launch
// takes them.
// ---------------------------------------------------------------------------
constexpr int kMixMin = 6, kMixMax = 10;
constexpr int kMixThreads = 256;
template <int LOG_N>
using MixPlan = RegPlan<LOG_N, 8, kMixThreads * 8 / (1 << LOG_N)>;

template <int LOG_N = kMixMin>
constexpr size_t mix_exchange()
{
    constexpr size_t here = MixPlan<LOG_N>::TW;
    if constexpr (LOG_N == kMixMax) {
        return here;
    } else {
        constexpr size_t rest = mix_exchange<LOG_N + 1>();
        return here > rest ? here : rest;
    }
}
// The exchange area, then the twiddle tables (that of 2^l from float2 2^l - 64
// on), then the threads' own values.
constexpr size_t kMixTw = mix_exchange();
constexpr size_t kMixHeld = kMixTw + sizeof(float2) * ((2 << kMixMax) - (1 << kMixMin));
constexpr size_t kMixSmem = kMixHeld + sizeof(float4) * 8 * kMixThreads;
static_assert(3 * (kMixSmem + 2048) <= 228 * 1024 && kMixHeld % 16 == 0, "three mixed CTAs fit on an SM");

// A size's tasks. (As functions of their own, not inlined, they spilled around
// the calls: 570 us against 531 for 64 oceans of 64^2 to 1024^2.)
template <int LOG_N, int NF, int AR>
__device__ __forceinline__ void mix_run(const MixedGroup& g, bool row, int ocean, int idx, unsigned char* smem, int tid,
                                     unsigned* const* pub)
{
    using P = MixPlan<LOG_N>;
    const Shared sh{smem, reinterpret_cast<const float2*>(smem + kMixTw) + (P::N - (1 << kMixMin)), smem + kMixHeld};
    float2* inter = g.a.inter + static_cast<size_t>(ocean % g.ring) * P::N * P::N * NF;
    if (row) {
        pair_row_task<P, NF, AR>(g.a, ocean, idx, inter, sh, tid, pub);
    } else {
        pair_col_task<P, NF, AR, false>(g.a, ocean, idx, inter, sh, tid, pub);
    }
}

__host__ __device__ constexpr unsigned mix_tasks(int log_n) { return (1u << (2 * log_n)) / (8u * kMixThreads); }
static_assert(mix_tasks(6) == MixPlan<6>::TASKS && mix_tasks(10) == MixPlan<10>::TASKS, "tasks of a size");
// Oceans that a size's rows run ahead of its columns in the one launch.
constexpr int mix_ahead(int log_n)
{
    const int tasks = static_cast<int>(mix_tasks(log_n));
    const int wave = (148 * 3 + tasks - 1) / tasks;
    return wave > 2 ? wave : 2;
}

template <int NF, int AR>
__global__ void __launch_bounds__(kMixThreads, 3) pair_mixed_kernel(const __grid_constant__ MixedArgs m)
{
    extern __shared__ float4 smem4[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(smem4);
    __shared__ unsigned s_ticket;
    __shared__ int s_ok, s_group, s_row, s_ocean, s_idx;
    __shared__ unsigned* s_publish;
    __shared__ unsigned* s_pub[2];
    __shared__ MixedGroup s_groups[kMaxMixedGroups];  // tasks index it by a runtime group
    unsigned r_next = 0;
    int r_have_next = 0;
    const int tid = threadIdx.x;
    for (int i = tid; i < static_cast<int>(m.groups * sizeof(MixedGroup) / sizeof(unsigned)); i += kMixThreads)
        reinterpret_cast<unsigned*>(s_groups)[i] = reinterpret_cast<const unsigned*>(m.g)[i];
    if (blockIdx.x == 0 && tid == 0 && m.clear_ticket != nullptr) *m.clear_ticket = 0u;
    for (int gi = 0; gi < m.groups; ++gi) {
        const MixedGroup& g = m.g[gi];
        clear_words(g.clear, g.clear_words, tid, kMixThreads);
        const int n = 1 << g.log_n;
        float2* tw = reinterpret_cast<float2*>(smem + kMixTw) + (n - (1 << kMixMin));
        for (int i = tid; i < n - 1; i += kMixThreads) tw[i] = g.a.twiddles[i];
    }
    if (tid == 0) {
        s_publish = nullptr;
        r_next = atomicAdd(m.ticket, 1u);
        r_have_next = 1;
    }
    while (true) {
        __syncthreads();
        if (tid == 0) {
            unsigned* prev = s_publish;
            const unsigned t = r_have_next ? r_next : atomicAdd(m.ticket, 1u);
            r_have_next = 0;
            int ok = 1;
            unsigned* pub = nullptr;
            unsigned* self = nullptr;
            const unsigned* dep = nullptr;
            unsigned need = 0;
            if (t < m.total) {
                if (t + 2u * gridDim.x < m.total) {
                    r_next = atomicAdd(m.ticket, 1u);
                    r_have_next = 1;
                }
                int gi = m.groups - 1;
                while (gi > 0 && t < m.g[gi].first) --gi;
                const MixedGroup& g = m.g[gi];
                need = mix_tasks(g.log_n);
                bool row;
                unsigned ocean, idx;
                decode(t - g.first, need, static_cast<unsigned>(g.ahead), static_cast<unsigned>(g.count), row, ocean, idx);
                if (row) {
                    if (ocean >= static_cast<unsigned>(g.ring)) dep = g.cols_done + (ocean - g.ring);
                    pub = g.rows_done + ocean;
                } else {
                    dep = g.rows_done + ocean;
                    self = g.cols_done + ocean;
                }
                s_group = gi;
                s_row = row ? 1 : 0;
                s_ocean = static_cast<int>(ocean);
                s_idx = static_cast<int>(idx);
            }
            if (t >= m.total || !m.defer || (dep != nullptr && ld_acquire(dep) < need)) {
                if (prev != nullptr) red_release_add(prev, 1u);
                prev = nullptr;
                if (dep != nullptr) ok = wait_at_least(dep, need, m.error, m.wait_ns);
            }
            s_pub[0] = prev;
            s_pub[1] = self;
            s_publish = pub;
            s_ticket = t;
            s_ok = ok;
        }
        __syncthreads();
        if (s_ticket >= m.total || !s_ok) break;
        const MixedGroup& g = s_groups[s_group];
        const bool row = s_row != 0;
        switch (g.log_n) {
            case 6: mix_run<6, NF, AR>(g, row, s_ocean, s_idx, smem, tid, s_pub); break;
            case 7: mix_run<7, NF, AR>(g, row, s_ocean, s_idx, smem, tid, s_pub); break;
            case 8: mix_run<8, NF, AR>(g, row, s_ocean, s_idx, smem, tid, s_pub); break;
            case 9: mix_run<9, NF, AR>(g, row, s_ocean, s_idx, smem, tid, s_pub); break;
            default: mix_run<10, NF, AR>(g, row, s_ocean, s_idx, smem, tid, s_pub); break;
        }
    }
}

template <int NF, int AR>
struct PairMixed {
    static cudaError_t prepare()
    {
        return cudaFuncSetAttribute(pair_mixed_kernel<NF, AR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(kMixSmem));
    }
    static int blocks_per_sm()
    {
        int n = 0;
        if (prepare() != cudaSuccess) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, pair_mixed_kernel<NF, AR>, kMixThreads, kMixSmem) !=
            cudaSuccess)
            return 0;
        return n;
    }
    static cudaError_t launch(const MixedArgs& m, int grid, cudaStream_t st)
    {
        cudaError_t e = prepare();
        if (e != cudaSuccess) return e;
        pair_mixed_kernel<NF, AR><<<grid, kMixThreads, kMixSmem, st>>>(m);
        return cudaGetLastError();
    }
};
template <typename Fn>
auto mixed_variant(int nf, int ar, Fn&& fn)
{
    if (ar == kArFast) return nf == 4 ? fn(PairMixed<4, kArFast>{}) : fn(PairMixed<6, kArFast>{});
    return nf == 4 ? fn(PairMixed<4, kArExact>{}) : fn(PairMixed<6, kArExact>{});
}

template <int LOG_N, int NF, int AR, bool FOAM>
struct PairLaunch {
    using P = PairPlan<LOG_N, AR, FOAM>;
    static constexpr size_t SMEM = P::SMEM;

    static cudaError_t prepare()
    {
        return cudaFuncSetAttribute(pair_frame_kernel<P, NF, AR, FOAM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(SMEM));
    }
    static int blocks_per_sm()
    {
        int n = 0;
        if (prepare() != cudaSuccess) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, pair_frame_kernel<P, NF, AR, FOAM>, P::T, SMEM) !=
            cudaSuccess)
            return 0;
        return n;
    }
    static cudaError_t launch(const FrameArgs& a, const QueueArgs& q, int grid, cudaStream_t st)
    {
        cudaError_t e = prepare();
        if (e != cudaSuccess) return e;
        pair_frame_kernel<P, NF, AR, FOAM><<<grid, P::T, SMEM, st>>>(a, q);
        return cudaGetLastError();
    }
};

// The variant of (log_n, nf, ar, foam) for `fn`.
template <int LOG_N, int AR, typename Fn>
auto variant_ar(int nf, bool foam, Fn&& fn)
{
    if (nf == 4) return fn(PairLaunch<LOG_N, 4, AR, false>{});
    if (foam) return fn(PairLaunch<LOG_N, 6, AR, true>{});
    return fn(PairLaunch<LOG_N, 6, AR, false>{});
}
template <int LOG_N, typename Fn>
auto variant(int nf, int ar, bool foam, Fn&& fn)
{
    if constexpr (LOG_N != 4 && LOG_N != 10) {
        if (ar == kArPrecise) return variant_ar<LOG_N, kArPrecise>(nf, foam, fn);
    }
    if (ar == kArFast) return variant_ar<LOG_N, kArFast>(nf, foam, fn);
    return variant_ar<LOG_N, kArExact>(nf, foam, fn);
}
template <typename Fn>
auto dispatch(int log_n, int nf, int ar, bool foam, Fn&& fn)
{
    switch (log_n) {
        case 4: return variant<4>(nf, ar, foam, fn);
        case 5: return variant<5>(nf, ar, foam, fn);
        case 6: return variant<6>(nf, ar, foam, fn);
        case 7: return variant<7>(nf, ar, foam, fn);
        case 8: return variant<8>(nf, ar, foam, fn);
        case 9: return variant<9>(nf, ar, foam, fn);
        default: return variant<10>(nf, ar, foam, fn);
    }
}

// Whether the size has a plan in this arithmetic.
bool has_plan(int log_n, int ar)
{
    return log_n >= 4 && log_n <= 10 && (ar != kArPrecise || (log_n != 4 && log_n != 10));
}

}  // namespace

// A ring no deeper than the rows ahead would have row tasks wait for later
// tickets.
bool pair_mixed_ok(int log_n, int ar, int count, int ring)
{
    return ar != kArPrecise && log_n >= kMixMin && log_n <= kMixMax && (ring >= count || ring > mix_ahead(log_n));
}

uint32_t pair_mixed_tasks(int log_n) { return mix_tasks(log_n); }

int pair_mixed_blocks_per_sm(int nf, int ar)
{
    return mixed_variant(nf, ar, [](auto L) { return decltype(L)::blocks_per_sm(); });
}

cudaError_t launch_pair_mixed(int nf, int ar, MixedArgs m, int grid, cudaStream_t st)
{
    m.total = 0;
    for (int i = 0; i < m.groups; ++i) {
        MixedGroup& g = m.g[i];
        if (!pair_mixed_ok(g.log_n, ar, g.count, g.ring)) return cudaErrorInvalidValue;
        const int ahead = mix_ahead(g.log_n);
        g.ahead = ahead < g.count ? ahead : g.count;
        g.first = m.total;
        m.total += 2u * static_cast<uint32_t>(g.count) * mix_tasks(g.log_n);
    }
    return mixed_variant(nf, ar, [&](auto L) { return decltype(L)::launch(m, grid, st); });
}

// A task takes its pairs one after the other, so a frame of few oceans, whose
// tasks do not fill the GPU, is a longer chain here than with a task's pairs side
// by side (frame_kernel). From the fourth ocean on that kernel waits for the three
// slots of its ring; at 512^2 and above a frame fills the GPU sooner. us a frame
// there / here on either side of each line, without velocity, with it, and with
// velocity and foam (where the lines differ, the first that holds for both):
//   FP32   16    3  9.3/10.4    9.3/12.8   10.3/13.4    4  14.4/10.3   14.5/12.4   15.1/13.5
//          32    3 12.4/13.4   15.4/15.7   15.4/17.0    4  19.6/13.4   23.7/15.9   23.9/17.2
//          64    3 10.3/13.4                            4  15.2/13.4
//                6             16.4/16.9   16.9/18.1    7              20.8/16.5   22.5/17.9
//         128    3 12.4/14.4   12.4/18.1   13.2/18.6    4  17.9/14.5   19.6/18.5   20.6/18.7
//         256    2 12.9/14.5                            3  18.5/16.5
//                3             20.6/21.9   20.9/22.8    4              32.8/21.8   32.9/22.8
//         512    1 18.2/18.1   22.7/22.6   24.7/26.0    2  28.3/24.7   36.5/32.9   40.1/35.7
//        1024    1 60.7/56.6   81.6/81.9   90.2/94.5    2 110.8/78.5  148.1/113.6 161.6/133.6
// The precise form's blocks of 16 indices (N = 128 and 256) leave four CTAs of 128
// threads on an SM, and its chain is longest:
//          32    3 14.5/17.8   17.5/22.0   17.5/22.7    4  21.9/18.2   27.5/22.2   27.7/22.7
//          64    6 18.5/19.1   19.3/24.7   19.6/25.6    7  23.3/19.3   24.7/24.7   25.8/25.3
//         128    9 30.9/31.4   37.5/47.2   39.4/48.0   10  40.8/31.3   48.7/47.2   50.9/48.0
//         256    6 37.0/43.1   53.5/61.9   59.7/64.3    7  48.8/43.1   62.7/61.7   64.9/64.5
//         512    1 24.6/26.8                            2  44.0/39.1
//               12             259/264     272/269     16              341/341     359/352
bool pair_frame_ok(int log_n, int ar, int nf, bool foam, int count)
{
    if (!has_plan(log_n, ar)) return false;
    const bool velocity = nf == 6;
    int line;
    if (ar == kArPrecise) {
        line = log_n == 9 ? (velocity ? 16 : 2) : log_n == 8 ? 7 : log_n == 7 ? 10 : log_n == 6 ? 7 : 4;
    } else {
        switch (log_n) {
            case 6: line = velocity ? 7 : 4; break;
            case 8: line = velocity ? 4 : 3; break;
            case 9: line = 2; break;
            case 10: line = foam ? 2 : 1; break;
            default: line = 4; break;
        }
    }
    return count >= line;
}

// 1024^2 in the FP32 forms has no other kernel without foam for a ring of three.
static_assert(PairPlan<10, kArExact, false>::ring(2) <= 3 && PairPlan<10, kArExact, true>::ring(2) <= 3);

int pair_frame_ring(int log_n, int ar, int slots)
{
    if (!has_plan(log_n, ar)) return 0;
    const unsigned s = static_cast<unsigned>(slots);
    int ring = 0;
    for (bool foam : {false, true}) {
        const int r = dispatch(log_n, 6, ar, foam, [&](auto L) { return static_cast<int>(decltype(L)::P::ring(s)); });
        ring = ring > r ? ring : r;
    }
    return ring;
}

int pair_frame_tasks(int log_n, int ar, bool fuse_foam)
{
    if (!has_plan(log_n, ar)) return 0;
    return dispatch(log_n, fuse_foam ? 6 : 4, ar, fuse_foam, [](auto L) { return decltype(L)::P::TASKS; });
}

int pair_frame_blocks_per_sm(int log_n, int nf, int ar, bool fuse_foam)
{
    if (!has_plan(log_n, ar)) return 0;
    return dispatch(log_n, nf, ar, fuse_foam, [](auto L) { return decltype(L)::blocks_per_sm(); });
}

cudaError_t launch_pair_frame(int log_n, int nf, int ar, bool fuse_foam, const FrameArgs& a, const QueueArgs& q, int grid,
                              cudaStream_t st)
{
    if (!has_plan(log_n, ar)) return cudaErrorInvalidValue;
    return dispatch(log_n, nf, ar, fuse_foam, [&](auto L) { return decltype(L)::launch(a, q, grid, st); });
}

}  // namespace ocean_b200
