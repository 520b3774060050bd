// RK4 steps in one resident kernel (plain form and no-allocation form, FP64 / FP32).
//
// On a grid of some thousand to some ten thousand nodes a stage takes a few
// microseconds, most of it the launch of the next kernel and chained L2 reads.  Here
// one cooperative launch runs all steps: CTA c (one per SM) owns nodes [c m, c m + m),
// keeps their stencil weights, pointwise records, base state and RK accumulator in
// shared memory and their gather rows in registers, and exchanges only the stage
// states through L2.  A stage is the node-per-lane kernel's work split (LPN lanes a
// node, stage_lane.cuh) with the same sums in the same order, so a step gives the
// bits that four stage launches with the same LPN give.
//
// Between stages the CTAs meet at one counter (a release-add each, then acquire-loads
// until all have added): 1.25 us for 148 CTAs, against 6.8 with a flag word per CTA in
// shared lines and 1.3-1.5 with a line per CTA and waits for the neighbours only.  K rows
// are read with plain loads, cached in L1: the acquire makes the rows that other SMs wrote
// visible.  Every wait is bounded: one that runs out raises an abort word that all CTAs
// see in theirs, sets a flag for the host and ends the kernel.  The first wait of a launch
// may be long, since other kernels may still hold some of the SMs.
//
// Weights that do not fit (FP64 from N = 27000 to 42600 on 148 SMs) are streamed from L2 in
// every stage, see kStagePairs.  N=40962: 7.15 us per stage against 8.2 with a launch per
// stage; 8.4 with plain loads of the nodes that do not fit, 7.9 with a copy per slot and
// warp, 7.5 with two smaller buffers filled four times a stage.
#pragma once

#include <type_traits>

#include "stage_lane.cuh"
#include "tcgen05.cuh"

namespace swe {
namespace res {

// threads of a CTA: 16 warps have 128 registers a thread, 20 have 96 (a few of them spilled
// with FP64)
constexpr int kFew = 512, kMost = 640;
constexpr int kSyncWords = 64;         // counter and abort word, a line each
constexpr int kPt = kPointFields;
constexpr unsigned long long kWaitNs = 2000000000ull, kFirstWaitNs = 60000000000ull;

template <typename T>
struct Args {
    int n, nnbr;
    int m;                             // nodes per CTA
    int nsteps;
    T *H, *Ka, *Kb;                    // [n][4]
    T gh0, c01, c2;                    // c01 = dt/2 (stages 0 and 1), c2 = dt (stage 2)
    double dt6;
    unsigned* counter;                 // arrivals of the CTAs, zero at launch; abort word 32 words on
    int* failed;                       // set when a wait ran out (pinned host or device memory)
    unsigned long long wait_ns = kWaitNs;
};

// Static data as swe_cuda_init packs it.
template <typename T, bool I16>
struct Packed {
    static constexpr bool kNodeFast = true;     // consecutive nodes of a slot are contiguous
    static constexpr bool kSmallRows = I16;     // rows lie within 32767 of their node
    const T* Wl;
    const int* idxl;
    const short* idxs;
    const T* PTl;
    __device__ static long at(long i, int slot) { return ((i / kLaneTile) * kSlots + slot) * kLaneTile + i % kLaneTile; }
    __device__ void weights(long i, int slot, int, T (&w)[4]) const { lane::weights(Wl + 4 * at(i, slot), lane::l2_normal(), w); }
    __device__ int row(long i, int slot, int, int) const {
        return I16 ? (int)i + lane::ld_stream(idxs + at(i, slot)) : lane::ld_stream(idxl + at(i, slot));
    }
    __device__ T point(long i, int f) const {
        return PTl[(i / kLaneTile * kPointFields + f) * kLaneTile + i % kLaneTile];
    }
};

// Streamed weights (FP64, two lanes a node): the two warps of a 32-node tile hold the weights
// of kHeldPairs slot pairs and stream the others through a buffer of kStagePairs pairs, filled
// by one bulk copy twice a stage: the first batch while the stage before ends and the CTAs
// meet, the second while the held pairs are summed.
constexpr int kStagePairs = 7, kHeldPairs = 2;
static_assert(2 * kStagePairs + kHeldPairs == kSlots / 2, "all slot pairs");
constexpr int kBatchBytes = 2 * kStagePairs * kLaneTile * 4 * 8;
constexpr uint32_t kCopyTries = 1u << 24;

// A stage state row: a plain L1-cached load (never the non-coherent path, the rows change
// between stages), one 32-byte sector.  FP64 rows of a caller's array (stage 0 reads H) may
// be only 16-byte aligned: two halves there.
__device__ __forceinline__ void load_state(const double* p, bool wide, double (&v)[4]) {
    if (wide) {
        asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                     : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
                     : "l"(p)
                     : "memory");
    } else {
        asm volatile("ld.global.v2.f64 {%0, %1}, [%4]; ld.global.v2.f64 {%2, %3}, [%4 + 16];"
                     : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
                     : "l"(p)
                     : "memory");
    }
}
__device__ __forceinline__ void load_state(const float* p, bool, float (&v)[4]) {
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "l"(p)
                 : "memory");
}

// shared memory of a CTA: weights [slot][16-byte unit][m], pointwise [kPt][m],
// base state and accumulator [8][m]
__host__ __device__ inline int slots_of(int nnbr, int lpn) { return (nnbr + lpn - 1) / lpn * lpn; }
// A slot's weights: FP64 as two 16-byte planes, so that neighbouring lanes read without
// bank conflicts.
__device__ __forceinline__ void put_weights(double* sw, int m, int slot, int ln, const double (&w)[4]) {
    double2* p = reinterpret_cast<double2*>(sw) + (long)2 * slot * m + ln;
    p[0] = make_double2(w[0], w[1]);
    p[m] = make_double2(w[2], w[3]);
}
__device__ __forceinline__ void get_weights(const double* sw, int m, int slot, int ln, double (&w)[4]) {
    const double2* p = reinterpret_cast<const double2*>(sw) + (long)2 * slot * m + ln;
    const double2 a = p[0], b = p[m];
    w[0] = a.x; w[1] = a.y; w[2] = b.x; w[3] = b.y;
}
__device__ __forceinline__ void put_weights(float* sw, int m, int slot, int ln, const float (&w)[4]) {
    reinterpret_cast<float4*>(sw)[(long)slot * m + ln] = make_float4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void get_weights(const float* sw, int m, int slot, int ln, float (&w)[4]) {
    const float4 a = reinterpret_cast<const float4*>(sw)[(long)slot * m + ln];
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
}

// Waits until every CTA has done its `stage`-th stage.
template <typename T>
__device__ __forceinline__ bool exchange(const Args<T>& a, unsigned stage, int* s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.counter) : "memory");
        volatile unsigned* abort_word = a.counter + 32;
        const unsigned all = stage * gridDim.x;
        unsigned long long t0 = 0;
        int ok = 1;
        for (unsigned tries = 1;; ++tries) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.counter) : "memory");
            if ((int)(v - all) >= 0) break;
            if ((tries & 63) == 0) {
                unsigned long long t;
                asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
                if (t0 == 0) t0 = t;
                if (*abort_word != 0 || t - t0 > (stage == 1 ? kFirstWaitNs : a.wait_ns)) {
                    *abort_word = 1;
                    *(volatile int*)a.failed = 1;
                    __threadfence_system();
                    ok = 0;
                    break;
                }
            }
        }
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// One block that waits, as after a step's second stage, for a block that was never launched:
// the path of a wait that runs out, without anything to run out of (swe_selftest_step_wait).
static __global__ void lone_block_kernel(Args<double> a) {
    __shared__ int ok;
    exchange(a, 2, &ok);
}

template <typename T, int LPN, int THREADS, class Src, bool STREAM>
__global__ void __launch_bounds__(THREADS, 1) steps_kernel(const Args<T> a, const Src src) {
    constexpr int kNpw = 32 / LPN;          // nodes per warp
    constexpr int kJpl = kSlots / LPN;      // slots per lane
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_ok;
    static_assert(!STREAM || (sizeof(T) == 8 && LPN == 2), "streamed weights are FP64, two lanes a node");
    __shared__ __align__(8) uint64_t s_bar[STREAM ? THREADS / 64 : 1];
    const int nst = STREAM ? 2 * kHeldPairs : slots_of(a.nnbr, LPN);   // slots in shared memory
    constexpr int kSlot0 = STREAM ? 2 * kStagePairs : 0;               // the first of them
    T* sw = reinterpret_cast<T*>(smem);
    T* sbuf = sw + (long)nst * 4 * a.m;                                // the tiles' buffers
    T* spt = sbuf + (STREAM ? 2 * kStagePairs * 4 * a.m : 0);
    T* shd = spt + kPt * a.m;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tl = lane % kNpw, sub = lane / kNpw;
    const long first = (long)blockIdx.x * a.m;
    const int cnt = (int)min((long)a.m, (long)a.n - first);
    // static data of the CTA's nodes
    for (int e = threadIdx.x; e < nst * a.m; e += blockDim.x) {
        const int slot = Src::kNodeFast ? e / a.m : e % nst, ln = Src::kNodeFast ? e % a.m : e / nst;
        T w[4] = {T(0), T(0), T(0), T(0)};
        if (ln < cnt && kSlot0 + slot < a.nnbr) src.weights(first + ln, kSlot0 + slot, a.nnbr, w);
        put_weights(sw, a.m, slot, ln, w);
    }
    for (int e = threadIdx.x; e < kPt * cnt; e += blockDim.x) spt[e / cnt * a.m + e % cnt] = src.point(first + e % cnt, e / cnt);
    // this lane's node
    const int ln = warp * kNpw + tl;
    const bool valid = ln < cnt;
    const bool active = (STREAM ? warp & ~1 : warp) * kNpw < cnt;      // warp-uniform; streamed: both or none of a tile's
    const int lnc = min(ln, cnt - 1);
    const int own = (int)first + lnc;
    constexpr bool kPack = Src::kSmallRows && kJpl > 8;      // two 16-bit offsets a register
    int rows[kPack ? kJpl / 2 : kJpl];
    if (active) {
#pragma unroll
        for (int jj = 0; jj < kJpl; ++jj) {
            const int slot = jj * LPN + sub;
            const int p = slot < a.nnbr ? src.row(own, slot, a.nnbr, a.n) : own;
            if constexpr (kPack) {
                if (jj & 1) rows[jj / 2] |= (p - own) << 16;
                else rows[jj / 2] = (p - own) & 0xffff;
            } else {
                rows[jj] = p;
            }
        }
    }
    // streamed weights: a batch of slot pairs from `pair0` on into the tile's buffer
    T* buf = sbuf + (warp >> 1) * (kBatchBytes / 8);
    uint64_t* bar = s_bar + (STREAM ? warp >> 1 : 0);
    unsigned batches = 0;                  // batches waited for
    bool pending = false;
    auto fill = [&](int pair0) {
        if constexpr (STREAM) {
            // both warps have read the buffer, and their reads come before the copy
            tc::fence_async_smem();
            asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp >> 1)) : "memory");
            if ((warp & 1) == 0 && lane == 0) {
                tc::mbar_arrive_expect_tx(bar, kBatchBytes);
                tc::bulk_g2s(buf, src.Wl + 4 * src.at(first + warp * kNpw, 2 * pair0), kBatchBytes, bar);
            }
            pending = true;
        }
    };
    auto filled = [&]() {
        if constexpr (STREAM) {
            if (!tc::mbar_wait_bounded(bar, batches & 1, kCopyTries)) {
                *(volatile unsigned*)(a.counter + 32) = 1;
                *(volatile int*)a.failed = 1;
            }
            ++batches;
            pending = false;
        }
    };
    if constexpr (STREAM) {
        if ((warp & 1) == 0 && lane == 0) tc::mbar_init(bar, 1);
        tc::fence_mbar_init();
        if (active) fill(0);
    }
    const bool wide_h = (reinterpret_cast<uintptr_t>(a.H) & 31) == 0;
    T q[4] = {};
    if (active) {
        load_state(a.H + 4L * own, wide_h, q);
        if (sub == 0 && valid)
#pragma unroll
            for (int x = 0; x < 4; ++x) shd[x * a.m + ln] = q[x];
    }
    __syncthreads();
    unsigned done = 0;

    auto stage = [&](auto mode_c, bool more) {
        constexpr int MODE = decltype(mode_c)::value;
        if (!active) return;
        const T* Kin = MODE == kStage0 ? a.H : MODE == kStage2 ? a.Kb : a.Ka;
        T* Kout = MODE == kStage3 ? a.H : MODE == kStage1 ? a.Kb : a.Ka;
        const bool wide = MODE != kStage0 || wide_h;
        // addresses are formed anew in every stage: kept over the step loop, the rows' addresses
        // in three buffers and the slots' in shared memory would spill
        int m = a.m;
        asm volatile("" : "+r"(m));
#pragma unroll
        for (int x = 0; x < (kPack ? kJpl / 2 : kJpl); ++x) asm volatile("" : "+r"(rows[x]));
        T acc[16];
#pragma unroll
        for (int x = 0; x < 16; ++x) acc[x] = T(0);
        // pairs (slots of this lane) [from, to), weights by get(pair, w)
        auto sum = [&](auto from_c, auto to_c, auto get) {
            constexpr int kFrom = decltype(from_c)::value, kTo = decltype(to_c)::value, kChunk = 4;
#pragma unroll
            for (int j0 = kFrom; j0 < kTo; j0 += kChunk) {
                if (j0 * LPN >= a.nnbr) break;
                T kv[kChunk][4];
#pragma unroll
                for (int u = 0; u < kChunk; ++u) {
                    const int jj = j0 + u;
                    if (jj >= kTo) continue;
                    int p;
                    if constexpr (kPack) p = own + (jj & 1 ? rows[jj / 2] >> 16 : (int)(short)rows[jj / 2]);
                    else p = rows[jj];
                    load_state(Kin + 4L * p, wide, kv[u]);
                }
#pragma unroll
                for (int u = 0; u < kChunk; ++u) {
                    if (j0 + u >= kTo) continue;
                    // (slots at or past nnbr: the own row with zero weights)
                    if (!STREAM && (j0 + u) * LPN >= nst) continue;
                    T w[4];
                    get(j0 + u, w);
#pragma unroll
                    for (int op = 0; op < 4; ++op)
#pragma unroll
                        for (int f = 0; f < 4; ++f) acc[op * 4 + f] += w[op] * kv[u][f];
                }
            }
        };
        auto held = [&](int jj, T (&w)[4]) { get_weights(sw, m, jj * LPN + sub - kSlot0, lnc, w); };
        if constexpr (STREAM) {
            // a node's four weights lie together: lanes 4..7 of each eight read their second
            // half first, so that a pass of 16-byte reads meets no bank twice
            const bool swap = tl & 4;
            int base = 0;
            auto streamed = [&](int jj, T (&w)[4]) {
                const double2* p = reinterpret_cast<const double2*>(buf + (((jj - base) * 2 + sub) * kLaneTile + (warp & 1) * kNpw + tl) * 4);
                const double2 x = p[swap], y = p[!swap];
                w[0] = swap ? y.x : x.x; w[1] = swap ? y.y : x.y;
                w[2] = swap ? x.x : y.x; w[3] = swap ? x.y : y.y;
            };
            using std::integral_constant;
            constexpr int kA = kStagePairs, kB = kStagePairs + kHeldPairs;
            filled();
            sum(integral_constant<int, 0>(), integral_constant<int, kA>(), streamed);
            fill(kB);
            sum(integral_constant<int, kA>(), integral_constant<int, kB>(), held);
            filled();
            base = kB;
            sum(integral_constant<int, kB>(), integral_constant<int, kJpl>(), streamed);
            if (more) fill(0);
        } else {
            sum(std::integral_constant<int, 0>(), std::integral_constant<int, kJpl>(), held);
        }
#pragma unroll
        for (int o = kNpw; o < 32; o <<= 1)
#pragma unroll
            for (int x = 0; x < 16; ++x) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], o);
        if (sub != 0 || !valid) return;
        T pt[kPointStride], F[4];
#pragma unroll
        for (int f = 0; f < kPt; ++f) pt[f] = spt[f * a.m + ln];
        pointwise_rhs(acc, q, pt, a.gh0, F);
        T* sh = shd + ln;
        T* sd = shd + 4 * a.m + ln;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            if (MODE == kStage0) {
                sd[x * a.m] = F[x];
                q[x] = Quad<T>::axpy(q[x], a.c01, F[x]);
            } else if (MODE != kStage3) {
                sd[x * a.m] = Quad<T>::axpy(sd[x * a.m], T(2), F[x]);
                q[x] = Quad<T>::axpy(sh[x * a.m], MODE == kStage1 ? a.c01 : a.c2, F[x]);
            } else {
                q[x] = Quad<T>::update_h(sh[x * a.m], a.dt6, Quad<T>::axpy(sd[x * a.m], T(1), F[x]));
                sh[x * a.m] = q[x];
            }
        }
        if (MODE != kStage3 || wide_h) lane::put_row(Kout + 4L * own, q);
        else Quad<T>::store_row(Kout + 4L * own, q);
    };

    for (int s = 0; s < a.nsteps; ++s) {
        const bool last = s + 1 == a.nsteps;
        stage(std::integral_constant<int, kStage0>(), true);
        if (!exchange(a, ++done, &s_ok)) break;
        stage(std::integral_constant<int, kStage1>(), true);
        if (!exchange(a, ++done, &s_ok)) break;
        stage(std::integral_constant<int, kStage2>(), true);
        if (!exchange(a, ++done, &s_ok)) break;
        stage(std::integral_constant<int, kStage3>(), !last);
        if (!last && !exchange(a, ++done, &s_ok)) break;
    }
    if (pending) filled();                 // after an abort: no copy in flight when the block ends
}

// How a grid of n nodes is split over the SMs with lpn lanes a node: nodes per CTA (a multiple
// of 8) and CTAs, and whether the weights are streamed (only where Src allows it: `streams`).
// False where a CTA's nodes exceed its threads or smem_max bytes.
template <typename T>
inline bool split(int n, int nnbr, int lpn, int sms, size_t smem_max, bool streams, int& m, int& ctas, size_t& smem,
                  bool& stream) {
    m = ((n + sms - 1) / sms + 7) / 8 * 8;
    smem = m * ((kPt + 8) * sizeof(T) + slots_of(nnbr, lpn) * 4 * sizeof(T));
    stream = false;
    if (smem > smem_max && streams && sizeof(T) == 8 && lpn == 2) {
        m = (m + kLaneTile - 1) / kLaneTile * kLaneTile;      // whole tiles
        smem = m * ((kPt + 8) * sizeof(T) + 2 * (kStagePairs + kHeldPairs) * 4 * sizeof(T));
        stream = true;
    }
    ctas = (n + m - 1) / m;
    return m * lpn <= kMost && smem <= smem_max;
}

template <typename T, int LPN, class Src>
inline cudaError_t launch(const Args<T>& a, const Src& src, int ctas, size_t smem, size_t smem_max, bool stream,
                          cudaStream_t st) {
    auto kernel = a.m * LPN <= kFew ? steps_kernel<T, LPN, kFew, Src, false> : steps_kernel<T, LPN, kMost, Src, false>;
    if constexpr (Src::kNodeFast && sizeof(T) == 8 && LPN == 2)
        if (stream) kernel = steps_kernel<T, LPN, kMost, Src, true>;
    // the device's limit in every call, never the call's own size: another thread may be
    // between its attribute and its launch
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(a.counter, 0, kSyncWords * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3((a.m * LPN + 31) / 32 * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;      // all CTAs resident together, or no launch
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a, src);
}

// shared memory a CTA of the current device may use
inline cudaError_t smem_limit(int& sms, size_t& most) {
    int dev = 0, v = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    most = v > 1024 ? v - 1024 : 0;                   // static shared memory aside
    return e;
}

}  // namespace res
}  // namespace swe
