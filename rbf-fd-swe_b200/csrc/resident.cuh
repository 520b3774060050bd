// RK4 steps in one resident kernel (plain form and no-allocation form, FP64 / FP32).
//
// On a grid of some thousand to some ten thousand nodes a stage takes a few
// microseconds, most of it the launch of the next kernel and chained L2 reads.  Here
// one launch runs all steps: CTA c (one per SM) owns nodes [c m, c m + m),
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
// see in theirs, sets a flag for the host and ends the kernel.
//
// The launch does not need all SMs: another stream's kernel may hold some of them for as long
// as it likes.  A CTA says that it has started; while some have not kGatherNs after the first
// stage, those that have go on without them (share_steps below): they deal all nodes out among
// themselves, with everything read from L2 as a stage launch reads it, and take in the CTAs
// that start later at every step's end.  A CTA that finds the work done ends at once.  Only a
// kernel that holds a part of every SM keeps the steps from running until it ends.  With 20 SMs
// held, us per stage: N=10242 FP64 7.9 (stage launches 4.1; nothing held 3.4 and 4.1), N=40962
// FP64 12.9 (9.7; 7.2 and 7.7): few warps an SM, for a state that ends with the other kernel.
//
// Weights that do not fit (31 neighbours, 148 SMs: FP64 from 27,233 to 42,624 nodes) are streamed
// from L2 in every stage, see kStagePairs.  N=40962: 7.2 us per stage against 7.7 with a launch
// per stage; before the pointwise values were transposed 7.15 against 8.2, 8.4 with plain loads
// of the nodes that do not fit, 7.9 with a copy per slot and warp, 7.5 with two smaller buffers
// filled four times a stage.
#pragma once

#include <type_traits>

#include "stage_lane.cuh"
#include "tcgen05.cuh"

namespace swe {
namespace res {

// threads of a CTA: 16 warps have 128 registers a thread, 20 have 96 (a few of them spilled
// with FP64)
constexpr int kFewThreads = 512, kMost = 640;
constexpr int kPt = kPointFields;
constexpr unsigned long long kWaitNs = 2000000000ull;
// CTAs of an idle GPU start within a few microseconds of one another, and their first stage
// comes after about 15 us of loading
constexpr unsigned long long kGatherNs = 100000ull;
// a launch runs at most this many steps: the kernels of other streams get a turn every few
// milliseconds, for less than 1 % in set-up
constexpr int kLaunchSteps = 200;

// words that the CTAs meet at, zero at launch, each on a line of its own
enum SyncWord {
    kArrived = 0,                      // CTAs done with their stages, counted over the launch
    kAbort = 32,
    kStarted = 64,                     // CTAs that have started; kShort: they go on without the others
    kShared = 96,                      // share_steps: CTAs done with their stages of a step
    kRoster = 128,                     // share_steps, 64 bits: step (from 1) << 32 | CTAs that take part
    kSyncSet = 160,
    kSyncWords = 2 * kSyncSet          // the launch's and finish_kernel's
};
constexpr unsigned kShort = 1u << 31;
enum Met { kFailed = 0, kAll = 1, kFew = 2 };

template <typename T>
struct Args {
    int n, nnbr;
    int m;                             // nodes per CTA
    int nsteps;
    T *H, *Ka, *Kb, *D;                // [n][4]; D: share_steps only
    T gh0, c01, c2;                    // c01 = dt/2 (stages 0 and 1), c2 = dt (stage 2)
    double dt6;
    unsigned* sync;                    // SyncWord
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

__device__ __forceinline__ unsigned long long time_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void add_release(unsigned* p) { asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory"); }
__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// One thread: waits until done() holds, looking at the clock and the abort word now and then;
// aborts when it has waited wait_ns.
template <typename T, class Done>
__device__ __forceinline__ bool wait_for(const Args<T>& a, Done done) {
    unsigned long long t0 = 0;
    for (unsigned tries = 1; !done(); ++tries) {
        if (tries & 63) continue;
        const unsigned long long t = time_ns();
        if (t0 == 0) t0 = t;
        if (*(volatile unsigned*)(a.sync + kAbort) != 0 || t - t0 > a.wait_ns) {
            *(volatile unsigned*)(a.sync + kAbort) = 1;
            *(volatile int*)a.failed = 1;
            __threadfence_system();
            return false;
        }
    }
    return true;
}

// Waits until every CTA has done its `stage`-th stage: kAll.  After the first stage also kFew,
// where some CTAs have not started: the bit kShort, which the CTA that gives up waiting sets
// together with the count of those that have, settles it for all of them -- a CTA that starts
// later finds it as it says so, and the count can no longer reach the grid's without it.
template <typename T>
__device__ __forceinline__ int exchange(const Args<T>& a, unsigned stage, int* s_met) {
    __syncthreads();
    if (threadIdx.x == 0) {
        add_release(a.sync + kArrived);
        const unsigned all = stage * gridDim.x;
        unsigned* started = a.sync + kStarted;
        auto arrived = [&]() { return (int)(load_acquire(a.sync + kArrived) - all) >= 0; };
        int met = kAll;
        if (stage == 1) {
            const unsigned long long t0 = time_ns();
            for (unsigned tries = 1; !arrived(); ++tries) {
                if (tries & 7) continue;
                const unsigned here = *(volatile unsigned*)started;
                if (here == gridDim.x) break;                 // none missing: wait for them below
                if ((here & kShort) ||
                    (time_ns() - t0 > kGatherNs && atomicCAS(started, here, here | kShort) == here)) {
                    met = kFew;
                    break;
                }
            }
        }
        if (met == kAll && !wait_for(a, arrived)) met = kFailed;
        *s_met = met;
    }
    __syncthreads();
    return *s_met;
}

// The steps of a launch some of whose CTAs cannot start: CTA `rank` (in the order they started;
// 0 leads) and the others on the roster take every stage's nodes in turn, a warp's nodes at a
// time.  Weights, rows and pointwise values are read as a stage launch reads them, base state
// and accumulator lie in H and D, and the sums have the resident stage's order: the same bits.
// Those who took part in the first stage have written K rows of this one's first stage, with
// its values, before they come here.
template <typename T, int LPN, class Src>
__device__ __forceinline__ void share_steps(const Args<T>& a, const Src& src, unsigned rank) {
    constexpr int kNpw = 32 / LPN, kJpl = kSlots / LPN;
    __shared__ unsigned long long s_roster;
    __shared__ int s_in, s_go;                               // of the wait for the roster, of a stage's
    unsigned long long* roster = reinterpret_cast<unsigned long long*>(a.sync + kRoster);
    unsigned* shared = a.sync + kShared;
    auto look = [&]() {
        unsigned long long v;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(roster) : "memory");
        return v;
    };
    auto publish = [&](unsigned step) {
        const unsigned long long v = (unsigned long long)step << 32 | (*(volatile unsigned*)(a.sync + kStarted) & ~kShort);
        asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(roster), "l"(v) : "memory");
    };
    const bool wide_h = (reinterpret_cast<uintptr_t>(a.H) & 31) == 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int tl = lane % kNpw, sub = lane / kNpw;
    if (rank == 0 && threadIdx.x == 0) publish(1);
    for (unsigned step = 0; step <= (unsigned)a.nsteps;) {
        // the next step that this CTA is on the roster of, or the end (step nsteps + 1)
        if (threadIdx.x == 0) {
            unsigned long long v = 0, before = 0;
            bool mine = false;
            do {                                              // the limit starts anew with every step of the others
                before = v;
                s_in = wait_for(a, [&]() {
                    v = look();
                    mine = (v >> 32) > step && ((unsigned)v > rank || (v >> 32) > (unsigned)a.nsteps);
                    return mine || v != before;
                });
            } while (s_in && !mine);
            s_roster = v;
        }
        __syncthreads();
        if (!s_in) return;
        step = (unsigned)(s_roster >> 32);
        const unsigned few = (unsigned)s_roster;
        if (step > (unsigned)a.nsteps) return;
        for (int mode = 0; mode < 4; ++mode) {
            const T* Kin = mode == kStage0 ? a.H : mode == kStage2 ? a.Kb : a.Ka;
            T* Kout = mode == kStage3 ? a.H : mode == kStage1 ? a.Kb : a.Ka;
            const bool wide = mode != kStage0 || wide_h;
            for (long u = (long)rank * warps + warp; u * kNpw < a.n; u += (long)few * warps) {
                const long i = u * kNpw + tl, own = min(i, (long)a.n - 1);
                // the lane's rows at once, then its gathers
                int rows[kJpl];
#pragma unroll
                for (int jj = 0; jj < kJpl; ++jj)
                    rows[jj] = jj * LPN + sub < a.nnbr ? src.row(own, jj * LPN + sub, a.nnbr, a.n) : (int)own;
                T acc[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) acc[x] = T(0);
#pragma unroll
                for (int jj = 0; jj < kJpl; ++jj) {
                    if (jj * LPN >= a.nnbr) break;
                    T w[4] = {T(0), T(0), T(0), T(0)}, kv[4];
                    if (jj * LPN + sub < a.nnbr) src.weights(own, jj * LPN + sub, a.nnbr, w);
                    load_state(Kin + 4L * rows[jj], wide, kv);
#pragma unroll
                    for (int op = 0; op < 4; ++op)
#pragma unroll
                        for (int f = 0; f < 4; ++f) acc[op * 4 + f] += w[op] * kv[f];
                }
#pragma unroll
                for (int o = kNpw; o < 32; o <<= 1)
#pragma unroll
                    for (int x = 0; x < 16; ++x) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], o);
                if (sub != 0 || i >= a.n) continue;
                T pt[kPointStride], q[4], F[4], h[4], d[4];
#pragma unroll
                for (int f = 0; f < kPt; ++f) pt[f] = src.point(i, f);
                load_state(Kin + 4 * i, wide, q);
                pointwise_rhs(acc, q, pt, a.gh0, F);
                if (mode == kStage0) {
#pragma unroll
                    for (int x = 0; x < 4; ++x) q[x] = Quad<T>::axpy(q[x], a.c01, F[x]);
                    lane::put_row(a.D + 4 * i, F);
                } else {
                    load_state(a.H + 4 * i, wide_h, h);
                    load_state(a.D + 4 * i, true, d);
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        d[x] = Quad<T>::axpy(d[x], mode == kStage3 ? T(1) : T(2), F[x]);
                        q[x] = mode == kStage3 ? Quad<T>::update_h(h[x], a.dt6, d[x])
                                               : Quad<T>::axpy(h[x], mode == kStage1 ? a.c01 : a.c2, F[x]);
                    }
                    if (mode != kStage3) lane::put_row(a.D + 4 * i, d);
                }
                if (mode != kStage3 || wide_h) lane::put_row(Kout + 4 * i, q);
                else Quad<T>::store_row(Kout + 4 * i, q);
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                add_release(shared);
                s_go = 1;
                if (mode < 3 || rank == 0)
                    s_go = wait_for(a, [&]() { return load_acquire(shared) >= few * (unsigned)(mode + 1); });
                if (mode == 3 && rank == 0 && s_go) {         // all are done: the next step's count and roster
                    *(volatile unsigned*)shared = 0;
                    publish(step + 1);
                }
            }
            __syncthreads();
            if (!s_go) return;
        }
    }
}

// One block that waits, as after a step's second stage, for a block that was never launched:
// the path of a wait that runs out, without anything to run out of (swe_selftest_step_wait).
static __global__ void lone_block_kernel(Args<double> a) {
    __shared__ int ok;
    exchange(a, 2, &ok);             // (two stages done by a grid of one block)
}

template <typename T, int LPN, int THREADS, class Src, bool STREAM>
__global__ void __launch_bounds__(THREADS, 1) steps_kernel(const __grid_constant__ Args<T> a, const __grid_constant__ Src src) {
    constexpr int kNpw = 32 / LPN;          // nodes per warp
    constexpr int kJpl = kSlots / LPN;      // slots per lane
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_met;
    __shared__ unsigned s_started;
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
    if (threadIdx.x == 0) s_started = atomicAdd(a.sync + kStarted, 1u);
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
                *(volatile unsigned*)(a.sync + kAbort) = 1;
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

    int met = s_started & kShort ? kFew : kAll;      // the others went on without this CTA
    for (int s = 0; s < a.nsteps && met == kAll; ++s) {
        const bool last = s + 1 == a.nsteps;
        stage(std::integral_constant<int, kStage0>(), true);
        if ((met = exchange(a, ++done, &s_met)) != kAll) break;
        stage(std::integral_constant<int, kStage1>(), true);
        if ((met = exchange(a, ++done, &s_met)) != kAll) break;
        stage(std::integral_constant<int, kStage2>(), true);
        if ((met = exchange(a, ++done, &s_met)) != kAll) break;
        stage(std::integral_constant<int, kStage3>(), !last);
        if (!last) met = exchange(a, ++done, &s_met);
    }
    if (pending) filled();                 // broken off: no copy in flight when the block ends
    // (the streamed form has no registers to spare for these: 7.47 us a stage with them at
    // N=40962, 7.22 without; it leaves the steps to finish_kernel)
    if constexpr (!STREAM)
        if (met == kFew) share_steps<T, LPN>(a, src, s_started & ~kShort);
}

// Follows a launch of the streamed form: nothing to do, unless some of its CTAs could not start.
constexpr int kFinishThreads = 128, kFinishPerSm = 4;
template <typename T, int LPN, class Src>
__global__ void __launch_bounds__(kFinishThreads, kFinishPerSm)
finish_kernel(const __grid_constant__ Args<T> a, const __grid_constant__ Src src) {
    __shared__ unsigned s_rank;
    if (!(a.sync[kStarted - kSyncSet] & kShort)) return;      // a.sync: the second set
    if (threadIdx.x == 0) s_rank = atomicAdd(a.sync + kStarted, 1u);
    __syncthreads();
    share_steps<T, LPN>(a, src, s_rank);
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
    auto kernel = a.m * LPN <= kFewThreads ? steps_kernel<T, LPN, kFewThreads, Src, false> : steps_kernel<T, LPN, kMost, Src, false>;
    if constexpr (Src::kNodeFast && sizeof(T) == 8 && LPN == 2)
        if (stream) kernel = steps_kernel<T, LPN, kMost, Src, true>;
    // the device's limit in every call, never the call's own size: another thread may be
    // between its attribute and its launch
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(a.sync, 0, kSyncWords * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3((a.m * LPN + 31) / 32 * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    e = cudaLaunchKernelEx(&cfg, kernel, a, src);
    if constexpr (Src::kNodeFast && sizeof(T) == 8 && LPN == 2)
        if (stream && e == cudaSuccess) {
            Args<T> rest = a;
            rest.sync += kSyncSet;
            finish_kernel<T, LPN, Src><<<ctas * kFinishPerSm, kFinishThreads, 0, st>>>(rest, src);
            e = cudaGetLastError();
        }
    return e;
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
