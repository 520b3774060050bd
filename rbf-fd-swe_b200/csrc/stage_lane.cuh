// Fused RK4 stage kernel, node-per-lane form (plain form, FP64 / FP32).
//
// Same stage semantics as stage_kernel.cuh (eval_RHS_swe plus the RK4 stage
// combine, swe_code/main/rk4_rbffd_swe.c:30-186 and :285-353), with a work split
// that needs little or no cross-lane reduction: each of a node's LPN lanes (1, 2
// or 4) sums the slots j = sub, sub + LPN, ... of the node serially, in the order
// of the packed arrays, and the LPN partial sums meet in a butterfly of
// log2(LPN) shuffle steps.  Lane sub 0 of every node then
// runs the pointwise part and the stage combine, so up to all 32 lanes of a warp
// are busy in the epilogue.
//
// The stencil weights and indices live in a second, tile-transposed copy
// (pack_stencils_kernel in pack.cuh): per 32-node tile, slot-major, node-minor,
// so one slot's weights of a warp's nodes are one contiguous 1024-byte (FP64) or
// 512-byte (FP32) row and one slot's indices a contiguous 64- or 128-byte row.
// Weights and FP64 state rows move as whole 32-byte sectors (256-bit loads): the L1
// data pipe is what the kernel spends most on when the data is in L2.  On small
// patches the slots are placed so that the lanes of a warp gather the same lines
// (pack_lanes_kernel has the rule).  N=40962 FP64: 10.2 us per stage with 128-bit
// loads, 8.7 with 256-bit loads, 7.7 with placed slots and the pointwise values
// transposed; N=10242 5.1 / 4.1 with 128- / 256-bit loads, N=655362 134.3 / 133.2.
// The pointwise values are transposed the same way: a record per node puts each field's
// load on 32 lines, a third of the L1 sectors of a whole stage: us per stage
// with records / transposed FP64 N=75000 13.3 / 11.8, N=163842 30.1 / 27.9, N=655362 126.5 /
// 120.6, FP32 N=655362 65.2 / 63.0.
// Weights and indices are streamed with L1 no-allocate loads; the
// neighbour gathers keep L1 to themselves.  One warp per unit of 32 / LPN nodes,
// no persistent loop: the hardware scheduler balances the tail.  MINB (4 or 5)
// is the register bound's CTAs per SM: 5 trades load depth for a grid that fits
// in one wave on mid-sized patches.  Programmatic dependent launch lets the next
// stage's CTAs take free SMs while the last wave of this stage finishes; every
// read of a state array comes after griddepcontrol.wait.  swe_cuda_init times
// the shapes (LPN x MINB x L2 prefetch) and keeps the fastest.
#pragma once

#include "stage_kernel.cuh"

namespace swe {

constexpr int kLaneThreads = 128;
constexpr int kLaneWarps = kLaneThreads / 32;
constexpr int kLaneTile = 32;      // nodes per transposed tile of the packed arrays

// Weights of more than 60 MB leave L2 (126 MB, shared with the state arrays, the pointwise
// records and the indices) between two stages when every stage reads them in the same order.
// From there on the stages alternate their direction and a quarter of the tiles is kept with
// L2 priority.  Microseconds per stage in one order without / alternating with priorities:
// FP64 N=40962 8.2 / 9.2 (weights 42 MB, below the line), N=60000 13.3 / 13.3, N=90000
// 21.0 / 17.6, N=163842 36.4 / 30.3, N=655362 131.7 / 126.1; FP32 N=125000 14.8 / 14.4,
// N=163842 18.4 / 14.9, N=655362 71.7 / 65.2.  Keeping 1/16, 1/8, 1/4, 1/2 or all of the
// tiles: 31.3, 30.8, 30.3, 31.3 and 32.6 (FP64 N=163842).  (Before the slots were placed and
// the pointwise values transposed; N=163842 28.2, N=655362 120.6 and FP32 14.9 and 63.6 since.)
constexpr int kLaneKeep = 16;      // tiles of every 64 kept in L2
inline bool lane_streams(long n, size_t fsize) { return n * kSlots * 4 * (long)fsize > 60L * 1000 * 1000; }

template <typename T>
struct LaneArgs {
    StageArgs<T> s;
    const T* Wl;       // [tile][slot][32 nodes][4] weights (Dx, Dy, Dz, L)
    const T* PTl;      // [tile][kPointFields][32 nodes] pointwise values
    const int* idxl;   // [tile][slot][32 nodes] gather rows
    const short* idxs; // the same as 16-bit offsets from the node's own row (clamped to n - 1)
    int l2_prefetch;   // 1: bulk L2 prefetch of each warp's contiguous blocks at its start
    int stream;        // 1: the weights do not fit in L2 (lane_streams)
    int nnbr;          // stencil slots in use: slots nnbr.. hold zero weights (a lane's last one is not read)
};

namespace lane {

__device__ __forceinline__ int ld_stream(const int* p) {
    int v;
    asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int ld_stream(const short* p) {
    short v;
    asm volatile("ld.global.nc.L1::no_allocate.b16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
// the four weights (Dx, Dy, Dz, L) of one slot of one node
__device__ __forceinline__ void weights(const double* p, uint64_t pol, double (&w)[4]) {
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f64 {%0, %1, %2, %3}, [%4], %5;"
                 : "=d"(w[0]), "=d"(w[1]), "=d"(w[2]), "=d"(w[3])
                 : "l"(p), "l"(pol));
}
__device__ __forceinline__ void weights(const float* p, uint64_t pol, float (&w)[4]) {
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3])
                 : "l"(p), "l"(pol));
}
// L2 priority of a tile's weights.  A patch whose weights do not fit in L2 reads them in
// alternating directions (LaneArgs::stream) and keeps kLaneKeep of every 64 tiles with
// priority, letting the others go first.
__device__ __forceinline__ uint64_t l2_normal() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_policy(int stream, long tile) {
    uint64_t last, first;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(last));
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(first));
    return !stream ? l2_normal() : (tile & 63) < kLaneKeep ? last : first;
}
// the pointwise values of node t of a tile
template <typename T>
__device__ __forceinline__ void points(const T* PTl, long tile, int t, T (&pt)[kPointFields]) {
    const T* p = PTl + tile * kPointFields * kLaneTile + t;
#pragma unroll
    for (int f = 0; f < kPointFields; ++f) pt[f] = __ldg(p + f * kLaneTile);
}
// one state row (u, v, w, h): a whole 32-byte sector in one load (FP64).  A coherent load: the
// stage before, resident beside this one, or this one itself writes the row.
__device__ __forceinline__ void state_row(const double* p, double (&v)[4]) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
                 : "l"(p));
}
__device__ __forceinline__ void state_row(const float* p, float (&v)[4]) { Quad<float>::load_row_rw(p, v); }
__device__ __forceinline__ void put_row(double* p, const double (&v)[4]) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3]) : "memory");
}
__device__ __forceinline__ void put_row(float* p, const float (&v)[4]) { Quad<float>::store_row(p, v); }
}  // namespace lane

// I16: read the gather rows from the 16-bit offsets (half the index bytes); every
// patch whose stencil rows lie within 32767 rows of their node (any RCM-ordered grid)
template <typename T, int MODE, int LPN, int MINB, bool I16>
__global__ void __launch_bounds__(kLaneThreads, MINB) stage_lane_kernel(const LaneArgs<T> la) {
    static_assert(LPN == 1 || LPN == 2 || LPN == 4, "1, 2 or 4 lanes per node");
    constexpr int kNpw = 32 / LPN;          // nodes per warp
    constexpr int kJpl = kSlots / LPN;      // slots per lane
    const StageArgs<T>& a = la.s;
    const int lane = threadIdx.x & 31;
    const int tl = lane % kNpw, sub = lane / kNpw;
    // odd stages run the tiles from the end: what the stage before read last is still in L2
    const long bid = (MODE & 1) && la.stream ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
    const long node0 = (bid * kLaneWarps + (threadIdx.x >> 5)) * kNpw;
    const int nvalid = (int)min((long)kNpw, (long)a.n - node0);
    // With l2_prefetch, one lane requests the warp's contiguous blocks into L2 up
    // front, so that the loads below wait on L2 rather than DRAM: this warp's share
    // of its tile's weight and index blocks (static: before the wait, overlapping
    // the previous stage), then its pointwise records and own / H / D rows.  On large
    // patches the extra requests compete with the demand loads; on small ones it
    // gains little now that the gather rows are read before the wait, so the
    // init-time timing keeps it only where it is clearly faster.
    constexpr uint32_t kTileW = kSlots * kLaneTile * 4 * sizeof(T), kTileI = kSlots * kLaneTile * (I16 ? 2 : 4);
    const bool pf = la.l2_prefetch != 0;
    if (pf && lane == 0 && nvalid > 0) {
        const long tb = node0 / kLaneTile;
        const int wt = (int)(node0 % kLaneTile) / kNpw;        // warp within its tile
        prefetch_l2_bulk(reinterpret_cast<const unsigned char*>(la.Wl) + tb * kTileW + wt * (kTileW / LPN), kTileW / LPN);
        const void* ib = I16 ? static_cast<const void*>(la.idxs) : static_cast<const void*>(la.idxl);
        prefetch_l2_bulk(reinterpret_cast<const unsigned char*>(ib) + tb * kTileI + wt * (kTileI / LPN), kTileI / LPN);
        if (wt == 0) prefetch_l2_bulk(la.PTl + tb * kPointFields * kLaneTile, (uint32_t)(kPointFields * kLaneTile * sizeof(T)));
    }
    // a warp's nodes lie in one tile of the packed arrays (kNpw divides 32); nodes
    // past n in the last tile have zero weights and gather a valid row
    const long i = node0 + tl;
    const long tile = i / kLaneTile;
    const int t = (int)(i % kLaneTile);
    const int* ip = la.idxl + (tile * kSlots + sub) * kLaneTile + t;
    const short* sp = la.idxs + (tile * kSlots + sub) * kLaneTile + t;
    const int own = (int)min(i, (long)a.n - 1) + a.pid0;   // the row the 16-bit offsets start from
    // the gather rows are static: with 2 or 4 lanes per node (16 or 8 rows a lane), or
    // at 3 CTAs per SM (168 registers), they are read before the wait, so that the
    // gathers issue as soon as the previous stage's states are visible (32 rows a
    // lane in 96 or 128 registers would spill)
    constexpr bool kEarlyRows = LPN > 1 || MINB <= 3;
    auto row = [&](int jj) {
        return I16 ? own + lane::ld_stream(sp + jj * LPN * kLaneTile) : lane::ld_stream(ip + jj * LPN * kLaneTile);
    };
    int prow[kEarlyRows ? kJpl : 1];
    if (kEarlyRows && nvalid > 0) {
#pragma unroll
        for (int jj = 0; jj < kJpl; ++jj)
            prow[kEarlyRows ? jj : 0] = jj < kJpl - 1 || jj * LPN + sub < la.nnbr ? row(jj) : own;
    }
    pdl_wait();                // neighbour states and H / D come from the previous stage
    pdl_trigger();
    if (nvalid <= 0) return;
    if (pf && lane == 0) {
        const uint32_t rows = (uint32_t)(nvalid * 4 * sizeof(T));
        prefetch_l2_bulk(a.Kin + 4 * (node0 + a.pid0), rows);
        if (MODE != kStage0 && MODE != kEvalOnly) {
            prefetch_l2_bulk(a.H + 4 * node0, rows);
            prefetch_l2_bulk(a.D + 4 * node0, rows);
        }
    }
    const T* wp = la.Wl + ((tile * kSlots + sub) * kLaneTile + t) * 4;
    const uint64_t pol = lane::l2_policy(la.stream, tile);
    T acc[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) acc[q] = T(0);
#pragma unroll
    for (int jj = 0; jj < kJpl; ++jj) {
        // a padding slot (zero weights) in a lane's last iteration moves no bytes (slot 31
        // of 31-neighbour stencils); a test in every iteration would keep the compiler
        // from issuing the other iterations' loads together
        if (jj == kJpl - 1 && jj * LPN + sub >= la.nnbr) continue;
        const int p = kEarlyRows ? prow[kEarlyRows ? jj : 0] : row(jj);
        T w[4], kv[4];
        lane::weights(wp + jj * LPN * kLaneTile * 4, pol, w);
        lane::state_row(a.Kin + 4L * p, kv);
#pragma unroll
        for (int op = 0; op < 4; ++op)
#pragma unroll
            for (int f = 0; f < 4; ++f) acc[op * 4 + f] += w[op] * kv[f];
    }
    if constexpr (LPN > 1) {
#pragma unroll
        for (int o = kNpw; o < 32; o <<= 1)
#pragma unroll
            for (int q = 0; q < 16; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
    }
    if (sub != 0 || i >= a.n) return;
    T q[4], F[4];
    lane::state_row(a.Kin + 4L * (i + a.pid0), q);
    T pt[kPointFields];
    lane::points(la.PTl, tile, t, pt);
    pointwise_rhs(acc, q, pt, a.gh0, F);
    if (MODE == kEvalOnly) {
        lane::put_row(a.F + 4 * i, F);
    } else if (MODE == kStage0) {
        // copy_fp_arr(D, F) and eval_K(H, K, F, dt/2): here K_in is H
        T kn[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) kn[x] = Quad<T>::axpy(q[x], a.c, F[x]);
        lane::put_row(a.D + 4 * i, F);
        lane::put_row(a.Kout + 4 * i, kn);
    } else {
        T h[4], d[4];
        lane::state_row(a.H + 4 * i, h);
        lane::state_row(a.D + 4 * i, d);
        if (MODE == kStage1 || MODE == kStage2) {
            // update_D(D, F, 2) and eval_K(H, K, F, c)
            T kn[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                d[x] = Quad<T>::axpy(d[x], T(2), F[x]);
                kn[x] = Quad<T>::axpy(h[x], a.c, F[x]);
            }
            lane::put_row(a.D + 4 * i, d);
            lane::put_row(a.Kout + 4 * i, kn);
        } else {
            // update_D(D, F, 1) and update_H(H, D, dt)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                d[x] = Quad<T>::axpy(d[x], T(1), F[x]);
                h[x] = Quad<T>::update_h(h[x], a.dt6, d[x]);
            }
            lane::put_row(a.H + 4 * i, h);
        }
    }
}

}  // namespace swe
