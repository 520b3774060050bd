// Device-side layout transforms of the static data (init of the plain form and
// grid registration of the serving form).
//
// The caller's arrays arrive in the reference's layouts: DM arrays (Dx, Dy, Dz, L,
// idx) of compute_size x padded_Nnbr values indexed by DM_LIN_ID, VECT arrays
// (p_u, p_v, p_w, gradghm) of compute_size x 3 values indexed by VECT_LIN_ID, and
// per-node arrays (x, y, z, f, ghm) -- swe_config.h:31-36.  They are copied to the
// device once and rearranged there by three kernels into every layout the stage
// kernels read:
//   * W / idx:   the 8-lanes-per-node layout (stage_kernel.cuh, stage_tma.cuh),
//   * Wl / idxl: the tile-transposed node-per-lane layout (stage_lane.cuh), the
//     slots of small patches placed so that neighbouring lanes gather the same
//     lines, and idxs, the same indices as 16-bit offsets from each node's own row,
//   * PT:        the pointwise records [node][kPointStride], and PTl, the same
//     values tile-transposed for the node-per-lane kernels.
// Slots j >= nnbr get zero weights and gather the node's own row; nodes past n in
// the last 32-node tile of Wl / idxl get zero weights and gather row pid0.  An
// index outside [0, rows) is reported as the first offending (node, slot) in
// row-major order.
#pragma once

#include <cuda_runtime.h>

#include <climits>
#include <vector>

#include "common.cuh"
#include "stage_kernel.cuh"
#include "stage_lane.cuh"

namespace swe {

template <typename T>
struct PackedStatic {
    T* W = nullptr;       // 8-lanes-per-node weights
    int* idx = nullptr;   // 8-lanes-per-node indices
    T* Wl = nullptr;      // tile-transposed weights
    int* idxl = nullptr;  // tile-transposed indices
    short* idxs = nullptr;  // the same as 16-bit offsets from the node's own row
    bool idxs_ok = false;   // every offset fits 16 bits
    T* PT = nullptr;      // pointwise records
    T* PTl = nullptr;     // tile-transposed pointwise values
    void release() {
        for (void* p : {(void*)W, (void*)idx, (void*)Wl, (void*)idxl, (void*)idxs, (void*)PT, (void*)PTl}) if (p) cudaFree(p);
        W = nullptr; idx = nullptr; Wl = nullptr; idxl = nullptr; idxs = nullptr; PT = PTl = nullptr;
        idxs_ok = false;
    }
};

// The 8-lanes-per-node layout: one thread per (node i, slot j), slots as given.
template <typename T>
__global__ void pack_stencils_kernel(const T* __restrict__ Dx, const T* __restrict__ Dy, const T* __restrict__ Dz,
                                     const T* __restrict__ L, const int* __restrict__ idx_raw, CallerLayout cl,
                                     int n, int nnbr, int rows, int pid0, T* __restrict__ W, int* __restrict__ idxp,
                                     unsigned long long* __restrict__ bad) {
    constexpr int U = Quad<T>::kUnits;
    constexpr int per_unit = 16 / (int)sizeof(T);
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)n * kSlots) return;
    const long i = t / kSlots;
    const int j = (int)(t % kSlots);
    T w[4] = {T(0), T(0), T(0), T(0)};
    int p = (int)i + pid0;
    if (j < nnbr) {
        const long dm = cl.dm(i, j);
        w[0] = Dx[dm]; w[1] = Dy[dm]; w[2] = Dz[dm]; w[3] = L[dm];
        const int q = idx_raw[dm];
        if (q < 0 || q >= rows) atomicMin(bad, ((unsigned long long)i << 32) | (unsigned)j);
        else p = q;
    }
    const int m = j / 8, k = j % 8;
#pragma unroll
    for (int op = 0; op < 4; ++op) {
        const long unit = ((i * kSlotChunks + m) * U + op / per_unit) * 8 + k;
        W[unit * per_unit + op % per_unit] = w[op];
    }
    idxp[(i * 8 + k) * 4 + m] = p;
}

// The node-per-lane layout: one warp per group of 128 / sizeof(row) consecutive nodes (4 in
// FP64, 8 in FP32), whose lanes gather one slot's rows in one pass of the L1 data pipe.  A
// pass costs a cycle per distinct 128-byte line, so with `place` the group's neighbours are
// placed to share lines: the first node's alternately from both ends of the ascending order
// of rows (neighbours on opposite sides cancel at once), every further node's into slots
// whose line another node of the group already reads, the rest into the slots left, in
// the same order.  Lines per 32 gathered rows, sorted slots / these (N=40962, reverse
// Cuthill-McKee order): FP64 19.0 / 15.1, FP32 10.9 / 9.4; on a spiral of 30000 nodes FP64
// 24.7 / 18.5, FP32 17.9 / 12.9.
//
// `place` is for kernels of two or more lanes a node, up to kPlacedNodes: their sums are as
// exact as in the caller's order or more so (FP32 right-hand side of N=40962 against 64 bits:
// 4.2e-5 in the caller's order, 2.2e-5 placed; two lanes' FP64 sums of N=10242 against longdouble:
// 5.2e-8 and, alternately from both ends, 3.3e-8).  Where one lane sums a node's 32 terms, the
// caller's order, nearest first, is the more exact one (N=163842: 1.8e-5 against 3.1e-5 placed,
// 3.6e-5 sorted), and past kPlacedNodes the gain is small: a stage of N=40962 FP64 takes 8.0 us
// in the caller's order and 7.2 placed, of 75,000 12.0 and 11.8, of 163,842 28.2 and 28.0,
// FP32 14.9 and 14.9, of 100,000 11.3 and 10.3.  The plain form packs again when the lanes of
// its kernel change (Plain::order_slots).
constexpr int kPlacedNodes = 148 * 5 * (kLaneThreads / 2);   // two lanes a node at 5 CTAs per SM fill the GPU once
inline bool places_slots(long n, int lanes) { return lanes > 1 && n <= kPlacedNodes; }
template <typename T>
__global__ void pack_lanes_kernel(const T* __restrict__ W, const int* __restrict__ idxp, int n, long npad, int nnbr,
                                  int pid0, bool place, T* __restrict__ Wl, int* __restrict__ idxl,
                                  short* __restrict__ idxs, int* __restrict__ wide) {
    constexpr int U = Quad<T>::kUnits, kPerUnit = 16 / (int)sizeof(T);
    constexpr int kGroup = 32 / (int)sizeof(T);      // nodes whose rows fill a pass
    constexpr int kRowsPerLine = 32 / (int)sizeof(T);
    constexpr int kWarps = 8;
    __shared__ int s_row[kWarps][32], s_src[kWarps][32], s_line[kWarps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long i0 = ((long)blockIdx.x * kWarps + warp) * kGroup;
    if (i0 >= npad) return;
    int have[kGroup];                                // lines this lane's slot reads so far
    for (int t = 0; t < kGroup; ++t) {
        const long i = i0 + t;
        // the node's rows, one a lane: alternately from both ends of their ascending order
        // (ties in slot order), or as given
        int p = i < n ? (int)i + pid0 : pid0, pos = lane, src = lane;
        if (i < n) {
            p = idxp[(i * 8 + lane % 8) * 4 + lane / 8];
            int rank = lane;
            if (place && lane < nnbr) {
                rank = 0;
                for (int o = 0; o < nnbr; ++o) {
                    const int q = __shfl_sync(nnbr < 32 ? (1u << nnbr) - 1 : 0xffffffffu, p, o);
                    rank += q < p || (q == p && o < lane);
                }
                rank = 2 * rank < nnbr ? 2 * rank : 2 * (nnbr - 1 - rank) + 1;
            }
            __syncwarp();
            s_row[warp][rank] = p;
            s_src[warp][rank] = lane;
            __syncwarp();
            p = s_row[warp][lane];
            src = s_src[warp][lane];
            const int line = p / kRowsPerLine;
            if (place && t > 0) {
                const unsigned used = nnbr < 32 ? (1u << nnbr) - 1 : 0xffffffffu;
                unsigned open = used;                // slots not taken
                pos = lane < nnbr ? -1 : lane;
                for (int k = 0; k < nnbr; ++k) {
                    const int want = __shfl_sync(0xffffffffu, line, k);
                    bool reads = false;
#pragma unroll
                    for (int u = 0; u < kGroup; ++u) reads = reads || (u < t && have[u] == want);
                    const unsigned m = __ballot_sync(0xffffffffu, reads) & open;
                    if (!m) continue;
                    const int slot = __ffs(m) - 1;
                    open &= ~(1u << slot);
                    if (lane == k) pos = slot;
                }
                const unsigned left = __ballot_sync(0xffffffffu, pos < 0);
                if (pos < 0) {                       // the k-th left over takes the k-th open slot
                    unsigned o = open;
                    for (int k = __popc(left & ((1u << lane) - 1)); k > 0; --k) o &= o - 1;
                    pos = __ffs(o) - 1;
                }
            }
            __syncwarp();
            s_line[warp][pos] = line;
            __syncwarp();
        }
#pragma unroll
        for (int u = 0; u < kGroup; ++u)
            if (u == t) have[u] = i < n ? s_line[warp][lane] : -1;
        const long b = i / kLaneTile, e = (b * kSlots + pos) * kLaneTile + i % kLaneTile;
        T w[4] = {T(0), T(0), T(0), T(0)};
        if (i < n)
#pragma unroll
            for (int op = 0; op < 4; ++op)
                w[op] = W[(((i * kSlotChunks + src / 8) * U + op / kPerUnit) * 8 + src % 8) * kPerUnit + op % kPerUnit];
#pragma unroll
        for (int op = 0; op < 4; ++op) Wl[4 * e + op] = w[op];
        idxl[e] = p;
        // 16-bit offset from the node's own row (past n: offset 0)
        const int off = i < n ? p - ((int)i + pid0) : 0;
        if (wide && (off < -32768 || off > 32767)) atomicOr(wide, 1);
        idxs[e] = (short)off;
    }
}

// The node-per-lane layout of n nodes from their 8-lanes-per-node layout, for a kernel of
// `lanes` lanes a node; wide: set where an offset does not fit 16 bits (null: not asked).
template <typename T>
inline cudaError_t pack_lanes(const T* W, const int* idx, int n, int nnbr, int pid0, int lanes, T* Wl, int* idxl,
                              short* idxs, int* wide, cudaStream_t st) {
    const long npad = ((long)n + kLaneTile - 1) / kLaneTile * kLaneTile, groups = npad * (long)sizeof(T) / 32;
    pack_lanes_kernel<T><<<(unsigned)((groups + 7) / 8), 256, 0, st>>>(W, idx, n, npad, nnbr, pid0, places_slots(n, lanes),
                                                                      Wl, idxl, idxs, wide);
    count_launch();
    return cudaGetLastError();
}

// One thread per node (and per place of the last tile).
template <typename T>
__global__ void pack_points_kernel(const T* __restrict__ x, const T* __restrict__ y, const T* __restrict__ z,
                                   const T* __restrict__ f, const T* __restrict__ ghm, const T* __restrict__ pu,
                                   const T* __restrict__ pv, const T* __restrict__ pw, const T* __restrict__ gg,
                                   CallerLayout cl, int n, long npad, T* __restrict__ PT, T* __restrict__ PTl) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npad) return;
    T r[kPointStride];
#pragma unroll
    for (int k = 0; k < kPointStride; ++k) r[k] = T(0);
    T* l = PTl + i / kLaneTile * kPointFields * kLaneTile + i % kLaneTile;
    if (i >= n) {                                    // past n in the last tile
#pragma unroll
        for (int k = 0; k < kPointFields; ++k) l[k * kLaneTile] = T(0);
        return;
    }
    r[PT_X] = x[i]; r[PT_Y] = y[i]; r[PT_Z] = z[i]; r[PT_F] = f[i]; r[PT_GHM] = ghm[i];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const long v = cl.vect(i, c);
        r[PT_PU + c] = pu[v]; r[PT_PV + c] = pv[v]; r[PT_PW + c] = pw[v]; r[PT_GG + c] = gg[v];
    }
#pragma unroll
    for (int k = 0; k < kPointStride; ++k) PT[i * kPointStride + k] = r[k];
#pragma unroll
    for (int k = 0; k < kPointFields; ++k) l[k * kLaneTile] = r[k];
}

namespace pack_detail {
// stream-ordered staging buffer: allocating and freeing it never waits for work
// on other streams (a persistent serving kernel may be running)
template <typename A>
inline cudaError_t upload(A** dst, const A* src, size_t count, cudaStream_t st, std::vector<void*>& owned) {
    cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(dst), count * sizeof(A), st);
    if (e != cudaSuccess) return e;
    owned.push_back(*dst);
    return cudaMemcpyAsync(*dst, src, count * sizeof(A), cudaMemcpyHostToDevice, st);
}
}  // namespace pack_detail

// Uploads the caller's static arrays (n nodes of a patch with `rows` gather rows,
// compute rows starting at pid0) and packs them on the device into `out` (which
// the caller releases).  Everything runs on a private non-blocking stream, so the
// call waits only for its own work.  Returns SWE_OK, SWE_ERR_INDEX (the message
// names the first out-of-range index) or SWE_ERR_CUDA / SWE_ERR_NOMEM.
template <typename T>
int pack_static_device(const CallerLayout& cl, int n, int rows, int pid0, int nnbr, const T* Dx, const T* Dy,
                       const T* Dz, const T* L, const int* idx, const T* x, const T* y, const T* z, const T* f,
                       const T* ghm, const T* pu, const T* pv, const T* pw, const T* gg, int lanes, PackedStatic<T>& out) {
    const size_t ndm = (size_t)n * cl.pnbr, nv = (size_t)n * 3;
    const long npad = ((long)n + kLaneTile - 1) / kLaneTile * kLaneTile;
    cudaStream_t st = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        set_error("static data packing: %s", cudaGetErrorString(e));
        return SWE_ERR_CUDA;
    }
    std::vector<void*> owned;
    auto drop_staging = [&]() {
        for (void* p : owned) cudaFreeAsync(p, st);
        owned.clear();
        cudaStreamSynchronize(st);
        cudaStreamDestroy(st);
    };
    auto fail = [&](cudaError_t err) {
        drop_staging();
        out.release();
        set_error("static data packing: %s", cudaGetErrorString(err));
        return err == cudaErrorMemoryAllocation ? SWE_ERR_NOMEM : SWE_ERR_CUDA;
    };
    T *tDx, *tDy, *tDz, *tL, *tx, *ty, *tz, *tf, *tghm, *tpu, *tpv, *tpw, *tgg;
    int* tidx;
    unsigned long long* bad = nullptr;
    using pack_detail::upload;
    if ((e = upload(&tDx, Dx, ndm, st, owned)) || (e = upload(&tDy, Dy, ndm, st, owned)) ||
        (e = upload(&tDz, Dz, ndm, st, owned)) || (e = upload(&tL, L, ndm, st, owned)) ||
        (e = upload(&tidx, idx, ndm, st, owned)) || (e = upload(&tx, x, (size_t)n, st, owned)) ||
        (e = upload(&ty, y, (size_t)n, st, owned)) || (e = upload(&tz, z, (size_t)n, st, owned)) ||
        (e = upload(&tf, f, (size_t)n, st, owned)) || (e = upload(&tghm, ghm, (size_t)n, st, owned)) ||
        (e = upload(&tpu, pu, nv, st, owned)) || (e = upload(&tpv, pv, nv, st, owned)) ||
        (e = upload(&tpw, pw, nv, st, owned)) || (e = upload(&tgg, gg, nv, st, owned)))
        return fail(e);
    constexpr int U = Quad<T>::kUnits;
    constexpr int per_unit = 16 / (int)sizeof(T);
    if ((e = cudaMalloc(&out.W, (size_t)n * kSlotChunks * U * 8 * per_unit * sizeof(T))) ||
        (e = cudaMalloc(&out.idx, (size_t)n * kSlots * sizeof(int))) ||
        (e = cudaMalloc(&out.Wl, (size_t)npad * kSlots * 4 * sizeof(T))) ||
        (e = cudaMalloc(&out.idxl, (size_t)npad * kSlots * sizeof(int))) ||
        (e = cudaMalloc(&out.idxs, (size_t)npad * kSlots * sizeof(short))) ||
        (e = cudaMalloc(&out.PT, (size_t)n * kPointStride * sizeof(T))) ||
        (e = cudaMalloc(&out.PTl, (size_t)npad * kPointFields * sizeof(T))))
        return fail(e);
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&bad), sizeof(*bad), st))) return fail(e);
    owned.push_back(bad);
    if ((e = cudaMemsetAsync(bad, 0xff, sizeof(*bad), st))) return fail(e);
    int* wide = nullptr;
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&wide), sizeof(int), st))) return fail(e);
    owned.push_back(wide);
    if ((e = cudaMemsetAsync(wide, 0, sizeof(int), st))) return fail(e);
    const long threads = (long)n * kSlots;
    pack_stencils_kernel<T><<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(tDx, tDy, tDz, tL, tidx, cl, n, nnbr,
                                                                              rows, pid0, out.W, out.idx, bad);
    if ((e = cudaGetLastError()) || (e = pack_lanes<T>(out.W, out.idx, n, nnbr, pid0, lanes, out.Wl, out.idxl, out.idxs, wide, st)))
        return fail(e);
    pack_points_kernel<T><<<(unsigned)((npad + 255) / 256), 256, 0, st>>>(tx, ty, tz, tf, tghm, tpu, tpv, tpw, tgg, cl,
                                                                         n, npad, out.PT, out.PTl);
    count_launch(2);
    unsigned long long hb = ULLONG_MAX;
    int hw = 1;
    if ((e = cudaGetLastError()) || (e = cudaMemcpyAsync(&hb, bad, sizeof(hb), cudaMemcpyDeviceToHost, st)) ||
        (e = cudaMemcpyAsync(&hw, wide, sizeof(hw), cudaMemcpyDeviceToHost, st)) || (e = cudaStreamSynchronize(st)))
        return fail(e);
    out.idxs_ok = hw == 0;
    drop_staging();
    if (hb != ULLONG_MAX) {
        const long i = (long)(hb >> 32);
        const int j = (int)(hb & 0xffffffffu);
        set_error("idx[node %ld][nbr %d] = %d outside the patch [0, %d)", i, j, idx[cl.dm(i, j)], rows);
        out.release();
        return SWE_ERR_INDEX;
    }
    return SWE_OK;
}

}  // namespace swe
