// Node ordering on the device: swe_dev_rcm_mapping.
//
// The reference orders nodes by reverse Cuthill-McKee on the host
// (swe_code/rcm/rcm.c:9-62; restated in host_layout.cu): breadth-first from
// node 0, each visited node appending its not yet mapped stencil neighbours in
// increasing order of their count of still-unmapped neighbours.  That count
// changes after every append, so each step depends on all earlier ones and the
// exact permutation is sequential.
//
// This is the same breadth-first level structure built one level at a time, in
// parallel within a level, and reversed at the end:
//   * offer: every node of the current level offers itself as parent to its
//     unmapped stencil neighbours (slots 1..nnbr-1); a neighbour keeps the
//     smallest key (parent position in the order, slot), so children follow
//     their first parent, nearest stencil slot first;
//   * place: an offer whose key its neighbour kept names one child; counting
//     them in (parent, slot) order gives every child its position behind the
//     current level.
// Keys are (parent position, slot), not the reference's dynamic degree, so the
// permutation differs from the reference's; its bandwidth (max and mean over
// nodes of max - min stencil index, as rcm.c:68-96 prints it) is of the same
// size, which is what the gathers' locality depends on.  A level may hold at
// most kMaxLevel nodes (the breadth-first rings of a quasi-uniform spherical
// grid hold a few thousand up to N ~ 10^7).
//
// One cluster of 16 CTAs (8 where the device cannot place 16 together) walks all
// levels (order_levels below): a level is a few thousand nodes, too little for the
// whole chip, and the cluster's hardware barrier costs less than a launch and a
// read-back per level.
#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include "common.cuh"

namespace swe {
namespace {

constexpr int kMaxLevel = 16384;         // nodes per breadth-first level
constexpr int kThreads = 1024, kWarps = kThreads / 32;
constexpr int kHeld = 16;                // parents whose neighbours a warp keeps in shared memory
enum { kOrdered = 0, kTooWide = 1, kDisconnected = 2 };

struct OrderResult {
    unsigned long long bad;              // first out-of-range entry of idx, ~0 if none
    int status, reached;
};

__global__ void check_indices(int n, long count, const int* __restrict__ idx, OrderResult* __restrict__ res) {
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += (long)gridDim.x * blockDim.x) {
        const int v = idx[t];
        if (v < 0 || v >= n) atomicMin(&res->bad, (unsigned long long)t);
    }
}

// Warp w of the cluster's CTAS x 32 takes the w-th run of the level's parents, lane j stencil slot
// j; its share's neighbours stay in shared memory between the two phases.  key[v] holds the
// offer v kept, and one below the level's first parent says that v is placed already.
// Bound by three dependent L2 reads (order, stencil row, key) and three cluster barriers a
// level: N=655362, 256 levels, 2.9 ms with 16 CTAs and 4.4 with 8; with two launches, a
// one-CTA sort (10.4 ms) and a read-back per level it took 25 ms.
template <int CTAS>
__global__ void __launch_bounds__(kThreads, 1)
order_levels(int n, int nnbr, const int* __restrict__ idx, unsigned* __restrict__ key, int* __restrict__ order,
             int* __restrict__ mapping, OrderResult* __restrict__ res) {
    namespace cg = cooperative_groups;
    constexpr int kAllWarps = CTAS * kWarps, kShare = kMaxLevel / kAllWarps;   // most parents of a warp
    extern __shared__ int held[];                    // [warp][kHeld][32]
    __shared__ unsigned masks[kWarps][kShare];       // children of each of the warp's parents, by slot
    __shared__ int warp_sum[kWarps], cta_sum[CTAS];
    if (res->bad != ~0ull) return;                   // the same for every thread of the cluster
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (rank == 0 && threadIdx.x == 0) {             // level 0: node 0, where the reference's search starts
        order[0] = 0;
        mapping[n - 1] = 0;
        key[0] = 0;
    }
    cluster.sync();
    const bool slot = lane >= 1 && lane < nnbr;
    int* mine = held + warp * kHeld * 32 + lane;
    int lv0 = 0, lv1 = 1, status = kOrdered;
    while (lv1 < n) {
        const unsigned placed = (unsigned)lv0 << 5;
        const int share = (lv1 - lv0 + kAllWarps - 1) / kAllWarps;
        const int p0 = min(lv0 + (rank * kWarps + warp) * share, lv1), np = min(share, lv1 - p0);
        auto neighbour = [&](int p) { return slot ? __ldg(idx + (long)__ldcg(order + p) * nnbr + lane) : -1; };
#pragma unroll 4
        for (int q = 0; q < np; ++q) {
            const int w = neighbour(p0 + q);
            if (q < kHeld) mine[q * 32] = w;
            if (w < 0) continue;
            const unsigned offer = (unsigned)(p0 + q) << 5 | (unsigned)lane, has = __ldcg(key + w);
            if (has >= placed && has > offer) atomicMin(key + w, offer);
        }
        cluster.sync();
        int children = 0;
#pragma unroll 4
        for (int q = 0; q < np; ++q) {
            const int w = q < kHeld ? mine[q * 32] : neighbour(p0 + q);
            const bool won = w >= 0 && __ldcg(key + w) == ((unsigned)(p0 + q) << 5 | (unsigned)lane);
            const unsigned m = __ballot_sync(0xffffffffu, won);
            if (lane == 0) masks[warp][q] = m;
            children += __popc(m);
        }
        if (lane == 0) warp_sum[warp] = children;
        __syncthreads();
        if (warp == 0) {                             // exclusive scan of the CTA's warps
            const int v = warp_sum[lane];
            int incl = v;
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            warp_sum[lane] = incl - v;
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            if (lane < CTAS) *cluster.map_shared_rank(cta_sum + rank, lane) = total;
        }
        cluster.sync();
        int at = lv1 + warp_sum[warp], level = 0;
        for (int r = 0; r < CTAS; ++r) {
            if (r < rank) at += cta_sum[r];
            level += cta_sum[r];
        }
        if (level == 0 || level > kMaxLevel) {
            status = level ? kTooWide : kDisconnected;
            break;
        }
        for (int q = 0; q < np; ++q) {
            const unsigned m = masks[warp][q];
            if (m >> lane & 1) {
                const int w = q < kHeld ? mine[q * 32] : neighbour(p0 + q);
                const int pos = at + __popc(m & ((1u << lane) - 1));
                order[pos] = w;
                mapping[n - 1 - pos] = w;            // reversed
            }
            at += __popc(m);
        }
        cluster.sync();
        lv0 = lv1;
        lv1 += level;
    }
    if (rank == 0 && threadIdx.x == 0) {
        res->status = status;
        res->reached = lv1;
    }
    cluster.sync();                                  // no CTA leaves while another may write its sums
}

constexpr int kOrderSmem = kWarps * kHeld * 32 * (int)sizeof(int);

// Launches order_levels as one cluster; false (and no launch) where the device cannot hold it.
template <int CTAS>
bool launch_order(int n, int nnbr, const int* idx, unsigned* key, int* order, int* mapping, OrderResult* res,
                  cudaStream_t st, cudaError_t& e) {
    auto kernel = order_levels<CTAS>;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kOrderSmem);
    if (e == cudaSuccess && CTAS > 8) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return true;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CTAS);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kOrderSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CTAS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess || fit < 1) {
        cudaGetLastError();
        return false;
    }
    e = cudaLaunchKernelEx(&cfg, kernel, n, nnbr, idx, key, order, mapping, res);
    return true;
}

}  // namespace
}  // namespace swe

using namespace swe;

extern "C" int swe_dev_rcm_mapping(int n, int nnbr, const int* idx, int* mapping) {
    if (n <= 0 || n >= (1 << 24) || nnbr < 2 || nnbr > kSlots || !idx || !mapping) {
        set_error("swe_dev_rcm_mapping: need 0 < n < 2^24, 2 <= nnbr <= %d and both arrays", kSlots);
        return SWE_ERR_ARG;
    }
    // one allocation: result words, stencils, keys, order and the reversed order
    const size_t count = (size_t)n * nnbr, words = count + 3 * (size_t)n;
    char* mem = nullptr;
    cudaStream_t st = nullptr;
    OrderResult res{~0ull, kOrdered, 0};
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&mem, sizeof(OrderResult) + words * sizeof(int));
    if (e == cudaSuccess) {
        OrderResult* d_res = reinterpret_cast<OrderResult*>(mem);
        int* d_idx = reinterpret_cast<int*>(d_res + 1);
        unsigned* d_key = reinterpret_cast<unsigned*>(d_idx + count);
        int* d_order = reinterpret_cast<int*>(d_key + n);
        int* d_map = d_order + n;
        auto run = [&]() {
            cudaError_t r;
            if ((r = cudaMemcpyAsync(d_res, &res, sizeof(res), cudaMemcpyHostToDevice, st))) return r;
            if ((r = cudaMemcpyAsync(d_idx, idx, count * sizeof(int), cudaMemcpyHostToDevice, st))) return r;
            if ((r = cudaMemsetAsync(d_key, 0xff, (size_t)n * sizeof(unsigned), st))) return r;
            check_indices<<<(int)(count / 4096 < 1184 ? count / 4096 + 1 : 1184), 256, 0, st>>>(n, (long)count, d_idx, d_res);
            if ((r = cudaGetLastError())) return r;
            if (!launch_order<16>(n, nnbr, d_idx, d_key, d_order, d_map, d_res, st, r) &&
                !launch_order<8>(n, nnbr, d_idx, d_key, d_order, d_map, d_res, st, r))
                return cudaErrorLaunchOutOfResources;
            if (r) return r;
            count_launch(2);
            if ((r = cudaMemcpyAsync(&res, d_res, sizeof(res), cudaMemcpyDeviceToHost, st))) return r;
            if ((r = cudaStreamSynchronize(st))) return r;
            if (res.bad == ~0ull && res.status == kOrdered) {
                if ((r = cudaMemcpyAsync(mapping, d_map, (size_t)n * sizeof(int), cudaMemcpyDeviceToHost, st))) return r;
                r = cudaStreamSynchronize(st);
            }
            return r;
        };
        e = run();
    }
    if (mem) cudaFree(mem);
    if (st) cudaStreamDestroy(st);
    // a bad index is reported before any CUDA error: where the device did not get to check
    // (no device, no memory), the host does
    if (e != cudaSuccess)
        for (size_t t = 0; t < count && res.bad == ~0ull; ++t)
            if (idx[t] < 0 || idx[t] >= n) res.bad = t;
    if (e != cudaSuccess && res.bad == ~0ull) {
        set_error("swe_dev_rcm_mapping: %s", cudaGetErrorString(e));
        return SWE_ERR_CUDA;
    }
    if (res.bad != ~0ull) {
        set_error("swe_dev_rcm_mapping: idx[%ld] = %d outside [0, %d)", (long)res.bad, idx[res.bad], n);
        return SWE_ERR_INDEX;
    }
    if (res.status == kTooWide) {
        set_error("swe_dev_rcm_mapping: a breadth-first level holds more than %d nodes", kMaxLevel);
        return SWE_ERR_ARG;
    }
    if (res.status == kDisconnected) {
        set_error("swe_dev_rcm_mapping: stencil graph is not connected (%d of %d nodes reached)", res.reached, n);
        return SWE_ERR_ARG;
    }
    return SWE_OK;
}
