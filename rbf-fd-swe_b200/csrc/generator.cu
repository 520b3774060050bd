// Offline input generator on the GPU: nearest-neighbour stencils and RBF-FD
// weights (swe_gen_* entry points of include/swe_b200.h).
//
// The reference ships one input file and not the tool that made it
// (io/input.c:189-414 reads the binary format).  swe_b200/gen.py builds inputs
// for the larger grids; these kernels are its native GPU path.
//
// Stencils: the k nearest nodes of every node by chordal distance, self first,
// then by increasing distance, ties by node index.  Nodes are counting-sorted
// into a uniform grid of cubic cells covering [-1, 1]^3 with an edge h chosen
// from the expected k-nearest radius; a query scans the cells within `ring`
// cells of its own and keeps the k best candidates.  Every node within ring * h
// of the query lies in the scanned block, so when the k-th distance found is at
// most ring * h the answer is exact; otherwise the query is repeated with a
// wider ring.
//
// Weights, per node c with stencil x_1..x_n (n <= 32), in FP64:
//   tangent frame e1 = c x a / |c x a| (a = z, or x near the poles), e2 = c x e1;
//   rho = max_j |x_j - c|; (xi_j, eta_j) = ((x_j - c).e1, (x_j - c).e2) / rho;
//   P = the 15 monomials xi^(t-b) eta^b, t <= 4, ordered by t then b.
//   Projected gradient: [[r_ij^7, P], [P^T, 0]] w = [[7 rc_j^5 (c (c.x_j) - x_j) / rho^2],
//     [0, e1/rho, e2/rho, 0...]] with r_ij = |x_i - x_j| / rho, rc_j = |x_j - c| / rho
//     (three right-hand sides: x, y, z).
//   Hyperviscosity Delta^4: [[s_ij^9, P], [P^T, 0]] w = [[9^2 7^2 5^2 3^2 s_j / rho^8], [0]]
//     with s the tangent-plane distances (s_j = |(xi_j, eta_j)|).
// Each system (n + 15 unknowns) is solved by Gauss-Jordan elimination with partial
// pivoting, one warp per node, the augmented matrix spread over the lanes' registers.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace swe {
namespace gen {

constexpr int kMaxK = 32;          // stencil size limit
constexpr int kNPoly = 15;         // degree-4 polynomials in two variables

// ---- kNN ---------------------------------------------------------------------------------

struct Grid {
    int G;          // cells per dimension
    double h;       // cell edge
};

__device__ __forceinline__ int cell_coord(double v, const Grid& g) {
    int c = (int)floor((v + 1.0) / g.h);
    return min(max(c, 0), g.G - 1);
}

__global__ void cell_of_kernel(const double* __restrict__ X, int n, Grid g, int* __restrict__ cell,
                               int* __restrict__ count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int cx = cell_coord(X[3 * i], g), cy = cell_coord(X[3 * i + 1], g), cz = cell_coord(X[3 * i + 2], g);
    const int c = (cz * g.G + cy) * g.G + cx;
    cell[i] = c;
    atomicAdd(count + c, 1);
}

// Exclusive scan of the cell counts in three launches: sums of kScanBlock counts, their
// scan by one block, and the scan within each block.  start[cells] = n; cursor: a copy of
// start for the scatter.
constexpr int kScanThreads = 256, kScanPer = 8, kScanBlock = kScanThreads * kScanPer;

// exclusive prefix of one value per thread over a block of kScanThreads or 1024 threads
__device__ __forceinline__ int block_exclusive(int v, int* total, int* warp_sums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int w = lane < nw ? warp_sums[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    *total = warp_sums[31];
    return incl - v + (warp ? warp_sums[warp - 1] : 0);
}

__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(const int* __restrict__ count, long cells,
                                                                 int* __restrict__ sums) {
    __shared__ int ws[32];
    const long c0 = (long)blockIdx.x * kScanBlock + threadIdx.x * kScanPer;
    int v = 0;
    for (int q = 0; q < kScanPer; ++q) v += c0 + q < cells ? count[c0 + q] : 0;
    int total;
    block_exclusive(v, &total, ws);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) scan_top_kernel(int* __restrict__ sums, int blocks) {
    __shared__ int ws[32];
    int base = 0;
    for (int b0 = 0; b0 < blocks; b0 += 1024) {
        const int b = b0 + threadIdx.x;
        const int v = b < blocks ? sums[b] : 0;
        int total;
        const int ex = block_exclusive(v, &total, ws);
        if (b < blocks) sums[b] = base + ex;
        base += total;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kScanThreads) scan_cells_kernel(const int* __restrict__ sums, long cells, int n,
                                                                  int* __restrict__ count, int* __restrict__ start) {
    __shared__ int ws[32];
    const long c0 = (long)blockIdx.x * kScanBlock + threadIdx.x * kScanPer;
    int v[kScanPer], sum = 0;
    for (int q = 0; q < kScanPer; ++q) {
        v[q] = c0 + q < cells ? count[c0 + q] : 0;
        sum += v[q];
    }
    int total;
    int at = sums[blockIdx.x] + block_exclusive(sum, &total, ws);
    for (int q = 0; q < kScanPer; ++q)
        if (c0 + q < cells) {
            start[c0 + q] = at;
            count[c0 + q] = at;        // the scatter's cursor
            at += v[q];
        }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) start[cells] = n;
}

struct __align__(32) CellNode {    // a node in cell order
    double x, y, z;
    long long j;                   // its index
};

__global__ void scatter_kernel(const double* __restrict__ X, const int* __restrict__ cell, int n,
                               int* __restrict__ cursor, CellNode* __restrict__ sorted) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    CellNode c;
    c.x = X[3 * (long)i]; c.y = X[3 * (long)i + 1]; c.z = X[3 * (long)i + 2];
    c.j = i;
    sorted[atomicAdd(cursor + cell[i], 1)] = c;
}

// squared distance of node s from (px, py, pz)
__device__ __forceinline__ double dist2(const CellNode& s, double px, double py, double pz) {
    const double dx = s.x - px, dy = s.y - py, dz = s.z - pz;
    return dx * dx + dy * dy + dz * dz;
}

// One warp per query (queries in cell order, so that neighbouring warps read the same
// cells): the lanes take the candidates of the 27 cells around it, keep those within one
// cell edge in shared memory -- the answer is exact if they are at least k, since every node
// that near lies in those cells -- and each lane ranks its share of them by (distance, index).
// A query with fewer than k or more than kNear of them goes to the list of the general
// kernel below.  On quasi-uniform nodes about 45 of 150 candidates are that near (k = 31).
// Bound by the latency of the candidates' loads; one thread per query keeping a sorted list
// in local memory took 1.61 ms at N=40962 (most of it in dependent local loads), this 0.077.
constexpr int kNear = 96, kKnnWarps = 8;
__global__ void __launch_bounds__(32 * kKnnWarps) knn_warp_kernel(int n, Grid g, const int* __restrict__ start,
                                                                  const CellNode* __restrict__ sorted, int k,
                                                                  int* __restrict__ idx, int* __restrict__ miss,
                                                                  int* __restrict__ nmiss) {
    __shared__ double sd[kKnnWarps][kNear];
    __shared__ int sj[kKnnWarps][kNear];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = blockIdx.x * kKnnWarps + warp;
    if (q >= n) return;
    const CellNode me = sorted[q];
    const int cx = cell_coord(me.x, g), cy = cell_coord(me.y, g), cz = cell_coord(me.z, g);
    const double reach2 = g.h * g.h;
    // lane r < 9: the r-th run of cells (x - 1 .. x + 1 are contiguous)
    int first = 0, len = 0;
    if (lane < 9) {
        const int y = cy + lane % 3 - 1, z = cz + lane / 3 - 1;
        if (y >= 0 && y < g.G && z >= 0 && z < g.G) {
            const long row = ((long)z * g.G + y) * g.G;
            first = start[row + max(cx - 1, 0)];
            len = start[row + min(cx + 1, g.G - 1) + 1] - first;
        }
    }
    int end = len;                          // inclusive prefix of the lengths
    for (int o = 1; o < 16; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += t;
    }
    const int total = __shfl_sync(0xffffffffu, end, 8);
    const int shift = first - (end - len);  // candidate t of run r is sorted[t + shift of r]
    int near = 0;
    for (int t0 = 0; t0 < total; t0 += 32) {
        const int t = t0 + lane;
        int sh = __shfl_sync(0xffffffffu, shift, 0);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int e = __shfl_sync(0xffffffffu, end, r), s = __shfl_sync(0xffffffffu, shift, r + 1);
            if (t >= e) sh = s;
        }
        double d = 0.0;
        int j = 0;
        bool in = false;
        if (t < total) {
            const CellNode c = sorted[t + sh];
            d = dist2(c, me.x, me.y, me.z);
            j = (int)c.j;
            in = d <= reach2;
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        const int at = near + __popc(m & ((1u << lane) - 1));
        if (in && at < kNear) {
            sd[warp][at] = d;
            sj[warp][at] = j;
        }
        near += __popc(m);
    }
    const int i = (int)me.j;
    if (near < k || near > kNear) {
        if (lane == 0) miss[atomicAdd(nmiss, 1)] = i;
        return;
    }
    __syncwarp();
    for (int a = lane; a < near; a += 32) {
        const double d = sd[warp][a];
        const int j = sj[warp][a];
        int rank = 0;
        for (int b = 0; b < near; ++b) {
            const double e = sd[warp][b];
            rank += e < d || (e == d && sj[warp][b] < j);
        }
        if (rank < k) idx[(long)i * k + rank] = j;
    }
}

// One thread per query of `todo`: the k best (d2, index) pairs over the cells within `ring`.
// Queries whose k-th distance is not within the scanned radius go to `miss`.
__global__ void knn_kernel(const double* __restrict__ X, Grid g, const int* __restrict__ start,
                           const CellNode* __restrict__ sorted, int k, int ring, const int* __restrict__ todo,
                           int ntodo, int* __restrict__ idx, int* __restrict__ miss, int* __restrict__ nmiss) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= ntodo) return;
    const long i = todo[q];
    const double px = X[3 * i], py = X[3 * i + 1], pz = X[3 * i + 2];
    double bd[kMaxK];
    int bi[kMaxK];
    int m = 0;
    const int cx = cell_coord(px, g), cy = cell_coord(py, g), cz = cell_coord(pz, g);
    for (int z = max(cz - ring, 0); z <= min(cz + ring, g.G - 1); ++z)
        for (int y = max(cy - ring, 0); y <= min(cy + ring, g.G - 1); ++y) {
            const long row = ((long)z * g.G + y) * g.G;
            const long c0 = row + max(cx - ring, 0), c1 = row + min(cx + ring, g.G - 1);
            for (int s = start[c0]; s < start[c1 + 1]; ++s) {
                const CellNode c = sorted[s];
                const int j = (int)c.j;
                const double d = dist2(c, px, py, pz);
                if (m == k && (d > bd[k - 1] || (d == bd[k - 1] && j > bi[k - 1]))) continue;
                // insert, keeping (d, j) ascending
                int p = m < k ? m++ : k - 1;
                while (p > 0 && (bd[p - 1] > d || (bd[p - 1] == d && bi[p - 1] > j))) {
                    bd[p] = bd[p - 1];
                    bi[p] = bi[p - 1];
                    --p;
                }
                bd[p] = d;
                bi[p] = j;
            }
        }
    const double reach = ring * g.h;
    const bool ok = m == k && bd[k - 1] <= reach * reach;
    if (!ok) miss[atomicAdd(nmiss, 1)] = (int)i;
    else
        for (int t = 0; t < k; ++t) idx[i * k + t] = bi[t];
}

// ---- weights -------------------------------------------------------------------------------

__device__ __forceinline__ double ipow(double x, int e) {
    double r = 1.0;
    for (int t = 0; t < e; ++t) r *= x;
    return r;
}

// One warp solves one node's two systems, the augmented matrix in its lanes' values.
//
// Lane (g, h), g = lane & 15, h = lane >> 4, holds rows g, g + 16, g + 32 of columns
// 2 i + h: 3 x 25 values, so the two half-warps share every row and the trailing columns
// of an elimination step stay spread over all lanes.  Rows and columns 0..31 are the RBF
// block, 32..46 the polynomials, columns 47..49 the right-hand sides; places k..31 of a
// stencil of k < 32 nodes hold zeros and their steps are skipped (from column 15 on; before,
// they hold a row of the identity, which costs the wide stencils no branch).
//
// A step picks the largest |entry| of its column among the rows not yet used (its leading
// bits and row number in one 32-bit maximum over the warp: the largest to within 2^-14,
// ties to the smaller row), leaves the row in place, hands it to all lanes through shared
// memory and subtracts it from every other row, used ones included (Gauss-Jordan): the
// lanes that hold them would idle otherwise, and no back substitution follows.
//
// Bound by the latency of the steps' chain (maximum, pivot row through shared memory,
// reciprocal) and the fetch of the unrolled code: issue slots 42 % busy, FP64 pipe 27 %,
// stalls per issue 1.9 on fixed latencies, 1.0 on instructions, 0.9 on shared memory
// (N=40962).  12 warps an SM have 168 registers a thread, and part of the 3 x 25 values
// spills (888 bytes of stores and 1316 of loads a thread in the compiled code, from L1):
// 6.9 ms at N=163842, k = 31, against 9.3 ms with 8 warps of 254 registers and no spill, and
// 29.6 ms with the matrix in shared memory, one lane per row.
constexpr int kNodesPerCta = 2;               // one warp each
constexpr int kLoc = 25;                      // columns a lane holds
constexpr int kPolyRow = 32;                  // first polynomial row / column
constexpr int kRhsCol = kPolyRow + kNPoly;    // first right-hand side column
constexpr int kPolyLd = 17;                   // row stride of the polynomial table

struct __align__(16) NodeWork {
    double prow[2][2][kLoc + 1];              // pivot row [step parity][h][i]
    double x[kMaxK], y[kMaxK], z[kMaxK];      // stencil node coordinates
    double xi[kMaxK], eta[kMaxK];             // tangent-plane coordinates
    double rc[kMaxK];                         // |x_j - c| / rho
    double poly[kMaxK * kPolyLd];
};

// The pivot row's buffer is the parity of its column.  A lane reads it after the step's one
// __syncwarp, so a buffer may be written again two steps on: the step between has a
// __syncwarp that follows those reads.  Where two steps that follow each other share a
// parity -- after the padding columns of an odd k, and from the last column of one system to
// the first of the other -- the second starts with a __syncwarp of its own.
__host__ __device__ constexpr bool eliminates(int p, int k) { return p < kNPoly || p >= kPolyRow || p < k; }
__host__ __device__ constexpr bool fenced(int p) { return p == 0 || p == kPolyRow; }
constexpr bool pivot_rows_ordered() {
    for (int k = 1; k <= kMaxK; ++k) {
        int before = -1;
        for (int q = 0; q < 2 * kRhsCol; ++q) {
            const int p = q % kRhsCol;
            if (!eliminates(p, k)) continue;
            if (before >= 0 && (before & 1) == (p & 1) && !fenced(p)) return false;
            before = p;
        }
    }
    return true;
}
static_assert(pivot_rows_ordered(), "a pivot row is overwritten while lanes may still read it");

__device__ __forceinline__ void poly15(double xi, double eta, double* out) {
    int col = 0;
    for (int t = 0; t <= 4; ++t)
        for (int b = 0; b <= t; ++b) out[col++] = ipow(xi, t - b) * ipow(eta, b);
}

// D: [4][n][k] (Dx, Dy, Dz, L) unit-sphere weights.
__global__ void __launch_bounds__(32 * kNodesPerCta, 6)
weights_kernel(const double* __restrict__ X, const int* __restrict__ idx, int n, int k, double* __restrict__ D,
               int* __restrict__ status) {
    __shared__ NodeWork works[kNodesPerCta];
    const int lane = threadIdx.x & 31;
    const int node = blockIdx.x * kNodesPerCta + (threadIdx.x >> 5);
    if (node >= n) return;
    NodeWork& w = works[threadIdx.x >> 5];
    const int g = lane & 15, h = lane >> 4;
    const double c0 = X[3 * (long)node], c1 = X[3 * (long)node + 1], c2 = X[3 * (long)node + 2];
    // tangent frame
    double ax0 = 0.0, ax1 = 0.0, ax2 = 1.0;
    if (fabs(c2) >= 0.9) { ax0 = 1.0; ax2 = 0.0; }
    double e10 = c1 * ax2 - c2 * ax1, e11 = c2 * ax0 - c0 * ax2, e12 = c0 * ax1 - c1 * ax0;
    const double en = sqrt(e10 * e10 + e11 * e11 + e12 * e12);
    e10 /= en; e11 /= en; e12 /= en;
    const double e20 = c1 * e12 - c2 * e11, e21 = c2 * e10 - c0 * e12, e22 = c0 * e11 - c1 * e10;
    // lane j: stencil node j; radius
    double px = 0.0, py = 0.0, pz = 0.0, dist = 0.0;
    if (lane < k) {
        const long s = idx[(long)node * k + lane];
        px = X[3 * s]; py = X[3 * s + 1]; pz = X[3 * s + 2];
        const double d0 = px - c0, d1 = py - c1, d2 = pz - c2;
        dist = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
    }
    double rho = dist;
    for (int o = 16; o > 0; o >>= 1) rho = fmax(rho, __shfl_xor_sync(0xffffffffu, rho, o));
    const double irho2 = 1.0 / (rho * rho);
    {
        const double d0 = px - c0, d1 = py - c1, d2 = pz - c2;
        const double xi = (d0 * e10 + d1 * e11 + d2 * e12) / rho, eta = (d0 * e20 + d1 * e21 + d2 * e22) / rho;
        w.x[lane] = px; w.y[lane] = py; w.z[lane] = pz;
        w.xi[lane] = xi; w.eta[lane] = eta; w.rc[lane] = dist / rho;
        poly15(xi, eta, w.poly + lane * kPolyLd);
    }
    __syncwarp();
    bool ok = true;
#pragma unroll 1
    for (int sys = 0; sys < 2 && ok; ++sys) {
        double m[3][kLoc];
        // RBF rows g and g + 16
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int r = g + 16 * s;
            const bool rv = r < k;
            const double rx = sys == 0 ? w.x[r] : w.xi[r], ry = sys == 0 ? w.y[r] : w.eta[r], rz = w.z[r];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int c = 2 * i + h;
                double v;
                if (sys == 0) {
                    const double d0 = rx - w.x[c], d1 = ry - w.y[c], d2 = rz - w.z[c];
                    const double t = (d0 * d0 + d1 * d1 + d2 * d2) * irho2;
                    v = t * t * t * sqrt(t);                      // r^7
                } else {
                    const double a = rx - w.xi[c], b = ry - w.eta[c];
                    const double t = a * a + b * b;
                    v = (t * t) * (t * t) * sqrt(t);              // r^9
                }
                m[s][i] = rv && c < k ? v : c == r && r < kNPoly ? 1.0 : 0.0;
            }
#pragma unroll
            for (int i = 16; i < 23; ++i) m[s][i] = rv ? w.poly[r * kPolyLd + 2 * (i - 16) + h] : 0.0;
            // column 46 (h = 0), the last polynomial; right-hand sides in columns 47 (h = 1), 48, 49
            double f0, f1, f2;
            if (sys == 0) {
                const double cdot = c0 * rx + c1 * ry + c2 * rz;
                const double f = 7.0 * ipow(w.rc[r], 5) / (rho * rho);
                f0 = f * (c0 * cdot - rx); f1 = f * (c1 * cdot - ry); f2 = f * (c2 * cdot - rz);
            } else {
                const double cl = (double)(9 * 7 * 5 * 3) * (double)(9 * 7 * 5 * 3);
                f0 = cl * sqrt(rx * rx + ry * ry) / ipow(rho, 8); f1 = 0.0; f2 = 0.0;
            }
            m[s][23] = rv ? (h == 0 ? w.poly[r * kPolyLd + 14] : f0) : 0.0;
            m[s][24] = rv ? (h == 0 ? f1 : f2) : 0.0;
        }
        // polynomial row 32 + g (g = 15: padding)
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int c = 2 * i + h;
            m[2][i] = g < kNPoly && c < k ? w.poly[c * kPolyLd + g] : 0.0;
        }
#pragma unroll
        for (int i = 16; i < kLoc; ++i) m[2][i] = 0.0;
        if (sys == 0 && (g == 1 || g == 2)) {
            if (h == 1) m[2][23] = (g == 1 ? e10 : e20) / rho;
            m[2][24] = h == 0 ? (g == 1 ? e11 : e21) / rho : (g == 1 ? e12 : e22) / rho;
        }
        int used = 0;                         // bit s: row g + 16 s has been a pivot row
        int pcol[3] = {-1, -1, -1};           // its column
        double pval[3] = {1.0, 1.0, 1.0};     // its pivot
#pragma unroll
        for (int p = 0; p < kRhsCol; ++p) {
            if (!eliminates(p, k)) continue;                      // padding of a narrower stencil
            const int hp = p & 1, ip = p >> 1;                    // where column p is held
            double v[3];
            unsigned key = 0;
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                v[s] = __shfl_sync(0xffffffffu, m[s][ip], hp * 16 + g);
                const unsigned hi = (unsigned)__double2hiint(v[s]) & 0x7fffffffu;
                // zeros and NaN are no pivots
                const bool can = !(used >> s & 1) && (hi | (unsigned)__double2loint(v[s])) != 0 && hi <= 0x7ff00000u;
                key = max(key, can ? max(hi & ~63u, 64u) | (unsigned)(63 - (g + 16 * s)) : 0u);
            }
            key = __reduce_max_sync(0xffffffffu, key);
            ok = ok && key >= 64u;
            const int br = 63 - (int)(key & 63u);
            double* pr = w.prow[p & 1][h];
            if (fenced(p)) __syncwarp();
#pragma unroll
            for (int s = 0; s < 3; ++s)
                if (br == g + 16 * s) {
#pragma unroll
                    for (int i = ip & ~1; i < kLoc; i += 2)
                        *reinterpret_cast<double2*>(pr + i) = make_double2(m[s][i], i + 1 < kLoc ? m[s][i + 1 < kLoc ? i + 1 : i] : 0.0);
                }
            __syncwarp();
            const double piv = w.prow[p & 1][hp][ip];
            const double rp = 1.0 / piv;
            double f[3];
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                // v / piv by the reciprocal and one correction: exactly 1 where v == piv, so
                // that the rows of coincident nodes cancel to zero
                const double q0 = v[s] * rp;
                f[s] = fma(fma(-q0, piv, v[s]), rp, q0);
                if (br == g + 16 * s) {
                    f[s] = 0.0;
                    used |= 1 << s;
                    pcol[s] = p;
                    pval[s] = piv;
                }
            }
#pragma unroll
            for (int i = (ip + hp) & ~1; i < kLoc; i += 2) {
                const double2 t = *reinterpret_cast<const double2*>(pr + i);
#pragma unroll
                for (int s = 0; s < 3; ++s) {
                    if (i >= ip + hp) m[s][i] -= f[s] * t.x;
                    if (i + 1 < kLoc) m[s][i + 1 < kLoc ? i + 1 : i] -= f[s] * t.y;
                }
            }
        }
        if (ok) {
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const int j = pcol[s];
                if (j < 0 || j >= k) continue;
                double* out = D + (long)node * k + j;
                const long op = (long)n * k;
                if (sys == 0) {
                    if (h == 1) {
                        out[0] = m[s][23] / pval[s];
                        out[2 * op] = m[s][24] / pval[s];
                    } else {
                        out[op] = m[s][24] / pval[s];
                    }
                } else if (h == 1) {
                    out[3 * op] = m[s][23] / pval[s];
                }
            }
        }
    }
    if (!ok && lane == 0) atomicExch(status, 1);
}

}  // namespace gen
}  // namespace swe

using namespace swe;
using namespace swe::gen;

extern "C" {

int swe_gen_stencils(int n, int k, const double* X, int* idx) {
    if (n <= 0 || k <= 0 || k > kMaxK || k > n || !X || !idx) {
        set_error("swe_gen_stencils: need n > 0, 1 <= k <= min(n, %d), device X and idx", kMaxK);
        return SWE_ERR_ARG;
    }
    // cell edge from the expected k-nearest radius of n quasi-uniform points on the unit sphere
    Grid g;
    // (at most 256^3 cells: beyond ~3M nodes cells hold more nodes, the answer stays exact)
    g.h = std::max(1.2 * std::sqrt(4.0 * k / n), 2.0 / 256.0);
    g.G = std::max(1, std::min(256, (int)std::ceil(2.0 / g.h)));
    g.h = 2.0 / g.G;
    const long cells = (long)g.G * g.G * g.G;
    const int blocks = ceil_div(cells, kScanBlock);
    // one allocation: nodes in cell order, then the cells' counts and starts, block sums, each
    // node's cell (later a list of queries), the other list, and the lists' lengths
    const size_t lists = (size_t)cells + (cells + 1) + blocks + 2 * (size_t)n + 2;
    char* mem = nullptr;
#define GEN_TRY(call)                                                                  \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess) {                                                       \
            set_error("%s: %s", #call, cudaGetErrorString(e_));                        \
            cudaFree(mem);                                                             \
            return SWE_ERR_CUDA;                                                       \
        }                                                                              \
    } while (0)
    GEN_TRY(cudaMalloc(&mem, n * sizeof(CellNode) + lists * sizeof(int)));
    CellNode* sorted = reinterpret_cast<CellNode*>(mem);
    int* count = reinterpret_cast<int*>(mem + n * sizeof(CellNode));
    int* start = count + cells;
    int* sums = start + cells + 1;
    int* list[2] = {sums + blocks, sums + blocks + n};
    int* nlist = list[1] + n;
    GEN_TRY(cudaMemsetAsync(count, 0, cells * sizeof(int), 0));
    GEN_TRY(cudaMemsetAsync(nlist, 0, 2 * sizeof(int), 0));
    const int T = 256;
    cell_of_kernel<<<ceil_div(n, T), T>>>(X, n, g, list[0], count);
    scan_sums_kernel<<<blocks, kScanThreads>>>(count, cells, sums);
    scan_top_kernel<<<1, 1024>>>(sums, blocks);
    scan_cells_kernel<<<blocks, kScanThreads>>>(sums, cells, n, count, start);
    scatter_kernel<<<ceil_div(n, T), T>>>(X, list[0], n, count, sorted);
    // within a cell the scatter order is arbitrary; the query's (distance, index)
    // ordering makes the result independent of it
    int cur = 1;
    knn_warp_kernel<<<ceil_div(n, kKnnWarps), 32 * kKnnWarps>>>(n, g, start, sorted, k, idx, list[cur], nlist + cur);
    count_launch(6);
    GEN_TRY(cudaGetLastError());
    int todo = 0;
    GEN_TRY(cudaMemcpy(&todo, nlist + cur, sizeof(int), cudaMemcpyDeviceToHost));
    for (int ring = 1; todo > 0; ++ring) {
        if (ring > g.G) {
            set_error("swe_gen_stencils: %d nodes found fewer than %d neighbours", todo, k);
            cudaFree(mem);
            return SWE_ERR_ARG;
        }
        const int next = 1 - cur;
        GEN_TRY(cudaMemsetAsync(nlist + next, 0, sizeof(int), 0));
        knn_kernel<<<ceil_div(todo, 128), 128>>>(X, g, start, sorted, k, ring, list[cur], todo, idx, list[next],
                                                 nlist + next);
        count_launch();
        GEN_TRY(cudaGetLastError());
        GEN_TRY(cudaMemcpy(&todo, nlist + next, sizeof(int), cudaMemcpyDeviceToHost));
        cur = next;
    }
#undef GEN_TRY
    cudaFree(mem);
    return SWE_OK;
}

int swe_gen_weights(int n, int k, const double* X, const int* idx, double* D) {
    if (n <= 0 || k <= 0 || k > kMaxK || !X || !idx || !D) {
        set_error("swe_gen_weights: need n > 0, 1 <= k <= %d and device X, idx, D", kMaxK);
        return SWE_ERR_ARG;
    }
    int* status = nullptr;
    SWE_CUDA_TRY(cudaMalloc(&status, sizeof(int)));
    SWE_CUDA_TRY(cudaMemset(status, 0, sizeof(int)));
    weights_kernel<<<ceil_div(n, kNodesPerCta), 32 * kNodesPerCta>>>(X, idx, n, k, D, status);
    count_launch();
    cudaError_t e = cudaGetLastError();
    int h = 0;
    if (e == cudaSuccess) e = cudaMemcpy(&h, status, sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(status);
    if (e != cudaSuccess) {
        set_error("swe_gen_weights: %s", cudaGetErrorString(e));
        return SWE_ERR_CUDA;
    }
    if (h) {
        set_error("swe_gen_weights: a local system was singular (coincident stencil nodes?)");
        return SWE_ERR_ARG;
    }
    return SWE_OK;
}

}  // extern "C"
