// RK4 steps with no device allocation: swe_cuda_step_noalloc.
//
// Some callers cannot call cudaMalloc: hosts whose device memory is owned by
// an outer framework's pool, and latency-critical loops where an allocation's
// implicit device synchronisation is not allowed.  They hand over every input
// and output as device pointers they already own; the only other memory this
// path needs -- the RK4 registers K (two ping-pong copies) and D -- lives in
// the file-scope array below, of SWE_NOALLOC_SCRATCH_BYTES.
//
// The array occupies that much memory on every GPU that loads this library,
// for the life of the process.  All calls share it: two calls whose kernels
// overlap on the GPU (different streams, or different host threads) race on
// it and give wrong results; serialise them.  Nothing in it has to start at
// zero: within one call every K and D value is written by a stage before any
// stage reads it, so the previous call's contents are never seen.
//
// The kernels are the fused stage kernel's math (stage_kernel.cuh) reading the
// caller's row-major arrays directly instead of the packed device layout that
// swe_cuda_init builds, so no packing buffer is needed either.  Grids of a few
// thousand nodes or more whose static data fits in the SMs' shared memory run a
// whole call in the resident kernel (resident.cuh), which lays it out there.
//
// The other entry points check every stencil index while packing it; here the
// indices are read straight from the caller's device array, so the kernel
// checks them as it gathers.  An index outside 0..n-1 is never dereferenced:
// the gather reads the node's own row instead (so that call's results are
// wrong), and the first such (node, slot, value) is kept in g_noalloc_bad.  A
// call with nsteps = 0 waits for `stream`, reports a kept record as
// SWE_ERR_INDEX and clears it.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "resident.cuh"
#include "stage_kernel.cuh"

namespace swe {
namespace {

constexpr size_t kNoallocScratchBytes = (size_t)4 << 20;
static_assert(kNoallocScratchBytes == SWE_NOALLOC_SCRATCH_BYTES, "header and file disagree");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocScratchBytes];

// First out-of-range stencil index met by a kernel: {seen, node, slot, value}.
// Zero at load; cleared by the nsteps = 0 call that reports it.
static __device__ int g_noalloc_bad[4];

// Arrival counter and abort word of the resident kernel, and its record of a wait that ran
// out (cleared by the nsteps = 0 call that reports it).
static __device__ __align__(128) unsigned g_noalloc_sync[res::kSyncWords];
static __device__ int g_noalloc_failed;

__device__ __forceinline__ int checked_neighbour(int v, int n, long node, int slot) {
    if ((unsigned)v < (unsigned)n) return v;
    if (atomicCAS(&g_noalloc_bad[0], 0, 1) == 0) {
        g_noalloc_bad[1] = (int)node;
        g_noalloc_bad[2] = slot;
        g_noalloc_bad[3] = v;
    }
    return (int)node;
}

// Device addresses of the scratch array, one per device, filled by the first
// call on that device (cudaGetSymbolAddress with that device current).  In
// host code the array's name is only a stand-in, so kernels get these.
constexpr int kMaxDevices = 64;
std::mutex g_setup_mu;
struct StaticArrays {
    void* scratch = nullptr;
    unsigned* sync = nullptr;
    int* failed = nullptr;
    int sms = 0;
    size_t smem = 0;          // shared memory a CTA may use
};
StaticArrays g_arrays[kMaxDevices];

template <typename T>
struct RowMajorArgs {
    int n, nnbr;
    const int* idx;                // [n][nnbr], 0-based
    const T *Dx, *Dy, *Dz, *L;     // [n][nnbr]
    const T *x, *y, *z, *f, *ghm;  // [n]
    const T *pu, *pv, *pw, *gg;    // [n][3]
    const T* Kin;                  // gather source [n][4]
    T* H;                          // [n][4] RK base state (the caller's buffer, in/out)
    T* D;                          // [n][4] scratch
    T* Kout;                       // [n][4] scratch
    T gh0;
    T c;                           // dt/2, dt/2, dt for stages 0-2
    double dt6;                    // dt/6
};

// One warp per 4 nodes, 8 lanes a node, slots j = k, k + 8, ... of lane k, as in
// stage_kernel.  Everything static -- weights, rows, pointwise values -- is requested
// before griddepcontrol.wait, so that a stage after the first starts on its gathers as
// soon as the previous stage's states are visible, with its other operands on the way or
// in place; the launches depend on one another programmatically (run_noalloc).
// Bound by the chain of dependent L2 reads and the hand-over between launches: N=10242
// FP64 6.4 us per stage, N=2562 3.1; 8.2 and 6.4 with plain launches and every load after
// the launch.  Grids that fit the resident kernel take that from a few thousand nodes on
// (resident_pays).
constexpr int kRowThreads = 128, kRowWarps = kRowThreads / 32;
template <typename T, int MODE>
__global__ void __launch_bounds__(kRowThreads, 4) rowmajor_stage_kernel(const RowMajorArgs<T> a) {
    constexpr bool kHD = MODE == kStage1 || MODE == kStage2 || MODE == kStage3;
    __shared__ __align__(16) T red[kRowWarps][4][16];
    __shared__ __align__(16) T ep[kRowWarps][4][kPointStride + 12];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 3, k = lane & 7;
    const long i = ((long)blockIdx.x * kRowWarps + warp) * 4 + g;
    const bool valid = i < a.n;
    const long ii = valid ? i : (long)a.n - 1;
    T* e = ep[warp][g];
    T w[kSlotChunks][4];
    int row[kSlotChunks];
#pragma unroll
    for (int m = 0; m < kSlotChunks; ++m) {
        const int j = 8 * m + k;
        row[m] = -1;
        if (j < a.nnbr) {
            const long x = ii * a.nnbr + j;
            row[m] = __ldg(a.idx + x);
            w[m][0] = __ldg(a.Dx + x); w[m][1] = __ldg(a.Dy + x); w[m][2] = __ldg(a.Dz + x); w[m][3] = __ldg(a.L + x);
        }
    }
    // pointwise values: lane k fetches the k-th scalar and the k-th vector
    if (k < 5) e[k] = __ldg((k == 0 ? a.x : k == 1 ? a.y : k == 2 ? a.z : k == 3 ? a.f : a.ghm) + ii);
    if (k < 4) {
        const T* v = (k == 0 ? a.pu : k == 1 ? a.pv : k == 2 ? a.pw : a.gg) + 3 * ii;
#pragma unroll
        for (int c = 0; c < 3; ++c) e[PT_PU + 3 * k + c] = __ldg(v + c);
    }
#pragma unroll
    for (int m = 0; m < kSlotChunks; ++m)
        if (8 * m + k < a.nnbr) row[m] = checked_neighbour(row[m], a.n, ii, 8 * m + k);
    pdl_wait();
    pdl_trigger();
    // (coherent loads: the stage before, resident beside this one, writes these rows)
    T kv[kSlotChunks][4];
#pragma unroll
    for (int m = 0; m < kSlotChunks; ++m)
        if (row[m] >= 0) Quad<T>::load_row_rw(a.Kin + 4L * row[m], kv[m]);
    // lanes 5-7: the own state and the H and D rows
    if (k == 5 || (kHD && k > 5)) {
        T r[4];
        Quad<T>::load_row_rw((k == 5 ? a.Kin : k == 6 ? a.H : a.D) + 4 * ii, r);
#pragma unroll
        for (int x = 0; x < 4; ++x) e[kPointStride + 4 * (k - 5) + x] = r[x];
    }
    T acc[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) acc[t] = T(0);
#pragma unroll
    for (int m = 0; m < kSlotChunks; ++m)
        if (row[m] >= 0) {
#pragma unroll
            for (int op = 0; op < 4; ++op)
#pragma unroll
                for (int fld = 0; fld < 4; ++fld) acc[op * 4 + fld] += w[m][op] * kv[m][fld];
        }
    T r0, r1;
    reduce_scatter8(acc, k, r0, r1);
    red[warp][g][2 * k] = r0;
    red[warp][g][2 * k + 1] = r1;
    __syncwarp();
    if (k != 0 || !valid) return;
    T s[16], q[4], F[4];
#pragma unroll
    for (int t = 0; t < 16; ++t) s[t] = red[warp][g][t];
#pragma unroll
    for (int t = 0; t < 4; ++t) q[t] = e[kPointStride + t];
    pointwise_rhs(s, q, e, a.gh0, F);
    const T* h = e + kPointStride + 4;
    const T* d = h + 4;
    T out[4], dn[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        if (MODE == kStage0) {
            dn[t] = F[t];
            out[t] = Quad<T>::axpy(q[t], a.c, F[t]);
        } else if (MODE != kStage3) {
            dn[t] = Quad<T>::axpy(d[t], T(2), F[t]);
            out[t] = Quad<T>::axpy(h[t], a.c, F[t]);
        } else {
            out[t] = Quad<T>::update_h(h[t], a.dt6, Quad<T>::axpy(d[t], T(1), F[t]));
        }
    }
    if (MODE != kStage3) Quad<T>::store_row(a.D + 4 * i, dn);
    Quad<T>::store_row((MODE == kStage3 ? a.H : a.Kout) + 4 * i, out);
}

// One stage on `stream`.  The call's first launch waits for everything before it on the
// stream; the others may start while the stage before them ends, and read nothing that a
// stage writes before their wait.
template <typename T, int MODE>
cudaError_t launch_stage(const RowMajorArgs<T>& a, bool first, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ceil_div(a.n, 4 * kRowWarps));
    cfg.blockDim = dim3(kRowThreads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = first ? 0 : 1;
    return cudaLaunchKernelEx(&cfg, rowmajor_stage_kernel<T, MODE>, a);
}

// First call on the current device: look up the static arrays' addresses.
int arrays_of_current_device(StaticArrays& out) {
    int dev = 0;
    SWE_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) {
        set_error("swe_cuda_step_noalloc: device %d beyond the %d supported", dev, kMaxDevices);
        return SWE_ERR_ARG;
    }
    std::lock_guard<std::mutex> lock(g_setup_mu);
    StaticArrays& A = g_arrays[dev];
    if (!A.scratch) {
        void *scratch = nullptr, *sync = nullptr, *failed = nullptr;
        SWE_CUDA_TRY(cudaGetSymbolAddress(&sync, g_noalloc_sync));
        SWE_CUDA_TRY(cudaGetSymbolAddress(&failed, g_noalloc_failed));
        SWE_CUDA_TRY(res::smem_limit(A.sms, A.smem));
        SWE_CUDA_TRY(cudaGetSymbolAddress(&scratch, g_noalloc_scratch));
        A.sync = (unsigned*)sync;
        A.failed = (int*)failed;
        A.scratch = scratch;
    }
    out = A;
    return SWE_OK;
}

// Static data in the caller's row-major arrays (resident.cuh), indices checked.
template <typename T>
struct RowMajor {
    static constexpr bool kNodeFast = false;    // a node's slots are contiguous
    static constexpr bool kSmallRows = false;
    const int* idx;
    const T *Dx, *Dy, *Dz, *L;
    const T *x, *y, *z, *f, *ghm;
    const T *pu, *pv, *pw, *gg;
    __device__ void weights(long i, int slot, int nnbr, T (&w)[4]) const {
        const long e = i * nnbr + slot;
        w[0] = __ldg(Dx + e); w[1] = __ldg(Dy + e); w[2] = __ldg(Dz + e); w[3] = __ldg(L + e);
    }
    __device__ int row(long i, int slot, int nnbr, int n) const {
        return checked_neighbour(__ldg(idx + i * nnbr + slot), n, i, slot);
    }
    __device__ T point(long i, int k) const {
        if (k >= PT_PU) {
            const int v = (k - PT_PU) / 3, c = (k - PT_PU) % 3;
            return __ldg((v == 0 ? pu : v == 1 ? pv : v == 2 ? pw : gg) + 3 * i + c);
        }
        return __ldg((k == 0 ? x : k == 1 ? y : k == 2 ? z : k == 3 ? f : ghm) + i);
    }
};

// Whether a grid steps in the resident kernel: its set-up, the static data's way into shared
// memory, takes about 15 us.  us per call, stage launches / resident: 20 steps FP64 N=2562 249 /
// 256, N=5000 361 / 278, N=10242 530 / 321, N=22000 923 / 486, FP32 N=2562 214 / 228, N=10242
// 328 / 254, N=40962 881 / 395; 2 steps FP64 N=2562 46 / 51, N=5000 55 / 53, FP32 N=10242 52 /
// 51; 1 step FP64 N=5000 38 / 41, N=10242 49 / 44, FP32 N=10242 37 / 40, N=20000 49 / 44.  By
// size alone: the two sum the slots in different orders, and the same steps give the same bits
// in one call or in several.
inline bool resident_pays(int n, size_t fsize) { return (size_t)n * fsize >= 40000; }

// Whole calls in the resident kernel: false where the grid does not fit it.
template <typename T>
bool run_resident(const RowMajorArgs<T>& r, T* Ka, T* Kb, T dt, int nsteps, const StaticArrays& A, cudaStream_t stream,
                  cudaError_t& e) {
    int m = 0, ctas = 0, lpn = 4;
    size_t smem = 0;
    bool stream_w = false;
    if (!res::split<T>(r.n, r.nnbr, 4, A.sms, A.smem, false, m, ctas, smem, stream_w)) {
        lpn = 2;
        if (!res::split<T>(r.n, r.nnbr, 2, A.sms, A.smem, false, m, ctas, smem, stream_w)) return false;
    }
    res::Args<T> a{};
    a.n = r.n;
    a.nnbr = r.nnbr;
    a.m = m;
    a.H = r.H;
    a.Ka = Ka;
    a.Kb = Kb;
    a.D = r.D;
    a.gh0 = r.gh0;
    a.c01 = (T)(dt / 2.0);
    a.c2 = dt;
    a.dt6 = r.dt6;
    a.sync = A.sync;
    a.failed = A.failed;
    const RowMajor<T> src{r.idx, r.Dx, r.Dy, r.Dz, r.L, r.x, r.y, r.z, r.f, r.ghm, r.pu, r.pv, r.pw, r.gg};
    for (int left = nsteps; left > 0 && e == cudaSuccess; left -= a.nsteps) {
        a.nsteps = std::min(left, res::kLaunchSteps);
        e = lpn == 4 ? res::launch<T, 4>(a, src, ctas, smem, A.smem, false, stream)
                     : res::launch<T, 2>(a, src, ctas, smem, A.smem, false, stream);
        count_launch();
    }
    return true;
}

// nsteps = 0: wait for the caller's stream, then report (and clear) the first
// out-of-range stencil index any earlier call met.
int report_bad_index(cudaStream_t stream) {
    SWE_CUDA_TRY(cudaStreamSynchronize(stream));
    int failed = 0;
    SWE_CUDA_TRY(cudaMemcpyFromSymbol(&failed, g_noalloc_failed, sizeof(failed)));
    if (failed) {
        failed = 0;
        SWE_CUDA_TRY(cudaMemcpyToSymbol(g_noalloc_failed, &failed, sizeof(failed)));
        set_error("swe_cuda_step_noalloc: a bounded wait of an earlier call's kernel ran out (calls that overlapped?)");
        return SWE_ERR_TIMEOUT;
    }
    int bad[4] = {0, 0, 0, 0};
    SWE_CUDA_TRY(cudaMemcpyFromSymbol(bad, g_noalloc_bad, sizeof(bad)));
    if (!bad[0]) return SWE_OK;
    const int zero[4] = {0, 0, 0, 0};
    SWE_CUDA_TRY(cudaMemcpyToSymbol(g_noalloc_bad, zero, sizeof(zero)));
    set_error("swe_cuda_step_noalloc: an earlier call met idx[node %d][nbr %d] = %d outside 0..n-1; it read the "
              "node's own row there, so its results are wrong", bad[1], bad[2], bad[3]);
    return SWE_ERR_INDEX;
}

template <typename T>
int run_noalloc(int n, int nnbr, double gh0, double dt, const int* idx, const void* Dx, const void* Dy,
                const void* Dz, const void* L, const void* x, const void* y, const void* z, const void* f,
                const void* ghm, const void* pu, const void* pv, const void* pw, const void* gg, void* H,
                int nsteps, bool stages, cudaStream_t stream) {
    StaticArrays A;
    SWE_TRY(arrays_of_current_device(A));
    T* Ka = reinterpret_cast<T*>(A.scratch);
    T* Kb = Ka + 4L * n;
    T* D = Kb + 4L * n;
    RowMajorArgs<T> a{};
    a.n = n;
    a.nnbr = nnbr;
    a.idx = idx;
    a.Dx = (const T*)Dx; a.Dy = (const T*)Dy; a.Dz = (const T*)Dz; a.L = (const T*)L;
    a.x = (const T*)x; a.y = (const T*)y; a.z = (const T*)z; a.f = (const T*)f; a.ghm = (const T*)ghm;
    a.pu = (const T*)pu; a.pv = (const T*)pv; a.pw = (const T*)pw; a.gg = (const T*)gg;
    a.H = (T*)H;
    a.D = D;
    a.gh0 = (T)gh0;
    const T dtT = (T)dt;
    a.dt6 = (double)dtT / 6.0;
    cudaError_t e = cudaSuccess;
    if (!stages && resident_pays(n, sizeof(T)) && run_resident<T>(a, Ka, Kb, dtT, nsteps, A, stream, e)) {
        SWE_CUDA_TRY(e);
        return SWE_OK;
    }
    for (int s = 0; s < nsteps; ++s) {
        a.Kin = a.H; a.Kout = Ka; a.c = (T)(dtT / 2.0);
        SWE_CUDA_TRY((launch_stage<T, kStage0>(a, s == 0, stream)));
        a.Kin = Ka; a.Kout = Kb;
        SWE_CUDA_TRY((launch_stage<T, kStage1>(a, false, stream)));
        a.Kin = Kb; a.Kout = Ka; a.c = dtT;
        SWE_CUDA_TRY((launch_stage<T, kStage2>(a, false, stream)));
        a.Kin = Ka; a.Kout = nullptr;
        SWE_CUDA_TRY((launch_stage<T, kStage3>(a, false, stream)));
        count_launch(4);
    }
    return SWE_OK;
}

int step_noalloc(int fsize, int n, int nnbr, double gh0, double dt, const int* idx, const void* Dx, const void* Dy,
                 const void* Dz, const void* L, const void* x, const void* y, const void* z, const void* f,
                 const void* ghm, const void* p_u, const void* p_v, const void* p_w, const void* gradghm, void* H,
                 int nsteps, bool stages, void* stream) {
    if (fsize != 8 && fsize != 4) { set_error("swe_cuda_step_noalloc: fsize must be 8 or 4, got %d", fsize); return SWE_ERR_ARG; }
    if (nnbr <= 0 || nnbr > kSlots) { set_error("swe_cuda_step_noalloc: nnbr %d not in 1..%d", nnbr, kSlots); return SWE_ERR_ARG; }
    if (nsteps < 0) { set_error("swe_cuda_step_noalloc: nsteps < 0"); return SWE_ERR_ARG; }
    const long max_nodes = (long)(kNoallocScratchBytes / (12L * fsize));
    if (n <= 0 || n > max_nodes) {
        set_error("swe_cuda_step_noalloc: n = %d nodes outside 1..%ld, the most the %zu-byte static scratch "
                  "holds at fsize %d (3 x n x 4 values)", n, max_nodes, kNoallocScratchBytes, fsize);
        return SWE_ERR_ARG;
    }
    if (!idx || !Dx || !Dy || !Dz || !L || !x || !y || !z || !f || !ghm || !p_u || !p_v || !p_w || !gradghm || !H) {
        set_error("swe_cuda_step_noalloc: null device pointer");
        return SWE_ERR_ARG;
    }
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (nsteps == 0) return report_bad_index(s);
    return fsize == 8 ? run_noalloc<double>(n, nnbr, gh0, dt, idx, Dx, Dy, Dz, L, x, y, z, f, ghm, p_u, p_v, p_w,
                                            gradghm, H, nsteps, stages, s)
                      : run_noalloc<float>(n, nnbr, gh0, dt, idx, Dx, Dy, Dz, L, x, y, z, f, ghm, p_u, p_v, p_w,
                                           gradghm, H, nsteps, stages, s);
}

}  // namespace
}  // namespace swe

using namespace swe;

extern "C" int swe_cuda_step_noalloc(int fsize, int n, int nnbr, double gh0, double dt, const int* idx,
                                     const void* Dx, const void* Dy, const void* Dz, const void* L,
                                     const void* x, const void* y, const void* z, const void* f,
                                     const void* ghm, const void* p_u, const void* p_v, const void* p_w,
                                     const void* gradghm, void* H, int nsteps, void* stream) {
    return step_noalloc(fsize, n, nnbr, gh0, dt, idx, Dx, Dy, Dz, L, x, y, z, f, ghm, p_u, p_v, p_w, gradghm, H, nsteps,
                        false, stream);
}

extern "C" int swe_cuda_step_noalloc_stages(int fsize, int n, int nnbr, double gh0, double dt, const int* idx,
                                            const void* Dx, const void* Dy, const void* Dz, const void* L,
                                            const void* x, const void* y, const void* z, const void* f,
                                            const void* ghm, const void* p_u, const void* p_v, const void* p_w,
                                            const void* gradghm, void* H, int nsteps, void* stream) {
    return step_noalloc(fsize, n, nnbr, gh0, dt, idx, Dx, Dy, Dz, L, x, y, z, f, ghm, p_u, p_v, p_w, gradghm, H, nsteps,
                        true, stream);
}
