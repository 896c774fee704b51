// noalloc.cu - the PPE conjugate-gradient solve for callers that cannot allocate device
// memory.
//
// Some callers of this library do not own the device allocator: a host application
// whose device memory is already reserved by its own caching allocator or arena (a
// deep-learning framework that pre-reserves the pool, an embedded solver inside a
// larger simulation that hands out fixed buffers), or code on a latency-critical path
// where cudaMalloc/cudaFree would implicitly synchronize the device.  Such callers keep
// their CSR system in their own device buffers and need a solve that allocates
// nothing.  This file provides that solve: the reference's FP64 CG
// (Computer::SolvePressurePoissonEquation, src/OpenMps/Computer.hpp:1359-1429) whose
// scratch vectors r, p, s, exchange words and scalars live in one file-scope static
// device array of fixed size (kNoallocMaxRows rows).  Every GPU that loads the library
// holds that array until the process exits.
//
// In host code the array's name stands for a host-side shadow, not a device address.
// Each call therefore asks the runtime for the array's address in the current device's
// context (cudaGetSymbolAddress, a lookup that allocates nothing) and passes it to the
// kernels.  The address is not cached: after cudaDeviceReset, or with another context
// current on the same device, the module is loaded again and the array can move, so a
// cached address would point at memory this context does not own.  The first call in a
// context may load the library's module (lazy module loading), so make that first call
// before any stream capture.  Every call shares the array and finds the previous
// call's contents; the parts that must start at zero are cleared at the start of each
// call.  Calls that overlap on the GPU (different streams or host threads at the same
// time) race on the array.
//
// A call is one launch: initial residual, iterations and the final true residual in one
// cluster of 16 blocks (small systems) or a cooperative grid of one block per SM, with the
// two exchanges per iteration of gridloop.cuh and the recurrence of cgloop.cu (s = A r +
// beta s).  Blocks own contiguous rows of equal entries; a few lanes share a row so that a
// warp reads consecutive entries of the CSR arrays, and their partial sums meet in a
// transposing exchange (four rows a lane, three additions instead of eight: the FP64 pipe
// takes a warp-wide addition every 64 cycles).  Before, one thread walked a row (a warp's
// loads touched 32 rows apart) in three kernels per iteration, and the host read the
// convergence flag every 16 iterations.
#include <cuda.h>

#include <cmath>

#include "gridloop.cuh"

namespace mpsgb {

namespace {

constexpr int64_t kNoallocMaxRows = MPS_NOALLOC_MAX_ROWS;
constexpr int kNoallocScalars = 16;  // doubles reserved for NoallocScalars
constexpr int64_t kNoallocDoubles = 3 * kNoallocMaxRows + kLoopSlots + kNoallocScalars;
// Rows up to which one cluster solves the system.  us per iteration on lattice operators,
// before and now: 500 rows of 13 entries 23.1 -> 5.5 and 2,000 of 48 30.9 -> 8.9 (cluster);
// 3,600 of 13 22.4 -> 7.7, 10,000 of 28 25.7 -> 9.5, 100,441 of 5 / 28 / 48 21.5 -> 10.3,
// 31.1 -> 17.9 and 44.1 -> 24.0 (grid: two exchanges of about 3 us, then the FP64 pipe, 5.3
// us at 28 entries).  Cluster / grid on either side of the line, 27 entries: 900 rows 6.3 / 7.3,
// 2,025 7.3 / 7.4, 4,096 9.6 / 7.6, 8,100 13.0 / 9.3.
constexpr int64_t kNoallocClusterRows = 2048;

struct NoallocScalars {
    double bb, true_rr;
    int iter, converged, timed_out, pad;
};
static_assert(sizeof(NoallocScalars) <= kNoallocScalars * sizeof(double), "scalars do not fit");

// The solver's whole scratch: r, p, s, exchange words, scalars.
static __device__ __align__(256) double g_noalloc_scratch[kNoallocDoubles];

struct CsrSystem {
    int n;
    const int64_t* rp;
    const int32_t* col;
    const double* val;
    const double* b;
    double* x;
    double *r, *p, *s, *slots;  // scratch
    NoallocScalars* S;
    double eps;
    int criterion, max_iter;
    int keep_rows;  // rows whose vectors fit the block's shared memory
    long long wait_clocks;  // bound of an exchange's wait
};

// How a block's warps walk its rows: LANES lanes share a row, GROUPS row groups of a warp at
// once.  Lane per row for short rows, four lanes in transposing groups of four for ordinary
// ones, fewer rows a warp when the block has few, a warp per row for long ones.
enum RowWalk { kLanePerRow, kFourByFour, kFourLanes, kEightLanes, kWarpPerRow };

__device__ __forceinline__ int walk_rows(int walk) {  // rows a warp takes at once
    return walk == kLanePerRow || walk == kFourByFour ? 32 : walk == kFourLanes ? 8 : walk == kEightLanes ? 4 : 1;
}

// f(row, (A v)_row) for rows [r0, r1), each in one lane
template <int LANES, int GROUPS, class F>
__device__ __forceinline__ void row_products(const CsrSystem& A, int r0, int r1, const double* v, F f) {
    static_assert(GROUPS == 1 || GROUPS == LANES, "the exchange transposes a square");
    constexpr int kPer = 32 / LANES;              // rows of a group
    constexpr int kDepth = GROUPS > 1 ? 2 : 8 / (LANES >= 8 ? 2 : 1);  // entries of a row a lane loads at once
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = static_cast<int>(blockDim.x >> 5);
    const int sub = lane % LANES, who = lane / LANES;
    for (int base = r0 + warp * kPer * GROUPS; base < r1; base += warps * kPer * GROUPS) {
        int64_t at[GROUPS];
        int left[GROUPS];
        double acc[GROUPS];
        int most = 0;
#pragma unroll
        for (int g = 0; g < GROUPS; g++) {
            const int row = base + g * kPer + who;
            const int64_t b = row < r1 ? A.rp[row] : 0, e = row < r1 ? A.rp[row + 1] : 0;
            at[g] = b + sub;
            left[g] = static_cast<int>(e - b) - sub;  // > 0: entries from this lane's on
            most = max(most, static_cast<int>(e - b));
            acc[g] = 0.0;
        }
        most = __reduce_max_sync(0xffffffffu, most);
        for (int k = 0; k < most; k += kDepth * LANES) {
            int c[GROUPS][kDepth];
            double a[GROUPS][kDepth];
#pragma unroll
            for (int g = 0; g < GROUPS; g++) {
#pragma unroll
                for (int d = 0; d < kDepth; d++) {
                    const bool in = k + d * LANES < left[g];
                    c[g][d] = in ? __ldg(A.col + at[g] + k + d * LANES) : 0;
                    a[g][d] = in ? __ldg(A.val + at[g] + k + d * LANES) : 0.0;
                }
            }
            double xv[GROUPS][kDepth];
#pragma unroll
            for (int g = 0; g < GROUPS; g++) {
#pragma unroll
                for (int d = 0; d < kDepth; d++) xv[g][d] = k + d * LANES < left[g] ? v[c[g][d]] : 0.0;
            }
#pragma unroll
            for (int d = 0; d < kDepth; d++) {
#pragma unroll
                for (int g = 0; g < GROUPS; g++)
                    if (k + d * LANES < left[g]) acc[g] = fma(a[g][d], xv[g][d], acc[g]);
            }
        }
        if constexpr (GROUPS == 4) {
            // lane `sub` of four ends with the row of group `sub`
            const bool hi = (sub & 2) != 0, odd = (sub & 1) != 0;
            const double m0 = hi ? acc[2] : acc[0], m1 = hi ? acc[3] : acc[1];
            const double o0 = hi ? acc[0] : acc[2], o1 = hi ? acc[1] : acc[3];
            const double t0 = m0 + __shfl_xor_sync(0xffffffffu, o0, 2), t1 = m1 + __shfl_xor_sync(0xffffffffu, o1, 2);
            const double mine = odd ? t1 : t0, other = odd ? t0 : t1;
            const double sum = mine + __shfl_xor_sync(0xffffffffu, other, 1);
            const int row = base + sub * kPer + who;
            if (row < r1) f(row, sum);
        } else {
            double sum = acc[0];
#pragma unroll
            for (int o = LANES / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (sub == 0 && base + who < r1) f(base + who, sum);
        }
    }
}

template <class F>
__device__ __forceinline__ void csr_product(const CsrSystem& A, int walk, int r0, int r1, const double* v, F f) {
    switch (walk) {
        case kLanePerRow: row_products<1, 1>(A, r0, r1, v, f); break;
        case kFourByFour: row_products<4, 4>(A, r0, r1, v, f); break;
        case kFourLanes: row_products<4, 1>(A, r0, r1, v, f); break;
        case kEightLanes: row_products<8, 1>(A, r0, r1, v, f); break;
        default: row_products<32, 1>(A, r0, r1, v, f); break;
    }
}

// The first row i with (entries before it) + a i >= share (rows 0 .. n).
__device__ __forceinline__ int row_at(const CsrSystem& A, int64_t a, int64_t share) {
    int lo = 0, hi = A.n;
    const int64_t first = A.rp[0];
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (A.rp[mid] - first + a * mid < share) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

template <bool kCluster>
__global__ void __launch_bounds__(kLoopThreads, 1) k_na_solve(CsrSystem A) {
    extern __shared__ __align__(16) double na_sm[];
    __shared__ LoopReduce red;
    __shared__ struct {
        double rr, alpha, beta, thr, bb, true_rr;
        int iter, conv;
    } sc;
    __shared__ int range[2];
    if (kCluster) loop_cluster_start();
    LoopSync ls{A.slots, gridDim.x, 0};
    const int t = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x);
    if (t == 0) red.wait_clocks = A.wait_clocks;
    {
        const int64_t nnz = A.rp[A.n] - A.rp[0];
        const int64_t a = max(static_cast<int64_t>(1), nnz / (4 * static_cast<int64_t>(A.n)));
        const int64_t total = nnz + a * A.n;
        if (t < 2) range[t] = row_at(A, a, (blockIdx.x + t) * total / gridDim.x);
    }
    __syncthreads();
    const int r0 = range[0], r1 = blockIdx.x + 1 == gridDim.x ? A.n : range[1], rows = r1 - r0;
    const int64_t entries = A.rp[r1] - A.rp[r0];
    const bool many = rows >= nt;
    const int walk = entries > 128 * static_cast<int64_t>(rows) ? kWarpPerRow
                     : many ? (entries <= 6 * static_cast<int64_t>(rows) ? kLanePerRow : kFourByFour)
                            : (rows >= nt / 4 ? kFourLanes : kEightLanes);
    const int warps_on = min(nt >> 5, (rows + walk_rows(walk) - 1) / walk_rows(walk));
    const int product_lanes = 32 * warps_on, row_lanes = min(nt, rows);
    // the block's rows of p, s, x and r, kept in shared memory when they fit
    const bool keep = rows <= A.keep_rows;
    double* P = keep ? na_sm - r0 : A.p;
    double* Q = keep ? na_sm + rows - r0 : A.s;
    double* X = keep ? na_sm + 2 * rows - r0 : A.x;
    double* R = keep ? na_sm + 3 * rows - r0 : A.r;
    bool ok;
    {
        // r = b - A x, p = s = 0, r.r, b.b, threshold (Computer.hpp:1382-1389)
        double v[2] = {0.0, 0.0};
        csr_product(A, walk, r0, r1, A.x, [&](int row, double ax) {
            const double bi = A.b[row], ri = bi - ax;
            P[row] = 0.0;
            Q[row] = 0.0;
            R[row] = ri;
            if (keep) {
                A.r[row] = ri;
                X[row] = A.x[row];
            }
            v[0] = fma(ri, ri, v[0]);
            v[1] = fma(bi, bi, v[1]);
        });
        ok = loop_reduce<kCluster, 2>(ls, red, v, product_lanes, [&](const double* tot) {
            if (threadIdx.x != 0) return;
            const double rr = tot[0], bb = tot[1];
            double thr = rr * A.eps * A.eps;
            if (A.criterion == MPS_CRIT_RHS && bb > 0) thr = bb * A.eps * A.eps;
            sc.rr = rr;
            sc.bb = bb;
            sc.thr = thr;
            sc.beta = 0.0;
            sc.iter = 0;
            sc.conv = A.criterion == MPS_CRIT_RHS ? (rr < thr || rr == 0) : thr == 0;
        });
    }
    while (ok && !sc.conv && sc.iter < A.max_iter) {
        // p = r + beta p; s = A r + beta s; alpha = r.r / p.s
        double v = 0.0;
        {
            const double beta = sc.beta;
            csr_product(A, walk, r0, r1, A.r, [&](int row, double ar) {
                const double p = fma(beta, P[row], R[row]);
                const double s = fma(beta, Q[row], ar);
                P[row] = p;
                Q[row] = s;
                v = fma(p, s, v);
            });
        }
        ok = loop_reduce<kCluster, 1>(ls, red, &v, product_lanes, [&](const double* tot) {
            const double alpha = ddiv_rn(sc.rr, tot[0]);
            if (threadIdx.x == 0) sc.alpha = alpha;
        });
        if (!ok) break;
        // x += alpha p; r -= alpha s; r.r; convergence; beta (Computer.hpp:1402-1420)
        v = 0.0;
        {
            const double alpha = sc.alpha;
            for (int row = r0 + t; row < r1; row += nt) {
                X[row] = fma(alpha, P[row], X[row]);
                const double ri = fma(-alpha, Q[row], R[row]);
                R[row] = ri;
                if (keep) A.r[row] = ri;
                v = fma(ri, ri, v);
            }
        }
        ok = loop_reduce<kCluster, 1>(ls, red, &v, row_lanes, [&](const double* tot) {
            const double beta = ddiv_rn(tot[0], sc.rr);
            __syncwarp();
            if (threadIdx.x != 0) return;
            sc.conv = tot[0] < sc.thr;
            if (!sc.conv) {
                sc.beta = beta;
                sc.rr = tot[0];
            }
            sc.iter++;
        });
    }
    // |b - A x|^2 of the x returned
    if (keep)
        for (int row = r0 + t; row < r1; row += nt) A.x[row] = X[row];
    ok = ok && loop_reduce<kCluster, 0>(ls, red, nullptr, 0, [](const double*) {});
    if (ok) {
        double v = 0.0;
        csr_product(A, walk, r0, r1, A.x, [&](int row, double ax) {
            const double ri = A.b[row] - ax;
            v = fma(ri, ri, v);
        });
        ok = loop_reduce<kCluster, 1>(ls, red, &v, product_lanes, [&](const double* tot) {
            if (threadIdx.x == 0) sc.true_rr = tot[0];
        });
    }
    if (blockIdx.x == 0 && t == 0) {
        A.S->bb = sc.bb;
        A.S->true_rr = sc.true_rr;
        A.S->iter = sc.iter;
        A.S->converged = ok ? sc.conv : 0;
        A.S->timed_out = ok ? 0 : 1;
    }
}

// Device address of g_noalloc_scratch in the current context, looked up on every call.
int scratch_for_current_context(double** out) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || !ptr) {
        cudaGetLastError();
        return MPS_ERR_CUDA;
    }
    *out = static_cast<double*>(ptr);
    return MPS_OK;
}

// SMs that work on the stream can use: `sms` (the device's), or the part that the stream's
// green context has.
int stream_sms(cudaStream_t s, int sms) {
    auto entry = [](const char* name, unsigned version) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion(name, &f, version, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return static_cast<void*>(nullptr);
        }
        return f;
    };
    static const auto stream_ctx = reinterpret_cast<CUresult (*)(CUstream, CUcontext*)>(entry("cuStreamGetCtx", 9020));
    static const auto resource = reinterpret_cast<CUresult (*)(CUcontext, CUdevResource*, CUdevResourceType)>(
        entry("cuCtxGetDevResource", 12040));
    CUcontext ctx = nullptr;
    CUdevResource r{};
    if (!stream_ctx || !resource || stream_ctx(s, &ctx) != CUDA_SUCCESS ||
        resource(ctx, &r, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS)
        return sms;
    const int part = static_cast<int>(r.sm.smCount);
    return part > 0 && part < sms ? part : sms;
}

// One cluster for small systems, else a block per SM; p, s, x, r of half as many rows again
// as the average block owns in shared memory.  All blocks must be resident at once: on a
// stream with a part of the SMs the grid is as many blocks as that part has (the blocks'
// shares of the rows follow from the grid; a cluster's 16 SMs must lie in one cluster of
// the chip, which a part need not have).
cudaError_t launch_na_solve(CsrSystem& A, cudaStream_t s) {
    int dev = 0, all = 0, most = 0, grid = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&all, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    const int sms = stream_sms(s, all);
    e = loop_grid_blocks(dev, sms, &grid);
    if (e != cudaSuccess) return e;
    bool cluster = A.n <= kNoallocClusterRows && sms == all;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.blockDim = dim3(kLoopThreads);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    for (;; cluster = false) {
        auto kernel = cluster ? k_na_solve<true> : k_na_solve<false>;
        const int blocks = cluster ? kLoopCluster : grid;
        const int64_t room = (most - 16 * 1024) / (4 * static_cast<int64_t>(sizeof(double)));
        const int64_t want = 3 * static_cast<int64_t>(A.n) / (2 * blocks) + 128;
        A.keep_rows = static_cast<int>(want < room ? want : room);
        cfg.gridDim = dim3(static_cast<unsigned>(blocks));
        cfg.dynamicSmemBytes = static_cast<size_t>(A.keep_rows) * 4 * sizeof(double);
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(cfg.dynamicSmemBytes));
        if (e != cudaSuccess) return e;
        if (!cluster) {
            at[0].id = cudaLaunchAttributeCooperative;
            at[0].val.cooperative = 1;
            cfg.numAttrs = blocks > 1 ? 1 : 0;
            e = cudaLaunchKernelEx(&cfg, kernel, A);
            if (e != cudaErrorCooperativeLaunchTooLarge || blocks == 1) return e;
            cudaGetLastError();  // fewer SMs than the device and the stream report
            grid = blocks / 2;
            continue;
        }
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kLoopCluster;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        int fit = 0;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) == cudaSuccess && fit > 0)
            return cudaLaunchKernelEx(&cfg, kernel, A);
        cudaGetLastError();  // no cluster of this size: the grid
    }
}

}  // namespace

}  // namespace mpsgb

extern "C" int mps_debug_cg_solve_csr_noalloc_wait(int64_t n, const int64_t* row_ptr,
                                                  const int32_t* col, const double* val,
                                                  const double* b, double* x, double eps,
                                                  int32_t criterion, int32_t max_iters,
                                                  void* stream, int32_t* iterations,
                                                  double* true_relres, int64_t wait_clocks) {
    using namespace mpsgb;
    if (n <= 0 || !row_ptr || !col || !val || !b || !x) return MPS_ERR_INVALID_ARGUMENT;
    if (n > kNoallocMaxRows) return MPS_ERR_NOALLOC_TOO_LARGE;
    if (criterion != MPS_CRIT_INITIAL_RESIDUAL && criterion != MPS_CRIT_RHS) return MPS_ERR_INVALID_ARGUMENT;
    double* base = nullptr;
    const int rc = scratch_for_current_context(&base);
    if (rc != MPS_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    CsrSystem A{};
    A.n = static_cast<int>(n);
    A.rp = row_ptr;
    A.col = col;
    A.val = val;
    A.b = b;
    A.x = x;
    A.r = base;
    A.p = base + kNoallocMaxRows;
    A.s = base + 2 * kNoallocMaxRows;
    A.slots = base + 3 * kNoallocMaxRows;
    A.S = reinterpret_cast<NoallocScalars*>(A.slots + kLoopSlots);
    A.eps = eps;
    A.criterion = criterion;
    A.max_iter = max_iters > 0 ? max_iters : static_cast<int>(n);
    A.wait_clocks = wait_clocks < 0 ? kLoopWaitClocks : wait_clocks;
    // the arrival counter starts from zero on every call
    NoallocScalars S{};
    if (cudaMemsetAsync(A.slots, 0, sizeof(double), s) != cudaSuccess || launch_na_solve(A, s) != cudaSuccess ||
        cudaMemcpyAsync(&S, A.S, sizeof(S), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
        cudaGetLastError();
        return MPS_ERR_CUDA;
    }
    if (S.timed_out) return MPS_ERR_TIMEOUT;
    if (iterations) *iterations = S.iter;
    if (true_relres) *true_relres = (S.bb > 0) ? std::sqrt(S.true_rr / S.bb) : std::sqrt(S.true_rr);
    return S.converged ? MPS_OK : MPS_ERR_CG_NOT_CONVERGED;
}

extern "C" int mps_cg_solve_csr_device_noalloc(int64_t n, const int64_t* row_ptr,
                                               const int32_t* col, const double* val,
                                               const double* b, double* x, double eps,
                                               int32_t criterion, int32_t max_iters,
                                               void* stream, int32_t* iterations,
                                               double* true_relres) {
    return mps_debug_cg_solve_csr_noalloc_wait(n, row_ptr, col, val, b, x, eps, criterion, max_iters, stream,
                                               iterations, true_relres, -1);
}
