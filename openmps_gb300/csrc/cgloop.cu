// cgloop.cu - the plain solvers' iteration loops (MPS_SOLVER_CG64, MPS_SOLVER_MIXED), each
// in one launch: one cluster of 16 blocks for small systems, a cooperative grid of one block
// per SM otherwise (gridloop.cuh).
//
// Work layout: a block owns a contiguous range of SELL chunks, cut so that matrix entries and
// rows are even over the blocks; chunks of identity rows with a zero residual (dummy and
// disabled particles: 84 % of the 3D dam break's chunks) keep x and stay out of the loop.
// The split stays the same through the solve, so a row's vectors are touched by one thread
// only, and the block keeps them in shared memory when they fit (the gathered vector has its
// global copy).
//
// CG64: the reference's conjugate gradient (Computer.hpp:1359-1429) with two grid-wide
// exchanges per iteration instead of three: the product is formed with the residual, and
// A p follows from s = A r + beta s (p = r + beta p), so p needs no exchange of its own.
// Both dot products are formed from the vectors themselves, as in the reference.
// MIXED: Chronopoulos-Gear CG in FP32 with FP64 dot products and reliable updates (cg.cu).
#include "cgloop.cuh"

namespace mpsgb {

namespace {

// dynamic shared memory: unit sums, tables, vectors.  (The gathered vector's rows around the
// block in shared memory too were measured: 42,226 rows 13.0 against 12.4 us, 90,050 rows
// 18.8 against 18.4, MIXED 13.9 against 14.0: loading them costs what the gathers wait.)
struct LoopPlan {
    int blocks;
    int tables;      // chunks the tables hold
    bool either;     // the direct form follows, for systems whose chunks in the loop pass them
    int keep_bytes;  // shared memory for the block's vectors
    size_t smem;
};

size_t table_bytes(int tables) {
    return part_room(tables) + table_room(tables);
}

// This block's chunks.  o.loop_w[c] is the width of a chunk the loop works on, 0 for one it
// leaves out.  With W entries per row in N chunks, chunk k of weight prefix P_k goes to block
// floor(P_k G / P_N), P_k = (widths before it) + a (chunks before it), a = W / (4 N) (a
// row's vector work is about ten matrix entries' at the 46 entries of the usual radius): a
// block then owns at most 5 N / G + 1 chunks, and even shares when the widths are alike.
template <bool kDirect>
__device__ __forceinline__ LoopView loop_view(const CgOperands& o, const LoopPlan& plan, unsigned char* sm,
                                             unsigned char** keep) {
    __shared__ int wsum[32], wcnt[32], first_pos, last_pos, first_chunk, last_chunk;
    LoopView L;
    L.lo = 0;
    L.hi = o.n;
    *keep = place_tables(L, sm, plan.tables);
    const int t = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x), lane = t & 31;
    L.warps = nt >> 5;
    const int seg = (o.nchunks + nt - 1) / nt;
    const int b = min(o.nchunks, t * seg), e = min(o.nchunks, b + seg);
    int w = 0, n = 0;
    for (int c = b; c < e; c++) {
        const int x = o.loop_w[c];
        w += x;
        n += x > 0 ? 1 : 0;
    }
    int ws = w, ns = n;
    for (int d = 1; d < 32; d <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, ws, d), y = __shfl_up_sync(0xffffffffu, ns, d);
        if (lane >= d) {
            ws += x;
            ns += y;
        }
    }
    if (lane == 31) {
        wsum[t >> 5] = ws;
        wcnt[t >> 5] = ns;
    }
    if (t == 0) {
        first_pos = first_chunk = 0x7fffffff;
        last_pos = last_chunk = -1;
    }
    __syncthreads();
    int W = 0, N = 0;
    for (int k = 0; k < L.warps; k++) {
        if (k == t >> 5) {
            ws += W;
            ns += N;
        }
        W += wsum[k];
        N += wcnt[k];
    }
    if (plan.either && (2 * (N / static_cast<int>(gridDim.x) + 1) + 2 > plan.tables) != kDirect) {
        L.nc = -1;  // the other form's (every block finds the same)
        return L;
    }
    const long long a = N > 0 ? max(1, W / (4 * N)) : 1;
    const long long total = W + a * N;
    const long long G = gridDim.x;
    for (int pass = 0; pass < 2; pass++) {
        int wp = ws - w, np = ns - n;
        for (int c = b; c < e; c++) {
            const int x = o.loop_w[c];
            if (x == 0) continue;
            if ((wp + a * np) * G / total == static_cast<long long>(blockIdx.x)) {
                if (pass == 0) {
                    atomicMin(&first_pos, np);
                    atomicMax(&last_pos, np);
                    atomicMin(&first_chunk, c);
                    atomicMax(&last_chunk, c);
                } else if (L.whole) {
                    L.info[np - first_pos].chunk = c;
                }
            }
            wp += x;
            np++;
        }
        __syncthreads();
        if (pass == 0) {
            const int mine = last_pos < 0 ? 0 : last_pos - first_pos + 1;
            L.whole = !kDirect && mine <= plan.tables;
            L.c0 = L.whole || mine == 0 ? 0 : first_chunk;
            L.nc = L.whole || mine == 0 ? mine : last_chunk - first_chunk + 1;
        }
    }
    split_tiles(L, plan.tables);
    if (L.whole) build_tables(o, L, L.nc);
    return L;
}

template <bool kCluster, bool kDirect>
__global__ void __launch_bounds__(kLoopThreads, 1) k_cg_loop(CgOperands o, LoopPlan plan) {
    extern __shared__ __align__(16) unsigned char loop_sm[];
    __shared__ LoopReduce red;
    __shared__ struct {
        double rr, alpha, beta, pap, rr_new;
        int iter, conv;
    } sc;
    CgScalars* S = o.S;
    if (S->converged || S->aborted || S->iter >= S->max_iter) return;
    unsigned char* keep_sm;
    const LoopView L = loop_view<kDirect>(o, plan, loop_sm, &keep_sm);
    if (L.nc < 0) return;
    if (kCluster) loop_cluster_start();
    LoopSync ls{o.slots, gridDim.x, 0};
    const double thr = S->thr;
    const int max_iter = S->max_iter;
    if (threadIdx.x == 0) {
        red.wait_clocks = loop_wait_clocks(o);
        sc.rr = S->rr;
        sc.beta = 0.0;
        sc.iter = S->iter;
        sc.conv = 0;
    }
    // the block's rows of p, s, x and r: index `a` of a row is its place in the block when
    // they are kept in shared memory, the row itself in the global arrays
    const int rows = L.nc * kSellRows;
    const bool keep = !kDirect && L.whole && 4 * static_cast<int64_t>(sizeof(double)) * rows <= plan.keep_bytes;
    double* kept = reinterpret_cast<double*>(keep_sm);
    double* P = keep ? kept : o.p;
    double* Q = keep ? kept + rows : o.Ap;
    double* X = keep ? kept + 2 * rows : o.x;
    double* R = keep ? kept + 3 * rows : o.r;
    own_rows<kDirect>(o, L, [&](int local, int row) {
        const int a = keep ? local : row;
        P[a] = 0.0;
        Q[a] = 0.0;
        if (keep) {
            X[a] = o.x[row];
            R[a] = o.r[row];
        }
    });
    __syncthreads();
    bool ok = true;
    while (ok) {
        // p = r + beta p; s = A r + beta s; p.s
        double v = 0.0;
        {
            const double beta = sc.beta;
            product<double, kDirect>(o, L, [&](int j) { return o.r[j]; }, [&](int local, int row, double ar) {
                const int a = keep ? local : row;
                const double p = fma(beta, P[a], R[a]);
                const double s = fma(beta, Q[a], ar);
                P[a] = p;
                Q[a] = s;
                v = fma(p, s, v);
            });
        }
        ok = loop_reduce<kCluster, 1>(ls, red, &v, L.active, [&](const double* tot) {
            const double a = ddiv_rn(sc.rr, tot[0]);
            if (threadIdx.x == 0) {
                sc.pap = tot[0];
                sc.alpha = a;
            }
        });
        if (!ok) break;
        // x += alpha p; r -= alpha s; r.r; convergence; beta (Computer.hpp:1402-1420)
        v = 0.0;
        {
            const double alpha = sc.alpha;
            own_rows<kDirect>(o, L, [&](int local, int row) {
                const int a = keep ? local : row;
                X[a] = fma(alpha, P[a], X[a]);
                const double ri = fma(-alpha, Q[a], R[a]);
                R[a] = ri;
                if (keep) o.r[row] = ri;
                v = fma(ri, ri, v);
            });
        }
        ok = loop_reduce<kCluster, 1>(ls, red, &v, L.active, [&](const double* tot) {
            const double b = ddiv_rn(tot[0], sc.rr);
            __syncwarp();
            if (threadIdx.x == 0) {
                sc.rr_new = tot[0];
                sc.conv = tot[0] < thr;
                if (!sc.conv) {
                    sc.beta = b;
                    sc.rr = tot[0];
                }
                sc.iter++;
            }
        });
        if (ok && (sc.conv || sc.iter >= max_iter)) break;
    }
    if (keep) own_rows<kDirect>(o, L, [&](int local, int row) { o.x[row] = X[local]; });
    if (!ok) {
        loop_timeout(o);
    } else if (blockIdx.x == 0 && threadIdx.x == 0) {
        S->rr_new = sc.rr_new;
        S->rr = sc.rr;
        S->pAp = sc.pap;
        S->alpha = sc.alpha;
        S->beta = sc.beta;
        S->iter = sc.iter;
        S->converged = sc.conv;
    }
}

template <bool kCluster, bool kDirect>
__global__ void __launch_bounds__(kLoopThreads, 1) k_mx_loop(CgOperands o, LoopPlan plan) {
    extern __shared__ __align__(16) unsigned char loop_sm[];
    __shared__ LoopReduce red;
    __shared__ CgScalars sc;  // the solve's scalars, as the per-phase kernels keep them
    __shared__ float alpha32, beta32;
    if (o.S->converged || o.S->aborted || o.S->iter >= o.S->max_iter) return;
    unsigned char* keep_sm;
    const LoopView L = loop_view<kDirect>(o, plan, loop_sm, &keep_sm);
    if (L.nc < 0) return;
    if (kCluster) loop_cluster_start();
    LoopSync ls{o.slots, gridDim.x, 0};
    if (threadIdx.x == 0) {
        red.wait_clocks = loop_wait_clocks(o);
        sc = *o.S;
        alpha32 = __double2float_rn(sc.alpha);
        beta32 = __double2float_rn(sc.beta);
    }
    // the block's rows of s, p, d, w and r (kept or global, as in k_cg_loop)
    const int rows = L.nc * kSellRows;
    const bool keep = !kDirect && L.whole && 5 * static_cast<int64_t>(sizeof(float)) * rows <= plan.keep_bytes;
    float* kept = reinterpret_cast<float*>(keep_sm);
    float* Sv = keep ? kept : o.s32;
    float* Pv = keep ? kept + rows : o.p32;
    float* Dv = keep ? kept + 2 * rows : o.d32;
    float* Wv = keep ? kept + 3 * rows : o.w32;
    float* Rv = keep ? kept + 4 * rows : o.r32;
    if (keep)
        own_rows<kDirect>(o, L, [&](int local, int row) {
            Sv[local] = o.s32[row];
            Pv[local] = o.p32[row];
            Dv[local] = o.d32[row];
            Wv[local] = o.w32[row];
            Rv[local] = o.r32[row];
        });
    __syncthreads();
    // w = A r (FP32); gamma = r.r and delta = w.r in FP64, and what follows from them
    auto spmv = [&](bool after_update) {
        double v[2] = {0.0, 0.0};
        product<float, kDirect>(o, L, [&](int j) { return o.r32[j]; }, [&](int local, int row, float w) {
            const int a = keep ? local : row;
            const double ri = widen(Rv[a]);
            Wv[a] = w;
            if (after_update) Dv[a] = 0.0f;
            v[0] = fma(ri, ri, v[0]);
            v[1] = fma(widen(w), ri, v[1]);
        });
        return loop_reduce<kCluster, 2>(ls, red, v, L.active, [&](const double* tot) {
            const double gam = tot[0], del = tot[1];
            // beta = gam / rr in lane 0 and beta gam / alpha = gam^2 / (rr alpha) in lane 1, so
            // that two divisions follow one another, not three
            const bool one = (threadIdx.x & 31) == 1;
            const double q = ddiv_rn(one ? gam * gam : gam, one ? sc.rr * sc.alpha : sc.rr);
            const double alpha = ddiv_rn(gam, del - __shfl_sync(0xffffffffu, q, 1));
            if (threadIdx.x != 0) return;
            sc.rr_new = gam;
            sc.do_update = !after_update && (gam < sc.delta2 * sc.rr_upd || gam < sc.thr);
            if (!sc.do_update) {
                sc.beta = q;
                sc.alpha = alpha;
                alpha32 = __double2float_rn(alpha);  // once: a conversion takes the pipe 64 cycles a warp
                beta32 = __double2float_rn(q);
                sc.iter += 1;
                if (sc.iter - sc.iter_upd > kMixedStallIter) sc.stalled = 1;
                sc.rr = gam;
                sc.pAp = del;
            }
            if (after_update) {
                // the true residual must at least halve in norm between reliable updates
                if (sc.true_rr > 0.25 * sc.prev_true_rr) sc.stalled = 1;
                sc.prev_true_rr = sc.true_rr;
            }
        });
    };
    bool ok = true;
    while (ok && !sc.stalled && sc.iter < sc.max_iter) {
        {
            // s = w + beta s; p = r + beta p; d += alpha p; r -= alpha s
            const float alpha = alpha32, beta = beta32;
            own_rows<kDirect>(o, L, [&](int local, int row) {
                const int a = keep ? local : row;
                const float si = fmaf(beta, Sv[a], Wv[a]);
                const float pi = fmaf(beta, Pv[a], Rv[a]);
                const float ri = fmaf(-alpha, si, Rv[a]);
                Sv[a] = si;
                Pv[a] = pi;
                Dv[a] = fmaf(alpha, pi, Dv[a]);
                Rv[a] = ri;
                if (keep) o.r32[row] = ri;
            });
        }
        ok = loop_reduce<kCluster, 0>(ls, red, nullptr, 0, [](const double*) {}) && spmv(false);
        if (!ok || !sc.do_update) continue;
        // reliable update: x' = x + d into the other buffer, r = b - A x' with the FP64 matrix
        const bool odd = (sc.updates & 1) != 0;
        const double* xc = odd ? o.x2 : o.x;
        double* xn = odd ? o.x : o.x2;
        own_rows<kDirect>(o, L, [&](int local, int row) {
            xn[row] = xc[row] + static_cast<double>(Dv[keep ? local : row]);
        });
        ok = loop_reduce<kCluster, 0>(ls, red, nullptr, 0, [](const double*) {});
        if (!ok) break;
        double v = 0.0;
        product<double, kDirect>(o, L, [&](int j) { return xn[j]; }, [&](int local, int row, double ax) {
            const double ri = o.b[row] - ax;
            const float rf = __double2float_rn(ri);
            Rv[keep ? local : row] = rf;
            if (keep) o.r32[row] = rf;
            v = fma(ri, ri, v);
        });
        ok = loop_reduce<kCluster, 1>(ls, red, &v, L.active, [&](const double* tot) {
            if (threadIdx.x != 0) return;
            sc.true_rr = sc.rr_upd = sc.rr_new = tot[0];
            sc.updates += 1;
            sc.iter_upd = sc.iter;
            sc.converged = tot[0] < sc.thr;
            if (sc.converged) sc.iter += 1;
        });
        if (!ok || sc.converged) break;
        ok = spmv(true);
    }
    if (keep) own_rows<kDirect>(o, L, [&](int local, int row) { o.d32[row] = Dv[local]; });
    if (!ok) {
        loop_timeout(o);
    } else if (blockIdx.x == 0) {
        store_scalars(o.S, sc);
    }
}

int g_loop_sms = 0;        // blocks of the grid form, set by cg_loop_prepare_device
int g_loop_cluster = 0;    // blocks of the cluster form (0: a cluster of that size cannot run)
size_t g_loop_smem = 0;    // largest dynamic shared memory of a block

// Chunks up to which the cluster form is used: its exchange is the cheaper one, but sixteen
// SMs have a tenth of the FP64 pipes and of the loads in flight.  And a cluster leaves the
// chip to other streams: grids of all SMs take turns, so four handles stepped from four
// threads take four times one's solve.  us a step, cluster against grid, of one handle and of
// each of four at once (dam breaks, r_e in l0; with kernels per phase four CG64 handles took
// 1,450 at 4,116 rows and 2.1 l0):
//   CG64   4,116 rows 2.1: 1,334 / 1,603, 363 / 1,433   3,745 rows 4.0: 2,260 / 2,205, 597 / 2,010
//          5,250 rows 2.1: 1,602 / 1,840, 424 / 1,721   5,250 rows 4.0: 3,004 / 2,667, 798 / 2,556
//   MIXED  5,250 rows 2.1: 1,786 / 2,100, 472 / 1,966   5,250 rows 4.0: 3,745 / 4,051, 1,029 / 3,970
//          a tall tank 6,925 rows 4.0: 2,925 / 2,697, 817 / 2,634
// Past the cluster four handles at once gain nothing over one after the other (CG64 at 10,920,
// 19,538 and 63,996 rows 2,697, 3,902 and 8,663 us a step each; kernels per phase 2,531, 3,664
// and 7,736, alone 9,275, 11,773 and 19,710); half grids would, but cost one handle 7 to 28 %.
// The grid form at 16,850, 42,226, 90,050 and 340,050 rows: CG64 9.4, 12.4, 18.4, 52.0
// (WHILE: 30.4, 31.5, 37.2, 73.7), MIXED 7.7, 9.4, 14.0 (20.6, 21.7, 25.1); the FP64 pipe
// bounds the large CG64 systems (one multiply-add per entry: 6.4 us at 90,050 rows), the
// exchanges the small ones.
// More chunks in the loop than a block's tables hold: whole chunks are walked without tables
// (kDirect).  CG64 / MIXED, us per iteration, with kernels per phase, with tables built again
// tile by tile in each product, and walked: 1.69 M rows of 28.9 entries 183 / 116, 170 / 134,
// 139 / 92; 2.4 M of 13 203 / 125, 176 / 133, 128 / 77; 4 M of 13 273 / 186, 339 / 278,
// 240 / 107 (DRAM's 6.8 TB/s bound these: 4 M rows are 624 / 416 MB of matrix an iteration).
constexpr int kClusterChunks64 = 128, kClusterChunks32 = 168;

LoopPlan loop_plan(int nchunks, bool cluster, int keep_row_bytes) {
    LoopPlan p{};
    p.blocks = cluster ? g_loop_cluster : g_loop_sms;
    if (!cluster && p.blocks > nchunks) p.blocks = nchunks;
    const int per = (nchunks + p.blocks - 1) / p.blocks;
    // two or three times the average share (a block of thin chunks alone can own five times
    // it, and then works in tiles); where that does not fit, as many as do: what the loop
    // leaves out (most rows in three dimensions) is known on the device only
    if (table_bytes(3 * per + 2) <= g_loop_smem / 2)
        p.tables = 3 * per + 2;
    else if (table_bytes(2 * per + 2) <= g_loop_smem / 4 * 3)
        p.tables = 2 * per + 2;
    else {
        p.either = true;
        p.tables = static_cast<int>((g_loop_smem / 4 * 3 - table_bytes(0)) / (table_bytes(1) - table_bytes(0)));
    }
    const size_t left = g_loop_smem - table_bytes(p.tables);
    // half as much again as the average block's vectors (the rest of the SM's memory is L1)
    const size_t want = (static_cast<size_t>(per) * 3 / 2 + 4) * kSellRows * keep_row_bytes;
    p.keep_bytes = static_cast<int>(want < left ? want : left);
    p.smem = table_bytes(p.tables) + p.keep_bytes;
    return p;
}

using LoopKernel = void (*)(CgOperands, LoopPlan);
struct LoopKernels {
    LoopKernel cluster, grid, direct;
};
constexpr LoopKernels kCgLoops{k_cg_loop<true, false>, k_cg_loop<false, false>, k_cg_loop<false, true>};
constexpr LoopKernels kMxLoops{k_mx_loop<true, false>, k_mx_loop<false, false>, k_mx_loop<false, true>};

cudaError_t launch_loop(const LoopKernels& k, const CgOperands& o, bool cluster, int keep_row_bytes, cudaStream_t s) {
    if (o.nchunks <= 0) return cudaErrorInvalidValue;
    const LoopPlan p = loop_plan(o.nchunks, cluster, keep_row_bytes);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(p.blocks));
    cfg.blockDim = dim3(kLoopThreads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    if (cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = static_cast<unsigned>(p.blocks);
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;  // every block resident: the exchanges need them all
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = p.blocks > 1 ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, cluster ? k.cluster : k.grid, o, p);
    if (e != cudaSuccess || !p.either) return e;
    cfg.dynamicSmemBytes = 0;
    return cudaLaunchKernelEx(&cfg, k.direct, o, p);
}

}  // namespace

cudaError_t cg_loop_prepare_device() {
    int dev = 0, sms = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    size_t room = static_cast<size_t>(most);
    for (auto k : {kCgLoops.cluster, kCgLoops.grid, kCgLoops.direct, kMxLoops.cluster, kMxLoops.grid, kMxLoops.direct}) {
        cudaFuncAttributes a{};
        e = cudaFuncGetAttributes(&a, k);
        if (e != cudaSuccess) return e;
        const size_t r = static_cast<size_t>(most) - a.sharedSizeBytes;
        if (r < room) room = r;
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(r));
        if (e != cudaSuccess) return e;
    }
    g_loop_smem = room;
    e = loop_grid_blocks(dev, sms, &g_loop_sms);
    if (e != cudaSuccess) return e;
    int cluster = kLoopCluster;
    for (auto k : {kCgLoops.cluster, kMxLoops.cluster}) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kLoopCluster);
        cfg.blockDim = dim3(kLoopThreads);
        cfg.dynamicSmemBytes = room;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kLoopCluster;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            cluster = 0;
        }
    }
    g_loop_cluster = cluster;
    return cudaSuccess;
}

int cg_loop_launches(int nchunks) {
    return nchunks > kClusterChunks32 && loop_plan(nchunks, false, 0).either ? 2 : 1;
}

cudaError_t launch_cg_loop(const CgOperands& o, cudaStream_t s) {
    const bool cluster = g_loop_cluster > 0 && o.nchunks <= kClusterChunks64;
    return launch_loop(kCgLoops, o, cluster, 4 * sizeof(double), s);
}

cudaError_t launch_mx_loop(const CgOperands& o, cudaStream_t s) {
    const bool cluster = g_loop_cluster > 0 && o.nchunks <= kClusterChunks32;
    return launch_loop(kMxLoops, o, cluster, 5 * sizeof(float), s);
}

}  // namespace mpsgb
