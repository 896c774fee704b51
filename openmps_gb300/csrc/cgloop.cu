// cgloop.cu - the plain solvers' iteration loops (MPS_SOLVER_CG64, MPS_SOLVER_MIXED), each
// in one launch: one cluster of 16 blocks for small systems, a cooperative grid of one block
// per SM otherwise (gridloop.cuh).
//
// Work layout: a block owns a contiguous range of SELL chunks, cut so that matrix entries and
// rows are even over the blocks; chunks of identity rows with a zero residual (dummy and
// disabled particles: 84 % of the 3D dam break's chunks) keep x and stay out of the loop.
// The split stays the same through the solve, so a row's vectors are touched by one thread
// only, and the block keeps them in shared memory when they fit (the gathered vector has
// its global copy).  For a product A v the block's chunks are cut into units of a few
// entries of a chunk's 32 rows (one warp per unit, one lane per row), the unit sums are
// parked in shared memory and the row's thread adds them: with whole chunks per warp, 17
// chunks of 46 entries (84k rows over 152 SMs) would occupy 17 of 32 warps, and a 58-chunk
// system (1,850 rows) would wait for one lane's 46 dependent multiply-adds.  Blocks with
// more chunks than the sums' room take them in tiles.
//
// CG64: the reference's conjugate gradient (Computer.hpp:1359-1429) with two grid-wide
// exchanges per iteration instead of three: the product is formed with the residual, and
// A p follows from s = A r + beta s (p = r + beta p), so p needs no exchange of its own.
// Both dot products are formed from the vectors themselves, as in the reference.
// MIXED: the Chronopoulos-Gear iteration of cg.cu (k_mx_axpy, k_mx_spmv, the reliable
// update of k_mx_fold and the FP64 true residual), phase by phase.

#include "cg.cuh"
#include "gridloop.cuh"

namespace mpsgb {

namespace {

constexpr int kStep = 8;         // matrix entries a lane loads at once
constexpr int kMaxUnits = 8;     // units of one chunk (longer rows take longer units)
constexpr int kTileChunks = 40;  // chunks whose unit sums fit a tile (40 x 8 x 32 doubles = 80 KB)

struct LoopPlan {
    int blocks;
    int tables;      // chunks the tables hold: all that a block can own, or one tile
    int keep_bytes;  // shared memory for the block's vectors
    size_t smem;
};

struct ChunkInfo {
    int chunk, off, width, first;  // first: its first unit
    int units, pad;
};

// dynamic shared memory: unit sums, chunk table, unit table, vectors
struct LoopView {
    double* part;     // kTileChunks * kMaxUnits * 32
    ChunkInfo* info;  // all chunks of the block (whole) or those of a tile
    int2* unit;       // {table index, first entry}
    unsigned char* keep;
    int c0, nc;  // whole: table entries are the chunks; else chunks c0 .. c0 + nc - 1
    int tile;    // chunks per tile
    int active;  // threads that own rows
    int warps;
    int cuts;  // units of a chunk, at most kMaxUnits
    bool whole;
};

size_t table_bytes(int tables) {
    return sizeof(double) * kTileChunks * kMaxUnits * 32 +
           (sizeof(ChunkInfo) + sizeof(int2) * kMaxUnits) * static_cast<size_t>(tables);
}

// Entries of a unit of a chunk `width` entries wide.  A block with chunks to spare takes
// them in few units (each unit past the first costs the row an addition); one with few
// cuts them so that its warps all have one.
__device__ __forceinline__ int unit_span(const LoopView& L, int width) {
    const int per = (width + L.cuts - 1) / L.cuts;
    return (per + kStep - 1) / kStep * kStep;
}

// Completes the table entries [0, m) whose chunks are set, and lists their units.
__device__ __forceinline__ void build_tables(const CgOperands& o, const LoopView& L, int m) {
    const int t = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x);
    for (int k = t; k < m; k += nt) {
        const int c = L.info[k].chunk;
        const int w = o.chunk[c] / kSellRows;
        L.info[k].off = o.off[c];
        L.info[k].width = w;
        L.info[k].units = w > 0 ? (w + unit_span(L, w) - 1) / unit_span(L, w) : 0;
    }
    __syncthreads();
    if (t < 32) {  // exclusive prefix sum of the unit counts
        int run = 0;
        for (int b = 0; b < m; b += 32) {
            const int u = b + t < m ? L.info[b + t].units : 0;
            int s = u;
            for (int d = 1; d < 32; d <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, s, d);
                if (t >= d) s += x;
            }
            if (b + t < m) L.info[b + t].first = run + s - u;
            run += __shfl_sync(0xffffffffu, s, 31);
        }
    }
    __syncthreads();
    for (int k = t; k < m; k += nt) {
        const ChunkInfo c = L.info[k];
        const int span = unit_span(L, c.width);
        for (int u = 0; u < c.units; u++) L.unit[c.first + u] = make_int2(k, u * span);
    }
    __syncthreads();
}

// This block's chunks.  o.loop_w[c] is the width of a chunk the loop works on, 0 for one it
// leaves out.  With W entries per row in N chunks, chunk k of weight prefix P_k goes to block
// floor(P_k G / P_N), P_k = (widths before it) + a (chunks before it), a = W / (4 N) (a
// row's vector work is about ten matrix entries' at the 46 entries of the usual radius): a
// block then owns at most 5 N / G + 1 chunks, and even shares when the widths are alike.
__device__ __forceinline__ LoopView loop_view(const CgOperands& o, const LoopPlan& plan, unsigned char* sm) {
    __shared__ int wsum[32], wcnt[32], first_pos, last_pos, first_chunk, last_chunk;
    LoopView L;
    L.part = reinterpret_cast<double*>(sm);
    L.info = reinterpret_cast<ChunkInfo*>(L.part + kTileChunks * kMaxUnits * 32);
    L.unit = reinterpret_cast<int2*>(L.info + plan.tables);
    L.keep = reinterpret_cast<unsigned char*>(L.unit + static_cast<size_t>(plan.tables) * kMaxUnits);
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
            L.whole = mine <= plan.tables;
            L.c0 = L.whole ? 0 : first_chunk;
            L.nc = L.whole ? mine : last_chunk - first_chunk + 1;
        }
    }
    const int tiles = max(1, (L.nc + kTileChunks - 1) / kTileChunks);
    L.tile = max(1, (L.nc + tiles - 1) / tiles);
    L.active = min(nt, L.nc * 32);
    L.cuts = min(kMaxUnits, max(1, (2 * L.warps + L.tile - 1) / L.tile));
    if (L.whole) build_tables(o, L, L.nc);
    return L;
}

// the SELL chunk of the block's k-th chunk
__device__ __forceinline__ int chunk_of(const LoopView& L, int k) { return L.whole ? L.info[k].chunk : L.c0 + k; }

__device__ __forceinline__ int ld_once(const int32_t* p) {
    int v;
    asm("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_once(const double* p) {
    double v;
    asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// A step of a unit: up to kStep entries of the lane's row.
template <class T>
struct UnitStep {
    int c[kStep];
    T a[kStep];
    int len;  // entries of the lane's row from the step on
    int out;  // the unit, when this is its last step (else -1)
};

// The warp's steps in order.
template <class T>
struct UnitCursor {
    const CgOperands& o;
    const LoopView& L;
    int u, u1, k0, end;
    ChunkInfo ci;

    __device__ __forceinline__ void open() {
        const int2 un = L.unit[u];
        ci = L.info[un.x];
        k0 = un.y;
        end = min(ci.width, k0 + unit_span(L, ci.width));
    }
    __device__ __forceinline__ UnitCursor(const CgOperands& o_, const LoopView& L_, int u_, int u1_)
        : o(o_), L(L_), u(u_), u1(u1_), k0(0), end(0) {
        if (u < u1) open();
    }
    __device__ __forceinline__ bool valid() const { return u < u1; }
    // Loads the current step and moves on.  Entries of a row past its length lie inside
    // the chunk: they are loaded, not used.
    __device__ __forceinline__ void load(UnitStep<T>& s) {
        const int lane = threadIdx.x & 31;
        s.len = o.len[ci.chunk * kSellRows + lane] - k0;
        const int64_t at = static_cast<int64_t>(ci.off) + static_cast<int64_t>(k0) * kSellRows + lane;
#pragma unroll
        for (int e = 0; e < kStep; e++) {
            s.c[e] = 0;
            s.a[e] = 0;
            if (k0 + e < ci.width) {
                if constexpr (sizeof(T) == 8) {
                    s.c[e] = ld_once(o.col + at + e * kSellRows);
                    s.a[e] = ld_once(o.val + at + e * kSellRows);
                } else {
                    const uint2 p = ld_sell_pair(o.cv32 + at + e * kSellRows);
                    s.c[e] = static_cast<int>(p.x);
                    s.a[e] = __uint_as_float(p.y);
                }
            }
        }
        s.out = -1;
        k0 += kStep;
        if (k0 >= end) {
            s.out = u;
            u += L.warps;
            if (u < u1) open();
        }
    }
};

// Unit sums of table chunks [a, b): T = double (FP64 matrix) or float (FP32 pairs).  Two
// steps in turn, each loaded while the other gathers and adds: a warp waits for one round
// trip to L2 per step (0.6 us across the dies), not for two.
template <class T>
__device__ __forceinline__ void unit_sums(const CgOperands& o, const LoopView& L, int a, int b, const T* v) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T* part = reinterpret_cast<T*>(L.part);
    const int u0 = L.info[a].first, u1 = L.info[b - 1].first + L.info[b - 1].units;
    UnitCursor<T> cur(o, L, u0 + warp, u1);
    if (!cur.valid()) return;
    T acc = 0;
    auto add = [&](const UnitStep<T>& s) {
        T xv[kStep];
#pragma unroll
        for (int e = 0; e < kStep; e++) xv[e] = e < s.len ? v[s.c[e]] : T(0);
#pragma unroll
        for (int e = 0; e < kStep; e++)
            if (e < s.len) {
                if constexpr (sizeof(T) == 8) acc = fma(s.a[e], xv[e], acc);
                else acc = fmaf(s.a[e], xv[e], acc);
            }
        if (s.out >= 0) {
            part[(s.out - u0) * 32 + lane] = acc;
            acc = 0;
        }
    };
    UnitStep<T> A, B;
    cur.load(A);
    while (true) {
        const bool b_next = cur.valid();
        if (b_next) cur.load(B);
        add(A);
        if (!b_next) break;
        const bool a_next = cur.valid();
        if (a_next) cur.load(A);
        add(B);
        if (!a_next) break;
    }
}

// f(local row, row, (A v)_row) for every row of the block, by the row's thread
template <class T, class F>
__device__ __forceinline__ void product(const CgOperands& o, const LoopView& L, const T* v, F f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const T* part = reinterpret_cast<const T*>(L.part);
    for (int k0 = 0; k0 < L.nc; k0 += L.tile) {
        const int k1 = min(L.nc, k0 + L.tile);
        const int table0 = L.whole ? 0 : k0;
        if (!L.whole) {
            for (int k = k0 + static_cast<int>(threadIdx.x); k < k1; k += static_cast<int>(blockDim.x))
                L.info[k - k0].chunk = L.c0 + k;
            __syncthreads();
            build_tables(o, L, k1 - k0);
        }
        unit_sums<T>(o, L, k0 - table0, k1 - table0, v);
        __syncthreads();
        const int u0 = L.info[k0 - table0].first;
        const int skip = k0 % L.warps;  // chunk k belongs to warp k % warps
        for (int k = k0 - skip + warp + (warp < skip ? L.warps : 0); k < k1; k += L.warps) {
            const ChunkInfo c = L.info[k - table0];
            const T* p = part + (c.first - u0) * 32 + lane;
            T s = c.units > 0 ? p[0] : T(0);  // two chains of additions
            if (c.units > 1) {
                T q = p[32];
                for (int u = 2; u < c.units; u++) {
                    if (u & 1) q += p[u * 32];
                    else s += p[u * 32];
                }
                s += q;
            }
            const int row = c.chunk * kSellRows + lane;
            if (row < o.n) f(k * kSellRows + lane, row, s);
        }
        if (k1 < L.nc) __syncthreads();  // the next tile overwrites the sums
    }
}

// g(local row, row) for every row of the block, by the thread product() gives it to
template <class G>
__device__ __forceinline__ void own_rows(const CgOperands& o, const LoopView& L, G g) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = warp; k < L.nc; k += L.warps) {
        const int row = chunk_of(L, k) * kSellRows + lane;
        if (row < o.n) g(k * kSellRows + lane, row);
    }
}

__device__ __forceinline__ void loop_timeout(const CgOperands& o) {
    if (threadIdx.x == 0) {
        if (o.status) atomicOr(&const_cast<DevStatus*>(o.status)->flags, kStatusWaitTimeout);
        o.S->aborted = 1;
    }
}

template <bool kCluster>
__global__ void __launch_bounds__(kLoopThreads, 1) k_cg_loop(CgOperands o, LoopPlan plan) {
    extern __shared__ __align__(16) unsigned char loop_sm[];
    __shared__ LoopReduce red;
    __shared__ struct {
        double rr, alpha, beta, pap, rr_new;
        int iter, conv;
    } sc;
    CgScalars* S = o.S;
    if (S->converged || S->aborted || S->iter >= S->max_iter) return;
    const LoopView L = loop_view(o, plan, loop_sm);
    if (kCluster) loop_cluster_start();
    LoopSync ls{o.slots, gridDim.x, 0};
    const double thr = S->thr;
    const int max_iter = S->max_iter;
    if (threadIdx.x == 0) {
        sc.rr = S->rr;
        sc.beta = 0.0;
        sc.iter = S->iter;
        sc.conv = 0;
    }
    // the block's rows of p, s, x and r: index `a` of a row is its place in the block when
    // they are kept in shared memory, the row itself in the global arrays
    const int rows = L.nc * kSellRows;
    const bool keep = L.whole && 4 * static_cast<int64_t>(sizeof(double)) * rows <= plan.keep_bytes;
    double* kept = reinterpret_cast<double*>(L.keep);
    double* P = keep ? kept : o.p;
    double* Q = keep ? kept + rows : o.Ap;
    double* X = keep ? kept + 2 * rows : o.x;
    double* R = keep ? kept + 3 * rows : o.r;
    own_rows(o, L, [&](int local, int row) {
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
            product<double>(o, L, o.r, [&](int local, int row, double ar) {
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
            own_rows(o, L, [&](int local, int row) {
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
    if (keep) own_rows(o, L, [&](int local, int row) { o.x[row] = X[local]; });
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

template <bool kCluster>
__global__ void __launch_bounds__(kLoopThreads, 1) k_mx_loop(CgOperands o, LoopPlan plan) {
    extern __shared__ __align__(16) unsigned char loop_sm[];
    __shared__ LoopReduce red;
    __shared__ CgScalars sc;  // the solve's scalars, as the per-phase kernels keep them
    if (o.S->converged || o.S->aborted || o.S->iter >= o.S->max_iter) return;
    const LoopView L = loop_view(o, plan, loop_sm);
    if (kCluster) loop_cluster_start();
    LoopSync ls{o.slots, gridDim.x, 0};
    if (threadIdx.x == 0) sc = *o.S;
    // the block's rows of s, p, d, w and r (kept or global, as in k_cg_loop)
    const int rows = L.nc * kSellRows;
    const bool keep = L.whole && 5 * static_cast<int64_t>(sizeof(float)) * rows <= plan.keep_bytes;
    float* kept = reinterpret_cast<float*>(L.keep);
    float* Sv = keep ? kept : o.s32;
    float* Pv = keep ? kept + rows : o.p32;
    float* Dv = keep ? kept + 2 * rows : o.d32;
    float* Wv = keep ? kept + 3 * rows : o.w32;
    float* Rv = keep ? kept + 4 * rows : o.r32;
    if (keep)
        own_rows(o, L, [&](int local, int row) {
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
        product<float>(o, L, o.r32, [&](int local, int row, float w) {
            const int a = keep ? local : row;
            const double ri = static_cast<double>(Rv[a]);
            Wv[a] = w;
            if (after_update) Dv[a] = 0.0f;
            v[0] = fma(ri, ri, v[0]);
            v[1] = fma(static_cast<double>(w), ri, v[1]);
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
            const float alpha = __double2float_rn(sc.alpha), beta = __double2float_rn(sc.beta);
            own_rows(o, L, [&](int local, int row) {
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
        own_rows(o, L, [&](int local, int row) {
            xn[row] = xc[row] + static_cast<double>(Dv[keep ? local : row]);
        });
        ok = loop_reduce<kCluster, 0>(ls, red, nullptr, 0, [](const double*) {});
        if (!ok) break;
        double v = 0.0;
        product<double>(o, L, xn, [&](int local, int row, double ax) {
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
    if (keep) own_rows(o, L, [&](int local, int row) { o.d32[row] = Dv[local]; });
    if (!ok) {
        loop_timeout(o);
    } else if (blockIdx.x == 0 && threadIdx.x == 0) {
        *o.S = sc;
    }
}

int g_loop_sms = 0;        // SMs of the device (one block each), set by cg_loop_prepare_device
int g_loop_cluster = 0;    // blocks of the cluster form (0: a cluster of that size cannot run)
size_t g_loop_smem = 0;    // largest dynamic shared memory of a block

// Chunks up to which the cluster form is used: its exchange is the cheaper one, but sixteen
// SMs have a tenth of the FP64 pipes and of the loads in flight.  us per iteration, cluster
// against grid (dam breaks at r_e = 4 l0; the WHILE node's kernels took 29-31 and 19-21):
//   rows      1,850        3,133        5,250         9,403
//   CG64    6.8 / 8.2    8.7 / 8.3   11.2 / 8.5    16.8 / 8.9
//   MIXED   5.5 / 7.1    6.7 / 7.3    8.2 / 7.2    11.1 / 7.2
// The grid form at 16,850, 42,226, 90,050 and 340,050 rows: CG64 10.2, 14.9, 23.0, 72.9
// (WHILE: 30.4, 31.5, 37.2, 73.7), MIXED 7.7, 10.7, 16.4 (20.6, 21.7, 25.1); the FP64 pipe
// bounds the large CG64 systems (one multiply-add per entry: 6.4 us at 90,050 rows), the
// exchanges the small ones.
constexpr int kClusterChunks64 = 80, kClusterChunks32 = 128;

LoopPlan loop_plan(int nchunks, bool cluster, int keep_row_bytes) {
    LoopPlan p{};
    p.blocks = cluster ? g_loop_cluster : g_loop_sms;
    if (!cluster && p.blocks > nchunks) p.blocks = nchunks;
    const int most = 5 * ((nchunks + p.blocks - 1) / p.blocks) + 2;
    p.tables = table_bytes(most) <= g_loop_smem ? most : kTileChunks;
    const size_t room = g_loop_smem - table_bytes(p.tables);
    // half as much again as the average block's vectors (the rest of the SM's memory is L1)
    const size_t want = (static_cast<size_t>(nchunks) * 3 / (2 * p.blocks) + 4) * kSellRows * keep_row_bytes;
    p.keep_bytes = static_cast<int>(want < room ? want : room);
    p.smem = table_bytes(p.tables) + p.keep_bytes;
    return p;
}

cudaError_t launch_loop(void (*kernel)(CgOperands, LoopPlan), const CgOperands& o, bool cluster, int keep_row_bytes,
                        cudaStream_t s) {
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
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, o, p);
}

}  // namespace

cudaError_t cg_loop_prepare_device() {
    int dev = 0, sms = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    size_t room = static_cast<size_t>(most);
    for (auto k : {k_cg_loop<false>, k_cg_loop<true>, k_mx_loop<false>, k_mx_loop<true>}) {
        cudaFuncAttributes a{};
        e = cudaFuncGetAttributes(&a, k);
        if (e != cudaSuccess) return e;
        const size_t r = static_cast<size_t>(most) - a.sharedSizeBytes;
        if (r < room) room = r;
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(r));
        if (e != cudaSuccess) return e;
    }
    g_loop_smem = room;
    g_loop_sms = sms < kLoopMaxBlocks ? sms : kLoopMaxBlocks;
    int cluster = kLoopCluster;
    for (auto k : {k_cg_loop<true>, k_mx_loop<true>}) {
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

cudaError_t launch_cg_loop(const CgOperands& o, cudaStream_t s) {
    const bool cluster = g_loop_cluster > 0 && o.nchunks <= kClusterChunks64;
    return launch_loop(cluster ? k_cg_loop<true> : k_cg_loop<false>, o, cluster, 4 * sizeof(double), s);
}

cudaError_t launch_mx_loop(const CgOperands& o, cudaStream_t s) {
    const bool cluster = g_loop_cluster > 0 && o.nchunks <= kClusterChunks32;
    return launch_loop(cluster ? k_mx_loop<true> : k_mx_loop<false>, o, cluster, 5 * sizeof(float), s);
}

}  // namespace mpsgb
