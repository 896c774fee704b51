// pcgloop.cu - the preconditioned iteration loop (MPS_SOLVER_MIXED_MG, MPS_SOLVER_LEARNED) in
// one launch: one cluster of 16 blocks for small scenes, a cooperative grid of one block per
// SM otherwise.  The iteration is cg.cu's preconditioned Chronopoulos-Gear CG with reliable
// updates, the preconditioner mg.cu's cell multigrid.
//
// As kernels under a WHILE node an iteration is a chain of five launches and their round
// trips whatever the size.  Here a block owns a contiguous range of search cells with their
// rows (PPE rows are in cell order) for the whole solve, and an iteration is
//   vector updates and the level-1 residuals of the own cells               | exchange
//   per level above the bottom: the own share of the next level's residuals | exchange each
//   the bottom levels, in every block at once from planes staged once per solve
//   per level between: the own share of the corrections                     | exchange each
//   level-1 corrections and u of the own cells and of the cells around them
//   w = A u for the own rows, three dot products                            | exchange (sum)
// A row's columns lie in the own cells and their neighbours: three ranges of rows, whose u
// the block computes itself into a window in shared memory (from the first row of the cells
// around to the last: a column is a place in it), so u needs no exchange and the SpMV
// gathers from shared memory.  If a block's window does not fit (cells much fuller than at
// rest) all blocks go through the global u and one more exchange.
//
// us per solve, the chain against this loop (GB300, dam breaks at r_e = 4 l0):
//   rows       1,850   3,133   5,250   9,403  16,850  42,226  90,050   hydrostatic 84,450
//   chain      1,684   1,861   1,882   2,087   2,075   2,752   2,896   2,634
//   loop         742     936   1,004   1,156   1,154   1,637   2,419   1,855
// An iteration's bound is latency: at 1,850 rows 5,000 of 24,000 cycles are the bottom
// levels' chain of shared-memory steps, 6,900 the sum and its divisions, 3,300 the SpMV's
// four dependent steps; at 84k rows 11,000 of 53,000 are the SpMV (28 MB from L2, which
// alone would stream in 4,000), 11,000 the sum, 10,000 the bottom levels.  From about 130,000
// rows window, own vectors and bottom levels pass the SM's shared memory, and the chain runs:
// with u (and the own vectors) in global memory this loop takes 142 us an iteration against
// the chain's 63 at 177,641 rows, and 333 against 73 at 340,050.
#include <algorithm>
#include <cmath>

#include "cgloop.cuh"
#include "mg.cuh"

namespace mpsgb {

namespace {

// Sizes of the dynamic shared memory: bottom levels, unit sums, tables, own rows, window,
// cells around.
struct PcgPlan {
    int blocks;
    int bottom_floats;
    int tables;  // chunks
    int rows;    // own rows whose vectors are kept (more: they stay in global memory)
    int window;  // rows of the window
    int cells;   // cells with rows among the window's
    int bottom;  // first of the levels that every block takes
    size_t smem;
};

// own rows' s, p, d, w, r; per window row u, Jacobi factor, cell; per cell its id and correction
constexpr int kRowBytes = 5 * 4, kWindowBytes = 4 + 4 + 2, kCellBytes = 4 + 4 + 4;

// A bottom level in shared memory: K[9][cells], 1 / diagonal, residual r, correction e, and
// the iterate x in a frame of zeros one cell wide, so that a stencil reads its neighbours at
// fixed offsets.  The last level: r, e and the dense inverse.
struct BottomLevel {
    int nx, nz, cells;
    int k, dinv, r, e, x;  // float offsets
    unsigned by_nz;        // of column_of
};

// c / nz for c nz < 2^32 (2^32 / 1 has no 32-bit multiplier)
__device__ __forceinline__ int column_of(const BottomLevel& B, int c) {
    return B.nz == 1 ? c : static_cast<int>(__umulhi(static_cast<unsigned>(c), B.by_nz));
}

__host__ __device__ inline int bottom_level_floats(const MgLevel& L, bool last) {
    const int64_t c = mg_round4(L.cells);
    if (last) return static_cast<int>(2 * c + mg_round4(static_cast<int64_t>(L.cells) * L.cells));
    return static_cast<int>(mg_round4(9 * static_cast<int64_t>(L.cells)) + 3 * c +
                            mg_round4(static_cast<int64_t>(L.nx + 2) * (L.nz + 2)));
}

// The block's share [first, last) of `cells`.
__device__ __forceinline__ int share_of(int cells, int b) {
    return static_cast<int>(static_cast<int64_t>(cells) * b / gridDim.x);
}

template <bool kCluster>
__global__ void __launch_bounds__(kLoopThreads, 1) k_pcg_loop(CgOperands o, MgHierarchy mg, PcgPlan plan) {
    extern __shared__ __align__(16) float pcg_sm[];
    __shared__ LoopReduce red;
    __shared__ CgScalars sc;  // the solve's scalars, as the per-phase kernels keep them
    __shared__ float alpha32, beta32;
    __shared__ int wsum[32], first_cell, last_cell, n_cells, own0, own1, windowed;
    __shared__ BottomLevel bl[kMgMaxLevels + 1];
    // the cells around, as up to three disjoint ranges of cells and of rows
    __shared__ struct {
        int ca[3], cb[3], ra[3], rb[3], before[3];
    } rg;
    // read by every phase: in registers they would spill, and spills miss L1 after each exchange
    __shared__ LoopView L;
    __shared__ float* vec[5];  // the own rows' s, p, d, w, r
    __shared__ float* uv;      // u: the window, or all of it
    if (o.S->converged || o.S->aborted || o.S->max_iter <= 0) return;
    if (kCluster) loop_cluster_start();
    LoopSync ls{o.slots, gridDim.x, 0};
    const int t = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x), lane = t & 31, warp = t >> 5;
    const MgLevel& L1 = mg.lv[1];
    const int nz1 = L1.nz;

    // ---- this block's cells: even shares of the cells' weights (mg.cell_w)
    const int seg = (L1.cells + nt - 1) / nt;
    const int sb = min(L1.cells, t * seg), se = min(L1.cells, sb + seg);
    int w = 0;
    for (int c = sb; c < se; c++) w += mg.cell_w[c];
    int ws = w;
    for (int d = 1; d < 32; d <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, ws, d);
        if (lane >= d) ws += x;
    }
    if (lane == 31) wsum[warp] = ws;
    if (t == 0) {
        red.wait_clocks = loop_wait_clocks(o);
        sc = *o.S;
        first_cell = 0x7fffffff;
        last_cell = -1;
        own0 = 0x7fffffff;
        own1 = 0;
        int at = 0;
        for (int l = plan.bottom; l <= mg.levels; l++) {
            const MgLevel& G = mg.lv[l];
            const int c4 = static_cast<int>(mg_round4(G.cells));
            BottomLevel B{G.nx, G.nz, G.cells, at, 0, 0, 0, 0, 0xffffffffu / static_cast<unsigned>(G.nz) + 1u};
            if (l == mg.levels) {
                B.r = at;
                B.e = at + c4;
                B.k = at + 2 * c4;
            } else {
                B.dinv = at + static_cast<int>(mg_round4(9 * static_cast<int64_t>(G.cells)));
                B.r = B.dinv + c4;
                B.e = B.r + c4;
                B.x = B.e + c4;
            }
            bl[l] = B;
            at += bottom_level_floats(G, l == mg.levels);
        }
    }
    __syncthreads();
    int W = 0;
    for (int k = 0; k < nt >> 5; k++) {
        if (k == warp) ws += W;
        W += wsum[k];
    }
    {
        long long wp = ws - w;
        for (int c = sb; c < se; c++) {
            const int x = mg.cell_w[c];
            if (x > 0 && wp * gridDim.x / W == static_cast<long long>(blockIdx.x)) {
                atomicMin(&first_cell, c);
                atomicMax(&last_cell, c);
            }
            wp += x;
        }
    }
    __syncthreads();
    const bool any = last_cell >= 0;
    const int c0 = any ? first_cell : 0, c1 = any ? last_cell + 1 : 0;
    const int r0 = any ? mg.cell_start[c0] : 0, r1 = any ? mg.cell_start[c1] : 0;
    const int rows = r1 - r0;
    if (t == 0) {
        const int lo[3] = {c0 - nz1 - 1, c0 - 1, c0 + nz1 - 1}, hi[3] = {c1 - nz1 + 1, c1 + 1, c1 + nz1 + 1};
        int end = 0, total = 0;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            rg.ca[q] = any ? min(L1.cells, max(max(lo[q], 0), end)) : 0;
            rg.cb[q] = any ? max(rg.ca[q], min(hi[q], L1.cells)) : 0;
            end = rg.cb[q];
            rg.ra[q] = any ? mg.cell_start[rg.ca[q]] : 0;
            rg.rb[q] = any ? mg.cell_start[rg.cb[q]] : 0;
            rg.before[q] = total;
            total += rg.rb[q] - rg.ra[q];
        }
    }
    __syncthreads();

    // ---- shared memory
    float* bot = pcg_sm;
    LoopView V;
    float* own = reinterpret_cast<float*>(place_tables(V, bot + plan.bottom_floats, plan.tables));
    ChunkInfo* const info = V.info;
    float* win_u = own + 5 * static_cast<size_t>(plan.rows);
    float* win_d = win_u + plan.window;
    int* cell_id = reinterpret_cast<int*>(win_d + plan.window);
    int* cell_row = cell_id + plan.cells;
    float* cell_e = reinterpret_cast<float*>(cell_row + plan.cells);
    uint16_t* win_c = reinterpret_cast<uint16_t*>(cell_e + plan.cells);

    // the cells with rows among them, in order, and each window row's cell and Jacobi factor
    bool fits = rg.rb[2] - rg.ra[0] <= plan.window;
    {
        int base = 0;
        for (int q = 0; q < 3; q++) {
            for (int at = rg.ca[q]; at < rg.cb[q]; at += nt) {
                const int c = at + t;
                const int b = c < rg.cb[q] ? mg.cell_start[c] : 0, e = c < rg.cb[q] ? mg.cell_start[c + 1] : 0;
                const unsigned m = __ballot_sync(0xffffffffu, e > b);
                __syncthreads();
                if (lane == 0) wsum[warp] = __popc(m);
                __syncthreads();
                int pos = base, all = 0;
                for (int k = 0; k < nt >> 5; k++) {
                    if (k < warp) pos += wsum[k];
                    all += wsum[k];
                }
                pos += __popc(m & ((1u << lane) - 1u));
                if (e > b && fits && pos < plan.cells) {
                    cell_id[pos] = c;
                    cell_row[pos] = b;
                    if (c >= c0 && c < c1) {
                        atomicMin(&own0, pos);
                        atomicMax(&own1, pos + 1);
                    }
                    for (int i = b; i < e; i++) {
                        const int a = rg.before[q] + i - rg.ra[q];
                        const float d = mg.dinv0[i];
                        win_c[a] = static_cast<uint16_t>(pos);
                        win_d[a] = mg.scale ? mg.scale[i] * d : d;
                    }
                }
                base += all;
            }
        }
        if (t == 0) n_cells = base;
    }
    __syncthreads();
    fits = fits && n_cells <= plan.cells;
    const bool listed = fits && any;
    // the bottom levels' planes and dense inverse
    for (int l = plan.bottom; l < mg.levels; l++) {
        const BottomLevel B = bl[l];
        for (int q = t; q < 9 * B.cells; q += nt) bot[B.k + q] = mg.lv[l].k32[q];
        for (int q = t; q < B.cells; q += nt) bot[B.dinv + q] = mg.lv[l].dinv[q];
        for (int q = t; q < (B.nx + 2) * (B.nz + 2); q += nt) bot[B.x + q] = 0.0f;
    }
    const int m_dense = mg.lv[mg.levels].cells;
    for (int q = t; q < m_dense * m_dense; q += nt) bot[bl[mg.levels].k + q] = mg.dense[q];

    // the rows as SELL chunks
    // the own rows' vectors, kept (index: row - r0) or global (index: row)
    const bool keep = rows <= plan.rows;
    if (t == 0) {
        V.warps = nt >> 5;
        V.lo = r0;
        V.hi = r1;
        V.c0 = r0 / kSellRows;
        V.nc = rows > 0 ? (r1 - 1) / kSellRows - V.c0 + 1 : 0;
        V.whole = V.nc <= plan.tables;
        split_tiles(V, plan.tables);
        L = V;
        float* const global[5] = {o.s32, o.p32, o.d32, o.w32, o.r32};
        for (int k = 0; k < 5; k++) vec[k] = keep ? own + k * plan.rows - r0 : global[k];
    }
    __syncthreads();
    if (L.whole) {
        for (int k = t; k < L.nc; k += nt) info[k].chunk = L.c0 + k;
        __syncthreads();
        build_tables(o, L, L.nc);
    }
    if (keep)
        for (int i = r0 + t; i < r1; i += nt) {
            for (int k = 0; k < 4; k++) vec[k][i] = 0.0f;
            vec[4][i] = o.r32[i];
        }
    const double misfit = t == 0 && !fits ? 1.0 : 0.0;
    bool ok = loop_reduce<kCluster, 1>(ls, red, &misfit, 1, [&](const double* tot) {
        if (threadIdx.x != 0) return;
        windowed = tot[0] == 0.0 ? 1 : 0;
        uv = windowed ? win_u - rg.ra[0] : o.u32;
    });
    const bool win = windowed != 0;

    auto barrier = [&] { return loop_reduce<kCluster, 0>(ls, red, nullptr, 0, [](const double*) {}); };
    // u = M r; with `axpy` the iteration's vector updates first
    auto cycle = [&](bool axpy) {
        if (axpy) {
            const float alpha = alpha32, beta = beta32;
            float *const Sv = vec[0], *const Pv = vec[1], *const Dv = vec[2], *const Wv = vec[3], *const Rv = vec[4];
            for (int i = L.lo + t; i < L.hi; i += nt) {
                const float ui = uv[i];
                const float si = fmaf(beta, Sv[i], Wv[i]);
                const float pi = fmaf(beta, Pv[i], ui);
                const float ri = fmaf(-alpha, si, Rv[i]);
                Sv[i] = si;
                Pv[i] = pi;
                Dv[i] = fmaf(alpha, pi, Dv[i]);
                Rv[i] = ri;
                if (keep) o.r32[i] = ri;
            }
        }
        __syncthreads();
        // level-1 residuals: eight lanes per cell (cells without rows keep their zero)
        const float* const Rv = vec[4];
        auto cell_sum = [&](int b, int e, int c) {
            float sum = 0.0f;
            for (int i = b + (t & 7); i < e; i += 8) sum += Rv[i];
#pragma unroll
            for (int d = 4; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
            if ((t & 7) == 0 && e > b) L1.r[c] = sum;
        };
        if (listed) {
            for (int k = own0 + (t >> 3); k - (t >> 3) < own1; k += nt >> 3) {
                const int b = k < own1 ? cell_row[k] : 0, e = k + 1 < own1 ? cell_row[k + 1] : k < own1 ? L.hi : 0;
                cell_sum(b, e, k < own1 ? cell_id[k] : 0);
            }
        } else {
            for (int c = c0 + (t >> 3); c - (t >> 3) < c1; c += nt >> 3)
                cell_sum(c < c1 ? mg.cell_start[c] : 0, c < c1 ? mg.cell_start[c + 1] : 0, c);
        }
        if (!barrier()) return false;
        if (win) {  // the residuals around, while the coarse levels run
            const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(win_u));
#pragma unroll
            for (int q = 0; q < 3; q++)
                for (int i = rg.ra[q] + t; i < rg.rb[q]; i += nt)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to + 4u * (i - rg.ra[0])), "l"(o.r32 + i) : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        // down to the bottom: four lanes per coarse cell, one child each
        for (int l = 1; l < plan.bottom; l++) {
            const MgLevel& f = mg.lv[l];
            const MgLevel& cl = mg.lv[l + 1];
            const int s0 = share_of(cl.cells, blockIdx.x), s1 = share_of(cl.cells, blockIdx.x + 1);
            for (int I = s0 + (t >> 2); I - (t >> 2) < s1; I += nt >> 2) {
                const int cell = min(I, cl.cells - 1);
                const int X = cell / cl.nz, Z = cell - (cell / cl.nz) * cl.nz;
                float v = child_residual(f.nx, f.nz, f.cells, f.k32, f.dinv, f.r, 2 * X + ((t >> 1) & 1), 2 * Z + (t & 1));
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if ((t & 3) == 0 && I < s1) cl.r[I] = v;
            }
            if (!barrier()) return false;
        }
        // the bottom levels, in every block
        {
            const BottomLevel B = bl[plan.bottom];
            const float* src = mg.lv[plan.bottom].r;
            for (int c = t; c < B.cells; c += nt) {
                const float r = src[c];
                bot[B.r + c] = r;
                if (plan.bottom < mg.levels) {
                    const int cx = column_of(B, c);
                    bot[B.x + (cx + 1) * (B.nz + 2) + c - cx * B.nz + 1] = bot[B.dinv + c] * r;
                }
            }
        }
        __syncthreads();
        // residual after the pre-smoothing x: r - K x at cell (cx, cz)
        auto residual = [&](const BottomLevel& B, int cx, int cz) {
            const int c = cx * B.nz + cz, pitch = B.nz + 2;
            const float* k = bot + B.k + c;
            const float* x = bot + B.x + cx * pitch + cz;
            float res = bot[B.r + c];
#pragma unroll
            for (int dx = 0; dx < 3; dx++) {
#pragma unroll
                for (int dz = 0; dz < 3; dz++) res -= k[(3 * dx + dz) * B.cells] * x[dx * pitch + dz];
            }
            return res;
        };
        for (int l = plan.bottom; l < mg.levels; l++) {  // four lanes per coarse cell, one child each
            const BottomLevel B = bl[l], C = bl[l + 1];
            for (int I = t >> 2; I - (t >> 2) < C.cells; I += nt >> 2) {
                const int cell = min(I, C.cells - 1);
                const int X = column_of(C, cell), Z = cell - X * C.nz;
                const int cx = 2 * X + ((t >> 1) & 1), cz = 2 * Z + (t & 1);
                float v = cx < B.nx && cz < B.nz ? residual(B, cx, cz) : 0.0f;
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if ((t & 3) == 0 && I < C.cells) {
                    bot[C.r + I] = v;
                    if (l + 1 < mg.levels) bot[C.x + (X + 1) * (C.nz + 2) + Z + 1] = bot[C.dinv + I] * v;
                }
            }
            __syncthreads();
        }
        {  // four lanes per row of the dense inverse
            const BottomLevel B = bl[mg.levels];
            const float* r = bot + B.r;
            for (int row = t >> 2; row - (t >> 2) < m_dense; row += nt >> 2) {
                const float* dn = bot + B.k + min(row, m_dense - 1) * m_dense;
                float v = 0.0f;
                for (int k = t & 3; k < m_dense; k += 4) v = fmaf(dn[k], r[k], v);
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if ((t & 3) == 0 && row < m_dense) bot[B.e + row] = v;
            }
        }
        __syncthreads();
        for (int l = mg.levels - 1; l >= plan.bottom; l--) {
            const BottomLevel B = bl[l], C = bl[l + 1];
            for (int c = t; c < B.cells; c += nt) {  // x += w e of the parent
                const int cx = column_of(B, c), cz = c - cx * B.nz;
                bot[B.x + (cx + 1) * (B.nz + 2) + cz + 1] += kMgCoarseWeight * bot[C.e + (cx >> 1) * C.nz + (cz >> 1)];
            }
            __syncthreads();
            for (int c = t; c < B.cells; c += nt) {  // and one Jacobi step
                const int cx = column_of(B, c), cz = c - cx * B.nz;
                bot[B.e + c] = bot[B.x + (cx + 1) * (B.nz + 2) + cz + 1] + bot[B.dinv + c] * residual(B, cx, cz);
            }
            __syncthreads();
        }
        // up to level 2
        for (int l = plan.bottom - 1; l >= 2; l--) {
            const MgLevel& f = mg.lv[l];
            const float* ec = l + 1 == plan.bottom ? bot + bl[plan.bottom].e : mg.lv[l + 1].e;
            const int s1 = share_of(f.cells, blockIdx.x + 1);
            for (int ch = share_of(f.cells, blockIdx.x) + t; ch < s1; ch += nt)
                f.e[ch] = smoothed_correction(f.nx, f.nz, f.cells, f.k32, f.dinv, f.r, mg.lv[l + 1].nz, ec, ch);
            if (!barrier()) return false;
        }
        // level 1 and u
        const float* eb = bot + bl[plan.bottom].e;
        const float* e2 = plan.bottom == 2 ? eb : mg.lv[2].e;
        auto level1 = [&](int c) {
            return plan.bottom == 1 ? eb[c]
                                  : smoothed_correction(L1.nx, L1.nz, L1.cells, L1.k32, L1.dinv, L1.r, mg.lv[2].nz, e2, c);
        };
        if (win) {
            for (int k = t; k < n_cells; k += nt) cell_e[k] = level1(cell_id[k]);
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 3; q++)
                for (int i = rg.ra[q] + t; i < rg.rb[q]; i += nt) {
                    const int a = rg.before[q] + i - rg.ra[q];
                    const float d = win_d[a];
                    float& ui = win_u[i - rg.ra[0]];
                    ui = d != 0.0f ? d * ui + cell_e[win_c[a]] : 0.0f;
                }
            __syncthreads();
            return true;
        }
        for (int c = c0 + t; c < c1; c += nt) {
            const int b = mg.cell_start[c], e = mg.cell_start[c + 1];
            if (e <= b) continue;
            const float ec = level1(c);
            for (int i = b; i < e; i++) {
                const float d = mg.dinv0[i];
                const float s = mg.scale ? mg.scale[i] : 1.0f;
                o.u32[i] = d != 0.0f ? s * d * Rv[i] + ec : 0.0f;
            }
        }
        return barrier();
    };
    // w = A u; gamma = r.u, delta = w.u, rho = r.r and what follows (pmx_finish in cg.cu).
    // mode 0: first, 1: an iteration, 2: after a reliable update
    auto spmv = [&](int mode) {
        double v[3] = {0.0, 0.0, 0.0};
        float *const Dv = vec[2], *const Wv = vec[3];
        const float *const Rv = vec[4], *const u = uv;
        auto row_done = [&](int, int row, float wi) {
            const double ri = widen(Rv[row]);
            const double ui = widen(u[row]);
            Wv[row] = wi;
            if (mode == 2) Dv[row] = 0.0f;
            v[0] = fma(ri, ui, v[0]);
            v[1] = fma(widen(wi), ui, v[1]);
            v[2] = fma(ri, ri, v[2]);
        };
        product<float>(o, L, [&](int j) { return u[j]; }, row_done);
        return loop_reduce<kCluster, 3>(ls, red, v, L.active, [&](const double* tot) {
            const double gam = tot[0], del = tot[1], rho = tot[2];
            // beta = gam / rr in lane 0, beta gam / alpha in lane 1
            const bool one = (threadIdx.x & 31) == 1;
            const double q = ddiv_rn(one ? gam * gam : gam, one ? sc.rr * sc.alpha : sc.rr);
            const double drop = __shfl_sync(0xffffffffu, q, 1);
            const double alpha = ddiv_rn(gam, mode == 0 ? del : del - drop);
            if (threadIdx.x != 0) return;
            sc.rr_new = rho;
            sc.do_update = mode == 1 && (rho < sc.delta2 * sc.rr_upd || rho < sc.thr);
            int stalled = 0;
            if (mode == 2) {
                stalled = sc.true_rr > 0.25 * sc.prev_true_rr;
                sc.prev_true_rr = sc.true_rr;
            }
            if (!sc.do_update && !stalled) {
                const double beta = mode == 0 ? 0.0 : q;
                if (mode != 0) sc.iter += 1;
                stalled = !(isfinite(alpha) && isfinite(beta) && alpha != 0.0);
                sc.alpha = alpha;
                sc.beta = beta;
                alpha32 = __double2float_rn(alpha);  // once: a conversion takes the pipe 64 cycles a warp
                beta32 = __double2float_rn(beta);
                sc.rr = gam;
                sc.pAp = del;
            }
            sc.stalled = stalled;
        });
    };
    ok = ok && cycle(false) && spmv(0);
    while (ok && !sc.stalled && sc.iter < sc.max_iter) {
        ok = cycle(true) && spmv(1);
        if (!ok || !sc.do_update) continue;
        // reliable update: x' = x + d into the other buffer, r = b - A x' with the FP64 matrix
        const bool odd = (sc.updates & 1) != 0;
        const double* xc = odd ? o.x2 : o.x;
        double* xn = odd ? o.x : o.x2;
        const float* const Dv = vec[2];
        float* const Rv = vec[4];
        for (int i = r0 + t; i < r1; i += nt) xn[i] = xc[i] + static_cast<double>(Dv[i]);
        ok = barrier();
        if (!ok) break;
        double v = 0.0;
        product<double>(o, L, [&](int j) { return xn[j]; }, [&](int, int row, double ax) {
            const double ri = o.b[row] - ax;
            const float rf = __double2float_rn(ri);
            Rv[row] = rf;
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
        ok = cycle(false) && spmv(2);
    }
    if (!ok) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        loop_timeout(o);
        return;
    }
    // the solution into x: the current buffer, with a correction not yet folded in (rows
    // outside every cell are identity rows, whose x stays)
    {
        const double* xc = (sc.updates & 1) != 0 ? o.x2 : o.x;
        const float* const Dv = vec[2];
        for (int i = r0 + t; i < r1; i += nt) o.x[i] = sc.converged ? xc[i] : xc[i] + static_cast<double>(Dv[i]);
    }
    if (blockIdx.x == 0) store_scalars(o.S, sc);
}

int g_pcg_sms = 0;       // blocks of the grid form, set by pcg_loop_prepare_device
bool g_pcg_cluster = false;
size_t g_pcg_smem = 0;   // largest dynamic shared memory of a block

// Rows of a full level-1 cell, about (21 in the dam breaks at rest).
constexpr int kCellRows = 24;

// Rows up to which the cluster form is used, and those up to which the grid is half the SMs.
// A grid of all SMs has the chip to itself: several handles' solves then take turns, where the
// kernel chain overlapped them.  us a step of one handle and of each of four stepped from four
// threads (dam breaks at r_e = 4 l0, another at 2.1, a tall tank):
//   rows                4,116 (2.1)  5,250      6,925 (tall)  10,920      19,538 (2.1)  63,996 (2.1)
//   cluster             895 / 249    1,068 / 304   1,186 / 345   1,465 / 423   1,870 / 525    -
//   half the SMs        973 / 438    1,076 / 467   1,118 / 516   1,308 / 650   1,500 / 731   2,417 / 1,270
//   all SMs             983 / 836    1,081 / 853   1,112 / 918   1,280 / 1,101 1,477 / 1,316 2,071 / 1,900
//   chain (2.1)       1,789 / 511        -             -         2,167 / 625   2,345 / 759   2,680 / 1,068
// Half the SMs cost one handle 1 to 3 % up to 20,000 rows and 17 % at 63,996.
constexpr int kPcgClusterRows = 5376, kPcgHalfRows = 12288;

// Largest level that every block takes by itself: a level costs 2,300 cycles per 512 cells
// in one block, and two exchanges and its round trips (9,000 cycles) when it is distributed.
// us per solve with 512, 1,024, 2,048 and 4,096 cells: 16,850 rows 1,311, 1,172, 1,174,
// 1,172; hydrostatic 84,450 rows 2,104, 2,105, 1,911, 1,913; 9,403 rows 1,240, 1,074, 1,172,
// 1,172.
constexpr int kPcgBottomCells = 2048;

bool pcg_plan(const MgHierarchy& mg, int blocks, PcgPlan* plan) {
    if (mg.levels <= 0 || mg.n <= 0 || blocks <= 0) return false;
    PcgPlan p{};
    p.blocks = blocks;
    const int each = mg.n / p.blocks + 1;
    p.rows = (each + each / 2 + 64 + 3) & ~3;
    p.tables = 2 * each / kSellRows + 4;
    // the own rows and two columns of cells
    p.window = (2 * each + 2 * mg.lv[1].nz * kCellRows + 64 + 3) & ~3;
    if (p.window > mg.n + 4) p.window = (mg.n + 3) & ~3;
    if (p.window > 65532) p.window = 65532;
    p.cells = (p.window / 4 + 3) & ~3;
    const size_t fixed = part_room(p.tables) + table_room(p.tables) +
                         static_cast<size_t>(kRowBytes) * p.rows + static_cast<size_t>(kWindowBytes) * p.window +
                         static_cast<size_t>(kCellBytes) * p.cells;
    for (p.bottom = mg.bottom; p.bottom <= mg.levels; p.bottom++) {
        int64_t floats = 0;
        for (int l = p.bottom; l <= mg.levels; l++) floats += bottom_level_floats(mg.lv[l], l == mg.levels);
        p.bottom_floats = static_cast<int>(floats);
        p.smem = fixed + sizeof(float) * static_cast<size_t>(floats);
        if (mg.lv[p.bottom].cells <= kPcgBottomCells && p.smem <= g_pcg_smem) break;
    }
    if (p.bottom > mg.levels) return false;
    *plan = p;
    return true;
}

// The form the rows take, where its blocks' shares fit.
bool pcg_choose(const MgHierarchy& mg, PcgPlan* plan, bool* cluster) {
    *cluster = g_pcg_cluster && mg.n <= kPcgClusterRows && pcg_plan(mg, kLoopCluster, plan);
    return *cluster || (mg.n <= kPcgHalfRows && pcg_plan(mg, g_pcg_sms / 2, plan)) || pcg_plan(mg, g_pcg_sms, plan);
}

}  // namespace

cudaError_t pcg_loop_prepare_device() {
    int dev = 0, sms = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    size_t room = static_cast<size_t>(most);
    for (auto k : {k_pcg_loop<false>, k_pcg_loop<true>}) {
        cudaFuncAttributes a{};
        e = cudaFuncGetAttributes(&a, k);
        if (e != cudaSuccess) return e;
        const size_t r = static_cast<size_t>(most) - a.sharedSizeBytes;
        if (r < room) room = r;
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(r));
        if (e != cudaSuccess) return e;
    }
    e = cudaFuncSetAttribute(k_pcg_loop<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    g_pcg_smem = room;
    e = loop_grid_blocks(dev, sms, &g_pcg_sms);
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
    g_pcg_cluster = cudaOccupancyMaxActiveClusters(&n, k_pcg_loop<true>, &cfg) == cudaSuccess && n > 0;
    if (!g_pcg_cluster) cudaGetLastError();
    return cudaSuccess;
}

bool pcg_loop_fits(const MgHierarchy& mg) {
    PcgPlan p;
    bool cluster;
    return mg.cell_w != nullptr && pcg_choose(mg, &p, &cluster);
}

cudaError_t launch_pcg_loop(const CgOperands& o, const MgHierarchy& mg, cudaStream_t s) {
    PcgPlan p;
    bool cluster;
    if (!pcg_choose(mg, &p, &cluster)) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(p.blocks));
    cfg.blockDim = dim3(kLoopThreads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    if (cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kLoopCluster;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = p.blocks > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, cluster ? k_pcg_loop<true> : k_pcg_loop<false>, o, mg, p);
}

}  // namespace mpsgb
