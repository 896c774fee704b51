// cgloop.cuh - the matrix products of the single-launch solver loops (cgloop.cu, pcgloop.cu).
//
// A block owns a range of SELL chunks.  For a product A v they are cut into units of a few
// entries of a chunk's 32 rows (one warp per unit, one lane per row), the unit sums are
// parked in shared memory and the row's thread adds them: with whole chunks per warp, 17
// chunks of 46 entries (84k rows over 152 SMs) would occupy 17 of 32 warps, and a 58-chunk
// system (1,850 rows) would wait for one lane's 46 dependent multiply-adds.  Blocks with
// more chunks than the sums' room take them in tiles.
#pragma once

#include "cg.cuh"
#include "gridloop.cuh"

namespace mpsgb {

namespace {

constexpr int kStep = 8;         // matrix entries a lane loads at once
constexpr int kMaxUnits = 8;     // units of one chunk (longer rows take longer units)
// Units a warp should have: with two, 18 chunks (84k rows over 152 SMs) are 36 units for 16
// warps and the last round is nearly empty.  us per iteration at two, three, four, six:
// CG64 23.4, 21.5, 21.9, 21.9 and MIXED 17.5, 15.9, 16.4, 16.4 at 90,050 rows; MIXED 20.2,
// 19.1, 18.5, 18.3 on a 3D dam break of 210,868 particles.
constexpr int kUnitsPerWarp = 4;

struct __align__(16) ChunkInfo {
    int chunk, off, width, span;  // span: entries of a unit
    int first, units;             // its first unit
    unsigned live;                // rows of the block with entries
    int pad;
};

// Shared memory of a table's chunk.
constexpr int kChunkBytes = static_cast<int>(sizeof(ChunkInfo) + sizeof(int2) * kMaxUnits);

struct LoopView {
    double* part;     // unit sums, `part_units` x 32
    ChunkInfo* info;  // all chunks of the block (whole) or those of a tile
    int2* unit;       // {table index, first entry}, kMaxUnits per chunk
    int c0, nc;  // whole: table entries are the chunks; else chunks c0 .. c0 + nc - 1
    int lo, hi;  // rows of the block (its first and last chunk may hold others' rows)
    int tile;    // chunks per tile
    int active;  // threads that own rows
    int warps;
    int cuts;  // units of a chunk, at most kMaxUnits
    bool whole;
};

// Entries of a unit of a chunk `width` entries wide.  A block with chunks to spare takes
// them in few units (each unit past the first costs the row an addition); one with few
// cuts them so that its warps all have one.
__device__ __forceinline__ int unit_span(const LoopView& L, int width) {
    const int per = (width + L.cuts - 1) / L.cuts;
    return (per + kStep - 1) / kStep * kStep;
}

// Lays the tables of `tables` chunks out at `at`; returns their end.
__device__ __forceinline__ unsigned char* place_tables(LoopView& L, void* at, int tables) {
    L.info = static_cast<ChunkInfo*>(at);
    L.unit = reinterpret_cast<int2*>(L.info + tables);
    return reinterpret_cast<unsigned char*>(L.unit + static_cast<size_t>(tables) * kMaxUnits);
}

// Completes the table entries [0, m) whose chunks are set, and lists their units.
__device__ __forceinline__ void build_tables(const CgOperands& o, const LoopView& L, int m) {
    const int t = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x);
    for (int k = t; k < m; k += nt) {
        const int c = L.info[k].chunk;
        const int w = o.chunk[c] / kSellRows;
        L.info[k].off = o.off[c];
        L.info[k].width = w;
        L.info[k].span = unit_span(L, w);
        L.info[k].units = w > 0 ? (w + L.info[k].span - 1) / L.info[k].span : 0;
    }
    for (int k = t >> 5; k < m; k += nt >> 5) {
        const int row = L.info[k].chunk * kSellRows + (t & 31);
        const unsigned live = __ballot_sync(0xffffffffu, row >= L.lo && row < L.hi && o.len[row] > 0);
        if ((t & 31) == 0) L.info[k].live = live;
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
        for (int u = 0; u < c.units; u++) L.unit[c.first + u] = make_int2(k, u * c.span);
    }
    __syncthreads();
}

// Tiles and cuts of a block with L.nc chunks whose unit sums have room for part_units and
// whose tables hold `tables` chunks.
__device__ __forceinline__ void split_tiles(LoopView& L, int part_units, int tables) {
    const int nc = max(1, L.nc);
    const int cuts = min(kMaxUnits, (kUnitsPerWarp * L.warps + nc - 1) / nc);
    int tiles = (nc * cuts + part_units - 1) / part_units;
    if (!L.whole) tiles = max(tiles, (nc + tables - 1) / tables);
    L.tile = (nc + tiles - 1) / tiles;
    L.cuts = min(min(kMaxUnits, (kUnitsPerWarp * L.warps + L.tile - 1) / L.tile), part_units / L.tile);
    L.active = min(static_cast<int>(blockDim.x), L.nc * 32);
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

// A step of a unit: kStep entries of the lane's row.
template <class T>
struct UnitStep {
    int c[kStep];
    T a[kStep];
    bool live;  // the lane's row is the block's and has entries
    int out;    // the unit, when this is its last step (else -1)
};

// The warp's steps in order.  A chunk's entries past a row's length are {the row itself, 0}
// (pad_row): a step loads and adds all of its entries without looking at the length.  With a
// test of each entry a step took 2,700 cycles of issue, not of memory, at 84k rows.
template <class T>
struct UnitCursor {
    const CgOperands& o;
    const LoopView& L;
    int u, u1, k0, end, row;
    bool live;
    int64_t at;  // the lane's first entry of the chunk

    __device__ __forceinline__ void open() {
        const int2 un = L.unit[u];
        const int lane = threadIdx.x & 31;
        const ChunkInfo& ci = L.info[un.x];
        at = static_cast<int64_t>(ci.off) + lane;
        row = ci.chunk * kSellRows + lane;
        k0 = un.y;
        end = min(ci.width, k0 + ci.span);
        live = (ci.live >> lane & 1u) != 0u;
    }
    __device__ __forceinline__ UnitCursor(const CgOperands& o_, const LoopView& L_, int u_, int u1_)
        : o(o_), L(L_), u(u_), u1(u1_), k0(0), end(0), row(0), live(false), at(0) {
        if (u < u1) open();
    }
    __device__ __forceinline__ bool valid() const { return u < u1; }
    __device__ __forceinline__ void entry(UnitStep<T>& s, int e, int64_t from) {
        if constexpr (sizeof(T) == 8) {
            s.c[e] = ld_once(o.col + from + e * kSellRows);
            s.a[e] = ld_once(o.val + from + e * kSellRows);
        } else {
            const uint2 p = ld_sell_pair(o.cv32 + from + e * kSellRows);
            s.c[e] = static_cast<int>(p.x);
            s.a[e] = __uint_as_float(p.y);
        }
    }
    // Loads the current step and moves on.
    __device__ __forceinline__ void load(UnitStep<T>& s) {
        const int64_t from = at + static_cast<int64_t>(k0) * kSellRows;
        s.live = live;
        s.out = -1;
        if (k0 + kStep <= end) {
#pragma unroll
            for (int e = 0; e < kStep; e++) entry(s, e, from);
        } else {  // the chunk's last entries
#pragma unroll
            for (int e = 0; e < kStep; e++) {
                s.c[e] = row;
                s.a[e] = 0;
                if (k0 + e < end) entry(s, e, from);
            }
        }
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
// trip to L2 per step (0.6 us across the dies), not for two.  Unit u's sums go to place
// u - base.
template <class T, class V>
__device__ __forceinline__ void unit_sums(const CgOperands& o, const LoopView& L, int a, int b, int base, V v) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T* part = reinterpret_cast<T*>(L.part);
    const int u0 = L.info[a].first, u1 = L.info[b - 1].first + L.info[b - 1].units;
    UnitCursor<T> cur(o, L, u0 + warp, u1);
    if (!cur.valid()) return;
    T acc = 0;
    auto add = [&](const UnitStep<T>& s) {
        if (s.live) {
            T xv[kStep];
#pragma unroll
            for (int e = 0; e < kStep; e++) xv[e] = v(s.c[e]);
#pragma unroll
            for (int e = 0; e < kStep; e++) {
                if constexpr (sizeof(T) == 8) acc = fma(s.a[e], xv[e], acc);
                else acc = fmaf(s.a[e], xv[e], acc);
            }
        }
        if (s.out >= 0) {
            part[(s.out - base) * 32 + lane] = acc;
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

// f(local row, row, (A v)_row) for every row of the block, by the row's thread; v(column)
// gathers the vector
template <class T, class V, class F>
__device__ __forceinline__ void product(const CgOperands& o, const LoopView& L, V v, F f) {
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
        const int u0 = L.info[k0 - table0].first;
        unit_sums<T>(o, L, k0 - table0, k1 - table0, u0, v);
        __syncthreads();
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
            if (row >= L.lo && row < L.hi) f(k * kSellRows + lane, row, s);
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
        if (row >= L.lo && row < L.hi) g(k * kSellRows + lane, row);
    }
}

// a wait of loop_reduce ran out: the step reports it
__device__ __forceinline__ void loop_timeout(const CgOperands& o) {
    if (threadIdx.x == 0) {
        if (o.status) atomicOr(&const_cast<DevStatus*>(o.status)->flags, kStatusWaitTimeout);
        o.S->aborted = 1;
    }
}

}  // namespace

}  // namespace mpsgb
