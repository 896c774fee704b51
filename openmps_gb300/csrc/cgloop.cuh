// cgloop.cuh - the matrix products of the single-launch solver loops (cgloop.cu, pcgloop.cu).
//
// A block owns a range of SELL chunks.  A product A v reads them in steps of eight entries of
// a chunk's 32 rows, one lane per row; the block's steps, chunk after chunk, are dealt to its
// warps in equal contiguous shares.  A unit is the part of one chunk in one warp's share: its
// sums are parked in shared memory and the row's thread adds them.  18 chunks of 41 entries
// (84k rows over 152 SMs) are 108 steps, seven for each of 16 warps at most; in units of 16
// entries dealt out whole (MIXED 16.4, CG64 21.9 us an iteration at 90,050 rows) the longest
// warp had ten.  A block with more chunks than its tables hold takes them in tiles; where the
// blocks' shares pass what tables fit, the loops walk whole chunks without (ChunkCursor).
#pragma once

#include <cstddef>

#include "cg.cuh"
#include "gridloop.cuh"

namespace mpsgb {

namespace {

constexpr int kStep = 8;         // matrix entries a lane loads at once

struct __align__(16) ChunkInfo {
    int chunk, off, width, steps;
    int first, units;  // its first unit
    unsigned live;     // rows of the block with entries
    int before;        // steps of the chunks before it
};

struct LoopView {
    double* part;     // unit sums, `parts` x 32
    ChunkInfo* info;  // all chunks of the block (whole) or those of a tile
    int4* unit;       // {table index, first entry, end}
    int2* share;      // per warp: its first unit and end
    int c0, nc;  // whole: table entries are the chunks; else chunks c0 .. c0 + nc - 1
    int lo, hi;  // rows of the block (its first and last chunk may hold others' rows)
    int tile;    // chunks per tile
    int active;  // threads that own rows
    int warps;
    bool whole;
};

// Shared memory of the tables of `tables` chunks: ChunkInfo and units (each chunk's last is
// its own or shared with a warp's end, so there are at most chunks + warps), shares.
__host__ __device__ constexpr size_t table_room(int tables) {
    return sizeof(ChunkInfo) * static_cast<size_t>(tables) +
           sizeof(int4) * static_cast<size_t>(tables + kLoopThreads / 32) + sizeof(int2) * (kLoopThreads / 32);
}
// and of their unit sums
__host__ __device__ constexpr size_t part_room(int tables) {
    return sizeof(double) * 32 * static_cast<size_t>(tables + kLoopThreads / 32);
}

// Lays unit sums and tables of `tables` chunks out at `at`; returns their end.
__device__ __forceinline__ unsigned char* place_tables(LoopView& L, void* at, int tables) {
    L.part = static_cast<double*>(at);
    L.info = reinterpret_cast<ChunkInfo*>(static_cast<unsigned char*>(at) + part_room(tables));
    L.unit = reinterpret_cast<int4*>(L.info + tables);
    L.share = reinterpret_cast<int2*>(L.unit + tables + kLoopThreads / 32);
    return reinterpret_cast<unsigned char*>(L.share + kLoopThreads / 32);
}

// Completes the table entries [0, m) whose chunks are set, and lists their units.
__device__ __forceinline__ void build_tables(const CgOperands& o, const LoopView& L, int m) {
    const int t = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x);
    const long long W = L.warps;
    for (int k = t; k < m; k += nt) {
        const int c = L.info[k].chunk;
        const int w = o.chunk[c] / kSellRows;
        L.info[k].off = o.off[c];
        L.info[k].width = w;
        L.info[k].steps = (w + kStep - 1) / kStep;
    }
    for (int k = t >> 5; k < m; k += nt >> 5) {
        const int row = L.info[k].chunk * kSellRows + (t & 31);
        const unsigned live = __ballot_sync(0xffffffffu, row >= L.lo && row < L.hi && o.len[row] > 0);
        if ((t & 31) == 0) L.info[k].live = live;
    }
    if (t < L.warps) L.share[t] = make_int2(0, 0);
    __shared__ int steps;
    __syncthreads();
    // exclusive prefix sums over the table, by one warp
    auto scan = [&](auto value, auto store) {
        int run = 0;
        for (int b = 0; b < m; b += 32) {
            const int u = b + t < m ? value(L.info[b + t]) : 0;
            int s = u;
            for (int d = 1; d < 32; d <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, s, d);
                if (t >= d) s += x;
            }
            if (b + t < m) store(L.info[b + t], run + s - u);
            run += __shfl_sync(0xffffffffu, s, 31);
        }
        return run;
    };
    if (t < 32) {
        const int T = scan([](const ChunkInfo& c) { return c.steps; }, [](ChunkInfo& c, int x) { c.before = x; });
        if (t == 0) steps = T;
        __syncwarp();
        scan(
            [&](ChunkInfo& c) {
                if (c.steps == 0) return c.units = 0;
                if (T < W) return c.units = c.steps;
                return c.units = static_cast<int>((c.before + c.steps - 1) * W / T - c.before * W / T) + 1;
            },
            [](ChunkInfo& c, int x) { c.first = x; });
    }
    __syncthreads();
    const int T = steps;  // step s is warp floor(s W / T)'s, whose first is start(warp)
    auto start = [&](int v) { return static_cast<int>((static_cast<long long>(v) * T + W - 1) / W); };
    for (int k = t; k < m; k += nt) {
        const ChunkInfo c = L.info[k];
        for (int u = 0; u < c.units; u++) {
            const int v = static_cast<int>((c.before + (T < W ? u : 0)) * W / T) + (T < W ? 0 : u);
            const int a = start(v), b = start(v + 1);
            const int s0 = max(c.before, a), s1 = min(c.before + c.steps, b);
            L.unit[c.first + u] = make_int4(k, (s0 - c.before) * kStep, min(c.width, (s1 - c.before) * kStep), 0);
            if (s0 == a) L.share[v].x = c.first + u;
            if (s1 == b) L.share[v].y = c.first + u + 1;
        }
    }
    __syncthreads();
}

// Tiles of a block with L.nc chunks whose tables hold `tables` chunks.
__device__ __forceinline__ void split_tiles(LoopView& L, int tables) {
    L.tile = L.whole ? max(1, L.nc) : tables;
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
    int out;    // the unit (ChunkCursor: chunk), when this is its last step (else -1)
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
        const int4 un = L.unit[u];
        const int lane = threadIdx.x & 31;
        const ChunkInfo& ci = L.info[un.x];
        at = static_cast<int64_t>(ci.off) + lane;
        row = ci.chunk * kSellRows + lane;
        k0 = un.y;
        end = un.z;
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
    // Loads the current step and moves past it.
    __device__ __forceinline__ void step(UnitStep<T>& s) {
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
    }
    __device__ __forceinline__ void load(UnitStep<T>& s) {
        step(s);
        if (k0 >= end) {
            s.out = u++;
            if (u < u1) open();
        }
    }
};

// The sums of a cursor's steps, T = double (FP64 matrix) or float (FP32 pairs): done(out, the
// lane's sum) at the last step of each unit or chunk.  Two steps in turn, each loaded while
// the other gathers and adds: a warp waits for one round trip to L2 per step (0.6 us across
// the dies), not for two.
template <class T, class Cursor, class V, class D>
__device__ __forceinline__ void walk_steps(Cursor& cur, V v, D done) {
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
            done(s.out, acc);
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

// The unit sums of the tables' chunks.
template <class T, class V>
__device__ __forceinline__ void unit_sums(const CgOperands& o, const LoopView& L, V v) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T* part = reinterpret_cast<T*>(L.part);
    const int2 mine = L.share[warp];
    UnitCursor<T> cur(o, L, mine.x, mine.y);
    walk_steps<T>(cur, v, [&](int unit, T sum) { part[unit * 32 + lane] = sum; });
}

// The steps of a block without tables: its chunks that the loop works on, dealt to the warps
// in turn, with a row's sum in its lane's register to the end.  A warp looks 32 of its chunks
// over at once, and loads the next one's place while the present one is read.
template <class T>
struct ChunkCursor : UnitCursor<T> {
    int k, next;              // the block's chunk, the warp's next one (nc: none)
    int next_off, next_size;
    int group;                // first of the chunks not looked over yet
    unsigned pending;         // chunks of the 32 before them to come

    __device__ __forceinline__ void take() {
        const int lane = threadIdx.x & 31, w = this->L.warps, nc = this->L.nc;
        while (pending == 0u) {
            if (group >= nc) {
                next = nc;
                return;
            }
            const int q = group + lane * w;
            pending = __ballot_sync(0xffffffffu, q < nc && this->o.loop_w[this->L.c0 + q] > 0);
            group += 32 * w;
        }
        next = group - 32 * w + (__ffs(static_cast<int>(pending)) - 1) * w;
        pending &= pending - 1u;
        next_off = this->o.off[this->L.c0 + next];
        next_size = this->o.chunk[this->L.c0 + next];
    }
    __device__ __forceinline__ void open() {
        k = next;
        if (!valid()) return;
        this->row = (this->L.c0 + k) * kSellRows + static_cast<int>(threadIdx.x & 31);
        this->at = static_cast<int64_t>(next_off) + (threadIdx.x & 31);
        this->k0 = 0;
        this->end = next_size / kSellRows;
        this->live = this->row >= this->L.lo && this->row < this->L.hi;
        take();
    }
    __device__ __forceinline__ ChunkCursor(const CgOperands& o_, const LoopView& L_)
        : UnitCursor<T>(o_, L_, 0, 0), next_off(0), next_size(0), group(static_cast<int>(threadIdx.x >> 5)), pending(0u) {
        take();
        open();
    }
    __device__ __forceinline__ bool valid() const { return k < this->L.nc; }
    __device__ __forceinline__ void load(UnitStep<T>& s) {
        this->step(s);
        if (this->k0 >= this->end) {
            s.out = k;
            open();
        }
    }
};

// f(local row, row, (A v)_row) for every row of the block, by the row's thread; v(column)
// gathers the vector (kDirect: a block without tables)
template <class T, bool kDirect = false, class V, class F>
__device__ __forceinline__ void product(const CgOperands& o, const LoopView& L, V v, F f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if constexpr (kDirect) {
        ChunkCursor<T> cur(o, L);
        walk_steps<T>(cur, v, [&](int k, T sum) {
            const int row = (L.c0 + k) * kSellRows + lane;
            if (row >= L.lo && row < L.hi) f(k * kSellRows + lane, row, sum);
        });
        return;
    }
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
        unit_sums<T>(o, L, v);
        __syncthreads();
        const int skip = k0 % L.warps;  // chunk k belongs to warp k % warps
        for (int k = k0 - skip + warp + (warp < skip ? L.warps : 0); k < k1; k += L.warps) {
            const ChunkInfo c = L.info[k - table0];
            const T* p = part + c.first * 32 + lane;
            T s = c.units > 0 ? p[0] : T(0);  // in ascending columns, as the units are
            for (int u = 1; u < c.units; u++) s += p[u * 32];
            const int row = c.chunk * kSellRows + lane;
            if (row >= L.lo && row < L.hi) f(k * kSellRows + lane, row, s);
        }
        if (k1 < L.nc) __syncthreads();  // the next tile overwrites the sums
    }
}

// g(local row, row) for every row of the block, by the thread product() gives it to
template <bool kDirect = false, class G>
__device__ __forceinline__ void own_rows(const CgOperands& o, const LoopView& L, G g) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if constexpr (kDirect) {
        for (int k0 = warp; k0 < L.nc; k0 += 32 * L.warps) {
            const int q = k0 + lane * L.warps;
            unsigned in = __ballot_sync(0xffffffffu, q < L.nc && o.loop_w[L.c0 + q] > 0);
            for (; in != 0u; in &= in - 1u) {
                const int k = k0 + (__ffs(static_cast<int>(in)) - 1) * L.warps;
                const int row = (L.c0 + k) * kSellRows + lane;
                if (row >= L.lo && row < L.hi) g(k * kSellRows + lane, row);
            }
        }
        return;
    }
    for (int k = warp; k < L.nc; k += L.warps) {
        const int row = chunk_of(L, k) * kSellRows + lane;
        if (row >= L.lo && row < L.hi) g(k * kSellRows + lane, row);
    }
}

// The bound of the loop's waits, by thread 0 before the first exchange.
__device__ __forceinline__ long long loop_wait_clocks(const CgOperands& o) {
    return o.limits ? o.limits->barrier_clocks : kDefaultBarrierClocks;
}

// A wait of loop_reduce ran out: the call reports it, and what the loop leaves counts as not
// converged (the FP64 CG finishes a mixed-precision solve).
__device__ __forceinline__ void loop_timeout(const CgOperands& o) {
    if (threadIdx.x == 0) {
        if (o.status) atomicOr(&const_cast<DevStatus*>(o.status)->flags, kStatusWaitTimeout);
        o.S->timed_out = 1;
    }
}

// The loop's scalars into the solve's, but for timed_out: any block may have set that.
__device__ __forceinline__ void store_scalars(CgScalars* S, const CgScalars& sc) {
    constexpr int kWords = static_cast<int>(offsetof(CgScalars, timed_out) / sizeof(uint32_t));
    const uint32_t* from = reinterpret_cast<const uint32_t*>(&sc);
    uint32_t* to = reinterpret_cast<uint32_t*>(S);
    for (int k = static_cast<int>(threadIdx.x); k < kWords; k += static_cast<int>(blockDim.x)) to[k] = from[k];
}

}  // namespace

}  // namespace mpsgb
