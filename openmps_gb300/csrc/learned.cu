// learned.cu - learned warm start / preconditioner scale: features, tensor-core
// inference (tcgen05, BF16 x BF16 -> FP32 in TMEM), warm start, training samples, and
// the FP32 forward/backward training kernels with Adam.
//
// Tensor-core inference (k_mlp_tc): one CTA of 128 threads per tile of 128 particles
// (persistent over tiles).  The four weight matrices live in shared memory in the
// canonical K-major no-swizzle layout of tcgen05 (8-row x 16-byte core matrices; LBO =
// byte distance of K-adjacent core matrices, SBO = distance of M/N-adjacent 8-row
// groups).  Per layer one thread issues the K/16 MMAs (M = 128, N = 64, or 16 for the
// padded output layer) into 64 TMEM columns and commits them to an mbarrier; every
// thread then reads its own row of the accumulator (tcgen05.ld 32x32b: warp w owns TMEM
// lanes 32w..32w+31), adds the bias, applies GELU, rounds to BF16 and writes the row
// back as the next layer's A operand.  Waits are bounded (WaitLimits::mma_clocks): a
// wait that gives up waits once more, within kMmaDrainClocks, for the MMAs it issued to
// complete, sets an error word, frees its TMEM and returns; the solve then uses no
// network output.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "learned.cuh"

namespace mpsgb {

namespace {

constexpr int kTile = 128;
constexpr int kTmemCols = 64;

// tensor-core weight image (bytes)
constexpr int kImgW1 = 0;                       // N 64 x K 16
constexpr int kImgW2 = kImgW1 + 64 * 16 * 2;    // N 64 x K 64
constexpr int kImgW3 = kImgW2 + 64 * 64 * 2;
constexpr int kImgW4 = kImgW3 + 64 * 64 * 2;    // N 16 (2 used) x K 64
constexpr int kImgBias = kImgW4 + 16 * 64 * 2;  // b1[64] b2[64] b3[64] b4[16] FP32
constexpr int kImgNorm = kImgBias + (64 * 3 + 16) * 4;  // mean[16] std[16]
constexpr int kImgBytes = ((kImgNorm + 32 * 4) + 15) / 16 * 16;

// shared-memory map of the inference kernel (the tail is slack: every address any
// descriptor can form stays inside the allocation)
constexpr int kSmA0 = 0;                        // 128 x 16 BF16
constexpr int kSmA = kSmA0 + kTile * 16 * 2;    // 128 x 64 BF16
constexpr int kSmImg = kSmA + kTile * 64 * 2;
constexpr int kSmBar = (kSmImg + kImgBytes + 15) / 16 * 16;
constexpr int kSmBytes = 48 * 1024;  // four CTAs per SM: the whole grid is resident

// byte offset of element (r, k) of a K-major operand with `rows` rows
__host__ __device__ constexpr int core_offset(int r, int k, int rows) {
    return ((k >> 3) * (rows >> 3) + (r >> 3)) * 128 + (r & 7) * 16 + (k & 7) * 2;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// tcgen05 shared-memory matrix descriptor, no swizzle
__device__ __forceinline__ uint64_t sm_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr >> 4) & 0x3FFFu);
    d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
    d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
    d |= static_cast<uint64_t>(1) << 46;  // descriptor version of tcgen05
    return d;                             // base offset 0, no swizzle
}

// instruction descriptor of kind::f16: BF16 A and B (K-major), FP32 D, M = 128
__host__ __device__ constexpr uint32_t idesc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(kTile >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ bool bar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16 consecutive FP32 accumulator columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const uint32_t lo = __bfloat16_as_ushort(__float2bfloat16_rn(a));
    const uint32_t hi = __bfloat16_as_ushort(__float2bfloat16_rn(b));
    return lo | (hi << 16);
}

// writes 8 consecutive K values of row r of a K-major operand (one 16-byte store)
__device__ __forceinline__ void store_row8(unsigned char* base, int rows, int r, int kc, const float* v) {
    uint4 q;
    q.x = pack_bf16(v[0], v[1]);
    q.y = pack_bf16(v[2], v[3]);
    q.z = pack_bf16(v[4], v[5]);
    q.w = pack_bf16(v[6], v[7]);
    *reinterpret_cast<uint4*>(base + core_offset(r, kc * 8, rows)) = q;
}

// ------------------------------------------------------------ inference (tcgen05)
__global__ void __launch_bounds__(kTile) k_mlp_tc(const unsigned char* __restrict__ image,
                                                  const float* __restrict__ feat, int n,
                                                  const double* sigma, float* __restrict__ out,
                                                  int32_t* error, const WaitLimits* limits) {
    extern __shared__ __align__(1024) unsigned char sm[];
    const int t = threadIdx.x, warp = t >> 5;
    unsigned char* A0 = sm + kSmA0;
    unsigned char* A = sm + kSmA;
    unsigned char* img = sm + kSmImg;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kSmBar);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + kSmBar + 8);

    for (int k = t; k < kImgBytes / 16; k += kTile)
        reinterpret_cast<uint4*>(img)[k] = reinterpret_cast<const uint4*>(image)[k];
    if (t == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    const float* bias = reinterpret_cast<const float*>(img + kImgBias);
    const float* mu = reinterpret_cast<const float*>(img + kImgNorm);
    const float* sd = mu + 16;
    const float inv_sigma = sigma ? static_cast<float>(1.0 / sigma[0]) : 1.0f;
    const long long wait_clocks = limits ? limits->mma_clocks : kDefaultMmaClocks;
    const uint32_t aA0 = smem_u32(A0), aA = smem_u32(A), aImg = smem_u32(img);
    uint32_t phase = 0;
    bool bad = false;
    const int ntiles = (n + kTile - 1) / kTile;

    // features of the CTA's next tile are loaded while the current tile runs its layers
    float4 nxt[4];
    auto load_tile = [&](int tile) {
        const int r = tile * kTile + t;
        if (tile < ntiles && r < n) {
            const float4* f4 = reinterpret_cast<const float4*>(feat + static_cast<int64_t>(r) * kMlpIn);
#pragma unroll
            for (int q = 0; q < 4; q++) nxt[q] = __ldg(f4 + q);
        }
    };
    load_tile(blockIdx.x);
    for (int tile = blockIdx.x; tile < ntiles && !bad; tile += gridDim.x) {
        const int row = tile * kTile + t;
        float x[16];
        if (row < n) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                x[4 * q] = nxt[q].x;
                x[4 * q + 1] = nxt[q].y;
                x[4 * q + 2] = nxt[q].z;
                x[4 * q + 3] = nxt[q].w;
            }
            x[8] *= inv_sigma;
            x[9] *= inv_sigma;
            x[10] *= inv_sigma;
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = (x[k] - mu[k]) / sd[k];
        } else {
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = 0.0f;
        }
        load_tile(tile + gridDim.x);
        store_row8(A0, kTile, t, 0, x);
        store_row8(A0, kTile, t, 1, x + 8);
        proxy_fence();
        tc_fence_before();
        __syncthreads();

        for (int layer = 0; layer < 4 && !bad; layer++) {
            if (t == 0) {
                tc_fence_after();
                if (layer == 0) {
                    mma_bf16(tmem, sm_desc(aA0, (kTile / 8) * 128, 128),
                             sm_desc(aImg + kImgW1, 64 / 8 * 128, 128), idesc_bf16(64), 0);
                } else {
                    const int nb = layer == 3 ? 16 : 64;
                    const uint32_t wb = aImg + (layer == 1 ? kImgW2 : layer == 2 ? kImgW3 : kImgW4);
                    const uint32_t lbo_a = (kTile / 8) * 128, lbo_b = (nb / 8) * 128;
#pragma unroll
                    for (int s = 0; s < 4; s++)
                        mma_bf16(tmem, sm_desc(aA + 2 * s * lbo_a, lbo_a, 128),
                                 sm_desc(wb + 2 * s * lbo_b, lbo_b, 128), idesc_bf16(nb), s > 0 ? 1u : 0u);
                }
                mma_commit(bar);
            }
            // the bound is checked before each poll, so a bound of 0 gives up at once
            const long long t0 = clock64();
            for (;;) {
                if (clock64() - t0 >= wait_clocks) {
                    bad = true;
                    break;
                }
                if (bar_try_wait(bar, phase)) break;
            }
            if (bad) {
                // the layer's MMAs may still be writing TMEM: wait for their commit
                // (bounded) before the CTA frees TMEM below
                const long long t1 = clock64();
                while (!bar_try_wait(bar, phase) && clock64() - t1 < kMmaDrainClocks) {
                }
            }
            phase ^= 1u;
            tc_fence_after();
            if (!bad) {
                if (layer < 3) {
                    const float* b = bias + 64 * layer;
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        float v[16];
                        tmem_ld16(lane_addr + 16 * q, v);
#pragma unroll
                        for (int k = 0; k < 16; k++) v[k] = gelu(v[k] + b[16 * q + k]);
                        store_row8(A, kTile, t, 2 * q, v);
                        store_row8(A, kTile, t, 2 * q + 1, v + 8);
                    }
                    proxy_fence();
                } else {
                    float v[16];
                    tmem_ld16(lane_addr, v);
                    if (row < n) {
                        out[2 * static_cast<int64_t>(row)] = v[0] + bias[192];
                        out[2 * static_cast<int64_t>(row) + 1] = v[1] + bias[193];
                    }
                }
            }
            tc_fence_before();
            bad = __syncthreads_or(bad) != 0;
        }
    }
    if (bad && t == 0) atomicExch(error, 1);
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols)
                     : "memory");
}

// ------------------------------------------------------------------ features
// Nothing to learn from when the step failed or the initial guess already solves it.
__device__ __forceinline__ bool lrn_skip(const CgScalars* S) { return S->aborted != 0 || S->converged != 0; }

// Per particle: density deviation, source term, free-surface deficiency, wall flag
// (neighbour-averaged below), the Jacobi term g = omega r0 / a_ii and the scaled p.
__global__ void __launch_bounds__(kBlock) k_lrn_q(LearnedOps L, CgOperands o, const float* dinv0,
                                                  const StepScalars* step, const CgScalars* S,
                                                  float4* q4, float2* q2) {
    // each solve starts with a clear tensor-core error word (read by the host after it)
    if (blockIdx.x == 0 && threadIdx.x == 0) *L.error = 0;
    if (lrn_skip(S)) return;
    const double dt = step->dt;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L.n; i += gridDim.x * blockDim.x) {
        const int q = L.particle_of ? L.particle_of[i] : i;  // row i holds particle q
        const double dev = (L.nd[q] - L.n0) / L.n0;
        double surf;
        if (L.flags & MPS_FLAG_SPP) {
            surf = (L.n0 - L.n_wo_spp[q]) / L.n0;
        } else {
            surf = (L.n0 - L.nd[q]) / L.n0;
        }
        surf = surf > 0.0 ? surf : 0.0;
        const float src = static_cast<float>(o.b[i] * dt * dt / L.rho);
        const float wall = L.type[q] == MPS_TYPE_WALL ? 1.0f : 0.0f;
        q4[i] = make_float4(static_cast<float>(dev), src, static_cast<float>(surf), wall);
        const float g = dinv0[i] * o.r32[i];
        q2[i] = make_float2(g, static_cast<float>(L.p[q] * dt * dt / L.rho_l02));
    }
}

__device__ double block_sum_d(double v, double* ws) {
    ws[threadIdx.x] = v;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (static_cast<int>(threadIdx.x) < s) ws[threadIdx.x] += ws[threadIdx.x + s];
        __syncthreads();
    }
    const double r = ws[0];
    __syncthreads();
    return r;
}

// Features (one warp per SELL chunk, lane per row; neighbour averages weighted by the
// FP32 PPE coefficients a_ij, j != i), the first preconditioned step c = alpha0 u0, FP64
// copy of x0, and sigma = RMS of g over active rows (last block).
__global__ void __launch_bounds__(kBlock) k_lrn_features(LearnedOps L, CgOperands o, const float* dinv0,
                                                         const StepScalars* step, const CgScalars* S,
                                                         const float4* q4, const float2* q2, float len_ref) {
    __shared__ double ws[kBlock];
    __shared__ bool last;
    if (lrn_skip(S)) return;
    const int lane = threadIdx.x & 31;
    const int warp = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int nwarps = static_cast<int>((gridDim.x * blockDim.x) >> 5);
    const double dt = step->dt;
    const float alpha0 = static_cast<float>(S->alpha);
    double g2 = 0.0, cnt = 0.0;
    for (int c = warp; c < o.nchunks; c += nwarps) {
        const int i = kSellRows * c + lane;
        if (i >= o.n) continue;
        const float d0 = dinv0[i];
        const bool active = d0 != 0.0f;
        L.active[i] = active ? 1 : 0;
        L.x0d[i] = o.x[i];
        float f[16];
#pragma unroll
        for (int k = 0; k < 16; k++) f[k] = 0.0f;
        float cc = 0.0f;
        if (active) {
            const int len = o.len[i];
            int64_t at = sell_index(o.off[c], lane, 0);
            float wsum = 0.0f, s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f, s4 = 0.0f, s5 = 0.0f;
            for (int k = 0; k < len; k++, at += kSellRows) {
                const uint2 e = o.cv32[at];
                const int j = static_cast<int>(e.x);
                if (j == i) continue;
                const float w = __uint_as_float(e.y);
                const float4 a = q4[j];
                const float2 b = q2[j];
                wsum += w;
                s0 += w * a.x;
                s1 += w * a.y;
                s2 += w * a.z;
                s3 += w * a.w;
                s4 += w * b.x;
                s5 += w * b.y;
            }
            const float inv = wsum > 0.0f ? 1.0f / wsum : 0.0f;
            const float4 a = q4[i];
            const float2 b = q2[i];
            cc = alpha0 * o.u32[i];
            f[0] = a.x;
            f[1] = s0 * inv;
            f[2] = a.y;
            f[3] = s1 * inv;
            f[4] = a.z;
            f[5] = s2 * inv;
            f[6] = a.w;
            f[7] = s3 * inv;
            f[8] = b.x;
            f[9] = s4 * inv;
            f[10] = cc;
            f[11] = static_cast<float>((kMgOmegaFine / d0) / L.a_ref) - 1.0f;
            f[12] = static_cast<float>(len) / len_ref - 1.0f;
            f[13] = b.y;
            f[14] = s5 * inv - b.y;
            f[15] = static_cast<float>(L.ecs[L.particle_of ? L.particle_of[i] : i] * dt);
            g2 += static_cast<double>(b.x) * b.x;
            cnt += 1.0;
        }
        float4* dst = reinterpret_cast<float4*>(L.feat + static_cast<int64_t>(i) * kMlpIn);
#pragma unroll
        for (int q = 0; q < 4; q++) dst[q] = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
        L.coarse[i] = cc;
    }
    const double sg = block_sum_d(g2, ws);
    const double sc = block_sum_d(cnt, ws);
    if (threadIdx.x == 0) {
        L.partials[2 * blockIdx.x] = sg;
        L.partials[2 * blockIdx.x + 1] = sc;
        __threadfence();
        last = atomicAdd(L.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    double a = 0.0, b = 0.0;
    for (int k = threadIdx.x; k < static_cast<int>(gridDim.x); k += blockDim.x) {
        a += __ldcg(L.partials + 2 * k);
        b += __ldcg(L.partials + 2 * k + 1);
    }
    a = block_sum_d(a, ws);
    b = block_sum_d(b, ws);
    if (threadIdx.x == 0) {
        *L.counter = 0;
        const double s = b > 0.0 ? sqrt(a / b) : 0.0;
        L.sigma[0] = s > 0.0 ? s : 1.0;
    }
}

// x += c + sigma out0 on active rows; scale = 1 + 0.25 tanh(out1) (1 without a usable output).
__global__ void __launch_bounds__(kBlock) k_lrn_apply(LearnedOps L, CgOperands o, const CgScalars* S) {
    if (lrn_skip(S)) return;
    const bool ok = *L.error == 0;
    const double sg = L.sigma[0];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L.n; i += gridDim.x * blockDim.x) {
        float s = 1.0f;
        if (ok && L.active[i]) {
            const float o0 = L.out[2 * static_cast<int64_t>(i)], o1 = L.out[2 * static_cast<int64_t>(i) + 1];
            if (isfinite(o0) && isfinite(o1)) {
                o.x[i] += static_cast<double>(L.coarse[i]) + sg * static_cast<double>(o0);
                s = 1.0f + kMlpScaleRange * tanhf(o1);
            }
        }
        L.scale[i] = s;
    }
}

// Training sample of each row after the solve: features (residual features in units of
// sigma), y = (x* - x0 - c) / sigma, g / sigma.
__global__ void __launch_bounds__(kBlock) k_lrn_targets(LearnedOps L, CgOperands o, const CgScalars* S) {
    if (lrn_skip(S)) {
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L.n; i += gridDim.x * blockDim.x)
            L.active[i] = 0;
        return;
    }
    const double sg = L.sigma[0];
    const float inv = static_cast<float>(1.0 / sg);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L.n; i += gridDim.x * blockDim.x) {
        float* dst = L.sample + static_cast<int64_t>(i) * kMlpSampleFloats;
        const float* f = L.feat + static_cast<int64_t>(i) * kMlpIn;
        for (int k = 0; k < kMlpIn; k++) dst[k] = (k >= 8 && k <= 10) ? f[k] * inv : f[k];
        dst[16] = L.active[i] ? static_cast<float>((o.x[i] - L.x0d[i] - static_cast<double>(L.coarse[i])) / sg) : 0.0f;
        dst[17] = f[8] * inv;
    }
}

// ------------------------------------------------------------------ training
// Forward, loss and gradient of a minibatch in FP32.  What bounds it is the chain of seven
// small matrix products per tile of samples (64 x 64 x 64) and their shared-memory reads
// (a 16-byte read takes the shared-memory pipe at least two cycles, broadcast or not).
// So a thread owns a register tile of each product, 2 samples x 4 units of a layer and 2 x 4
// entries of a weight gradient, and a tile of 64 samples is split over a cluster of two
// blocks: each runs forward and backward for 32 samples and writes its activations and
// deltas into both blocks' shared memory, then sums half of the gradient's entries over all
// 64 (so a minibatch of 4,096 fills 128 SMs with the sums over runs of 64 samples that one
// block per 64 made).  GELU and its derivative come from one erf, evaluated in the forward
// pass.  The weights arrive in 16-byte loads issued together, and the first samples before
// the wait for the kernel that writes the weights.  GB300, 4,096 samples: 53.6 -> 18.8 us
// (before: 64 blocks of 64 samples, one output per thread and step, the gradient accumulated
// in shared memory; one unit a thread over eight samples measured 22.4, 4 x 4 tiles on 128
// threads 32.2).  Every sum keeps its order, so the weights are the same bit for bit.
constexpr int kTrainThreads = 256;
constexpr int kTrainS = 32;         // samples of a block
constexpr int kTileS = 64;          // samples of a cluster of two
constexpr int kTrainClusters = 76;  // a block per SM
constexpr int kTrainParts = 148;    // partial gradients of a large batch
// floats of a 64-unit and a 16-feature row in shared memory: 16-byte aligned, rows shifted by
// four banks
constexpr int kPitch = 68, kPitchX = 20;
// shared-memory floats of the training kernel
constexpr int kTrWt1 = 0;                          // [16][kPitch] transposed (forward)
constexpr int kTrWt2 = kTrWt1 + 16 * kPitch;       // [64][kPitch] transposed (forward)
constexpr int kTrW2 = kTrWt2 + 64 * kPitch;        // [64][kPitch] (backward)
constexpr int kTrWt3 = kTrW2 + 64 * kPitch;
constexpr int kTrW3 = kTrWt3 + 64 * kPitch;
constexpr int kTrW4 = kTrW3 + 64 * kPitch;         // [2][64]
constexpr int kTrB = kTrW4 + 128;                  // b1[64] b2[64] b3[64] b4[2]
constexpr int kTrX = kTrB + 196;                   // [64][kPitchX]
constexpr int kTrA1 = kTrX + kTileS * kPitchX;     // activations [64][kPitch] x 3
constexpr int kTrA2 = kTrA1 + kTileS * kPitch;
constexpr int kTrA3 = kTrA2 + kTileS * kPitch;
constexpr int kTrD1 = kTrA3 + kTileS * kPitch;     // gelu'(z) (own samples), then delta [64][kPitch] x 3
constexpr int kTrD2 = kTrD1 + kTileS * kPitch;
constexpr int kTrD3 = kTrD2 + kTileS * kPitch;
constexpr int kTrO = kTrD3 + kTileS * kPitch;      // [64][2] outputs (own samples), then their deltas
constexpr int kTrY = kTrO + kTileS * 2;            // [32][2]: y, g
constexpr int kTrFloats = kTrY + kTrainS * 2;
constexpr size_t kTrBytes = kTrFloats * sizeof(float);
static_assert(kTrWt2 % 4 == 0 && kTrB % 4 == 0 && kTrX % 4 == 0 && kTrA1 % 4 == 0, "16-byte rows");

// gradient offsets (relative to blob W1)
constexpr int gW1 = 0, gB1 = gW1 + 1024, gW2 = gB1 + 64, gB2 = gW2 + 4096, gW3 = gB2 + 64,
              gB3 = gW3 + 4096, gW4 = gB3 + 64, gB4 = gW4 + 128;

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

// Shared memory of the block and, at the same offsets, of its peer in the cluster.
struct PairMem {
    float* own;
    uint32_t peer;  // shared::cluster address
    __device__ __forceinline__ void put(int at, float v) const {
        own[at] = v;
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(peer + 4u * at), "f"(v) : "memory");
    }
    __device__ __forceinline__ void put4(int at, float a, float b, float c, float d) const {
        st4(own + at, make_float4(a, b, c, d));
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(peer + 4u * at), "f"(a), "f"(b), "f"(c),
                     "f"(d)
                     : "memory");
    }
};

__device__ __forceinline__ void pair_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// acc[i][j] += sum_k In[s0 + i][k] Wk[k][j0 + j] for the thread's 2 samples and 4 units
template <int K, int PITCH_IN>
__device__ __forceinline__ void tile_product(const float* In, const float* Wk, int s0, int j0, float (&acc)[2][4]) {
#pragma unroll 4
    for (int k = 0; k < K; k += 4) {
        float4 a[2], w[4];
#pragma unroll
        for (int i = 0; i < 2; i++) a[i] = ld4(In + (s0 + i) * PITCH_IN + k);
#pragma unroll
        for (int q = 0; q < 4; q++) w[q] = ld4(Wk + (k + q) * kPitch + j0);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float av[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
#pragma unroll
            for (int q = 0; q < 4; q++) {
                acc[i][0] = fmaf(w[q].x, av[q], acc[i][0]);
                acc[i][1] = fmaf(w[q].y, av[q], acc[i][1]);
                acc[i][2] = fmaf(w[q].z, av[q], acc[i][2]);
                acc[i][3] = fmaf(w[q].w, av[q], acc[i][3]);
            }
        }
    }
}

// A = gelu(In Wk + b) for both blocks, D = gelu'(In Wk + b) for this one (samples row0 ..)
template <int K, int PITCH_IN>
__device__ __forceinline__ void dense_fwd(const PairMem& M, int row0, int in, int wk, int b, int A, int D) {
    const int j0 = 4 * (threadIdx.x & 15), s0 = row0 + 2 * (threadIdx.x >> 4);
    const float4 b4 = ld4(M.own + b + j0);
    float acc[2][4] = {{b4.x, b4.y, b4.z, b4.w}, {b4.x, b4.y, b4.z, b4.w}};
    tile_product<K, PITCH_IN>(M.own + in, M.own + wk, s0, j0, acc);
#pragma unroll
    for (int i = 0; i < 2; i++) {
        float a[4], d[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float z = acc[i][j];
            const float e1 = 1.0f + erff(z * 0.70710678118654752f);
            a[j] = 0.5f * z * e1;
            d[j] = 0.5f * e1 + z * 0.39894228040143268f * expf(-0.5f * z * z);
        }
        M.put4(A + (s0 + i) * kPitch + j0, a[0], a[1], a[2], a[3]);
        st4(M.own + D + (s0 + i) * kPitch + j0, make_float4(d[0], d[1], d[2], d[3]));
    }
}

// delta of the layer below for both blocks, in place of its gelu': D[s][k] *= sum_j Delta[s][j] W[j][k]
__device__ __forceinline__ void dense_back(const PairMem& M, int row0, int Delta, int W, int D) {
    const int k0 = 4 * (threadIdx.x & 15), s0 = row0 + 2 * (threadIdx.x >> 4);
    float acc[2][4] = {};
    tile_product<64, kPitch>(M.own + Delta, M.own + W, s0, k0, acc);
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int at = D + (s0 + i) * kPitch + k0;
        const float4 g = ld4(M.own + at);
        M.put4(at, acc[i][0] * g.x, acc[i][1] * g.y, acc[i][2] * g.z, acc[i][3] * g.w);
    }
}

// g[i][k] += sum_s Delta[s][j0 + i] In[s][k0 + k] over the tile, for the thread's 2 x 4 entries
__device__ __forceinline__ void dense_wgrad(const float* Delta, const float* In, int j0, int k0, float (&g)[2][4]) {
    float t[2][4] = {};
#pragma unroll 8
    for (int s = 0; s < kTileS; s++) {
        const float2 d2 = *reinterpret_cast<const float2*>(Delta + s * kPitch + j0);
        const float4 x = ld4(In + s * kPitch + k0);
        const float d[2] = {d2.x, d2.y};
#pragma unroll
        for (int i = 0; i < 2; i++) {
            t[i][0] = fmaf(d[i], x.x, t[i][0]);
            t[i][1] = fmaf(d[i], x.y, t[i][1]);
            t[i][2] = fmaf(d[i], x.z, t[i][2]);
            t[i][3] = fmaf(d[i], x.w, t[i][3]);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int k = 0; k < 4; k++) g[i][k] += t[i][k];
}

// Losses of `n` samples (rows order[0 .. n - 1] of `samples`, or its first n rows without an
// order) and the gradient of their mean: `parts` partial gradients, part p of the tiles p,
// p + parts, .. in FP32 (kTrainParts parts whatever the grid: fewer make longer FP32 sums).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kTrainThreads)
    k_mlp_grad(const float* __restrict__ w, const float* __restrict__ samples, const int64_t* __restrict__ order,
               int64_t n, int parts, float* partials, float* losses) {
    extern __shared__ __align__(16) float sh[];
    const int t = threadIdx.x, rank = static_cast<int>(blockIdx.x & 1u), row0 = kTrainS * rank;
    PairMem M{sh, smem_u32(sh)};
    asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(M.peer) : "r"(rank ^ 1));
    const int clusters = static_cast<int>(gridDim.x >> 1);
    const int64_t stride = static_cast<int64_t>(parts) * kTileS;
    const int fk = t & 15;  // the feature this thread loads
    // features of this block's samples (t >> 4) and (t >> 4) + 16, y or g of threads fk < 2
    float feat[2], target[2];
    auto fetch = [&](int64_t first) {
        int64_t row[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int64_t at = first + row0 + (t >> 4) + 16 * q;
            row[q] = at < n ? (order ? order[at] : at) : -1;
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            feat[q] = row[q] >= 0 ? samples[row[q] * kMlpSampleFloats + fk] : 0.0f;
            target[q] = row[q] >= 0 && fk < 2 ? samples[row[q] * kMlpSampleFloats + 16 + fk] : 0.0f;
        }
    };
    int part = static_cast<int>(blockIdx.x >> 1);
    int64_t tile = static_cast<int64_t>(part) * kTileS;
    fetch(tile);
    pdl_begin();  // the weights come from the update just before
    {
        float4 w2[4], w3[4];
        const float4 w1 = ld4(w + kMlpOffW1 + 4 * t);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            w2[q] = ld4(w + kMlpOffW2 + 4 * (t + kTrainThreads * q));
            w3[q] = ld4(w + kMlpOffW3 + 4 * (t + kTrainThreads * q));
        }
        const float bias = t < 192 ? w[t < 64 ? kMlpOffB1 + t : t < 128 ? kMlpOffB2 + t - 64 : kMlpOffB3 + t - 128] : 0.0f;
        const float out = t < 128 ? w[kMlpOffW4 + t] : t < 130 ? w[kMlpOffB4 + t - 128] : 0.0f;
        {
            const int j = t >> 2, k = 4 * (t & 3);
            const float v[4] = {w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int c = 0; c < 4; c++) sh[kTrWt1 + (k + c) * kPitch + j] = v[c];
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int e = t + kTrainThreads * q, j = e >> 4, k = 4 * (e & 15);
            st4(sh + kTrW2 + j * kPitch + k, w2[q]);
            st4(sh + kTrW3 + j * kPitch + k, w3[q]);
            const float v2[4] = {w2[q].x, w2[q].y, w2[q].z, w2[q].w}, v3[4] = {w3[q].x, w3[q].y, w3[q].z, w3[q].w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                sh[kTrWt2 + (k + c) * kPitch + j] = v2[c];
                sh[kTrWt3 + (k + c) * kPitch + j] = v3[c];
            }
        }
        if (t < 192) sh[kTrB + t] = bias;
        if (t < 128) sh[kTrW4 + t] = out;
        else if (t < 130) sh[kTrB + 64 + t] = out;  // b4 after b1, b2, b3
    }
    const float mu = w[kMlpOffMu + fk], sd = w[kMlpOffSd + fk];
    // this block's half of the gradient: units [32 rank, 32 rank + 32) of W1, W2, W3 and the
    // biases, output `rank` of W4
    const int gj = row0 + 2 * (t >> 4), gk = 4 * (t & 15);
    float g2[2][4] = {}, g3[2][4] = {}, g1[2] = {};
    float gb = 0.0f, g4 = 0.0f, gb4 = 0.0f;
    const float inv_total = 1.0f / static_cast<float>(n);
    while (tile < n) {
        int64_t next = tile + stride;  // the part's next tile, or the first of the cluster's next part
        const bool last = next >= n;
        if (last) next = part + clusters < parts ? static_cast<int64_t>(part + clusters) * kTileS : n;
        pair_barrier();  // the peer has started, and is done with the tile before
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int s = (t >> 4) + 16 * q;
            M.put(kTrX + (row0 + s) * kPitchX + fk, tile + row0 + s < n ? (feat[q] - mu) / sd : 0.0f);
            if (fk < 2) sh[kTrY + 2 * s + fk] = target[q];
        }
        __syncthreads();
        dense_fwd<16, kPitchX>(M, row0, kTrX, kTrWt1, kTrB, kTrA1, kTrD1);
        if (next < n) fetch(next);
        __syncthreads();
        dense_fwd<64, kPitch>(M, row0, kTrA1, kTrWt2, kTrB + 64, kTrA2, kTrD2);
        __syncthreads();
        dense_fwd<64, kPitch>(M, row0, kTrA2, kTrWt3, kTrB + 128, kTrA3, kTrD3);
        __syncthreads();
        if (t < 2 * kTrainS) {
            const int s = row0 + (t >> 1), o = t & 1;
            float acc = sh[kTrB + 192 + o];
#pragma unroll
            for (int k = 0; k < 64; k += 4) {
                const float4 a = ld4(sh + kTrA3 + s * kPitch + k);
                const float4 v = ld4(sh + kTrW4 + 64 * o + k);
                acc = fmaf(v.x, a.x, acc);
                acc = fmaf(v.y, a.y, acc);
                acc = fmaf(v.z, a.z, acc);
                acc = fmaf(v.w, a.w, acc);
            }
            sh[kTrO + 2 * s + o] = acc;
        }
        __syncthreads();
        if (t < kTrainS) {
            const bool valid = tile + row0 + t < n;
            const int at = kTrO + 2 * (row0 + t);
            const float o0 = sh[at], o1 = sh[at + 1];
            const float y = sh[kTrY + 2 * t], g = sh[kTrY + 2 * t + 1];
            const float th = tanhf(o1);
            const float sc = 1.0f + kMlpScaleRange * th;
            const float r0 = o0 - y, r1 = y - sc * g;
            if (valid) losses[tile + row0 + t] = r0 * r0 + r1 * r1;
            M.put(at, valid ? 2.0f * r0 * inv_total : 0.0f);
            M.put(at + 1, valid ? -2.0f * r1 * g * kMlpScaleRange * (1.0f - th * th) * inv_total : 0.0f);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 2; q++) {  // the last layer's deltas
            const int e = t + kTrainThreads * q, s = row0 + (e >> 4), k = 4 * (e & 15);
            const float4 g = ld4(sh + kTrD3 + s * kPitch + k);
            const float4 w0 = ld4(sh + kTrW4 + k), w1 = ld4(sh + kTrW4 + 64 + k);
            const float d0 = sh[kTrO + 2 * s], d1 = sh[kTrO + 2 * s + 1];
            M.put4(kTrD3 + s * kPitch + k, (w0.x * d0 + w1.x * d1) * g.x, (w0.y * d0 + w1.y * d1) * g.y,
                   (w0.z * d0 + w1.z * d1) * g.z, (w0.w * d0 + w1.w * d1) * g.w);
        }
        __syncthreads();
        dense_back(M, row0, kTrD3, kTrW3, kTrD2);
        __syncthreads();
        dense_back(M, row0, kTrD2, kTrW2, kTrD1);
        pair_barrier();  // both blocks' activations and deltas
        dense_wgrad(sh + kTrD3, sh + kTrA2, gj, gk, g3);
        dense_wgrad(sh + kTrD2, sh + kTrA1, gj, gk, g2);
        {  // W1[j][k] and W1[j][k + 1] of thread t: j = 32 rank + t / 8, k = 2 (t % 8)
            const int j = row0 + (t >> 3), k = 2 * (t & 7);
            float a = 0.0f, b = 0.0f;
#pragma unroll 8
            for (int s = 0; s < kTileS; s++) {
                const float d = sh[kTrD1 + s * kPitch + j];
                const float2 x = *reinterpret_cast<const float2*>(sh + kTrX + s * kPitchX + k);
                a = fmaf(d, x.x, a);
                b = fmaf(d, x.y, b);
            }
            g1[0] += a;
            g1[1] += b;
        }
        if (t < 96) {  // b1, b2 and b3
            const float* D = sh + (t < 32 ? kTrD1 : t < 64 ? kTrD2 : kTrD3) + row0 + (t & 31);
            float b = 0.0f;
#pragma unroll 8
            for (int s = 0; s < kTileS; s++) b += D[s * kPitch];
            gb += b;
        } else if (t >= 128 && t < 192) {  // W4[rank][k]
            float a = 0.0f;
#pragma unroll 8
            for (int s = 0; s < kTileS; s++) a = fmaf(sh[kTrO + 2 * s + rank], sh[kTrA3 + s * kPitch + t - 128], a);
            g4 += a;
        } else if (t == 192) {
            float b = 0.0f;
#pragma unroll 8
            for (int s = 0; s < kTileS; s++) b += sh[kTrO + 2 * s + rank];
            gb4 += b;
        }
        if (last) {
            float* dst = partials + static_cast<int64_t>(part) * kMlpParams;
#pragma unroll
            for (int i = 0; i < 2; i++) {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    dst[gW2 + (gj + i) * 64 + gk + k] = g2[i][k];
                    dst[gW3 + (gj + i) * 64 + gk + k] = g3[i][k];
                }
            }
            dst[gW1 + 16 * row0 + 2 * t] = g1[0];
            dst[gW1 + 16 * row0 + 2 * t + 1] = g1[1];
            if (t < 96) dst[(t < 32 ? gB1 : t < 64 ? gB2 : gB3) + row0 + (t & 31)] = gb;
            else if (t >= 128 && t < 192) dst[gW4 + 64 * rank + t - 128] = g4;
            else if (t == 192) dst[gB4 + rank] = gb4;
#pragma unroll
            for (int i = 0; i < 2; i++) {
#pragma unroll
                for (int k = 0; k < 4; k++) g2[i][k] = g3[i][k] = 0.0f;
                g1[i] = 0.0f;
            }
            gb = g4 = gb4 = 0.0f;
            part += clusters;
        }
        tile = next;
    }
}

// The draws of one Fisher-Yates shuffle of 0 .. n - 1 by SplitMix64 (Steele, Lea, Flood
// 2014): pick[i] in [0, i] for i = n - 1 .. 1, in that order from state `state`.
__global__ void __launch_bounds__(256) k_mlp_draws(uint64_t state, int64_t n, int64_t* pick) {
    const int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;  // k-th draw
    if (k >= n - 1) return;
    uint64_t z = state + static_cast<uint64_t>(k + 1) * 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z ^= z >> 31;
    const int64_t i = n - 1 - k;
    pick[i] = static_cast<int64_t>(z % static_cast<uint64_t>(i + 1));
}

// grad = sum of the block partials in a fixed order (FP64), loss likewise; with kAdam the
// Adam step of the entry follows.  32 entries a block, eight warps sharing the partials:
// one thread per entry took 13.4 us for 64 partials (a chain of FP64 additions) and Adam
// 3.5 us in its own launch; together now 7.3 us.  The last block adds the
// losses: FP32 within runs of 64 samples (of every kLossGroups-th run), FP64 over those.
constexpr int kUpdateThreads = 256;
constexpr int kUpdateBlocks = (kMlpParams + 31) / 32;
constexpr int kLossRun = 64, kLossGroups = 148;

template <bool kAdam>
__global__ void __launch_bounds__(kUpdateThreads) k_mlp_update(const float* partials, int blocks, const float* losses,
                                                               int64_t n, float* grad, double* loss, float* w,
                                                               float* m, float* v, float lr, float bc1, float bc2) {
    __shared__ double part[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_begin();
    if (blockIdx.x == kUpdateBlocks) {
        const int64_t runs = (n + kLossRun - 1) / kLossRun;
        float sum = 0.0f;
        if (threadIdx.x < kLossGroups)
            for (int64_t r = threadIdx.x; r < runs; r += runs < kLossGroups ? runs : kLossGroups) {
                float x[kLossRun];
#pragma unroll
                for (int k = 0; k < kLossRun; k++) x[k] = kLossRun * r + k < n ? __ldcg(losses + kLossRun * r + k) : 0.0f;
#pragma unroll
                for (int k = 0; k < kLossRun; k++) sum += x[k];
            }
        double acc = sum;
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) part[0][warp] = acc;
        __syncthreads();
        if (threadIdx.x == 0)
            *loss = ((part[0][0] + part[0][1]) + (part[0][2] + part[0][3])) +
                    ((part[0][4] + part[0][5]) + (part[0][6] + part[0][7]));
        return;
    }
    const int e = blockIdx.x * 32 + lane;
    // all of the warp's partials in flight, then two chains of additions
    constexpr int kMost = (kTrainParts + 7) / 8;
    float x[kMost];
#pragma unroll
    for (int k = 0; k < kMost; k++) {
        const int b = warp + 8 * k;
        x[k] = b < blocks && e < kMlpParams ? __ldcg(partials + static_cast<int64_t>(b) * kMlpParams + e) : 0.0f;
    }
    double acc = 0.0, odd = 0.0;
#pragma unroll
    for (int k = 0; k < kMost; k += 2) {
        if (warp + 8 * k < blocks) acc += widen(x[k]);
        if (k + 1 < kMost && warp + 8 * (k + 1) < blocks) odd += widen(x[k + 1]);
    }
    acc += odd;
    part[warp][lane] = acc;
    __syncthreads();
    if (warp != 0 || e >= kMlpParams) return;
    acc = ((part[0][lane] + part[1][lane]) + (part[2][lane] + part[3][lane])) +
          ((part[4][lane] + part[5][lane]) + (part[6][lane] + part[7][lane]));
    const float g = static_cast<float>(acc);
    const int p = kMlpOffW1 + e;
    if (!kAdam) {
        grad[p] = g;
        return;
    }
    const float mm = fmaf(0.1f, g, 0.9f * m[p]);
    const float vv = fmaf(0.001f * g, g, 0.999f * v[p]);
    m[p] = mm;
    v[p] = vv;
    w[p] -= lr * (mm / bc1) / (sqrtf(vv / bc2) + 1e-8f);
}

}  // namespace

size_t mlp_packed_bytes() { return kImgBytes; }

void mlp_pack_weights(const float* blob, void* image) {
    unsigned char* img = static_cast<unsigned char*>(image);
    std::memset(img, 0, kImgBytes);
    auto bf16 = [](float f) -> uint16_t {  // round to nearest even
        uint32_t u;
        std::memcpy(&u, &f, 4);
        if ((u & 0x7f800000u) == 0x7f800000u) return static_cast<uint16_t>(u >> 16);
        u += 0x7fffu + ((u >> 16) & 1u);
        return static_cast<uint16_t>(u >> 16);
    };
    auto put = [&](int off, int rows, int kdim, const float* W, int used_rows) {
        for (int r = 0; r < used_rows; r++)
            for (int k = 0; k < kdim; k++) {
                const uint16_t h = bf16(W[r * kdim + k]);
                std::memcpy(img + off + core_offset(r, k, rows), &h, 2);
            }
    };
    put(kImgW1, 64, 16, blob + kMlpOffW1, 64);
    put(kImgW2, 64, 64, blob + kMlpOffW2, 64);
    put(kImgW3, 64, 64, blob + kMlpOffW3, 64);
    put(kImgW4, 16, 64, blob + kMlpOffW4, 2);
    float* bias = reinterpret_cast<float*>(img + kImgBias);
    std::memcpy(bias, blob + kMlpOffB1, 64 * 4);
    std::memcpy(bias + 64, blob + kMlpOffB2, 64 * 4);
    std::memcpy(bias + 128, blob + kMlpOffB3, 64 * 4);
    std::memcpy(bias + 192, blob + kMlpOffB4, 2 * 4);
    std::memcpy(img + kImgNorm, blob + kMlpOffMu, 32 * 4);
}

cudaError_t mlp_prepare_device() {
    return cudaFuncSetAttribute(k_mlp_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmBytes);
}

cudaError_t mlp_train_prepare_device() {
    return cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(kTrBytes));
}

void launch_learned_q(const LearnedOps& L, const CgOperands& o, const CgScalars* S, cudaStream_t s) {
    k_lrn_q<<<grid_for(L.n), kBlock, 0, s>>>(L, o, L.dinv0, L.step, S, L.q4, L.q2);
}

void launch_learned_feature_rows(const LearnedOps& L, const CgOperands& o, const CgScalars* S, cudaStream_t s) {
    k_lrn_features<<<o.grid_spmv, kBlock, 0, s>>>(L, o, L.dinv0, L.step, S, L.q4, L.q2, L.len_ref);
}

void launch_learned_features(const LearnedOps& L, const CgOperands& o, const CgScalars* S,
                             cudaStream_t s) {
    launch_learned_q(L, o, S, s);
    launch_learned_feature_rows(L, o, S, s);
}

void launch_learned_apply(const LearnedOps& L, const CgOperands& o, const CgScalars* S, cudaStream_t s) {
    k_lrn_apply<<<grid_for(L.n), kBlock, 0, s>>>(L, o, S);
}

void launch_learned_targets(const LearnedOps& L, const CgOperands& o, const CgScalars* S,
                            cudaStream_t s) {
    k_lrn_targets<<<grid_for(L.n), kBlock, 0, s>>>(L, o, S);
}

void launch_mlp_infer(const void* packed, const float* feat, int n, const double* sigma, float* out,
                      int32_t* error, cudaStream_t s, const WaitLimits* limits) {
    const int tiles = (n + kTile - 1) / kTile;
    const int grid = tiles < 4 * 152 ? (tiles > 0 ? tiles : 1) : 4 * 152;
    k_mlp_tc<<<grid, kTile, kSmBytes, s>>>(static_cast<const unsigned char*>(packed), feat, n, sigma, out, error,
                                           limits);
}

int mlp_train_partials(int64_t n) {
    const int64_t c = (n + kTileS - 1) / kTileS;
    return static_cast<int>(c < kTrainParts ? (c > 0 ? c : 1) : kTrainParts);
}

void launch_mlp_loss_grad(const MlpTrainer& T, const float* samples, int64_t n, cudaStream_t s) {
    const int parts = mlp_train_partials(n);
    k_mlp_grad<<<2 * std::min(parts, kTrainClusters), kTrainThreads, kTrBytes, s>>>(T.w, samples, nullptr, n, parts,
                                                                                T.partials, T.losses);
    k_mlp_update<false><<<kUpdateBlocks + 1, kUpdateThreads, 0, s>>>(T.partials, parts, T.losses, n, T.grad, T.loss,
                                                                   nullptr, nullptr, nullptr, 0.0f, 0.0f, 0.0f);
}

void launch_mlp_draws(uint64_t state, int64_t n, int64_t* pick, cudaStream_t s) {
    k_mlp_draws<<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(state, n, pick);
}

void launch_mlp_train_step(const MlpTrainer& T, const int64_t* order, int64_t n, float lr, int step, double* loss,
                           cudaStream_t s) {
    const float bc1 = 1.0f - std::pow(0.9f, static_cast<float>(step));
    const float bc2 = 1.0f - std::pow(0.999f, static_cast<float>(step));
    const int parts = mlp_train_partials(n);
    launch_pdl(k_mlp_grad, 2 * std::min(parts, kTrainClusters), kTrainThreads, kTrBytes, s, T.w, T.samples, order, n,
               parts, T.partials, T.losses);
    launch_pdl(k_mlp_update<true>, kUpdateBlocks + 1, kUpdateThreads, 0, s, T.partials, parts, T.losses, n, nullptr,
               loss, T.w, T.m, T.v, lr, bc1, bc2);
}

}  // namespace mpsgb
