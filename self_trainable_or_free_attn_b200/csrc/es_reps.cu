// Four representatives per 64-token kv block, clustered in the query metric
// (reference: echosparse/kernels/representatives.py:1-166).
//
//   G_h = Q_h^T Q_h / (D L) + 1e-3 mean(diag) I;  M_h = chol(G_h) (lower, pivots clamped), stored bf16
//   64 probes per head: scaled means of evenly spaced 64-row query blocks, bf16
//   per kv block: X = K M, token weights from the probes' softmaxes, weighted Lloyd from four 16-token groups,
//   output = plain means of K and V over each final cluster (bf16) and log2 of the cluster sizes (-inf when empty).
//
// The Gram matrix is accumulated as per-split partial sums that the Cholesky kernel adds in a fixed order, so the
// metric is reproducible bit for bit (the reference adds with atomics).
#include "es_ptx.cuh"
#include "es_api_internal.h"

#include <cuda_bf16.h>
#include <math.h>

namespace es {

constexpr int HD = 128;
constexpr int NP = 64;            // probes per head

__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// ------------------------------------------------------------------------------------------------ Gram partials
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
// 16-byte asynchronous copy global -> shared; `bytes` = 0 fills the destination with zeros
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// parts[h][split] = sum over the split's rows of q_r q_r^T (bf16 products, float32 sums in tensor memory). A 64-row tile of Q
// ([d half][64 rows][128 B], by TMA, rows past L zero) is both operands of a tcgen05.mma, MN-major: A = Q^T, B = Q. The tensor pipe
// needs 256 clocks a tile of 16 KB, less than HBM takes to bring it, so the ring is there to keep loads on their way: six tiles,
// two CTAs per SM: 0.132 ms for 75,600 tokens x 40 heads, 5.9 TB/s (mma.sync from two cp.async tiles: 0.364 ms), and the same error
// against fp64 (3.4e-6, the float32 sums over a split).
//   warps 0-3  the result: row m of the accumulator is stored as column m (the matrix is symmetric), a whole line per store
//   warp 4     MMAs; warp 5 loads
constexpr int GRAM_SLOTS = 6;
constexpr uint32_t GRAM_HALF = 64 * 128, GRAM_TILE = 2 * GRAM_HALF, GRAM_CTL = GRAM_SLOTS * GRAM_TILE, GRAM_SMEM = GRAM_CTL + 256;
struct GramCtl {
    uint64_t full[GRAM_SLOTS], empty[GRAM_SLOTS], done;
    uint32_t tmem_base;
    int abort;
};
static_assert(sizeof(GramCtl) <= 256, "control block");

__global__ void __launch_bounds__(192, 2)
gram_kernel(const __grid_constant__ CUtensorMap tmQ, float* __restrict__ parts, int L, int rows_per_split, int nsplit, int* status) {
    extern __shared__ __align__(1024) uint8_t gram_smem[];
    const int h = blockIdx.x, sp = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = smem_u32(gram_smem);
    GramCtl* ctl = reinterpret_cast<GramCtl*>(gram_smem + GRAM_CTL);
    volatile int* abort_flag = &ctl->abort;
    // a split is a multiple of 64 rows, so that only rows past L fill up its last tile
    const int r_begin = sp * rows_per_split, nt = (min(L - r_begin, rows_per_split) + 63) / 64;
    if (tid == 0) {
        for (int i = 0; i < GRAM_SLOTS; ++i) {
            mbar_init(smem_u32(&ctl->full[i]), 1);
            mbar_init(smem_u32(&ctl->empty[i]), 1);
        }
        mbar_init(smem_u32(&ctl->done), 1);
        ctl->abort = (base & 1023u) ? 1 : 0;              // the swizzled tiles need a 1024-byte aligned base
        if (base & 1023u) atomicCAS(status, 0, 904);
        mbar_fence_init();
        fence_proxy_async_smem();
    }
    if (warp == 4) {
        tmem_alloc(smem_u32(&ctl->tmem_base), HD);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base, full0 = smem_u32(&ctl->full[0]), empty0 = smem_u32(&ctl->empty[0]);
    bool ok = *abort_flag == 0;
    int issued = 0;
    if (warp == 5) {
        for (int c = 0; c < nt && ok; ++c) {
            const uint32_t slot = c % GRAM_SLOTS, bar = full0 + 8 * slot;
            ok = mbar_wait_warp(empty0 + 8 * slot, ((c / GRAM_SLOTS) & 1) ^ 1, abort_flag, status, 601);
            if (!ok) break;
            if (lane == 0) mbar_arrive_expect_tx(bar, GRAM_TILE);
            __syncwarp();
            if (lane < 2) tma_load_3d(base + slot * GRAM_TILE + lane * GRAM_HALF, &tmQ, bar, 64 * lane, r_begin + 64 * c, h);
            issued = c + 1;
        }
    } else if (warp == 4) {
        constexpr uint32_t IDESC = umma_idesc_bf16(HD, HD, 1) | (1u << 15);      // both operands MN-major
        const uint64_t d0 = umma_desc_sw128(0, GRAM_HALF, 1024);
        const uint32_t d_hi = (uint32_t)(d0 >> 32), d_lo = (uint32_t)d0;
        for (int c = 0; c < nt && ok; ++c) {
            const uint32_t slot = c % GRAM_SLOTS;
            ok = mbar_wait_warp(full0 + 8 * slot, (c / GRAM_SLOTS) & 1, abort_flag, status, 602);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t t = d_lo + ((base + slot * GRAM_TILE) >> 4);
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                    umma_ss_lohi(tmem, t + ((ks * 2048) >> 4), d_hi, t + ((ks * 2048) >> 4), d_hi, IDESC, (c > 0 || ks > 0) ? 1u : 0u);
                umma_commit(empty0 + 8 * slot);
            }
            __syncwarp();
        }
        // after the last product, or what was issued of them: tensor memory is freed below
        if (elect_one()) umma_commit(smem_u32(&ctl->done));
        __syncwarp();
        mbar_wait(smem_u32(&ctl->done), 0, abort_flag, status, 603);
    } else {
        ok = ok && mbar_wait_warp(smem_u32(&ctl->done), 0, abort_flag, status, 604) && *abort_flag == 0;
        tc_fence_after();
        float* out = parts + ((size_t)h * nsplit + sp) * HD * HD + 32 * warp + lane;
#pragma unroll 1
        for (int p = 0; p < HD / 32; ++p) {
            uint32_t r[32];
            tmem_ld32(tmem + ((uint32_t)(32 * warp) << 16) + 32 * p, r);
            tmem_wait_ld_regs(r);
#pragma unroll
            for (int j = 0; j < 32; ++j) out[(32 * p + j) * HD] = ok ? __uint_as_float(r[j]) : NAN;
        }
        tc_fence_before();
    }
    __syncwarp();
    if (warp == 5 && lane == 0 && *abort_flag) {
        // a wait gave up: give the loads a moment (100 us in all) to land before shared memory goes away
        const uint64_t t_end = global_timer_ns() + 100000ull;
        for (int c = max(0, issued - GRAM_SLOTS); c < issued; ++c)
            while (!mbar_try_wait(full0 + 8 * (c % GRAM_SLOTS), (c / GRAM_SLOTS) & 1) && global_timer_ns() < t_end) {}
    }
    __syncthreads();
    if (warp == 4) {
        tc_fence_after();
        tmem_dealloc(tmem, HD);
    }
}

// ------------------------------------------------------------------------------------------------ metric
// Sum of the Gram partials of a head, scaled: parts[h][0] <- norm * sum_p parts[h][p], in the fixed order the sums have
// always been taken in (four running sums over p % 4, then (s0 + s1) + (s2 + s3)). Sixteen CTAs per head, so that the
// reduction of the 2 MB of partials is not one CTA's chain of loads (with a handful of heads per GPU it was).
__global__ void __launch_bounds__(256)
gram_reduce_kernel(float* __restrict__ parts, int nsplit, float norm) {
    const int h = blockIdx.x, e0 = (blockIdx.y * 256 + threadIdx.x) * 4;
    float* src = parts + (size_t)h * nsplit * HD * HD + e0;
    float4 s4[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) s4[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    int p = 0;
    for (; p + 4 <= nsplit; p += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float4 x = *reinterpret_cast<const float4*>(src + (size_t)(p + u) * HD * HD);
            s4[u].x += x.x; s4[u].y += x.y; s4[u].z += x.z; s4[u].w += x.w;
        }
    }
    for (int u = 0; p < nsplit; ++p, ++u) {
        const float4 x = *reinterpret_cast<const float4*>(src + (size_t)p * HD * HD);
        s4[u].x += x.x; s4[u].y += x.y; s4[u].z += x.z; s4[u].w += x.w;
    }
    float4 r;
    r.x = ((s4[0].x + s4[1].x) + (s4[2].x + s4[3].x)) * norm;
    r.y = ((s4[0].y + s4[1].y) + (s4[2].y + s4[3].y)) * norm;
    r.z = ((s4[0].z + s4[1].z) + (s4[2].z + s4[3].z)) * norm;
    r.w = ((s4[0].w + s4[1].w) + (s4[2].w + s4[3].w)) * norm;
    *reinterpret_cast<float4*>(src) = r;              // the slot of split 0: only this thread reads or writes these elements
}

// ------------------------------------------------------------------------------------------------ probes
// Probe i of a head = scale * mean of the query rows of 64-row block floor(i (nb - 1) / 63 + 0.5) (representatives.py:36-46): a warp
// each, four dimensions a lane, 32 rows requested at a time. The probes need only q, so they are more CTAs of the launch that makes
// the metric, beside its one chain per head. As a kernel of their own (a dimension per thread, a few loads on their way) they took
// 57 us a branch at Wan-14B, 20 us at Wan-1.3B, 6.7 us and a launch at 4,152 tokens.
constexpr int PROBES_PER_CTA = 8;
__device__ __forceinline__ void probe_block(const __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ probes, int cta, int L,
                                            int H, int nb, float scale) {
    const int at = cta * PROBES_PER_CTA + (threadIdx.x >> 5), d = 4 * (threadIdx.x & 31), i = at % NP, h = at / NP;
    const int blk = (int)((float)(i * (nb - 1)) / (float)(NP - 1) + 0.5f), n = min(64, L - blk * 64);
    const __nv_bfloat16* src = q + ((size_t)blk * 64 * H + h) * HD + d;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r0 = 0; r0 < 64; r0 += 32) {
        uint2 w[32];
#pragma unroll
        for (int r = 0; r < 32; ++r) w[r] = r0 + r < n ? __ldg(reinterpret_cast<const uint2*>(src + (size_t)(r0 + r) * H * HD)) : make_uint2(0u, 0u);
#pragma unroll
        for (int r = 0; r < 32; ++r)
            if (r0 + r < n) { s[0] += bf_lo(w[r].x); s[1] += bf_hi(w[r].x); s[2] += bf_lo(w[r].y); s[3] += bf_hi(w[r].y); }
    }
    const float c = fmaxf((float)n, 1.0f);
#pragma unroll
    for (int e = 0; e < 4; ++e) probes[(size_t)at * HD + d + e] = __float2bfloat16_rn(s[e] * scale / c);
}

// ------------------------------------------------------------------------------------------------ metric
// G (from gram_reduce_kernel) regularised, then its Cholesky factor with clamped pivots (representatives.py:49-63,
// 163-165), one CTA per head, the matrix in shared memory, blocked by panels of 16 columns. What bounds it is one chain of
// 128 square roots, divisions and broadcasts; everything else is kept off that chain:
//   panel     every warp factors the 16 x 16 diagonal block for itself in registers (a lane per row, broadcasts by shuffle), and
//             thread r solves its own row r of the panel in the same loop with the same broadcasts, so that the rows below the
//             block cost one multiply-add per broadcast and no barrier; the panel's columns of the result leave from there;
//   trailing  A -= L_panel L_panel^T on the lower triangle in 4 x 4 tiles from a transposed copy of the panel.
// Two barriers per panel. An element takes its 128 multiply-adds in ascending order whatever the blocking, so the bits do not
// depend on it. 26 us with two heads, 82 us with the rows below, the update and the stores as phases of their own.
constexpr int CH_PANEL = 16, CH_LD = 132;
constexpr int METRIC_SMEM = (HD + CH_PANEL) * CH_LD * (int)sizeof(float);
__global__ void __launch_bounds__(256)
metric_kernel(const float* __restrict__ parts, __nv_bfloat16* __restrict__ metric, float* __restrict__ gram_out,
              int nsplit, const __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ probes, int L, int H, float scale) {
    if ((int)blockIdx.x >= H) {
        probe_block(q, probes, (int)blockIdx.x - H, L, H, (L + 63) / 64, scale);
        return;
    }
    extern __shared__ __align__(16) float sm[];
    float* A = sm;                    // [128][CH_LD]
    float* P = A + HD * CH_LD;        // [16][CH_LD]: the panel, transposed
    __shared__ float red[8];
    __shared__ float s_eps, s_diag;
    const int h = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const float* src = parts + (size_t)h * nsplit * HD * HD;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int e = (u * 256 + tid) * 4;
        *reinterpret_cast<float4*>(A + (e >> 7) * CH_LD + (e & 127)) = *reinterpret_cast<const float4*>(src + e);
    }
    __syncthreads();
    float dg = tid < HD ? A[tid * CH_LD + tid] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dg += __shfl_xor_sync(0xffffffffu, dg, o);
    if (lane == 0) red[warp] = dg;
    __syncthreads();
    if (tid == 0) s_diag = (((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]))) / HD;
    __syncthreads();
    if (tid < HD) A[tid * CH_LD + tid] += 1e-3f * s_diag;
    __syncthreads();
    if (gram_out)
        for (int e = tid; e < HD * HD; e += 256) gram_out[(size_t)h * HD * HD + e] = A[(e >> 7) * CH_LD + (e & 127)];
    dg = tid < HD ? A[tid * CH_LD + tid] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dg += __shfl_xor_sync(0xffffffffu, dg, o);
    __syncthreads();
    if (lane == 0) red[warp] = dg;
    __syncthreads();
    if (tid == 0)
        s_eps = (((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]))) / HD * 1e-12f;
    __syncthreads();
    const float eps = s_eps;
    for (int j0 = 0; j0 < HD; j0 += CH_PANEL) {
        if (tid < HD) {
            const int i = lane & 15, r = tid;
            if (warp * 32 + 31 >= j0) {                    // uniform over the warp: some row of it is not above the panel
                float d[CH_PANEL], x[CH_PANEL];            // row i of the diagonal block; this thread's row of the panel
#pragma unroll
                for (int c = 0; c < CH_PANEL; c += 4) {
                    *reinterpret_cast<float4*>(d + c) = *reinterpret_cast<const float4*>(A + (j0 + i) * CH_LD + j0 + c);
                    *reinterpret_cast<float4*>(x + c) = *reinterpret_cast<const float4*>(A + r * CH_LD + j0 + c);
                }
#pragma unroll
                for (int j = 0; j < CH_PANEL; ++j) {
                    const float root = sqrtf(fmaxf(__shfl_sync(0xffffffffu, d[j], j), eps));
                    const float l = d[j] / root;           // lanes above the pivot, and x right of the diagonal, hold values
                    x[j] /= root;                          // that nothing reads
#pragma unroll
                    for (int c = j + 1; c < CH_PANEL; ++c) {
                        const float lc = __shfl_sync(0xffffffffu, l, c);
                        d[c] = fmaf(-l, lc, d[c]);
                        x[c] = fmaf(-x[j], lc, x[c]);
                    }
                }
                uint32_t w[CH_PANEL / 2];
#pragma unroll
                for (int c = 0; c < CH_PANEL; ++c) {
                    x[c] = j0 + c <= r ? x[c] : 0.f;
                    P[c * CH_LD + r] = x[c];
                }
#pragma unroll
                for (int c = 0; c < CH_PANEL / 2; ++c) {
                    const __nv_bfloat162 v = __floats2bfloat162_rn(x[2 * c], x[2 * c + 1]);
                    w[c] = *reinterpret_cast<const uint32_t*>(&v);
                }
                uint4* dst = reinterpret_cast<uint4*>(metric + (size_t)h * HD * HD + r * HD + j0);
                dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
                dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
            } else {
                uint4* dst = reinterpret_cast<uint4*>(metric + (size_t)h * HD * HD + r * HD + j0);
                dst[0] = dst[1] = make_uint4(0, 0, 0, 0);
            }
        }
        __syncthreads();
        const int first = j0 + CH_PANEL, T = (HD - first) / 4;
        for (int t = tid; t < T * (T + 1) / 2; t += 256) {
            int tr = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);      // tile (tr, tc), tc <= tr
            if (tr * (tr + 1) / 2 > t) --tr;
            if ((tr + 1) * (tr + 2) / 2 <= t) ++tr;
            const int tc = t - tr * (tr + 1) / 2, R0 = first + 4 * tr, C0 = first + 4 * tc;
            float4 acc[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[u] = *reinterpret_cast<const float4*>(A + (R0 + u) * CH_LD + C0);
#pragma unroll
            for (int k = 0; k < CH_PANEL; ++k) {
                const float4 b = *reinterpret_cast<const float4*>(P + k * CH_LD + C0);
                const float4 a4 = *reinterpret_cast<const float4*>(P + k * CH_LD + R0);
                const float a[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    acc[u].x = fmaf(-a[u], b.x, acc[u].x);
                    acc[u].y = fmaf(-a[u], b.y, acc[u].y);
                    acc[u].z = fmaf(-a[u], b.z, acc[u].z);
                    acc[u].w = fmaf(-a[u], b.w, acc[u].w);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) *reinterpret_cast<float4*>(A + (R0 + u) * CH_LD + C0) = acc[u];
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------------ k-means
// One CTA (8 warps) per (kv block, head), several blocks in turn. Every contraction runs on the tensor cores
// (mma.sync m16n8k16 with float32 sums): the probe scores and X = K M on bf16 inputs (the arithmetic of the reference's
// tl.dot on bf16), the Lloyd iterations on float32 values split into two bf16 halves, x = hi + lo with lo = bf16(x - hi),
// 16 mantissa bits (the reference's tl.dot on float32 inputs runs as TF32 on a GPU, 10 bits; the golden outputs come
// from exact float32):
//   distances   X C^T: the warp's X fragments (hi, lo) stay in registers from the X = K M accumulators; the right operand
//               has the centroids' upper halves in columns 0-3 and their lower halves in columns 4-7, so two MMAs per
//               k-step give all four cross products and no column is padding;
//   centroids   (w X)^T (0 / 1 membership): the token weights are folded into Y = w X once per block, so the membership
//               operand is exact and two products (Y hi, Y lo) suffice; Y is read back by transposing loads;
//   final means (0 / 1 membership)^T K and V, exact products.
constexpr int KS = 136;           // bf16 row stride of the K tile: 272 B, so the 8 rows of an ldmatrix hit distinct banks
constexpr int XB = 136;           // bf16 row stride of the two halves of Y and of the centroids
constexpr int PS = 65;            // float row stride of the probe scores
constexpr int MS = 136;           // bf16 row stride of the metric in shared memory
constexpr int OS = 72;            // bf16 row stride of the (cluster, token) membership matrix
constexpr int KM_BLOCKS = 4;      // kv blocks per CTA: the metric is loaded into shared memory once for all of them
constexpr int VS = 136;           // bf16 row stride of the V tile (it takes the place of the probe scores)
constexpr int KM_SMEM = 128 * MS * 2 + 64 * KS * 2 + 2 * 64 * XB * 2 + 64 * VS * 2 + 8 * XB * 2 + 4 * 64 * 4 + 64 * 4 +
                        64 * 4 + 2 * 64 * 8 * 4 + 8 * OS * 2;
static_assert(64 * VS * 2 >= 64 * PS * 4, "the V tile and the probe scores share one area");

__device__ __forceinline__ void split_bf16(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h2 = __floats2bfloat162_rn(x, y);
    const float2 hf = __bfloat1622float2(h2);
    const __nv_bfloat162 l2 = __floats2bfloat162_rn(x - hf.x, y - hf.y);
    hi = *reinterpret_cast<const uint32_t*>(&h2);
    lo = *reinterpret_cast<const uint32_t*>(&l2);
}

__global__ void __launch_bounds__(256, 2)
kmeans_kernel(const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
              const __nv_bfloat16* __restrict__ metric, const __nv_bfloat16* __restrict__ probes,
              __nv_bfloat16* __restrict__ k4, __nv_bfloat16* __restrict__ v4, float* __restrict__ c4,
              __nv_bfloat16* __restrict__ km, __nv_bfloat16* __restrict__ vm, int L, int H, int nb4, int iters,
              int blocks_per_cta) {
    extern __shared__ __align__(16) uint8_t raw[];
    __nv_bfloat16* sM = reinterpret_cast<__nv_bfloat16*>(raw);                     // [128][MS] the head's metric
    __nv_bfloat16* sK = sM + 128 * MS;                                             // [64][KS]
    __nv_bfloat16* sYh = sK + 64 * KS;                                             // [64][XB] Y = w X, upper halves
    __nv_bfloat16* sYl = sYh + 64 * XB;                                            // [64][XB] Y, lower halves
    float* sP = reinterpret_cast<float*>(sYl + 64 * XB);                           // [64 probes][PS]
    __nv_bfloat16* cen = reinterpret_cast<__nv_bfloat16*>(sP) + 64 * VS;           // [8][XB] centroids: rows 0-3 upper, 4-7 lower halves
    float* wpart = reinterpret_cast<float*>(cen + 8 * XB);                         // [4][64]
    float* w = wpart + 4 * 64;                                                     // [64]
    int* lab = reinterpret_cast<int*>(w + 64);                                     // [64]
    float* dpart = reinterpret_cast<float*>(lab + 64);                             // [2 d halves][64 tokens][8 columns]
    __nv_bfloat16* oh = reinterpret_cast<__nv_bfloat16*>(dpart + 2 * 64 * 8);      // [8][OS] (cluster, token) membership, rows 4-7 zero
    __shared__ float cw[4], cwp[4][4], nnp[8][4];
    __shared__ float s_cnt[4];
    const int h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tg = lane & 3;
    const int nb = (L + 63) / 64;
    // the metric of this head: 128 x 128 bf16, once per CTA
    for (int e = tid; e < 128 * 16; e += 256) {
        const int r = e >> 4, c16 = e & 15;
        cp_async16_zfill((uint32_t)__cvta_generic_to_shared(sM + r * MS + c16 * 8),
                         metric + ((size_t)h * HD + r) * HD + c16 * 8, 16);
    }
    cp_async_commit();
    // rows 4-7 of the membership matrix pad the four clusters to the 8 columns of an MMA: zero for good
    for (int e = tid; e < 8 * OS / 2; e += 256) reinterpret_cast<uint32_t*>(oh)[e] = 0u;
    const int mt = warp & 3, nh = warp >> 2;
    const int lj = lane & 7, lm = lane >> 3;
    const __nv_bfloat16 one = __float2bfloat16_rn(1.0f), zero = __float2bfloat16_rn(0.0f);
  for (int j = blockIdx.x * blocks_per_cta; j < min(nb, (int)(blockIdx.x + 1) * blocks_per_cta); ++j) {
    const int nvalid = min(L - j * 64, 64);
    __syncthreads();                       // the previous block's readers of the shared tiles are done
    // K tile (rows past L are zero)
    for (int e = tid; e < 64 * 16; e += 256) {
        const int r = e >> 4, c16 = e & 15;
        const bool okr = r < nvalid;
        cp_async16_zfill((uint32_t)__cvta_generic_to_shared(sK + r * KS + c16 * 8),
                         k + ((size_t)(j * 64 + (okr ? r : 0)) * H + h) * HD + c16 * 8, okr ? 16 : 0);
    }
    cp_async_commit();
    // this thread's A fragments of the probe scores (probes 16 mt .. +15), requested while the K tile travels
    uint32_t pa[8][4];
    {
        const __nv_bfloat16* p0 = probes + ((size_t)h * NP + 16 * mt + g) * HD + 2 * tg;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            pa[ks][0] = __ldg(reinterpret_cast<const uint32_t*>(p0 + ks * 16));
            pa[ks][1] = __ldg(reinterpret_cast<const uint32_t*>(p0 + 8 * HD + ks * 16));
            pa[ks][2] = __ldg(reinterpret_cast<const uint32_t*>(p0 + ks * 16 + 8));
            pa[ks][3] = __ldg(reinterpret_cast<const uint32_t*>(p0 + 8 * HD + ks * 16 + 8));
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    {
        // probe scores: probes 16 mt .. +15 (A, in registers), tokens 32 nh .. +31 (B = K rows, from shared memory)
        float acc[4][4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[nt][x] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            const uint32_t a0 = pa[ks][0], a1 = pa[ks][1], a2 = pa[ks][2], a3 = pa[ks][3];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const __nv_bfloat16* kr = sK + (32 * nh + 8 * nt + g) * KS + ks * 16 + 2 * tg;
                mma16816(acc[nt], a0, a1, a2, a3, *reinterpret_cast<const uint32_t*>(kr),
                         *reinterpret_cast<const uint32_t*>(kr + 8));
            }
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const int col = 32 * nh + 8 * nt + 2 * tg;
            sP[(16 * mt + g) * PS + col] = acc[nt][0];
            sP[(16 * mt + g) * PS + col + 1] = acc[nt][1];
            sP[(16 * mt + g + 8) * PS + col] = acc[nt][2];
            sP[(16 * mt + g + 8) * PS + col + 1] = acc[nt][3];
        }
    }
    __syncthreads();
    // each probe's softmax over the block's valid tokens (natural exponent): four threads per probe, 16 tokens each
    {
        float* row = sP + (tid >> 2) * PS + (tid & 3) * 16;
        const int t0 = (tid & 3) * 16;
        float mx = -INFINITY;
#pragma unroll
        for (int t = 0; t < 16; ++t) mx = (t0 + t < nvalid) ? fmaxf(mx, row[t]) : mx;
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        float e[16], sum = 0.f;
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            e[t] = (t0 + t < nvalid) ? expf(row[t] - mx) : 0.f;
            sum += e[t];
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        const float inv = 1.0f / sum;
#pragma unroll
        for (int t = 0; t < 16; ++t) row[t] = e[t] * inv;
    }
    __syncthreads();
    // token weights: sum over the probes (four partial sums of 16 probes, added in a fixed order)
    {
        const int t = tid & 63, qp = tid >> 6;
        float sacc = 0.f;
#pragma unroll
        for (int p = 0; p < 16; ++p) sacc += sP[(16 * qp + p) * PS + t];
        wpart[qp * 64 + t] = sacc;
    }
    __syncthreads();
    if (tid < 64) {
        const float sacc = (wpart[tid] + wpart[64 + tid]) + (wpart[128 + tid] + wpart[192 + tid]);
        w[tid] = tid < nvalid ? sacc * ((float)nvalid / (float)NP) : 0.f;
    }
    __syncthreads();
    // Warp mt of the first four owns tokens 16 mt .. +15: lane (g, tg) keeps the labels of tokens g and g + 8 and writes
    // cluster tg's column of their rows of the membership matrix; the cluster weights of the 16 tokens are added over the
    // lanes in a fixed order.
    const float w_a = w[16 * mt + g], w_b = w[16 * mt + g + 8];
    int lab_a = mt, lab_b = mt;                       // the initial clusters are the four token quarters
    auto publish = [&]() {
        oh[tg * OS + 16 * mt + g] = lab_a == tg ? one : zero;
        oh[tg * OS + 16 * mt + g + 8] = lab_b == tg ? one : zero;
        if (tg == 0) { lab[16 * mt + g] = lab_a; lab[16 * mt + g + 8] = lab_b; }
        float ws = (lab_a == tg ? w_a : 0.f) + (lab_b == tg ? w_b : 0.f);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) ws += __shfl_xor_sync(0xffffffffu, ws, o);
        if (g == 0) cwp[mt][tg] = ws;
    };
    if (nh == 0) publish();
    // The probe scores are dead now: their area receives the V tile (64 x 128 bf16), copied asynchronously while the
    // Lloyd iterations run, so the final cluster means do not wait on global memory.
    __nv_bfloat16* sV = reinterpret_cast<__nv_bfloat16*>(sP);
    for (int e = tid; e < 64 * 16; e += 256) {
        const int r = e >> 4, c16 = e & 15;
        const bool okr = r < nvalid;
        cp_async16_zfill((uint32_t)__cvta_generic_to_shared(sV + r * VS + c16 * 8),
                         v + ((size_t)(j * 64 + (okr ? r : 0)) * H + h) * HD + c16 * 8, okr ? 16 : 0);
    }
    cp_async_commit();

    // X = K M: rows 16 mt .. +15, columns 64 nh .. +63. The accumulators of column tiles 2 ks, 2 ks + 1 are, split in two
    // bf16 halves, this warp's A fragment of k-step ks of the distance products (rows = tokens, k = these 64 dims); the
    // rows times their tokens' weights go to shared memory for the centroid sums.
    uint32_t xa_h[4][4], xa_l[4][4];
    {
        float acc[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[nt][x] = 0.f;
        const uint32_t a_addr = (uint32_t)__cvta_generic_to_shared(sK + (16 * mt + (lane & 15)) * KS + (lane >> 4) * 8);
        const uint32_t m_addr = (uint32_t)__cvta_generic_to_shared(sM);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            uint32_t a0, a1, a2, a3;
            ldmatrix_x4(a_addr + ks * 32, a0, a1, a2, a3);
#pragma unroll
            for (int np = 0; np < 4; ++np) {
                // B[k][n] = M[k][n], row-major in shared memory: transposed 8 x 8 loads, matrices (k lo, n0), (k hi, n0),
                // (k lo, n0 + 8), (k hi, n0 + 8)
                const int row = ks * 16 + lj + (lm & 1) * 8, col = 64 * nh + 16 * np + (lm >> 1) * 8;
                uint32_t b0, b1, b2, b3;
                ldmatrix_x4_trans(m_addr + (uint32_t)(row * MS + col) * 2, b0, b1, b2, b3);
                mma16816(acc[2 * np], a0, a1, a2, a3, b0, b1);
                mma16816(acc[2 * np + 1], a0, a1, a2, a3, b2, b3);
            }
        }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            uint32_t h0, l0, h1, l1;
            split_bf16(acc[nt][0], acc[nt][1], h0, l0);        // row g
            split_bf16(acc[nt][2], acc[nt][3], h1, l1);        // row g + 8
            xa_h[nt >> 1][(nt & 1) * 2] = h0; xa_h[nt >> 1][(nt & 1) * 2 + 1] = h1;
            xa_l[nt >> 1][(nt & 1) * 2] = l0; xa_l[nt >> 1][(nt & 1) * 2 + 1] = l1;
            split_bf16(acc[nt][0] * w_a, acc[nt][1] * w_a, h0, l0);
            split_bf16(acc[nt][2] * w_b, acc[nt][3] * w_b, h1, l1);
            const int col = 64 * nh + 8 * nt + 2 * tg;
            *reinterpret_cast<uint32_t*>(sYh + (16 * mt + g) * XB + col) = h0;
            *reinterpret_cast<uint32_t*>(sYh + (16 * mt + g + 8) * XB + col) = h1;
            *reinterpret_cast<uint32_t*>(sYl + (16 * mt + g) * XB + col) = l0;
            *reinterpret_cast<uint32_t*>(sYl + (16 * mt + g + 8) * XB + col) = l1;
        }
    }
    __syncthreads();

    // Weighted centroids of the current labels, transposed: rows = this warp's 16 dims, columns = clusters. The warp's
    // fragments of Y^T (all 64 tokens, both halves) are fetched once per block by transposing loads: matrices (tokens lo,
    // dims lo), (tokens lo, dims hi), (tokens hi, dims lo), (tokens hi, dims hi). keep_old: an emptied cluster keeps its
    // centroid (and its squared norm).
    uint32_t ya_h[4][4], ya_l[4][4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        const uint32_t off = (uint32_t)((16 * ks + lj + (lm >> 1) * 8) * XB + 16 * warp + (lm & 1) * 8) * 2;
        ldmatrix_x4_trans((uint32_t)__cvta_generic_to_shared(sYh) + off, ya_h[ks][0], ya_h[ks][1], ya_h[ks][2], ya_h[ks][3]);
        ldmatrix_x4_trans((uint32_t)__cvta_generic_to_shared(sYl) + off, ya_l[ks][0], ya_l[ks][1], ya_l[ks][2], ya_l[ks][3]);
    }
    auto update_centroids = [&](bool keep_old) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            const uint32_t b0 = *reinterpret_cast<const uint32_t*>(oh + g * OS + 16 * ks + 2 * tg);
            const uint32_t b1 = *reinterpret_cast<const uint32_t*>(oh + g * OS + 16 * ks + 8 + 2 * tg);
            mma16816(acc, ya_h[ks][0], ya_h[ks][1], ya_h[ks][2], ya_h[ks][3], b0, b1);
            mma16816(acc, ya_l[ks][0], ya_l[ks][1], ya_l[ks][2], ya_l[ks][3], b0, b1);
        }
        // lanes with tg < 2: dims 16 warp + g and + 8 of clusters 2 tg and 2 tg + 1
        const int ca = (2 * tg) & 3, cb = ca + 1;
        const float wa = (cwp[0][ca] + cwp[1][ca]) + (cwp[2][ca] + cwp[3][ca]);
        const float wb = (cwp[0][cb] + cwp[1][cb]) + (cwp[2][cb] + cwp[3][cb]);
        const bool wr_a = tg < 2 && (!keep_old || wa > 0.f), wr_b = tg < 2 && (!keep_old || wb > 0.f);
        const float ia = 1.0f / fmaxf(wa, 1e-6f), ib = 1.0f / fmaxf(wb, 1e-6f);
        uint32_t ha, la, hb, lb;
        split_bf16(acc[0] * ia, acc[2] * ia, ha, la);          // cluster a: dims g, g + 8
        split_bf16(acc[1] * ib, acc[3] * ib, hb, lb);          // cluster b
        const int d = 16 * warp + g;
        float na = 0.f, nb2 = 0.f;
        if (wr_a) {
            cen[ca * XB + d] = __ushort_as_bfloat16((unsigned short)(ha & 0xFFFFu));
            cen[ca * XB + d + 8] = __ushort_as_bfloat16((unsigned short)(ha >> 16));
            cen[(4 + ca) * XB + d] = __ushort_as_bfloat16((unsigned short)(la & 0xFFFFu));
            cen[(4 + ca) * XB + d + 8] = __ushort_as_bfloat16((unsigned short)(la >> 16));
            const float c0 = bf_lo(ha) + bf_lo(la), c1 = bf_hi(ha) + bf_hi(la);
            na = c0 * c0 + c1 * c1;
        }
        if (wr_b) {
            cen[cb * XB + d] = __ushort_as_bfloat16((unsigned short)(hb & 0xFFFFu));
            cen[cb * XB + d + 8] = __ushort_as_bfloat16((unsigned short)(hb >> 16));
            cen[(4 + cb) * XB + d] = __ushort_as_bfloat16((unsigned short)(lb & 0xFFFFu));
            cen[(4 + cb) * XB + d + 8] = __ushort_as_bfloat16((unsigned short)(lb >> 16));
            const float c0 = bf_lo(hb) + bf_lo(lb), c1 = bf_hi(hb) + bf_hi(lb);
            nb2 = c0 * c0 + c1 * c1;
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            na += __shfl_xor_sync(0xffffffffu, na, o);
            nb2 += __shfl_xor_sync(0xffffffffu, nb2, o);
        }
        if (g == 0) {                                  // the squared norms' shares of these 16 dims
            if (wr_a) nnp[warp][ca] = na;
            if (wr_b) nnp[warp][cb] = nb2;
        }
        if (warp == 0 && g == 0 && tg < 2) { cw[ca] = wa; cw[cb] = wb; }
        __syncthreads();
    };
    update_centroids(false);
    for (int it = 0; it < iters; ++it) {
        // the warp's 16 tokens against the four centroids over its 64 dims: columns 0-3 x . c_hi, columns 4-7 x . c_lo
        {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                const int d = 64 * nh + 16 * ks + 2 * tg;
                const uint32_t b0 = *reinterpret_cast<const uint32_t*>(cen + g * XB + d);
                const uint32_t b1 = *reinterpret_cast<const uint32_t*>(cen + g * XB + d + 8);
                mma16816(acc, xa_h[ks][0], xa_h[ks][1], xa_h[ks][2], xa_h[ks][3], b0, b1);
                mma16816(acc, xa_l[ks][0], xa_l[ks][1], xa_l[ks][2], xa_l[ks][3], b0, b1);
            }
            float* mine = dpart + (nh * 64 + 16 * mt + g) * 8 + 2 * tg;
            *reinterpret_cast<float2*>(mine) = make_float2(acc[0], acc[1]);
            *reinterpret_cast<float2*>(mine + 64) = make_float2(acc[2], acc[3]);
        }
        __syncthreads();
        int differs = 0;
        if (nh == 0) {
            // this warp's 16 tokens: both d halves, then upper + lower centroid halves (lanes tg and tg ^ 2), then the
            // smaller distance of the lane's two clusters against that of lane tg ^ 1 (ties to the smaller cluster)
            const float* p0 = dpart + (16 * mt + g) * 8 + 2 * tg;
            const float2 a0 = *reinterpret_cast<const float2*>(p0), a1 = *reinterpret_cast<const float2*>(p0 + 64 * 8);
            const float2 b0 = *reinterpret_cast<const float2*>(p0 + 64), b1 = *reinterpret_cast<const float2*>(p0 + 64 * 8 + 64);
            float da[2] = {a0.x + a1.x, a0.y + a1.y}, db[2] = {b0.x + b1.x, b0.y + b1.y};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                da[e] += __shfl_xor_sync(0xffffffffu, da[e], 2);
                db[e] += __shfl_xor_sync(0xffffffffu, db[e], 2);
            }
            const int c0 = (2 * tg) & 3;              // lanes tg and tg ^ 2 hold clusters c0, c0 + 1
            float dist_a[2], dist_b[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int cc = c0 + e;
                const float nn = ((nnp[0][cc] + nnp[1][cc]) + (nnp[2][cc] + nnp[3][cc])) +
                                 ((nnp[4][cc] + nnp[5][cc]) + (nnp[6][cc] + nnp[7][cc]));
                const bool live = cw[cc] > 0.f;
                dist_a[e] = live ? nn - 2.0f * da[e] : INFINITY;
                dist_b[e] = live ? nn - 2.0f * db[e] : INFINITY;
            }
            auto pick = [&](const float (&d)[2]) -> int {
                float bd = d[0];
                int bi = c0;
                if (d[1] < bd) { bd = d[1]; bi = c0 + 1; }
                const float od = __shfl_xor_sync(0xffffffffu, bd, 1);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, 1);
                return (od < bd || (od == bd && oi < bi)) ? oi : bi;
            };
            const int na = pick(dist_a), nb_ = pick(dist_b);
            differs = (16 * mt + g < nvalid && na != lab_a) || (16 * mt + g + 8 < nvalid && nb_ != lab_b);
            lab_a = na; lab_b = nb_;
            publish();
        }
        const int changed = __syncthreads_or(differs);
        update_centroids(true);
        if (changed == 0) break;
    }

    // plain means of K and V over the final clusters, and the block means when asked for
    if (warp == 0) {
        const int l0 = lane < nvalid ? lab[lane] : -1, l1 = lane + 32 < nvalid ? lab[lane + 32] : -1;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int n = __popc(__ballot_sync(0xffffffffu, l0 == c)) + __popc(__ballot_sync(0xffffffffu, l1 == c));
            if (lane == c) {
                s_cnt[c] = (float)n;
                c4[(size_t)h * nb4 + j * 4 + c] = n > 0 ? log2f((float)n) : -INFINITY;
            }
            // membership of the valid tokens only (the last readers passed the barrier that ended the iterations)
            oh[c * OS + lane] = l0 == c ? one : zero;
            oh[c * OS + lane + 32] = l1 == c ? one : zero;
        }
    }
    cp_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int which = 0; which < 2; ++which) {
        // (membership)^T K and (membership)^T V: rows = clusters (4 of 16), columns = this warp's 16 dims; products with
        // 0 / 1 are exact, the sums are float32
        float acc[2][4];
#pragma unroll
        for (int jj = 0; jj < 2; ++jj)
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[jj][x] = 0.f;
        const uint32_t src = (uint32_t)__cvta_generic_to_shared(which ? sV : sK);
        const int stride = which ? VS : KS;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            const uint32_t a0 = *reinterpret_cast<const uint32_t*>(oh + g * OS + 16 * ks + 2 * tg);
            const uint32_t a2 = *reinterpret_cast<const uint32_t*>(oh + g * OS + 16 * ks + 8 + 2 * tg);
            uint32_t b0, b1, b2, b3;
            ldmatrix_x4_trans(src + (uint32_t)((16 * ks + lj + (lm & 1) * 8) * stride + 16 * warp + (lm >> 1) * 8) * 2, b0, b1, b2, b3);
            mma16816(acc[0], a0, 0u, a2, 0u, b0, b1);
            mma16816(acc[1], a0, 0u, a2, 0u, b2, b3);
        }
        const float inv = g < 4 ? 1.0f / fmaxf(s_cnt[g], 1.0f) : 0.f;
        __nv_bfloat16* o = (which ? v4 : k4) + ((size_t)h * nb4 + j * 4 + (g & 3)) * HD + 16 * warp + 2 * tg;
        __nv_bfloat16* mo = which ? vm : km;
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
            if (g < 4) *reinterpret_cast<__nv_bfloat162*>(o + 8 * jj) = __floats2bfloat162_rn(acc[jj][0] * inv, acc[jj][1] * inv);
            // block mean: the four clusters' sums, (0 + 1) + (2 + 3), held by lanes 4 c + tg
            float t0 = acc[jj][0], t1 = acc[jj][1];
            t0 += __shfl_xor_sync(0xffffffffu, t0, 4); t1 += __shfl_xor_sync(0xffffffffu, t1, 4);
            t0 += __shfl_xor_sync(0xffffffffu, t0, 8); t1 += __shfl_xor_sync(0xffffffffu, t1, 8);
            if (mo && g == 0)
                *reinterpret_cast<__nv_bfloat162*>(mo + ((size_t)j * H + h) * HD + 16 * warp + 8 * jj + 2 * tg) =
                    __floats2bfloat162_rn(t0 / (float)nvalid, t1 / (float)nvalid);
        }
    }
  }
}

}  // namespace es

using namespace es;

static int launch_gram(const void* q, float* parts, int L, int H, int rows_per_split, int nsplit, cudaStream_t st) {
    int* status = device_status_ptr();
    if (!status) return set_error(-2, "es_reps_metric: the device status word is not available on this device");
    // (L, H, 128) bf16 viewed as dims {128 d, L, H}; a box is 64 d x 64 rows, 128-byte swizzled
    CUtensorMap tq;
    cuuint64_t dims[3] = {(cuuint64_t)HD, (cuuint64_t)L, (cuuint64_t)H};
    cuuint64_t strides[2] = {(cuuint64_t)H * HD * 2, (cuuint64_t)HD * 2};
    cuuint32_t box[3] = {64, 64, 1}, estr[3] = {1, 1, 1};
    if (int rc = encode_tensor_map(&tq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, estr,
                                   CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    if (int rc = opt_in_shared_memory((const void*)gram_kernel, (int)GRAM_SMEM)) return rc;
    gram_kernel<<<dim3(H, nsplit), 192, GRAM_SMEM, st>>>(tq, parts, L, rows_per_split, nsplit, status);
    ES_CHECK_LAUNCH("gram");
    return 0;
}

// Rows of q per Gram partial, as the reference splits them (representatives.py:160).
static int gram_rows_per_split(int L) { return ((((L + 31) / 32) + 63) / 64) * 64; }

extern "C" int es_reps_gram_splits(int32_t L) {
    if (L <= 0) return 0;
    const int rps = gram_rows_per_split(L);
    return (L + rps - 1) / rps;
}

// q (L, H, 128) bf16 -> metric (H, 128, 128) bf16 (Cholesky factor) and probes (H, 64, 128) bf16.
// gram_parts: scratch of es_reps_gram_splits(L) * H * 128 * 128 floats; gram (H, 128, 128) fp32 receives the
// regularised Gram matrix when not null.
extern "C" int es_reps_metric(const void* q, float* gram_parts, float* gram, void* metric, void* probes, int32_t L,
                              int32_t H, void* stream) {
    if (!q || !gram_parts || !metric || !probes) return set_error(-1, "es_reps_metric: null pointer");
    if (L <= 0 || H <= 0) return set_error(-1, "es_reps_metric: L and H must be positive");
    if (!aligned(16, q, gram_parts, metric)) return set_error(-1, "es_reps_metric: q, gram_parts and metric must be 16-byte aligned");
    const int rps = gram_rows_per_split(L), nsplit = (L + rps - 1) / rps;
    cudaStream_t st = (cudaStream_t)stream;
    if (int rc = launch_gram(q, gram_parts, L, H, rps, nsplit, st)) return rc;
    const int smem = METRIC_SMEM;
    if (int rc = opt_in_shared_memory((const void*)metric_kernel, smem)) return rc;
    const float scale = 1.0f / sqrtf((float)HD);
    gram_reduce_kernel<<<dim3(H, HD * HD / 1024), 256, 0, st>>>(gram_parts, nsplit, scale * scale / (float)L);
    ES_CHECK_LAUNCH("gram_reduce");
    metric_kernel<<<H + NP / PROBES_PER_CTA * H, 256, smem, st>>>(gram_parts, (__nv_bfloat16*)metric, gram, nsplit, (const __nv_bfloat16*)q,
                                                                  (__nv_bfloat16*)probes, L, H, scale);
    ES_CHECK_LAUNCH("metric");
    return 0;
}

// k, v (L, H, 128) bf16 -> k_rep, v_rep (H, (nb + 1) * 4, 128) bf16 and log_counts (H, (nb + 1) * 4) fp32; block nb of
// the tables is left as the caller initialised it (zeros, -inf). k_mean / v_mean (nb, H, 128) are written when given.
extern "C" int es_reps_kmeans(const void* k, const void* v, const void* metric, const void* probes, void* k_rep,
                              void* v_rep, float* log_counts, void* k_mean, void* v_mean, int32_t L, int32_t H,
                              int32_t iters, void* stream) {
    if (!k || !v || !metric || !probes || !k_rep || !v_rep || !log_counts)
        return set_error(-1, "es_reps_kmeans: null pointer");
    if (L <= 0 || H <= 0) return set_error(-1, "es_reps_kmeans: L and H must be positive");
    if (!aligned(16, k, v, metric)) return set_error(-1, "es_reps_kmeans: k, v and metric must be 16-byte aligned");
    if (!aligned(4, probes, k_rep, v_rep, k_mean, v_mean)) return set_error(-1, "es_reps_kmeans: probes, tables and means must be 4-byte aligned");
    if ((k_mean == nullptr) != (v_mean == nullptr)) return set_error(-1, "es_reps_kmeans: give both means or neither");
    const int nb = (L + 63) / 64;
    if (int rc = opt_in_shared_memory((const void*)kmeans_kernel, KM_SMEM)) return rc;
    // kv blocks per CTA: KM_BLOCKS share one load of the head's metric; fewer when that would leave the GPU with only a
    // few waves of CTAs (a handful of heads per GPU), where the last, partly filled wave costs more than the reloads
    int per = KM_BLOCKS;
    while (per > 1 && (long long)((nb + per - 1) / per) * H < 8LL * 2 * 148) per >>= 1;
    kmeans_kernel<<<dim3((nb + per - 1) / per, H), 256, KM_SMEM, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, (const __nv_bfloat16*)metric, (const __nv_bfloat16*)probes,
        (__nv_bfloat16*)k_rep, (__nv_bfloat16*)v_rep, log_counts, (__nv_bfloat16*)k_mean, (__nv_bfloat16*)v_mean, L, H,
        (nb + 1) * 4, iters, per);
    ES_CHECK_LAUNCH("kmeans");
    return 0;
}

// ------------------------------------------------------------------------------------------------ no-allocation variant
// Scratch for es_reps_metric_static: room for ES_STATIC_GRAM_PARTS partial Gram matrices (128 x 128 floats each), held by
// every GPU that loads this library from load to exit.
#define ES_STATIC_GRAM_PARTS 256
static __device__ __align__(256) float g_static_gram_parts[ES_STATIC_GRAM_PARTS * HD * HD];

// Device address of the scratch array on the current device. In host code the array's name is only a handle for the
// runtime, not an address a kernel could use, so the address is asked for once per device (with that device current).
static float* static_gram_parts() {
    static float* ptrs[64] = {nullptr};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (!ptrs[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_static_gram_parts) != cudaSuccess) return nullptr;
        ptrs[dev] = static_cast<float*>(p);
    }
    return ptrs[dev];
}

extern "C" int es_reps_metric_static_max_heads(void) { return ES_STATIC_GRAM_PARTS; }

extern "C" int es_reps_metric_static(const void* q, float* gram, void* metric, void* probes, int32_t L, int32_t H,
                                     void* stream) {
    if (!q || !metric || !probes) return set_error(-1, "es_reps_metric_static: null pointer");
    if (L <= 0 || H <= 0) return set_error(-1, "es_reps_metric_static: L and H must be positive");
    if (!aligned(16, q, metric)) return set_error(-1, "es_reps_metric_static: q and metric must be 16-byte aligned");
    if (H > ES_STATIC_GRAM_PARTS)
        return set_error(-1, "es_reps_metric_static: more than 256 heads do not fit the built-in scratch; use es_reps_metric");
    float* parts = static_gram_parts();
    if (!parts) return set_error(-2, "es_reps_metric_static: the address of the built-in scratch is not available");
    // as many row splits as the scratch holds for this head count (at most the usual number)
    int nsplit = ES_STATIC_GRAM_PARTS / H;
    const int usual = es_reps_gram_splits(L);
    if (nsplit > usual) nsplit = usual;
    const int rps = (((L + nsplit - 1) / nsplit + 63) / 64) * 64;
    nsplit = (L + rps - 1) / rps;
    cudaStream_t st = (cudaStream_t)stream;
    if (int rc = launch_gram(q, parts, L, H, rps, nsplit, st)) return rc;
    const int smem = METRIC_SMEM;
    if (int rc = opt_in_shared_memory((const void*)metric_kernel, smem)) return rc;
    const float scale = 1.0f / sqrtf((float)HD);
    gram_reduce_kernel<<<dim3(H, HD * HD / 1024), 256, 0, st>>>(parts, nsplit, scale * scale / (float)L);
    ES_CHECK_LAUNCH("gram_reduce");
    metric_kernel<<<H + NP / PROBES_PER_CTA * H, 256, smem, st>>>(parts, (__nv_bfloat16*)metric, gram, nsplit, (const __nv_bfloat16*)q,
                                                                  (__nv_bfloat16*)probes, L, H, scale);
    ES_CHECK_LAUNCH("metric");
    return 0;
}
