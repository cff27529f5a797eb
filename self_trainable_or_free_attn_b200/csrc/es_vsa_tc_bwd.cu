// VSA2 backward on the 5th-generation tensor cores: one kernel for both passes, one CTA per owner block (64 tokens) walking
// the blocks of its list two at a time. No atomics: every output row has one owner, so results are reproducible bit for bit.
// Conventions: es_vsa_tc_fwd.cu; padded rows receive zero gradient. The coarse branch runs here too.
//
// With X1, X2 the walked tiles (128 rows: two blocks; one at the end of an odd list) and Y1, Y2 the owner's (64 rows):
//   dK / dV pass (KV = true):  X1 = Q, X2 = dO, Y1 = K, Y2 = V, rows are queries, columns are the owner's keys
//   dQ pass     (KV = false):  X1 = K, X2 = V,  Y1 = Q, Y2 = dO, rows are keys, columns are the owner's queries
//   S = X1 Y1^T, dP = X2 Y2^T (128 x 64), P = exp(scale S - lse), dS = P (dP - delta)
//   G1^T (d x 64) += X1^T dS  (dK or dQ),   G2^T (d x 64) += X2^T P  (dV, only in the dK / dV pass)
// Both kinds of product have 64 columns; M is the 128 walked rows, then the head dimension. That makes P and dS operands with
// 64 contiguous columns per row, which is what a thread of the accumulator's layout holds (half a row each), and the owner's
// gradient the accumulator, kept in tensor memory over the whole list. (Rows and columns the other way round, S would be an
// M = 64 product, which uses half of the tensor pipe.)
//
//   warps 0-7  P and dS: warp w owns rows 32 (w % 4) .. + 31 and columns 32 (w / 4) .. + 31
//   warp 8     issues the MMAs; warp 9 issues the TMA loads
// Tensor memory: (S, dP) of even and of odd iterations (4 x 64 columns), G1^T, G2^T (2 x 64). S and dP of iteration i + 1 are
// computed while the warps work on iteration i. X tiles (32 KB at D = 128) go through a ring of five slots (ten at D = 64).
//
// What bounds it: shared memory. At D = 128 the MMAs read 96 KB per pair of blocks (72 KB in the dQ pass) and the loads fill 32
// KB, 1,000 (830) clocks at 128 B/clock; the ring's five slots leave the X2 tile of the next iteration half an iteration of
// lead. 32,768 tokens x 12 heads, 32 blocks per list: dK / dV 1.20 ms, dQ 1.09 ms (mma.sync: 2.27 and 1.68 ms); at D = 64 0.94
// and 0.78 ms (1.29 and 0.91 ms), where M = D = 64 gradient products take half of the tensor pipe.
#include "es_vsa_tc.cuh"

namespace es {
namespace vsa {

namespace {
constexpr int TB = 64;
constexpr float kLog2e = 1.4426950408889634f;
constexpr int BW_THREADS = 320;
constexpr uint32_t Y_HALF = TB * 128, X_HALF = 128 * 128;                // 64 d of an owner / a walked tile
constexpr uint32_t DS_BYTES = 128 * 128;                                 // P, dS: [128 rows][64 columns] 16-bit
template <int D, bool KV> struct BwdCfg {
    static constexpr int DH = D / 64, NSLOT = D == 128 ? 5 : 10;
    static constexpr uint32_t Y_TILE = DH * Y_HALF, X_TILE = DH * X_HALF;   // [d half][rows][128 B]
    static constexpr uint32_t Y1 = 0, Y2 = Y_TILE, DS = 2 * Y_TILE, P = DS + DS_BYTES;
    static constexpr uint32_t RING = P + (KV ? DS_BYTES : 0u), CTL = RING + NSLOT * X_TILE, BYTES = CTL + 1024;
    static constexpr int LD = D + 4;                                     // epilogue staging: floats per token row
};

struct BwdCtl {
    uint64_t yfull, full[10], empty[10], sfull[2], pfull, pvdone, drain;
    uint32_t tmem_base;
    int abort;
    alignas(16) float lse2[TB], delta[TB];       // dQ pass: the owner's rows
};
static_assert(sizeof(BwdCtl) <= 1024, "control block");

struct BwdTcArgs {
    const float *lse, *delta;
    void *d0, *d1;                 // dK, dV / dQ, unused
    float *f0, *f1;                // fp32 outputs instead, when not null
    const float *add0, *add1;      // optional per-block gradients [BH, add_nb, D], added as add / count to every valid token
    int add_nb;
    const int *row_ptr, *col_idx, *blk_cnt;
    int L, NB;
    int rows;                      // coarse branch (no lists, row_ptr null): real rows of the sequence, the rest of L is padding
    float scale, scale_log2;
    // Split-KV task mode over the walked lists (es_vsa_tc_fwd.cu): slot >= 0 writes fp32 partial gradients to part0 / part1
    // [slot] [64, D] without the per-block add (the merge adds it once and zeroes the padded rows).
    const int *tasks, *task_info;
    float *part0, *part1;
    int* status;
    int wide;                      // every output pointer is 16-byte aligned
};

__device__ __forceinline__ void store4(float* dst, float4 v, int wide) {
    if (wide) {
        *reinterpret_cast<float4*>(dst) = v;
    } else {
        reinterpret_cast<float2*>(dst)[0] = make_float2(v.x, v.y);
        reinterpret_cast<float2*>(dst)[1] = make_float2(v.z, v.w);
    }
}
}  // namespace

template <typename T, int D, bool KV>
__global__ void __launch_bounds__(BW_THREADS, 1)
attn_bwd_tc_kernel(const __grid_constant__ CUtensorMap tmX1, const __grid_constant__ CUtensorMap tmX2,
                   const __grid_constant__ CUtensorMap tmY1, const __grid_constant__ CUtensorMap tmY2, const BwdTcArgs a) {
    using C = BwdCfg<D, KV>;
    constexpr int NSLOT = C::NSLOT, DH = C::DH;
    constexpr uint32_t Y_TILE = C::Y_TILE, X_TILE = C::X_TILE;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int ob, bh, beg, end, slot_out;
    if (a.tasks) {
        if ((int)blockIdx.x >= a.task_info[0]) return;
        const int4 t = reinterpret_cast<const int4*>(a.tasks)[blockIdx.x];
        bh = t.x / a.NB; ob = t.x - bh * a.NB; beg = t.y; end = t.z; slot_out = t.w;
    } else {
        ob = blockIdx.x; bh = blockIdx.y; slot_out = -1;
        beg = a.row_ptr ? a.row_ptr[(size_t)bh * (a.NB + 1) + ob] : 0;
        end = a.row_ptr ? a.row_ptr[(size_t)bh * (a.NB + 1) + ob + 1] : a.NB;
    }
    auto block_at = [&](int e) { return a.col_idx ? __ldg(a.col_idx + beg + e) : e; };
    auto tokens_of = [&](int j) { return a.blk_cnt ? __ldg(a.blk_cnt + j) : min(TB, a.rows - TB * j); };
    const int n = end - beg, nt = (n + 1) >> 1;
    const uint32_t base = smem_u32(smem);
    BwdCtl* ctl = reinterpret_cast<BwdCtl*>(smem + C::CTL);
    volatile int* abort_flag = &ctl->abort;
    const int row0 = bh * a.L;                               // first row of this (b, h) in the [BH L, D] view
    const int cnt_o = tokens_of(ob);
    if (tid == 0) {
        mbar_init(smem_u32(&ctl->yfull), 1);
        for (int i = 0; i < NSLOT; ++i) {
            mbar_init(smem_u32(&ctl->full[i]), 1);
            mbar_init(smem_u32(&ctl->empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&ctl->sfull[i]), 1);
        mbar_init(smem_u32(&ctl->pfull), 256);
        mbar_init(smem_u32(&ctl->pvdone), 1);
        mbar_init(smem_u32(&ctl->drain), 1);
        ctl->abort = (base & 1023u) ? 1 : 0;                 // the swizzled tiles need a 1024-byte aligned base
        if (base & 1023u) atomicCAS(a.status, 0, 903);
        mbar_fence_init();
        fence_proxy_async_smem();
    }
    if (!KV && tid >= 64 && tid < 128) {
        const int r = tid - 64;
        const size_t g = (size_t)row0 + (size_t)ob * TB + r;
        const float l = a.lse[g];
        // an offset of +inf makes P of a padded or empty query 0
        ctl->lse2[r] = r < cnt_o && l != -INFINITY ? l * kLog2e : INFINITY;
        ctl->delta[r] = a.delta[g];
    }
    if (warp == 8) {
        tmem_alloc(smem_u32(&ctl->tmem_base), 512);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    constexpr uint32_t G1 = 256, G2 = 320;                   // accumulator columns
    const uint32_t full0 = smem_u32(&ctl->full[0]), empty0 = smem_u32(&ctl->empty[0]);
    uint32_t pseq = 0;                                       // load warp: tiles issued

    if (warp == 9) {
        // ------------------------------------------------------------ loads: Y1, Y2, then X1(i), X2(i)
        bool ok = *abort_flag == 0;
        if (ok && nt > 0) {
            if (lane == 0) {
                tma_prefetch_desc(&tmX1);
                tma_prefetch_desc(&tmX2);
                mbar_arrive_expect_tx(smem_u32(&ctl->yfull), 2 * Y_TILE);
                for (int d = 0; d < DH; ++d) {
                    tma_load_2d(base + C::Y1 + d * Y_HALF, &tmY1, smem_u32(&ctl->yfull), 64 * d, row0 + ob * TB);
                    tma_load_2d(base + C::Y2 + d * Y_HALF, &tmY2, smem_u32(&ctl->yfull), 64 * d, row0 + ob * TB);
                }
            }
            int win = lane < n ? block_at(lane) : 0;          // a window of 32 list entries
            uint32_t slot = 0, par = 1;
            for (int i = 0; i < nt && ok; ++i) {
                const int e = 2 * i;
                if (e > 0 && (e & 31) == 0) win = e + lane < n ? block_at(e + lane) : 0;
                const int j0 = __shfl_sync(0xffffffffu, win, e & 31), j1 = __shfl_sync(0xffffffffu, win, (e + 1) & 31);
                const int nb = e + 1 < n ? 2 : 1;
#pragma unroll 1
                for (int x = 0; x < 2; ++x) {
                    if (lane == 0) ok = mbar_wait(empty0 + 8 * slot, par, abort_flag, a.status, 501);
                    ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
                    if (!ok) break;
                    if (lane == 0) mbar_arrive_expect_tx(full0 + 8 * slot, nb * Y_TILE);
                    __syncwarp();
                    // the d halves of the first block, then of the second
                    if (lane < DH * nb) {
                        const int d = lane % DH, b = lane / DH;
                        tma_load_2d(base + C::RING + slot * X_TILE + d * X_HALF + b * Y_HALF, x ? &tmX2 : &tmX1,
                                    full0 + 8 * slot, 64 * d, row0 + (b ? j1 : j0) * TB);
                    }
                    __syncwarp();
                    ++pseq;
                    if (++slot == NSLOT) { slot = 0; par ^= 1; }
                }
            }
        }
    } else if (warp == 8) {
        // ------------------------------------------------------------ MMAs
        constexpr uint32_t ID_S = umma_idesc<T>(128, TB, 0, 0);       // walked rows x owner rows, both K-major
        constexpr uint32_t ID_G = umma_idesc<T>(D, TB, 1, 1);         // d x owner rows: both operands MN-major
        const uint64_t dk0 = umma_desc_sw128(0, 16, 1024), dx0 = umma_desc_sw128(0, X_HALF, 1024);
        const uint32_t k_hi = (uint32_t)(dk0 >> 32), k_lo = (uint32_t)dk0, x_hi = (uint32_t)(dx0 >> 32), x_lo = (uint32_t)dx0;
        bool ok = *abort_flag == 0;
        if (nt > 0) ok = ok && mbar_wait_warp(smem_u32(&ctl->yfull), 0, abort_flag, a.status, 502);
        // tile number s of the ring sits in slot s % NSLOT, its full barrier in phase (s / NSLOT) & 1
        auto issue_s = [&](int i) {
#pragma unroll 1
            for (int x = 0; x < 2; ++x) {
                const uint32_t seq = 2 * i + x, s = seq % NSLOT;
                ok = ok && mbar_wait_warp(full0 + 8 * s, (seq / NSLOT) & 1, abort_flag, a.status, 503);
                if (!ok) return;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t xa = k_lo + ((base + C::RING + s * X_TILE) >> 4);
                    const uint32_t yb = k_lo + ((base + (x ? C::Y2 : C::Y1)) >> 4);
                    const uint32_t d = tmem + (i & 1) * 128 + x * 64;
#pragma unroll
                    for (int ks = 0; ks < D / 16; ++ks)
                        umma_ss_lohi(d, xa + (((ks >> 2) * X_HALF + (ks & 3) * 32) >> 4), k_hi,
                                     yb + (((ks >> 2) * Y_HALF + (ks & 3) * 32) >> 4), k_hi, ID_S, ks > 0);
                    if (!KV && x == 1) umma_commit(empty0 + 8 * s);   // the dQ pass needs V no more
                    if (x == 1) umma_commit(smem_u32(&ctl->sfull[i & 1]));
                }
                __syncwarp();
            }
        };
        if (nt > 0 && ok) issue_s(0);
        for (int i = 0; i < nt && ok; ++i) {
            if (i + 1 < nt) issue_s(i + 1);       // its S / dP columns were read before P and dS of iteration i - 1 were stored
            ok = ok && mbar_wait_warp(smem_u32(&ctl->pfull), i & 1, abort_flag, a.status, 504);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const int ksteps = 2 * i + 1 < n ? 8 : 4;      // an odd end has 64 rows: the other half of the slot is stale
#pragma unroll 1
                for (int x = 0; x < (KV ? 2 : 1); ++x) {
                    const uint32_t s = (uint32_t)(2 * i + x) % NSLOT;
                    const uint32_t xa = x_lo + ((base + C::RING + s * X_TILE) >> 4);
                    const uint32_t pb = k_lo + ((base + (x ? C::P : C::DS)) >> 4);
                    for (int ks = 0; ks < ksteps; ++ks)
                        umma_ss_lohi(tmem + (x ? G2 : G1), xa + ((ks * 2048) >> 4), x_hi, pb + ((ks * 2048) >> 4), k_hi, ID_G,
                                     (i > 0 || ks > 0) ? 1u : 0u);
                    umma_commit(empty0 + 8 * s);
                }
                umma_commit(smem_u32(&ctl->pvdone));
            }
            __syncwarp();
        }
        // every MMA issued above has finished before tensor memory is freed
        if (elect_one()) umma_commit(smem_u32(&ctl->drain));
        __syncwarp();
        mbar_wait(smem_u32(&ctl->drain), 0, abort_flag, a.status, 505);
    } else {
        // ------------------------------------------------------------ P, dS and epilogue
        const int rq = warp & 3, ch = warp >> 2;
        const int r = 32 * rq + lane;                        // row of the walked tile
        const uint32_t tw = tmem + ((uint32_t)(32 * rq) << 16);
        const uint32_t prow = base + r * 128, psw = r & 7;
        bool ok = *abort_flag == 0;
        // the walked row's block, and in the dK / dV pass its offset and delta, one iteration ahead
        auto fetch = [&](int i, bool& valid, float& off, float& dl) {
            const int e = 2 * i + (r >> 6);
            valid = e < n;
            off = dl = 0.f;
            if (!valid) return;
            const int j = block_at(e);
            valid = (r & 63) < tokens_of(j);
            if (KV) {
                const size_t g = (size_t)row0 + (size_t)j * TB + (r & 63);
                const float l = __ldg(a.lse + g);
                valid = valid && l != -INFINITY;
                off = -l * kLog2e;
                dl = __ldg(a.delta + g);
            }
        };
        bool nv = false;
        float noff = 0.f, ndl = 0.f;
        if (nt > 0) fetch(0, nv, noff, ndl);
        for (int i = 0; i < nt && ok; ++i) {
            const bool valid = nv;
            const float off = noff, dl = ndl;
            if (i + 1 < nt) fetch(i + 1, nv, noff, ndl);
            ok = mbar_wait_warp(smem_u32(&ctl->sfull[i & 1]), (i >> 1) & 1, abort_flag, a.status, 506);
            if (!ok) break;
            tc_fence_after();
            uint32_t s[32], dp[32];
            tmem_ld32(tw + (i & 1) * 128 + 32 * ch, s);
            tmem_ld32(tw + (i & 1) * 128 + 64 + 32 * ch, dp);
            tmem_wait_ld();
            uint32_t pk[16], dk[16];
            const float2 sc = make_float2(a.scale_log2, a.scale_log2);
            const float4* lse4 = reinterpret_cast<const float4*>(ctl->lse2 + 32 * ch);
            const float4* dl4 = reinterpret_cast<const float4*>(ctl->delta + 32 * ch);
#pragma unroll
            for (int c4 = 0; c4 < 8; ++c4) {
                float4 o4 = make_float4(off, off, off, off), d4 = make_float4(dl, dl, dl, dl);
                if (!KV) {
                    o4 = lse4[c4];
                    o4 = make_float4(-o4.x, -o4.y, -o4.z, -o4.w);
                    d4 = dl4[c4];
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = 4 * c4 + 2 * h;
                    const float2 x = __ffma2_rn(make_float2(__uint_as_float(s[c]), __uint_as_float(s[c + 1])), sc,
                                                h ? make_float2(o4.z, o4.w) : make_float2(o4.x, o4.y));
                    float2 p = make_float2(ex2_approx(x.x), ex2_approx(x.y));
                    // rows without a query / key are 0; a padded column only reaches its own (zeroed) gradient row
                    p.x = valid ? p.x : 0.f;
                    p.y = valid ? p.y : 0.f;
                    const float2 g = make_float2(__uint_as_float(dp[c]) - (h ? d4.z : d4.x),
                                                 __uint_as_float(dp[c + 1]) - (h ? d4.w : d4.y));
                    const float gx = p.x * g.x, gy = p.y * g.y;
                    if (KV) pk[c / 2] = pack2<T>(p.x, p.y);
                    dk[c / 2] = pack2<T>(valid ? gx : 0.f, valid ? gy : 0.f);
                }
            }
            if (i > 0) {
                // the products of iteration i - 1 have read the previous P and dS
                ok = mbar_wait_warp(smem_u32(&ctl->pvdone), (i - 1) & 1, abort_flag, a.status, 507);
                if (!ok) break;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t sw = ((uint32_t)(4 * ch + j) ^ psw) << 4;
                st_shared16(prow + C::DS + sw, dk[4 * j], dk[4 * j + 1], dk[4 * j + 2], dk[4 * j + 3]);
                if (KV) st_shared16(prow + C::P + sw, pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
            }
            tc_fence_before();
            fence_proxy_async_smem();
            mbar_arrive(smem_u32(&ctl->pfull));
        }
        if (nt > 0) ok = ok && mbar_wait_warp(smem_u32(&ctl->pvdone), (nt - 1) & 1, abort_flag, a.status, 508);
        // all products have finished and every load has been consumed: the ring holds the transposed gradients now,
        // [64 tokens][LD] floats each
        tc_fence_after();
        float* stage = reinterpret_cast<float*>(smem + C::RING);
#pragma unroll
        for (int x = 0; x < (KV ? 2 : 1); ++x) {
            uint32_t g[32];
#pragma unroll
            for (int c = 0; c < 32; ++c) g[c] = 0;
            float* dst = stage + x * TB * C::LD + (32 * ch) * C::LD;
            if (D == 128) {
                if (nt > 0) {
                    tmem_ld32(tw + (x ? G2 : G1) + 32 * ch, g);
                    tmem_wait_ld_regs(g);
                }
#pragma unroll
                for (int c = 0; c < 32; ++c) dst[c * C::LD + r] = __uint_as_float(g[c]);     // lane r is head dimension r
            } else {
                // an M = 64 accumulator: 16 rows of head dimensions per warp, see tmem_ld_16x64
                if (nt > 0) {
                    tmem_ld_16x32(tw + (x ? G2 : G1) + 32 * ch, g);
                    tmem_wait_ld_regs(g);
                }
                const int d = 16 * rq + (lane >> 2), c0 = 2 * (lane & 3);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    dst[(8 * j + c0) * C::LD + d] = __uint_as_float(g[4 * j]);
                    dst[(8 * j + c0 + 1) * C::LD + d] = __uint_as_float(g[4 * j + 1]);
                    dst[(8 * j + c0) * C::LD + d + 8] = __uint_as_float(g[4 * j + 2]);
                    dst[(8 * j + c0 + 1) * C::LD + d + 8] = __uint_as_float(g[4 * j + 3]);
                }
            }
        }
        tc_fence_before();
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const float inv = 1.f / (float)cnt_o;
#pragma unroll
        for (int x = 0; x < (KV ? 2 : 1); ++x) {
            const float mul = x ? 1.f : a.scale;
            const float* add = x ? a.add1 : a.add0;
            const int d = 4 * (lane % (D / 4));                  // D / 4 lanes share a token
            float4 ad = make_float4(0.f, 0.f, 0.f, 0.f);
            if (add && slot_out < 0) {
                const float* src = add + ((size_t)bh * a.add_nb + ob) * D + d;
                ad = make_float4(__ldg(src), __ldg(src + 1), __ldg(src + 2), __ldg(src + 3));
                ad.x *= inv; ad.y *= inv; ad.z *= inv; ad.w *= inv;
            }
            float* part = x ? a.part1 : a.part0;
            float* f = x ? a.f1 : a.f0;
            T* e = static_cast<T*>(x ? a.d1 : a.d0);
            if (!ok) continue;
#pragma unroll
            for (int t = warp * (128 / D) + lane / (D / 4); t < TB; t += 8 * (128 / D)) {
                float4 v = *reinterpret_cast<const float4*>(stage + x * TB * C::LD + t * C::LD + d);
                v.x *= mul; v.y *= mul; v.z *= mul; v.w *= mul;
                if (slot_out >= 0) {
                    store4(part + ((size_t)slot_out * TB + t) * D + d, v, a.wide);
                    continue;
                }
                v.x += ad.x; v.y += ad.y; v.z += ad.z; v.w += ad.w;
                if (t >= cnt_o) v = make_float4(0.f, 0.f, 0.f, 0.f);
                const size_t g = ((size_t)row0 + (size_t)ob * TB + t) * D + d;
                if (f) {
                    store4(f + g, v, a.wide);
                } else {
                    const uint32_t w0 = pack2<T>(v.x, v.y), w1 = pack2<T>(v.z, v.w);
                    uint32_t* dst = reinterpret_cast<uint32_t*>(e + g);
                    if (a.wide) *reinterpret_cast<uint2*>(dst) = make_uint2(w0, w1);
                    else { dst[0] = w0; dst[1] = w1; }
                }
            }
        }
    }

    // ---------------------------------------------------------------- teardown
    __syncwarp();
    if (warp == 9 && lane == 0 && *abort_flag) {
        // a wait gave up: give the loads of this warp a moment (100 us in all) to land before shared memory goes away
        const uint64_t t_end = global_timer_ns() + 100000ull;
        for (uint32_t back = 1; back <= (uint32_t)NSLOT && back <= pseq; ++back) {
            const uint32_t sq = pseq - back;
            while (!mbar_try_wait(full0 + 8 * (sq % NSLOT), (sq / NSLOT) & 1) && global_timer_ns() < t_end) {}
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <typename T, int D, bool KV>
static int launch_bwd(const void* x1, const void* x2, const void* y1, const void* y2, const BwdTcArgs& a, int BH, dim3 grid,
                      cudaStream_t st) {
    CUtensorMap t[4];
    const void* p[4] = {x1, x2, y1, y2};
    for (int i = 0; i < 4; ++i)
        if (int rc = make_token_map<T>(&t[i], p[i], D, (long long)BH * a.L)) return rc;
    auto kern = attn_bwd_tc_kernel<T, D, KV>;
    if (int rc = opt_in_shared_memory((const void*)kern, (int)BwdCfg<D, KV>::BYTES)) return rc;
    kern<<<grid, BW_THREADS, BwdCfg<D, KV>::BYTES, st>>>(t[0], t[1], t[2], t[3], a);
    ES_CHECK_LAUNCH("attn_bwd_tc_kernel");
    return 0;
}

template <bool KV>
static int dispatch_bwd(const void* x1, const void* x2, const void* y1, const void* y2, const BwdTcArgs& a, int BH, int D,
                        int dtype, dim3 grid, cudaStream_t st) {
    if (D == 128)
        return dtype == 0 ? launch_bwd<__nv_bfloat16, 128, KV>(x1, x2, y1, y2, a, BH, grid, st)
                          : launch_bwd<__half, 128, KV>(x1, x2, y1, y2, a, BH, grid, st);
    return dtype == 0 ? launch_bwd<__nv_bfloat16, 64, KV>(x1, x2, y1, y2, a, BH, grid, st)
                      : launch_bwd<__half, 64, KV>(x1, x2, y1, y2, a, BH, grid, st);
}

// The caller has checked the pointers and sizes (D = 64 or 128). kv: the dK / dV pass (out0 = dK, out1 = dV), else the dQ pass
// (out0 = dQ). tasks == nullptr: one CTA per (owner block, bh). row_ptr and tasks null: every block with every block, the
// sequence's real rows are `rows`.
int attn_bwd_tc(bool kv, const void* q, const void* k, const void* v, const void* dout, const float* lse, const float* delta,
                void* out0, void* out1, float* f0, float* f1, const float* add0, const float* add1, int add_nb,
                const int* row_ptr, const int* col_idx, const int* blk_cnt, int BH, int L, int rows, int D, int dtype, const int* tasks,
                const int* task_info, int n_tasks, float* part0, float* part1, cudaStream_t st) {
    int* status = device_status_ptr();
    if (!status) return set_error(-2, "attn_bwd_tc: the device status word is not available on this device");
    const float scale = 1.f / sqrtf((float)D);
    const int wide = (((uintptr_t)out0 | (uintptr_t)out1 | (uintptr_t)f0 | (uintptr_t)f1 | (uintptr_t)part0 | (uintptr_t)part1) & 15) == 0;
    const BwdTcArgs a{lse, delta, out0, out1, f0, f1, add0, add1, add_nb, row_ptr, col_idx, blk_cnt, L, L / TB, rows, scale,
                      kLog2e * scale, tasks, task_info, part0, part1, status, wide};
    const dim3 grid = tasks ? dim3(n_tasks, 1) : dim3(L / TB, BH);
    return kv ? dispatch_bwd<true>(q, dout, k, v, a, BH, D, dtype, grid, st)
              : dispatch_bwd<false>(k, v, q, dout, a, BH, D, dtype, grid, st);
}

}  // namespace vsa
}  // namespace es
