// VSA2 fine / coarse forward on the 5th-generation tensor cores: online-softmax attention of one 64-row query block over the
// 64-token kv blocks of its list, two CTAs per SM.
//
// Conventions (reference: csrc/vsa/vsa2_kernels.h:1-12 of shaoshitong/self_trainable_or_free_attn): token tensors [BH, L, D],
// L = NB * 64, blk_cnt [NB] valid tokens per block (valid tokens first); CSR row_ptr [BH * (NB + 1)] absolute offsets into
// col_idx; lse [BH, L] natural log, -inf for rows without a key and for padded rows, which output 0. The coarse branch runs
// here too (block means as a sequence of 64-row tiles with their own counts).
//
// An iteration covers two kv blocks (128 keys; one at the end of an odd list):
//   warps 0-3  softmax: warp w owns rows 16 w .. 16 w + 15 (an M = 64 accumulator sits in 16 lanes of each quarter)
//   warp 4     issues the MMAs; warp 5 issues the TMA loads
//   S (64 x 128) = Q K^T as two N = 64 products, one per kv block, and O (64 x D) += P V as four K = 16 steps per block;
//   Q, K, V and P all come from shared memory, S (columns 0-127) and O (128-255) live in tensor memory.
// S is read into registers at once and handed back, so QK of iteration i + 1 runs during the softmax of iteration i, and the
// other CTA of the SM fills what is left. A warp rescales its rows of O (64 registers through tensor memory) only in the
// iterations in which one of its maxima grew: a row's does in iteration i with a chance of 1 / i if its logits come in no order, one
// of sixteen rows in 85 % of the 16 iterations of a list of 32 blocks, in 67 % of those of 64 blocks. Waiting until a maximum has grown by a factor
// 256 is no faster and loses the exact P = 1 of a row's largest term (error against fp64 2.48e-3 instead of 2.40e-3). K and V
// blocks (16 KB each) go through one ring of five slots.
//
// What bounds it: shared memory. Per pair of a query and a kv block an SM fills 32 KB (256 clocks at 128 B/clock), the MMAs
// read 56 KB (448) and P is written once (64): 0.53 ms for the 196,608 pairs of 32,768 tokens x 12 heads at 32 blocks per list.
// Measured there, with the coarse branch's launch: 0.71 ms; the mma.sync kernel took 1.35 ms. Wan-1.3B 480p, 64 blocks per
// list: 1.49 ms, 3.10 ms before. D = 64 at the first shape: 0.51 ms, 0.74 ms before.
//
// TIER: the same walk over three tiers of resolution (es_vsa_tc.cuh), one softmax over all; a mean's column has the bias log2 of
// its tokens. K and V have a load warp each, with one copy of the code that finds and loads a unit: 512 blocks x 12 heads, 32 + 102
// blocks in tiers A and B of every query block, 1.25 ms (2.26 ms with that code inlined at six places, mma.sync 2.37 ms).
#include "es_vsa_tc.cuh"

namespace es {
namespace vsa {

namespace {
constexpr int TB = 64;
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
constexpr int FW_THREADS = 192, FW_THREADS_TIER = 224;

template <int D> struct FwdCfg {
    static constexpr uint32_t HALF = TB * 128;                   // 64 rows x 64 d: one TMA box
    static constexpr uint32_t TILE = TB * D * 2;                 // one block: [d half][64 rows][128 B]
    static constexpr int NSLOT = 5;
    static constexpr uint32_t Q = 0, P = TILE, RING = P + 2 * HALF, CTL = RING + NSLOT * TILE;
    static constexpr uint32_t COUNTS = CTL + 256;                // tiers: [UNIT_RING][64] bytes
    static constexpr uint32_t BYTES = CTL + 256, BYTES_TIER = COUNTS + UNIT_RING * TB;
};
struct FwdCtl {
    uint64_t qfull, full[5], empty[5], sfull, sfree, pfull, pvdone, drain;
    uint32_t tmem_base;
    int abort;
    int2 tiers;                    // tier-B and tier-C blocks of the query block
};
static_assert(sizeof(FwdCtl) <= 256, "control block");

struct FwdTcArgs {
    void* o;
    float* lse;
    const int *row_ptr, *col_idx, *blk_cnt;
    int L, NB;
    int rows;                      // coarse branch (no lists, row_ptr null): real rows of the sequence, the rest of L is padding
    float scale_log2;
    // Split-KV task mode (es_vsa_split_plan), all null in the plain (block, bh) grid: tasks[t] = {row = bh * NB + block,
    // first edge, one past the last edge, slot}; slot < 0 writes o / lse, slot >= 0 writes the fp32 normalised partial
    // part_o[slot] [64, D] and its log2-domain lse part_lse[slot] [64].
    const int* tasks;
    const int* task_info;
    float *part_o, *part_lse;
    int* status;
    TierMaps tier;
};
}  // namespace

template <typename T, int D, bool TIER>
__global__ void __launch_bounds__(TIER ? FW_THREADS_TIER : FW_THREADS, 2)
attn_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmKm,
                   const __grid_constant__ CUtensorMap tmVm, const __grid_constant__ CUtensorMap tmKt,
                   const __grid_constant__ CUtensorMap tmVt, const __grid_constant__ FwdTcArgs a) {
    using C = FwdCfg<D>;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int qb, bh, beg, end, slot_out;
    if (a.tasks) {
        if ((int)blockIdx.x >= a.task_info[0]) return;
        const int4 t = reinterpret_cast<const int4*>(a.tasks)[blockIdx.x];
        bh = t.x / a.NB; qb = t.x - bh * a.NB; beg = t.y; end = t.z; slot_out = t.w;
    } else {
        qb = blockIdx.x; bh = blockIdx.y; slot_out = -1;
        beg = a.row_ptr ? a.row_ptr[(size_t)bh * (a.NB + 1) + qb] : 0;
        end = a.row_ptr ? a.row_ptr[(size_t)bh * (a.NB + 1) + qb + 1] : a.NB;
    }
    auto block_at = [&](int e) { return a.col_idx ? __ldg(a.col_idx + beg + e) : e; };
    auto tokens_of = [&](int j) { return a.blk_cnt ? __ldg(a.blk_cnt + j) : min(TB, a.rows - TB * j); };
    const uint32_t base = smem_u32(smem);
    uint8_t* counts = smem + C::COUNTS;
    FwdCtl* ctl = reinterpret_cast<FwdCtl*>(smem + C::CTL);
    volatile int* abort_flag = &ctl->abort;
    if (tid == 0) {
        const int earlier = *reinterpret_cast<volatile int*>(a.status);      // (on its way during the set-up)
        mbar_init(smem_u32(&ctl->qfull), 1);
        for (int i = 0; i < C::NSLOT; ++i) {
            mbar_init(smem_u32(&ctl->full[i]), 1);
            mbar_init(smem_u32(&ctl->empty[i]), 1);
        }
        mbar_init(smem_u32(&ctl->sfull), 1);
        mbar_init(smem_u32(&ctl->sfree), 4);
        mbar_init(smem_u32(&ctl->pfull), 128);
        mbar_init(smem_u32(&ctl->pvdone), 1);
        mbar_init(smem_u32(&ctl->drain), 1);
        ctl->abort = (base & 1023u) || earlier ? 1 : 0;      // the swizzled tiles need a 1024-byte aligned base
        if (base & 1023u) atomicCAS(a.status, 0, 902);
        mbar_fence_init();
        fence_proxy_async_smem();
    }
    if (TIER && warp == 5) {
        const int2 t = tier_sizes(a.tier, bh, a.NB, qb, lane);
        if (lane == 0) ctl->tiers = t;
    }
    if (warp == 4) {
        tmem_alloc(smem_u32(&ctl->tmem_base), 256);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    // units of 64 columns: the list's blocks, then (tiers) gathered group means, then block means
    const int nA = TIER && !(a.tier.phases & PH_A) ? 0 : end - beg;
    const int nM = TIER ? nA + (ctl->tiers.x * a.tier.RM + TB - 1) / TB : nA;
    const int n = TIER ? nM + tail_units(a.tier, a.NB, ctl->tiers.y) : nM;
    const int nt = (n + 1) >> 1;
    const uint32_t full0 = smem_u32(&ctl->full[0]), empty0 = smem_u32(&ctl->empty[0]);
    const int row0 = bh * a.L;                               // first row of this (b, h) in the [BH L, D] view
    uint32_t pseq = 0;                                       // load warps: one past the last tile issued

    if (warp == 5 || (TIER && warp == 6)) {
        // ------------------------------------------------------------ loads: Q, K(0), then K(i + 1), V(i) for every i
        // Tile numbers in the ring are in the order of use. With tiers K and V have a warp each: a gathered unit is up to 64 small
        // boxes per tensor.
        const bool k_warp = warp == 5;
        bool ok = *abort_flag == 0;
        if (ok && nt > 0) {
            if (lane == 0) {
                tma_prefetch_desc(&tmK);
                tma_prefetch_desc(&tmV);
                if (k_warp) {
                    mbar_arrive_expect_tx(smem_u32(&ctl->qfull), C::TILE);
                    for (int d = 0; d < D / 64; ++d)
                        tma_load_2d(base + C::Q + d * C::HALF, &tmQ, smem_u32(&ctl->qfull), 64 * d, row0 + qb * TB);
                }
            }
            int kwin = lane < nA ? block_at(lane) : 0, kbase = 0;   // a window of 32 list entries per tensor
            int vwin = kwin, vbase = 0;
            uint32_t next_slot = 0, next_par = 1;
            TierWalk walk;
            if (TIER) walk.start(a.tier, bh, a.NB, qb, lane);
            auto put = [&](bool is_v, int& win, int& wbase, int e) {
                if (!ok || e >= n) return;
                // with one warp for both, the next slot; else the tile's number in the order of use
                const uint32_t seq = !TIER ? pseq : is_v ? e + min(n, (e & ~1) + 4) : e + max(0, (e & ~1) - 2);
                const uint32_t slot = TIER ? seq % C::NSLOT : next_slot, par = TIER ? ((seq / C::NSLOT) & 1) ^ 1 : next_par;
                int j = 0;
                int2 id = make_int2(-1, -1), tokens = make_int2(0, 0);
                if (!TIER || e < nA) {
                    if ((e & ~31) != wbase) {
                        wbase = e & ~31;
                        win = wbase + lane < nA ? block_at(wbase + lane) : 0;
                    }
                    j = __shfl_sync(0xffffffffu, win, e & 31);
                } else {
                    id = unit_blocks(walk, a.tier, bh, a.NB, qb, e < nM, e < nM ? e - nA : e - nM, lane);
                    if (!is_v) tokens = unit_tokens(a.blk_cnt, a.tier, bh, a.NB, qb, e < nM, id, e - nM, lane);
                }
                if (lane == 0) ok = mbar_wait(empty0 + 8 * slot, par, abort_flag, a.status, 401);
                ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
                if (!ok) return;
                const uint32_t dst = base + C::RING + slot * C::TILE, bar = full0 + 8 * slot;
                if (TIER && e >= nA) {
                    // the counts of unit e - 8 have been read: the tile whose ring slot this is belonged to V(i - 3), i = e / 2
                    if (!is_v) write_counts(counts + (e % UNIT_RING) * TB, tokens, a.tier.RM, e < nM, lane);
                    __syncwarp();
                    if (lane == 0) mbar_arrive_expect_tx(bar, C::TILE);
                    __syncwarp();
                    load_means<D / 64>(dst, C::HALF, is_v ? &tmVm : &tmKm, is_v ? &tmVt : &tmKt, bar, a.tier, bh, e < nM, id, e - nM, lane);
                } else if (lane == 0) {
                    mbar_arrive_expect_tx(bar, C::TILE);
#pragma unroll
                    for (int d = 0; d < D / 64; ++d) tma_load_2d(dst + d * C::HALF, is_v ? &tmV : &tmK, bar, 64 * d, row0 + j * TB);
                }
                __syncwarp();
                pseq = seq + 1;
                if (!TIER && ++next_slot == C::NSLOT) { next_slot = 0; next_par ^= 1; }
            };
            if (TIER) {
#pragma unroll 1
                for (int e = 0; e < n && ok; ++e) put(!k_warp, kwin, kbase, e);
            } else {
                put(false, kwin, kbase, 0);
                put(false, kwin, kbase, 1);
                for (int i = 0; i < nt; ++i) {
                    put(false, kwin, kbase, 2 * i + 2);
                    put(false, kwin, kbase, 2 * i + 3);
                    put(true, vwin, vbase, 2 * i);
                    put(true, vwin, vbase, 2 * i + 1);
                }
            }
        }
    } else if (warp == 4) {
        // ------------------------------------------------------------ MMAs
        constexpr uint32_t ID_QK = umma_idesc<T>(64, 64, 0, 0), ID_PV = umma_idesc<T>(64, D, 0, 1);
        const uint64_t dk0 = umma_desc_sw128(0, 16, 1024), dv0 = umma_desc_sw128(0, C::HALF, 1024);
        const uint32_t k_hi = (uint32_t)(dk0 >> 32), k_lo = (uint32_t)dk0, v_hi = (uint32_t)(dv0 >> 32), v_lo = (uint32_t)dv0;
        const uint32_t q_lo = k_lo + ((base + C::Q) >> 4), p_lo = k_lo + ((base + C::P) >> 4);
        uint32_t slot = 0, par = 0;
        bool ok = *abort_flag == 0;
        if (nt > 0) ok = ok && mbar_wait_warp(smem_u32(&ctl->qfull), 0, abort_flag, a.status, 402);
        auto take = [&]() -> uint32_t {
            const uint32_t s = slot;
            ok = ok && mbar_wait_warp(full0 + 8 * s, par, abort_flag, a.status, 403);
            if (++slot == C::NSLOT) { slot = 0; par ^= 1; }
            return s;
        };
        auto issue_qk = [&](int i) {
#pragma unroll 1
            for (int b = 0; b < 2; ++b) {
                if (2 * i + b >= n) break;
                const uint32_t s = take();
                if (!ok) return;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t kb = k_lo + ((base + C::RING + s * C::TILE) >> 4);
#pragma unroll
                    for (int ks = 0; ks < D / 16; ++ks) {
                        const uint32_t off = ((ks >> 2) * C::HALF + (ks & 3) * 32) >> 4;
                        umma_ss_lohi(tmem + 64 * b, q_lo + off, k_hi, kb + off, k_hi, ID_QK, ks > 0);
                    }
                    umma_commit(empty0 + 8 * s);
                }
                __syncwarp();
            }
            if (elect_one()) umma_commit(smem_u32(&ctl->sfull));
            __syncwarp();
        };
        if (nt > 0 && ok) issue_qk(0);
        for (int i = 0; i < nt && ok; ++i) {
            if (i + 1 < nt) {
                ok = mbar_wait_warp(smem_u32(&ctl->sfree), i & 1, abort_flag, a.status, 404);
                if (ok) issue_qk(i + 1);
                if (!ok) break;
            }
            ok = mbar_wait_warp(smem_u32(&ctl->pfull), i & 1, abort_flag, a.status, 405);
            if (!ok) break;
#pragma unroll 1
            for (int b = 0; b < 2; ++b) {
                if (2 * i + b >= n) break;
                const uint32_t s = take();
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t vb = v_lo + ((base + C::RING + s * C::TILE) >> 4), pb = p_lo + ((b * C::HALF) >> 4);
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)
                        umma_ss_lohi(tmem + 128, pb + ((ks * 32) >> 4), k_hi, vb + ((ks * 2048) >> 4), v_hi, ID_PV,
                                     (i > 0 || b > 0 || ks > 0) ? 1u : 0u);
                    umma_commit(empty0 + 8 * s);
                }
                __syncwarp();
            }
            if (!ok) break;
            if (elect_one()) umma_commit(smem_u32(&ctl->pvdone));
            __syncwarp();
        }
        // every MMA issued above has finished before tensor memory is freed
        if (elect_one()) umma_commit(smem_u32(&ctl->drain));
        __syncwarp();
        mbar_wait(smem_u32(&ctl->drain), 0, abort_flag, a.status, 406);
    } else {
        // ------------------------------------------------------------ softmax and epilogue
        const uint32_t tw = tmem + ((uint32_t)(32 * warp) << 16);
        const int cnt_q = tokens_of(qb);
        float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;      // offsets in use (log2) and row sums relative to them
        bool ok = *abort_flag == 0;
        // columns of unit e that are not masked here (the means' come with their biases below)
        auto width = [&](int e) { return e < nA ? tokens_of(block_at(e)) : e < n ? TB : 0; };
        int ca = width(0), cb = width(1);
        // stmatrix: lane l gives the address of row (l & 7) of 8 x 8 matrix l >> 3: (rows 0-7, 8-15) x (chunk 2 j, 2 j + 1)
        const int prow = 16 * warp + (lane & 7) + ((lane >> 3) & 1) * 8;
        const uint32_t paddr = base + C::P + prow * 128, psw = prow & 7, pch = lane >> 4;
        for (int i = 0; i < nt && ok; ++i) {
            const int cnt_a = ca, cnt_b = cb;
            ca = width(2 * i + 2);
            cb = width(2 * i + 3);
            ok = mbar_wait_warp(smem_u32(&ctl->sfull), i & 1, abort_flag, a.status, 407);
            if (!ok) break;
            tc_fence_after();
            uint32_t s[64];
            tmem_ld_16x64(tw, s);
            tmem_ld_16x64(tw + 64, s + 32);
            tmem_wait_ld_regs(s);
            tmem_wait_ld_regs(s + 32);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ctl->sfree));
            if ((cnt_a & cnt_b) != TB) {                     // (counts are 1 .. 64) a short block, or none: mask its keys
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int c = (j & 7) * 8 + 2 * (lane & 3), cnt = j < 8 ? cnt_a : cnt_b;
                    if (c >= cnt) s[4 * j] = s[4 * j + 2] = 0xff800000u;
                    if (c + 1 >= cnt) s[4 * j + 1] = s[4 * j + 3] = 0xff800000u;
                }
            }
            if (TIER) {
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int e = 2 * i + b;
                    if (e < nA || e >= n) continue;
                    const uint8_t* c8 = counts + (e % UNIT_RING) * TB + 2 * (lane & 3);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t cc = *reinterpret_cast<const uint16_t*>(c8 + 8 * j);
                        const float b0 = a.tier.bias[cc & 255u], b1 = a.tier.bias[cc >> 8];
                        uint32_t* x = s + 32 * b + 4 * j;
                        x[0] = __float_as_uint(__uint_as_float(x[0]) + b0);
                        x[1] = __float_as_uint(__uint_as_float(x[1]) + b1);
                        x[2] = __float_as_uint(__uint_as_float(x[2]) + b0);
                        x[3] = __float_as_uint(__uint_as_float(x[3]) + b1);
                    }
                }
            }
            float x0 = -INFINITY, x1 = -INFINITY;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                x0 = fmaxf(x0, fmaxf(__uint_as_float(s[4 * j]), __uint_as_float(s[4 * j + 1])));
                x1 = fmaxf(x1, fmaxf(__uint_as_float(s[4 * j + 2]), __uint_as_float(s[4 * j + 3])));
            }
            x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 1));
            x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 1));
            x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 2)) * a.scale_log2;
            x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 2)) * a.scale_log2;
            float al0 = 1.f, al1 = 1.f;
            const bool grow = __any_sync(0xffffffffu, x0 > m0 || x1 > m1);
            if (grow) {
                const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
                al0 = n0 == -INFINITY ? 0.f : ex2_approx(m0 - n0);
                al1 = n1 == -INFINITY ? 0.f : ex2_approx(m1 - n1);
                m0 = n0; m1 = n1;
            }
            const float o0 = m0 == -INFINITY ? 0.f : -m0, o1 = m1 == -INFINITY ? 0.f : -m1;
            const float2 sc = make_float2(a.scale_log2, a.scale_log2);
            float2 r0 = make_float2(0.f, 0.f), r1 = make_float2(0.f, 0.f);
            uint32_t p[32];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float2 y0 = __ffma2_rn(make_float2(__uint_as_float(s[4 * j]), __uint_as_float(s[4 * j + 1])), sc,
                                             make_float2(o0, o0));
                const float2 y1 = __ffma2_rn(make_float2(__uint_as_float(s[4 * j + 2]), __uint_as_float(s[4 * j + 3])), sc,
                                             make_float2(o1, o1));
                const float2 p0 = make_float2(ex2_approx(y0.x), ex2_approx(y0.y));
                const float2 p1 = make_float2(ex2_approx(y1.x), ex2_approx(y1.y));
                r0 = __fadd2_rn(r0, p0);
                r1 = __fadd2_rn(r1, p1);
                p[2 * j] = pack2<T>(p0.x, p0.y);
                p[2 * j + 1] = pack2<T>(p1.x, p1.y);
            }
            l0 = l0 * al0 + (r0.x + r0.y);
            l1 = l1 * al1 + (r1.x + r1.y);
            if (i > 0) {
                // PV(i - 1) has read the previous P and written O
                ok = mbar_wait_warp(smem_u32(&ctl->pvdone), (i - 1) & 1, abort_flag, a.status, 408);
                if (!ok) break;
                if (grow) {
                    tc_fence_after();
#pragma unroll
                    for (int h = 0; h < D / 64; ++h) {
                        tmem_ld_16x64(tw + 128 + 64 * h, s);
                        tmem_wait_ld_regs(s);
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            s[4 * j] = __float_as_uint(__uint_as_float(s[4 * j]) * al0);
                            s[4 * j + 1] = __float_as_uint(__uint_as_float(s[4 * j + 1]) * al0);
                            s[4 * j + 2] = __float_as_uint(__uint_as_float(s[4 * j + 2]) * al1);
                            s[4 * j + 3] = __float_as_uint(__uint_as_float(s[4 * j + 3]) * al1);
                        }
                        tmem_st_16x64(tw + 128 + 64 * h, s);
                    }
                    tmem_wait_st();
                    tc_fence_before();
                }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t ch = 2 * (j & 3) + pch;
                stsm4(paddr + (j >> 2) * C::HALF + ((ch ^ psw) << 4), p[4 * j], p[4 * j + 1], p[4 * j + 2], p[4 * j + 3]);
            }
            fence_proxy_async_smem();
            mbar_arrive(smem_u32(&ctl->pfull));
        }
        l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
        l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
        l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
        l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
        if (nt > 0) ok = ok && mbar_wait_warp(smem_u32(&ctl->pvdone), (nt - 1) & 1, abort_flag, a.status, 409);
        if (ok) {
            tc_fence_after();
            const int r0 = warp * 16 + (lane >> 2), r1 = r0 + 8;
            // a chunk of a split row writes every row (the merge masks the padded ones)
            const bool part = slot_out >= 0;
            // a row sum of 0 is a row without a key; one that is NaN (a NaN or infinite logit) stays NaN in O and in the LSE
            const bool ok0 = (part || r0 < cnt_q) && l0 != 0.f, ok1 = (part || r1 < cnt_q) && l1 != 0.f;
            const float i0 = ok0 ? 1.f / l0 : 0.f, i1 = ok1 ? 1.f / l1 : 0.f;
            T* out = static_cast<T*>(a.o) + ((size_t)row0 + (size_t)qb * TB) * D;
            float* po = part ? a.part_o + (size_t)slot_out * TB * D : nullptr;
#pragma unroll
            for (int h = 0; h < D / 64; ++h) {
                uint32_t o[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) o[j] = 0;
                if (nt > 0) {
                    tmem_ld_16x64(tw + 128 + 64 * h, o);
                    tmem_wait_ld_regs(o);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int c = 64 * h + j * 8 + 2 * (lane & 3);
                    // a row without a key, or a padded one, is 0 whatever its products hold
                    const float v0 = ok0 ? __uint_as_float(o[4 * j]) * i0 : 0.f, v1 = ok0 ? __uint_as_float(o[4 * j + 1]) * i0 : 0.f;
                    const float v2 = ok1 ? __uint_as_float(o[4 * j + 2]) * i1 : 0.f, v3 = ok1 ? __uint_as_float(o[4 * j + 3]) * i1 : 0.f;
                    if (part) {
                        *reinterpret_cast<float2*>(po + (size_t)r0 * D + c) = make_float2(v0, v1);
                        *reinterpret_cast<float2*>(po + (size_t)r1 * D + c) = make_float2(v2, v3);
                    } else {
                        *reinterpret_cast<uint32_t*>(out + (size_t)r0 * D + c) = pack2<T>(v0, v1);
                        *reinterpret_cast<uint32_t*>(out + (size_t)r1 * D + c) = pack2<T>(v2, v3);
                    }
                }
            }
            if ((lane & 3) == 0) {
                if (part) {
                    a.part_lse[(size_t)slot_out * TB + r0] = ok0 ? m0 + log2f(l0) : -INFINITY;
                    a.part_lse[(size_t)slot_out * TB + r1] = ok1 ? m1 + log2f(l1) : -INFINITY;
                } else {
                    float* lse = a.lse + (size_t)row0 + (size_t)qb * TB;
                    lse[r0] = ok0 ? (m0 + log2f(l0)) * kLn2 : -INFINITY;
                    lse[r1] = ok1 ? (m1 + log2f(l1)) * kLn2 : -INFINITY;
                }
            }
            tc_fence_before();
        }
    }

    // ---------------------------------------------------------------- teardown
    __syncwarp();
    if (warp >= 5 && lane == 0 && *abort_flag) {
        // a wait gave up: give the loads of this warp a moment (100 us in all) to land before shared memory goes away
        const uint64_t t_end = global_timer_ns() + 100000ull;
        for (uint32_t back = 1; back <= (uint32_t)C::NSLOT && back <= pseq; ++back) {
            const uint32_t sq = pseq - back;
            while (!mbar_try_wait(full0 + 8 * (sq % C::NSLOT), (sq / C::NSLOT) & 1) && global_timer_ns() < t_end) {}
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 4) {
        tc_fence_after();
        tmem_dealloc(tmem, 256);
    }
    if (*abort_flag) {
        const size_t row = slot_out >= 0 ? (size_t)slot_out * TB : (size_t)row0 + (size_t)qb * TB;
        if (slot_out >= 0) fill_nan(a.part_o + row * D, TB * D, kNaN32);
        else fill_nan(static_cast<T*>(a.o) + row * D, TB * D / 2, kNaN16x2);
        fill_nan((slot_out >= 0 ? a.part_lse : a.lse) + row, TB, kNaN32);
    }
}

template <typename T, int D>
static int launch_fwd(const void* q, const void* k, const void* v, FwdTcArgs a, int BH, dim3 grid, cudaStream_t st) {
    CUtensorMap tq, tk, tv;
    int rc;
    const long long rows = (long long)BH * a.L;
    if ((rc = make_token_map<T>(&tq, q, D, rows)) || (rc = make_token_map<T>(&tk, k, D, rows)) ||
        (rc = make_token_map<T>(&tv, v, D, rows)))
        return rc;
    auto kern = attn_fwd_tc_kernel<T, D, false>;
    if ((rc = opt_in_shared_memory((const void*)kern, (int)FwdCfg<D>::BYTES))) return rc;
    kern<<<grid, FW_THREADS, FwdCfg<D>::BYTES, st>>>(tq, tk, tv, tk, tv, tk, tv, a);
    ES_CHECK_LAUNCH("attn_fwd_tc_kernel");
    return 0;
}

// The caller has checked the pointers and sizes (D = 64 or 128). tasks == nullptr: one CTA per (query block, bh). row_ptr and
// tasks null: every block attends to every block, the sequence's real rows are `rows`.
int attn_fwd_tc(const void* q, const void* k, const void* v, void* o, float* lse, const int* row_ptr, const int* col_idx,
                const int* blk_cnt, int BH, int L, int rows, int D, int dtype, const int* tasks, const int* task_info, int n_tasks,
                float* part_o, float* part_lse, cudaStream_t st) {
    if (!aligned(4, o) || !aligned(8, part_o)) return set_error(-1, "attn_fwd_tc: o must be 4-byte, part_o 8-byte aligned");
    int* status = device_status_ptr();
    if (!status) return set_error(-2, "attn_fwd_tc: the device status word is not available on this device");
    const FwdTcArgs a{o, lse, row_ptr, col_idx, blk_cnt, L, L / TB, rows, kLog2e / sqrtf((float)D), tasks, task_info, part_o, part_lse, status, {}};
    const dim3 grid = tasks ? dim3(n_tasks, 1) : dim3(L / TB, BH);
    if (D == 64)
        return dtype == 0 ? launch_fwd<__nv_bfloat16, 64>(q, k, v, a, BH, grid, st) : launch_fwd<__half, 64>(q, k, v, a, BH, grid, st);
    return dtype == 0 ? launch_fwd<__nv_bfloat16, 128>(q, k, v, a, BH, grid, st) : launch_fwd<__half, 128>(q, k, v, a, BH, grid, st);
}

template <typename T, int D>
static int launch_tier_fwd(const void* q, const void* k, const void* v, const void* k_mid, const void* v_mid, const void* k_tail,
                           const void* v_tail, const FwdTcArgs& a, int BH, cudaStream_t st) {
    CUtensorMap t[7];
    const long long tok = (long long)BH * a.L, mid = (long long)BH * a.tier.mid_stride, tail = (long long)BH * a.tier.tail_stride;
    const void* p[7] = {q, k, v, k_mid, v_mid, k_tail, v_tail};
    const long long rows[7] = {tok, tok, tok, mid, mid, tail, tail};
    for (int i = 0; i < 7; ++i)
        if (int rc = make_token_map<T>(&t[i], p[i], D, rows[i], i >= 5 ? a.tier.tail_box() : i >= 3 ? a.tier.RM : TB)) return rc;
    auto kern = attn_fwd_tc_kernel<T, D, true>;
    if (int rc = opt_in_shared_memory((const void*)kern, (int)FwdCfg<D>::BYTES_TIER)) return rc;
    kern<<<dim3(a.NB, BH), FW_THREADS_TIER, FwdCfg<D>::BYTES_TIER, st>>>(t[0], t[1], t[2], t[3], t[4], t[5], t[6], a);
    ES_CHECK_LAUNCH("attn_fwd_tc_kernel");
    return 0;
}

// The three-tier forward; the caller has checked the pointers and sizes.
int tier_fwd_tc(const void* q, const void* k, const void* v, const void* k_mid, const void* v_mid, const void* k_tail,
                const void* v_tail, void* o, float* lse, const int* row_ptr, const int* col_idx, const TierMaps& tier,
                const int* blk_cnt, int BH, int L, int D, int dtype, cudaStream_t st) {
    if (!aligned(4, o)) return set_error(-1, "tier_fwd_tc: o must be 4-byte aligned");
    int* status = device_status_ptr();
    if (!status) return set_error(-2, "tier_fwd_tc: the device status word is not available on this device");
    FwdTcArgs a{o, lse, row_ptr, col_idx, blk_cnt, L, L / TB, 0, kLog2e / sqrtf((float)D), nullptr, nullptr, nullptr, nullptr,
                status, tier};
    a.tier.set_bias(a.scale_log2);                            // S is scaled after the bias has been added
    if (D == 64)
        return dtype == 0 ? launch_tier_fwd<__nv_bfloat16, 64>(q, k, v, k_mid, v_mid, k_tail, v_tail, a, BH, st)
                          : launch_tier_fwd<__half, 64>(q, k, v, k_mid, v_mid, k_tail, v_tail, a, BH, st);
    return dtype == 0 ? launch_tier_fwd<__nv_bfloat16, 128>(q, k, v, k_mid, v_mid, k_tail, v_tail, a, BH, st)
                      : launch_tier_fwd<__half, 128>(q, k, v, k_mid, v_mid, k_tail, v_tail, a, BH, st);
}

}  // namespace vsa
}  // namespace es
