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
//   warp 8     issues the MMAs; warps 9 and 10 issue the TMA loads (X1 and X2; warp 9 alone where they share a ring)
// Tensor memory: (S, dP) of even and of odd iterations (4 x 64 columns), G1^T, G2^T (2 x 64). S and dP of iteration i + 1 are
// computed while the warps work on iteration i. X1 and X2 tiles (32 KB at D = 128) have a ring each, of three and two slots (five
// and five at D = 64): the dQ passes free X2 as soon as dP has read it. Where the second products need both (dK / dV at D = 128),
// one ring of five in the order of use is 2 to 6 % faster.
//
// What bounds it: the hand-overs. The MMAs take 1,024 (768) clocks per two blocks at D = 128 and their operands 1,500 (1,150) of
// shared memory's, of 3,300 (2,400) measured: a tile's load, its products, P / dS and the second products follow one another
// with too few slots to have more than one and a half iterations on their way. 32,768 tokens x 12 heads, 32 random blocks
// per list, one launch after the other: dK / dV 1.12 ms, dQ 0.89 ms (mma.sync: 2.27 and 1.68 ms); at D = 64 0.84 and 0.71 ms (1.29 and
// 0.91 ms), where M = D = 64 gradient products take half of the tensor pipe. In a training step, with routed lists: 1.19 and 0.91 ms.
//
// BWD_TIER_Q, BWD_REP: the three tiers of resolution, see the modes below. 512 blocks x 12 heads, 32 + 102 blocks in tiers A and B:
// dQ 1.83 ms, tables 1.08 ms (mma.sync: 2.66 and 2.94 ms).
#include "es_vsa_tc.cuh"

namespace es {
namespace vsa {

namespace {
constexpr int TB = 64;
constexpr float kLog2e = 1.4426950408889634f;
constexpr uint32_t Y_HALF = TB * 128, X_HALF = 128 * 128;                // 64 d of an owner / a walked tile
constexpr int COUNT_RING = 16;                                           // units whose column counts are staged
constexpr int REP_WORDS = 4096 / 32;                                     // the entry points take up to 4096 blocks
constexpr uint32_t DS_BYTES = 128 * 128;                                 // P, dS: [128 rows][64 columns] 16-bit
// BWD_TIER_Q: the dQ pass over the units of all three tiers. BWD_REP: the dK / dV pass for 64 consecutive rows of a table of
// representatives (group means, then block means) as the owner; it walks the query blocks that use one of them, masked by the tier
// of each (query block, table row), and writes fp32 tables.
enum BwdMode { BWD_KV, BWD_Q, BWD_TIER_Q, BWD_REP };
template <int D, int MODE> struct BwdCfg {
    static constexpr bool KV = MODE == BWD_KV || MODE == BWD_REP;
    static constexpr int DH = D / 64, N1 = D == 128 ? 3 : 5, N2 = D == 128 ? 2 : 5;   // slots of X1 and of X2
    static constexpr bool SHARED = KV && D == 128;                       // one ring of N1 + N2 slots instead, filled by one warp
    static constexpr int THREADS = SHARED ? 320 : 352;
    static constexpr uint32_t Y_TILE = DH * Y_HALF, X_TILE = DH * X_HALF;   // [d half][rows][128 B]
    static constexpr uint32_t Y1 = 0, Y2 = Y_TILE, DS = 2 * Y_TILE, P = DS + DS_BYTES;
    static constexpr uint32_t RING = P + (KV ? DS_BYTES : 0u), CTL = RING + (N1 + N2) * X_TILE, COUNTS = CTL + 1024;
    // BWD_TIER_Q: column counts of the units; BWD_REP: a bit per query block
    static constexpr uint32_t BYTES = COUNTS + (MODE == BWD_TIER_Q ? COUNT_RING * TB : MODE == BWD_REP ? REP_WORDS * 4 : 0);
    static constexpr int LD = D + 4;                                     // epilogue staging: floats per token row
};

struct BwdCtl {
    uint64_t yfull, full[10], empty[10], sfull[2], pfull, pvdone, drain;
    uint32_t tmem_base;
    int abort;
    int2 tiers;                                  // BWD_TIER_Q: tier-B and tier-C blocks of the query block
    alignas(16) float lse2[TB], delta[TB];       // the owner's columns: minus their additive terms of the exponent; delta
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
    TierMaps tier;
    int wide;                      // every output pointer is 16-byte aligned
};

// The set bits of a bitmap in shared memory, ascending.
struct BitWalk {
    const uint32_t* words;
    int w;
    uint32_t bits;
    __device__ __forceinline__ BitWalk(const uint32_t* words_, bool any) : words(words_), w(0), bits(any ? words_[0] : 0u) {}
    __device__ __forceinline__ int next() {                  // the caller knows that there is one
        while (bits == 0) bits = words[++w];
        const int b = __ffs(bits) - 1;
        bits &= bits - 1;
        return 32 * w + b;
    }
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

template <typename T, int D, int MODE>
__global__ void __launch_bounds__((BwdCfg<D, MODE>::THREADS), 1)
attn_bwd_tc_kernel(const __grid_constant__ CUtensorMap tmX1, const __grid_constant__ CUtensorMap tmX2,
                   const __grid_constant__ CUtensorMap tmY1, const __grid_constant__ CUtensorMap tmY2,
                   const __grid_constant__ CUtensorMap tmM1, const __grid_constant__ CUtensorMap tmM2,
                   const __grid_constant__ CUtensorMap tmT1, const __grid_constant__ CUtensorMap tmT2, const __grid_constant__ BwdTcArgs a) {
    // tmM, tmT: tables of group and of block means, walked (BWD_TIER_Q; tmM in boxes of RM rows) or the owner (BWD_REP)
    constexpr bool TIER = MODE == BWD_TIER_Q, REP = MODE == BWD_REP;
    using C = BwdCfg<D, MODE>;
    constexpr bool KV = C::KV;
    constexpr int N1 = C::N1, N2 = C::N2, DH = C::DH;
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
        // BWD_REP: ob is a tile of 64 table rows
        beg = a.row_ptr ? a.row_ptr[(size_t)bh * (a.NB + 1) + ob] : 0;
        end = a.row_ptr ? a.row_ptr[(size_t)bh * (a.NB + 1) + ob + 1] : a.NB;
    }
    auto block_at = [&](int e) { return a.col_idx ? __ldg(a.col_idx + beg + e) : e; };
    auto tokens_of = [&](int j) { return a.blk_cnt ? __ldg(a.blk_cnt + j) : min(TB, a.rows - TB * j); };
    const uint32_t base = smem_u32(smem);
    BwdCtl* ctl = reinterpret_cast<BwdCtl*>(smem + C::CTL);
    volatile int* abort_flag = &ctl->abort;
    const int row0 = bh * a.L;                               // first row of this (b, h) in the [BH L, D] view
    uint8_t* counts = smem + C::COUNTS;
    uint32_t* use_words = reinterpret_cast<uint32_t*>(smem + C::COUNTS);
    // BWD_REP: the owner's table and tile in it, and the first block that the tile covers
    const int mid_tiles = REP && (a.tier.phases & PH_B) ? (a.NB * a.tier.RM + TB - 1) / TB : 0;
    const bool rep_mid = REP && ob < mid_tiles;
    const int rep_tile = rep_mid ? ob : ob - mid_tiles, rep_per = rep_mid ? TB / a.tier.RM : TB, rep_blk = rep_tile * rep_per;
    const int rep_row0 = REP ? bh * (rep_mid ? a.tier.mid_stride : a.tier.tail_stride) + rep_tile * TB : 0;
    const int cnt_o = REP ? min(TB, (rep_mid ? a.NB * a.tier.RM : a.NB) - rep_tile * TB) : tokens_of(ob);
    if (tid == 0) {
        const int earlier = *reinterpret_cast<volatile int*>(a.status);      // (on its way during the set-up)
        mbar_init(smem_u32(&ctl->yfull), 2);
        for (int i = 0; i < N1 + N2; ++i) {
            mbar_init(smem_u32(&ctl->full[i]), 1);
            mbar_init(smem_u32(&ctl->empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&ctl->sfull[i]), 1);
        mbar_init(smem_u32(&ctl->pfull), 256);
        mbar_init(smem_u32(&ctl->pvdone), 1);
        mbar_init(smem_u32(&ctl->drain), 1);
        ctl->abort = (base & 1023u) || earlier ? 1 : 0;      // the swizzled tiles need a 1024-byte aligned base
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
    if (REP && tid >= 64 && tid < 128) {
        // additive term of a table row: log2 of the tokens it stands for, -inf for none
        const int r = tid - 64, j = rep_blk + (rep_mid ? r / a.tier.RM : r), R = TB / a.tier.RM;
        int c = j < a.NB ? __ldg(a.blk_cnt + j) : 0;
        if (rep_mid) c = min(max(c - (r % a.tier.RM) * R, 0), R);
        ctl->lse2[r] = -a.tier.bias[c];
    }
    if (REP) {
        // bit i: query block i uses a row of this tile
        const uint32_t* bit_row = a.tier.bits_ab + (size_t)bh * a.NB * a.tier.W;
        const uint32_t* bit_row_a = a.tier.bits_a + (size_t)bh * a.NB * a.tier.W;
        const int w0 = rep_blk >> 5, left = a.NB - rep_blk;
        const uint32_t lo = left >= 32 ? 0xFFFFFFFFu : (1u << left) - 1u, hi = left >= 64 ? 0xFFFFFFFFu : left > 32 ? (1u << (left - 32)) - 1u : 0u;
        const uint32_t mid_mask = (rep_per >= 32 ? 0xFFFFFFFFu : (1u << rep_per) - 1u) & lo;
#pragma unroll 2
        for (int w = warp; w < a.tier.W; w += C::THREADS / 32) {
            const int i = 32 * w + lane;
            bool used = false;
            if (i < a.NB) {
                const size_t at = (size_t)i * a.tier.W + w0;
                const uint32_t ab = __ldg(bit_row + at);
                if (rep_mid) used = ((ab & ~__ldg(bit_row_a + at)) >> (rep_blk & 31)) & mid_mask;
                else used = (~ab & lo) || (hi && (~__ldg(bit_row + at + 1) & hi));
            }
            const uint32_t word = __ballot_sync(0xffffffffu, used);
            if (lane == 0) use_words[w] = word;
        }
    }
    if (TIER && warp == 9) {
        const int2 t = tier_sizes(a.tier, bh, a.NB, ob, lane);
        if (lane == 0) ctl->tiers = t;
    }
    if (warp == 8) {
        tmem_alloc(smem_u32(&ctl->tmem_base), 512);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    // walked units of 64 rows: the list's blocks (the query blocks of the bitmap for BWD_REP), then the tiers' means as in the forward
    int nA = TIER && !(a.tier.phases & PH_A) ? 0 : end - beg;
    if (REP) {
        int used = 0;
        for (int w = lane; w < a.tier.W; w += 32) used += __popc(use_words[w]);
        nA = __reduce_add_sync(0xffffffffu, used);
    }
    const int nM = TIER ? nA + (ctl->tiers.x * a.tier.RM + TB - 1) / TB : nA;
    const int n = TIER ? nM + tail_units(a.tier, a.NB, ctl->tiers.y) : nM;
    const int nt = (n + 1) >> 1;
    constexpr uint32_t G1 = 256, G2 = 320;                   // accumulator columns
    const uint32_t full0 = smem_u32(&ctl->full[0]), empty0 = smem_u32(&ctl->empty[0]);
    int issued[2] = {0, 0};                                  // load warps: X1 and X2 tiles issued
    // tile number i of X1 / X2: its index among the slots and barriers, and the phase of its full barrier
    auto slot_of = [&](int x, int i) { return C::SHARED ? (2 * i + x) % (N1 + N2) : x ? N1 + i % N2 : i % N1; };
    auto phase_of = [&](int x, int i) { return (uint32_t)(C::SHARED ? (2 * i + x) / (N1 + N2) : i / (x ? N2 : N1)) & 1u; };

    if (warp == 9 || warp == 10) {
        // ------------------------------------------------------------ loads: Y1, X1(i) by warp 9, Y2, X2(i) by warp 10 or, into one
        // ring, all by warp 9. A tile's load is 600 clocks of a warp: with one warp for both dQ took 0.94 ms of a training step instead of 0.91; two
        // warps into the one ring made dK / dV slower, 1.24 -> 1.285 ms.
        const int x_first = warp - 9, x_last = C::SHARED ? 1 : x_first;
        bool ok = *abort_flag == 0;
        if (ok && nt > 0) {
            for (int x = x_first; x <= x_last && lane == 0; ++x) {
                const CUtensorMap* y = !REP ? (x ? &tmY2 : &tmY1) : rep_mid ? (x ? &tmM2 : &tmM1) : (x ? &tmT2 : &tmT1);
                const int yrow = REP ? rep_row0 : row0 + ob * TB;
                tma_prefetch_desc(x ? &tmX2 : &tmX1);
                mbar_arrive_expect_tx(smem_u32(&ctl->yfull), Y_TILE);
                for (int d = 0; d < DH; ++d) tma_load_2d(base + (x ? C::Y2 : C::Y1) + d * Y_HALF, y, smem_u32(&ctl->yfull), 64 * d, yrow);
            }
            int win = !REP && lane < nA ? block_at(lane) : 0;  // a window of 32 list entries
            BitWalk used(use_words, REP);
            TierWalk walk;
            if (TIER) walk.start(a.tier, bh, a.NB, ob, lane);
            for (int i = 0; i < nt && ok; ++i) {
                const int e = 2 * i;
                const int nb = e + 1 < n ? 2 : 1;
                int j0, j1;
                if (REP) {
                    j0 = used.next();
                    j1 = nb > 1 ? used.next() : j0;
                } else {
                    if (e > 0 && (e & 31) == 0) win = e + lane < nA ? block_at(e + lane) : 0;
                    j0 = __shfl_sync(0xffffffffu, win, e & 31);
                    j1 = __shfl_sync(0xffffffffu, win, (e + 1) & 31);
                }
                const bool lists = !TIER || e + nb <= nA;
#pragma unroll 1
                for (int x = x_first; x <= x_last; ++x) {
                    const uint32_t slot = slot_of(x, i), par = phase_of(x, i) ^ 1, bar = full0 + 8 * slot;
                    const uint32_t dst = base + C::RING + slot * X_TILE;
                    if (lists) {
                        if (lane == 0) ok = mbar_wait(empty0 + 8 * slot, par, abort_flag, a.status, 501);
                        ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
                        if (!ok) break;
                        if (lane == 0) mbar_arrive_expect_tx(bar, nb * Y_TILE);
                        __syncwarp();
                        // the d halves of the first block, then of the second
                        if (lane < DH * nb) {
                            const int d = lane % DH, b = lane / DH;
                            tma_load_2d(dst + d * X_HALF + b * Y_HALF, x ? &tmX2 : &tmX1, bar, 64 * d, row0 + (b ? j1 : j0) * TB);
                        }
                    } else {
                        // unit by unit; one copy of the code that finds and loads a unit's means (two: 4 % slower)
#pragma unroll 1
                        for (int b = 0; b < nb; ++b) {
                            const int u = e + b;
                            int2 id = make_int2(-1, -1), tokens = make_int2(0, 0);
                            if (u >= nA) {
                                id = unit_blocks(walk, a.tier, bh, a.NB, ob, u < nM, u < nM ? u - nA : u - nM, lane);
                                if (x == 0) tokens = unit_tokens(a.blk_cnt, a.tier, bh, a.NB, ob, u < nM, id, u - nM, lane);
                            }
                            if (b == 0) {
                                if (lane == 0) ok = mbar_wait(empty0 + 8 * slot, par, abort_flag, a.status, 501);
                                ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
                                if (!ok) break;
                            }
                            // the counts' slot is free: the tile this one replaces was released after iteration i - N1
                            if (x == 0 && u >= nA) write_counts(counts + (u % COUNT_RING) * TB, tokens, a.tier.RM, u < nM, lane);
                            __syncwarp();
                            // one arrival, after the counts of both units (bytes may land before they are expected)
                            if (lane == 0 && b + 1 == nb) mbar_arrive_expect_tx(bar, nb * Y_TILE);
                            if (u >= nA)
                                load_means<DH>(dst + b * Y_HALF, X_HALF, x ? &tmM2 : &tmM1, x ? &tmT2 : &tmT1, bar, a.tier, bh, u < nM, id,
                                               u - nM, lane);
                            else if (lane < DH)
                                tma_load_2d(dst + lane * X_HALF, x ? &tmX2 : &tmX1, bar, 64 * lane, row0 + j0 * TB);
                        }
                        if (!ok) break;
                    }
                    __syncwarp();
                    issued[x] = i + 1;
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
        auto ready = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_test_wait(bar, parity)) != 0; };
        auto issue_s = [&](int x, int i) {                  // x = 0: S(i), x = 1: dP(i)
            tc_fence_after();
            if (elect_one()) {
                const uint32_t slot = slot_of(x, i);
                const uint32_t xa = k_lo + ((base + C::RING + slot * X_TILE) >> 4);
                const uint32_t yb = k_lo + ((base + (x ? C::Y2 : C::Y1)) >> 4);
                const uint32_t d = tmem + (i & 1) * 128 + x * 64;
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_ss_lohi(d, xa + (((ks >> 2) * X_HALF + (ks & 3) * 32) >> 4), k_hi,
                                 yb + (((ks >> 2) * Y_HALF + (ks & 3) * 32) >> 4), k_hi, ID_S, ks > 0);
                if (!KV && x == 1) umma_commit(empty0 + 8 * slot);    // the dQ passes need V no more
                if (x == 1) umma_commit(smem_u32(&ctl->sfull[i & 1]));
            }
            __syncwarp();
        };
        auto issue_g = [&](int i) {
            tc_fence_after();
            if (elect_one()) {
                const int ksteps = 2 * i + 1 < n ? 8 : 4;      // an odd end has 64 rows: the other half of the slot is stale
#pragma unroll 1
                for (int x = 0; x < (KV ? 2 : 1); ++x) {
                    const uint32_t slot = slot_of(x, i);
                    const uint32_t xa = x_lo + ((base + C::RING + slot * X_TILE) >> 4);
                    const uint32_t pb = k_lo + ((base + (x ? C::P : C::DS)) >> 4);
                    for (int ks = 0; ks < ksteps; ++ks)
                        umma_ss_lohi(tmem + (x ? G2 : G1), xa + ((ks * 2048) >> 4), x_hi, pb + ((ks * 2048) >> 4), k_hi, ID_G,
                                     (i > 0 || ks > 0) ? 1u : 0u);
                    umma_commit(empty0 + 8 * slot);
                }
                umma_commit(smem_u32(&ctl->pvdone));
            }
            __syncwarp();
        };
        if (C::SHARED) {
            // in the order of the ring (choosing as below is 8 % slower here)
            auto issue_both = [&](int i) {
                for (int x = 0; x < 2; ++x) {
                    ok = ok && mbar_wait_warp(full0 + 8 * slot_of(x, i), phase_of(x, i), abort_flag, a.status, 504);
                    if (ok) issue_s(x, i);
                }
            };
            if (nt > 0) issue_both(0);
            for (int i = 0; i < nt && ok; ++i) {
                if (i + 1 < nt) issue_both(i + 1);
                ok = ok && mbar_wait_warp(smem_u32(&ctl->pfull), i & 1, abort_flag, a.status, 509);
                if (ok) issue_g(i);
            }
        }
        // Whatever is ready goes next: in a fixed order the second products of one iteration waited for the X2 tile of the next
        // but one, and that tile for the slot they free. S and dP of iteration i write the columns of i - 2, which the P / dS
        // warps had read when they handed over P and dS of i - 2 (seen here before the second products of i - 2 were issued).
        int si = 0, di = 0, gi = 0;                            // next S, dP and second products
        uint32_t idle = 0, late = 0;
        int64_t t0 = 0;
        while (!C::SHARED && ok && gi < nt) {
            bool did = false;
            if (gi < di && ready(smem_u32(&ctl->pfull), gi & 1)) { issue_g(gi++); did = true; }
            if (si < nt && si <= gi + 1 && ready(full0 + 8 * slot_of(0, si), phase_of(0, si))) { issue_s(0, si++); did = true; }
            if (di < si && ready(full0 + 8 * slot_of(1, di), phase_of(1, di))) { issue_s(1, di++); did = true; }
            if (did) {
                idle = 0;
                continue;
            }
            // a bounded wait, as mbar_wait
            if (idle == 0) {
                t0 = (int64_t)global_timer_ns();
                late = 0;
            }
            if ((++idle & 255u) == 0) {
                const bool gone = (int64_t)global_timer_ns() - t0 > (int64_t)kWaitLimitNs;
                late = gone ? late + 1 : 0;
                const bool stop = *abort_flag || *reinterpret_cast<volatile int*>(a.status) != 0 || late >= 2;
                if (__any_sync(0xffffffffu, stop)) {
                    if (lane == 0) {
                        *abort_flag = 1;
                        atomicCAS(a.status, 0, 503 + 1000 * (int)(blockIdx.x % 100000));
                    }
                    ok = false;
                }
            }
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
        // The walked row's block id is requested two iterations ahead and what hangs on it (the block's tokens, in the dK / dV
        // pass the row's LSE and delta) one ahead, and nothing is computed from a loaded value before its own iteration: a warp
        // issues in order, so one use of a load that is still on its way would stall the current iteration's exponentials.
        BitWalk used(use_words, REP);
        auto walked = [&](int i) -> int {                    // called for i = 0, 1, 2, ...
            const int e = 2 * i + (r >> 6);
            if (REP) {
                if (i >= nt) return -1;
                const int j0 = used.next(), j1 = 2 * i + 1 < nA ? used.next() : -1;
                return r >> 6 ? j1 : j0;
            }
            return i < nt && e < nA ? block_at(e) : -1;
        };
        int n_blk = walked(0), n2_blk = walked(1), n_cnt = 0;
        float n_lse = 0.f, n_delta = 0.f;
        // BWD_REP: the tier words of (this warp's query block, the tile's columns)
        uint32_t n_wa = 0, n_wab = 0;
        const int rep_word = (rep_blk >> 5) + (rep_mid ? 0 : ch);
        auto request = [&](int jb) {
            if (jb < 0) return;
            n_cnt = tokens_of(jb);
            if (KV) {
                const size_t g = (size_t)row0 + (size_t)jb * TB + (r & 63);
                n_lse = __ldg(a.lse + g);
                n_delta = __ldg(a.delta + g);
            }
            if (REP && rep_word < a.tier.W) {
                const size_t at = ((size_t)bh * a.NB + jb) * a.tier.W + rep_word;
                n_wab = __ldg(a.tier.bits_ab + at);
                n_wa = __ldg(a.tier.bits_a + at);
            }
        };
        request(n_blk);
        for (int i = 0; i < nt && ok; ++i) {
            const int blk = n_blk, cnt_w = n_cnt;
            const float lse_w = n_lse, dl = n_delta;
            const uint32_t wa = n_wa, wab = n_wab;
            n_blk = n2_blk;
            request(n_blk);
            n2_blk = walked(i + 2);
            ok = mbar_wait_warp(smem_u32(&ctl->sfull[i & 1]), (i >> 1) & 1, abort_flag, a.status, 506);
            if (!ok) break;
            tc_fence_after();
            bool valid = blk >= 0 && (r & 63) < cnt_w && (!KV || lse_w != -INFINITY);
            float off = KV ? -lse_w * kLog2e : 0.f;
            uint32_t use = 0xFFFFFFFFu;                      // bit c: this thread's column c is used by the row's block
            if (REP) {
                const uint32_t bits = blk < 0 || rep_word >= a.tier.W ? 0u : rep_mid ? (wab & ~wa) >> (rep_blk & 31) : ~wab;
                const int b = rep_mid ? (32 * ch + lane) / a.tier.RM : lane;
                use = __ballot_sync(0xffffffffu, (bits >> b) & 1u);
            }
            if (TIER && 2 * i + (r >> 6) >= nA && 2 * i + (r >> 6) < n) {
                const int c = counts[((2 * i + (r >> 6)) % COUNT_RING) * TB + (r & 63)];
                valid = c > 0;
                off = a.tier.bias[max(c, 1)];
            }
            uint32_t s[32], dp[32];
            tmem_ld32(tw + (i & 1) * 128 + 32 * ch, s);
            tmem_ld32(tw + (i & 1) * 128 + 64 + 32 * ch, dp);
            tmem_wait_ld_regs(s);
            tmem_wait_ld_regs(dp);
            uint32_t pk[16], dk[16];
            const float2 sc = make_float2(a.scale_log2, a.scale_log2);
            const float4* lse4 = reinterpret_cast<const float4*>(ctl->lse2 + 32 * ch);
            const float4* dl4 = reinterpret_cast<const float4*>(ctl->delta + 32 * ch);
#pragma unroll
            for (int c4 = 0; c4 < 8; ++c4) {
                float4 o4 = make_float4(off, off, off, off), d4 = make_float4(dl, dl, dl, dl);
                if (!KV || REP) {
                    const float4 l4 = lse4[c4];
                    if (TIER || REP) o4 = make_float4(off - l4.x, off - l4.y, off - l4.z, off - l4.w);
                    else o4 = make_float4(-l4.x, -l4.y, -l4.z, -l4.w);
                }
                if (!KV) d4 = dl4[c4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = 4 * c4 + 2 * h;
                    const float2 x = __ffma2_rn(make_float2(__uint_as_float(s[c]), __uint_as_float(s[c + 1])), sc,
                                                h ? make_float2(o4.z, o4.w) : make_float2(o4.x, o4.y));
                    float2 p = make_float2(ex2_approx(x.x), ex2_approx(x.y));
                    // rows without a query / key are 0; a padded column only reaches its own (zeroed) gradient row
                    p.x = valid && (!REP || ((use >> c) & 1u)) ? p.x : 0.f;
                    p.y = valid && (!REP || ((use >> (c + 1)) & 1u)) ? p.y : 0.f;
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
        // the per-block gradients to add, on their way during the last products (fetched where they are added they cost a tile 1,500 clocks: dK / dV of a training step 1.24 -> 1.19 ms)
        float4 adds[KV ? 2 : 1];
        const float inv = 1.f / (float)cnt_o;
#pragma unroll
        for (int x = 0; x < (KV ? 2 : 1); ++x) {
            const float* add = x ? a.add1 : a.add0;
            adds[x] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (add && slot_out < 0) {
                const float* src = add + ((size_t)bh * a.add_nb + ob) * D + 4 * (lane % (D / 4));
                adds[x] = make_float4(__ldg(src) * inv, __ldg(src + 1) * inv, __ldg(src + 2) * inv, __ldg(src + 3) * inv);
            }
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
#pragma unroll
        for (int x = 0; x < (KV ? 2 : 1); ++x) {
            const float mul = x ? 1.f : a.scale;
            const float4 ad = adds[x];
            const int d = 4 * (lane % (D / 4));                  // D / 4 lanes share a token
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
                if (REP) {
                    // rows past the table's real size are left to the caller
                    if (t < cnt_o)
                        store4((rep_mid ? (x ? a.part1 : a.part0) : f) + ((size_t)rep_row0 + t) * D + d, v, a.wide);
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
    if (warp >= 9 && lane == 0 && *abort_flag) {
        // a wait gave up: give the loads of this warp a moment (100 us in all) to land before shared memory goes away
        const uint64_t t_end = global_timer_ns() + 100000ull;
        for (int x = 0; x < 2; ++x)
            for (int i = max(0, issued[x] - N1); i < issued[x]; ++i)
                while (!mbar_try_wait(full0 + 8 * slot_of(x, i), phase_of(x, i)) && global_timer_ns() < t_end) {}
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (*abort_flag) {
        for (int x = 0; x < (KV ? 2 : 1); ++x) {
            float* part = x ? a.part1 : a.part0;
            float* f = x ? a.f1 : a.f0;
            const size_t row = (size_t)row0 + (size_t)ob * TB;
            if (slot_out >= 0) fill_nan(part + (size_t)slot_out * TB * D, TB * D, kNaN32);
            else if (REP) fill_nan((rep_mid ? part : f) + (size_t)rep_row0 * D, cnt_o * D, kNaN32);
            else if (f) fill_nan(f + row * D, TB * D, kNaN32);
            else fill_nan(static_cast<T*>(x ? a.d1 : a.d0) + row * D, TB * D / 2, kNaN16x2);
        }
    }
}

template <typename T, int D, int MODE>
static int launch_bwd(const void* x1, const void* x2, const void* y1, const void* y2, const BwdTcArgs& a, int BH, dim3 grid,
                      cudaStream_t st) {
    CUtensorMap t[4];
    const void* p[4] = {x1, x2, y1, y2};
    for (int i = 0; i < 4; ++i)
        if (int rc = make_token_map<T>(&t[i], p[i], D, (long long)BH * a.L)) return rc;
    auto kern = attn_bwd_tc_kernel<T, D, MODE>;
    if (int rc = opt_in_shared_memory((const void*)kern, (int)BwdCfg<D, MODE>::BYTES)) return rc;
    kern<<<grid, BwdCfg<D, MODE>::THREADS, BwdCfg<D, MODE>::BYTES, st>>>(t[0], t[1], t[2], t[3], t[2], t[3], t[2], t[3], a);
    ES_CHECK_LAUNCH("attn_bwd_tc_kernel");
    return 0;
}

template <int MODE>
static int dispatch_bwd(const void* x1, const void* x2, const void* y1, const void* y2, const BwdTcArgs& a, int BH, int D,
                        int dtype, dim3 grid, cudaStream_t st) {
    if (D == 128)
        return dtype == 0 ? launch_bwd<__nv_bfloat16, 128, MODE>(x1, x2, y1, y2, a, BH, grid, st)
                          : launch_bwd<__half, 128, MODE>(x1, x2, y1, y2, a, BH, grid, st);
    return dtype == 0 ? launch_bwd<__nv_bfloat16, 64, MODE>(x1, x2, y1, y2, a, BH, grid, st)
                      : launch_bwd<__half, 64, MODE>(x1, x2, y1, y2, a, BH, grid, st);
}

// The caller has checked the pointers and sizes (D = 64 or 128). kv: the dK / dV pass (out0 = dK, out1 = dV), else the dQ pass
// (out0 = dQ). tasks == nullptr: one CTA per (owner block, bh). row_ptr and tasks null: every block with every block, the
// sequence's real rows are `rows`.
int attn_bwd_tc(bool kv, const void* q, const void* k, const void* v, const void* dout, const float* lse, const float* delta,
                void* out0, void* out1, float* f0, float* f1, const float* add0, const float* add1, int add_nb,
                const int* row_ptr, const int* col_idx, const int* blk_cnt, int BH, int L, int rows, int D, int dtype, const int* tasks,
                const int* task_info, int n_tasks, float* part0, float* part1, cudaStream_t st) {
    if (!aligned(4, out0, out1) || !aligned(8, f0, f1, part0, part1))
        return set_error(-1, "attn_bwd_tc: 16-bit gradients must be 4-byte, fp32 gradients and partials 8-byte aligned");
    int* status = device_status_ptr();
    if (!status) return set_error(-2, "attn_bwd_tc: the device status word is not available on this device");
    const float scale = 1.f / sqrtf((float)D);
    const int wide = (((uintptr_t)out0 | (uintptr_t)out1 | (uintptr_t)f0 | (uintptr_t)f1 | (uintptr_t)part0 | (uintptr_t)part1) & 15) == 0;
    const BwdTcArgs a{lse, delta, out0, out1, f0, f1, add0, add1, add_nb, row_ptr, col_idx, blk_cnt, L, L / TB, rows, scale,
                      kLog2e * scale, tasks, task_info, part0, part1, status, {}, wide};
    const dim3 grid = tasks ? dim3(n_tasks, 1) : dim3(L / TB, BH);
    return kv ? dispatch_bwd<BWD_KV>(q, dout, k, v, a, BH, D, dtype, grid, st)
              : dispatch_bwd<BWD_Q>(k, v, q, dout, a, BH, D, dtype, grid, st);
}

template <typename T, int D, int MODE>
static int launch_tier_bwd(const void* x1, const void* x2, const void* y1, const void* y2, const void* k_mid, const void* v_mid,
                           const void* k_tail, const void* v_tail, const BwdTcArgs& a, int BH, int grid_x, cudaStream_t st) {
    CUtensorMap t[8];
    const long long tok = (long long)BH * a.L, mid = (long long)BH * a.tier.mid_stride, tail = (long long)BH * a.tier.tail_stride;
    const void* p[8] = {x1, x2, y1, y2, k_mid, v_mid, k_tail, v_tail};
    const long long rows[8] = {tok, tok, tok, tok, mid, mid, tail, tail};
    for (int i = 0; i < 8; ++i) {
        if (MODE == BWD_REP && (i == 2 || i == 3)) { t[i] = t[i - 2]; continue; }            // the owner is a table
        const int box = MODE != BWD_TIER_Q || i < 4 ? TB : i < 6 ? a.tier.RM : a.tier.tail_box();
        if (int rc = make_token_map<T>(&t[i], p[i], D, rows[i], box)) return rc;
    }
    auto kern = attn_bwd_tc_kernel<T, D, MODE>;
    if (int rc = opt_in_shared_memory((const void*)kern, (int)BwdCfg<D, MODE>::BYTES)) return rc;
    kern<<<dim3(grid_x, BH), BwdCfg<D, MODE>::THREADS, BwdCfg<D, MODE>::BYTES, st>>>(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], a);
    ES_CHECK_LAUNCH("attn_bwd_tc_kernel");
    return 0;
}

template <int MODE>
static int dispatch_tier_bwd(const void* x1, const void* x2, const void* y1, const void* y2, const void* k_mid, const void* v_mid,
                             const void* k_tail, const void* v_tail, const BwdTcArgs& a, int BH, int D, int dtype, int grid_x,
                             cudaStream_t st) {
    if (D == 128)
        return dtype == 0 ? launch_tier_bwd<__nv_bfloat16, 128, MODE>(x1, x2, y1, y2, k_mid, v_mid, k_tail, v_tail, a, BH, grid_x, st)
                          : launch_tier_bwd<__half, 128, MODE>(x1, x2, y1, y2, k_mid, v_mid, k_tail, v_tail, a, BH, grid_x, st);
    return dtype == 0 ? launch_tier_bwd<__nv_bfloat16, 64, MODE>(x1, x2, y1, y2, k_mid, v_mid, k_tail, v_tail, a, BH, grid_x, st)
                      : launch_tier_bwd<__half, 64, MODE>(x1, x2, y1, y2, k_mid, v_mid, k_tail, v_tail, a, BH, grid_x, st);
}

// The three-tier dQ pass, and the gradients of the tables of representatives (fp32, like the tables); the caller has checked the
// pointers and sizes.
int tier_bwd_q_tc(const void* q, const void* k, const void* v, const void* k_mid, const void* v_mid, const void* k_tail,
                  const void* v_tail, const void* dout, const float* lse, const float* delta, void* dq, const float* add, int add_nb,
                  const int* row_ptr, const int* col_idx, const TierMaps& tier, const int* blk_cnt, int BH, int L, int D, int dtype,
                  cudaStream_t st) {
    if (!aligned(4, dq)) return set_error(-1, "tier_bwd_q_tc: dq must be 4-byte aligned");
    int* status = device_status_ptr();
    if (!status) return set_error(-2, "tier_bwd_q_tc: the device status word is not available on this device");
    const float scale = 1.f / sqrtf((float)D);
    BwdTcArgs a{lse, delta, dq, nullptr, nullptr, nullptr, add, nullptr, add_nb, row_ptr, col_idx, blk_cnt, L, L / TB, 0, scale,
                      kLog2e * scale, nullptr, nullptr, nullptr, nullptr, status, tier, ((uintptr_t)dq & 15) == 0};
    a.tier.set_bias(1.0);
    return dispatch_tier_bwd<BWD_TIER_Q>(k, v, q, dout, k_mid, v_mid, k_tail, v_tail, a, BH, D, dtype, L / TB, st);
}

int tier_rep_bwd_tc(const void* q, const void* k_mid, const void* v_mid, const void* k_tail, const void* v_tail, const void* dout,
                    const float* lse, const float* delta, float* dk_mid, float* dv_mid, float* dk_tail, float* dv_tail,
                    const TierMaps& tier, const int* blk_cnt, int BH, int L, int D, int dtype, int tiles, cudaStream_t st) {
    if (!aligned(8, dk_mid, dv_mid, dk_tail, dv_tail)) return set_error(-1, "tier_rep_bwd_tc: the tables' gradients must be 8-byte aligned");
    int* status = device_status_ptr();
    if (!status) return set_error(-2, "tier_rep_bwd_tc: the device status word is not available on this device");
    const float scale = 1.f / sqrtf((float)D);
    const int wide = (((uintptr_t)dk_mid | (uintptr_t)dv_mid | (uintptr_t)dk_tail | (uintptr_t)dv_tail) & 15) == 0;
    // no lists: the kernel finds the query blocks to walk; the group means' gradients travel as part0 / part1
    BwdTcArgs a{lse, delta, nullptr, nullptr, dk_tail, dv_tail, nullptr, nullptr, 0, nullptr, nullptr, blk_cnt, L, L / TB, 0,
                      scale, kLog2e * scale, nullptr, nullptr, dk_mid, dv_mid, status, tier, wide};
    a.tier.set_bias(1.0);
    return dispatch_tier_bwd<BWD_REP>(q, dout, nullptr, nullptr, k_mid, v_mid, k_tail, v_tail, a, BH, D, dtype, tiles, st);
}

}  // namespace vsa
}  // namespace es
