// Pieces shared by the tcgen05 kernels of the VSA2 fine branch (es_vsa_tc_fwd.cu, es_vsa_tc_bwd.cu): tensor maps over
// [BH, L, 128] token tensors, instruction descriptors for bf16 and fp16, the tensor-memory load / store of a 64-row
// accumulator, bounded waits of a warp, and the teardown after a wait that gave up.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cmath>
#include <string>
#include <type_traits>

#include "es_api_internal.h"
#include "es_ptx.cuh"

namespace es {
namespace vsa {

// kind::f16 with fp32 accumulation; a_mn / b_mn = 1 when M / N is the contiguous direction of the operand in shared memory.
template <typename T> __host__ __device__ constexpr uint32_t umma_idesc(int m, int n, int a_mn, int b_mn);
template <> __host__ __device__ constexpr uint32_t umma_idesc<__nv_bfloat16>(int m, int n, int a_mn, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
template <> __host__ __device__ constexpr uint32_t umma_idesc<__half>(int m, int n, int a_mn, int b_mn) {
    return (1u << 4) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}

template <typename T> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) { return pack_bf16x2(lo, hi); }
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// An M = 64 accumulator occupies lanes 0 .. 15 of every warp's quarter of tensor memory: warp w holds rows 16 w .. 16 w + 15.
// The 16x256b shape hands 8 columns to a thread as (row lane / 4, columns 2 (lane % 4), + 1) and the same of row + 8:
// registers 4 i .. 4 i + 3 belong to columns 8 i .. 8 i + 7. 64 columns here, 32 registers.
__device__ __forceinline__ void tmem_ld_16x64(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_16x64(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x8.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
          "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
          "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void stsm4(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};"
                 ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}
__device__ __forceinline__ void st_shared16(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y)
        : "memory");
}

// Four rows y of a 2-D tensor, 128 bytes each, one below the other in shared memory; the map's box is one row high.
__device__ __forceinline__ void tma_gather4(uint32_t dst, const CUtensorMap* m, uint32_t bar, int x, const int (&y)[4]) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3])
        : "memory");
}

// Token tensor [BH, L, D] as dims {D, BH L}; a box is 64 d x one 64-token block, 128-byte swizzled (8 KB), or fewer rows.
template <typename T> static int make_token_map(CUtensorMap* m, const void* ptr, int D, long long rows, int box_rows = 64) {
    cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)D * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return encode_tensor_map(m, std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                                                : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                             2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_SWIZZLE_128B);
}

// A CTA whose wait gave up, or that starts while the status word of an earlier one is set, leaves NaN in all it owns: its caller's
// memory is not initialised, and without this could pass for a result until the word is read. The whole CTA, `words` 32-bit words.
constexpr uint32_t kNaN16x2 = 0x7FFF7FFFu, kNaN32 = 0x7FFFFFFFu;      // bf16 and fp16 alike; fp32
__device__ __forceinline__ void fill_nan(void* p, int words, uint32_t nan) {
    for (int i = threadIdx.x; i < words; i += blockDim.x) static_cast<uint32_t*>(p)[i] = nan;
}

// ---------------------------------------------------------------- 64 / RM / 1 representative tiers
// Per query block every kv block is in one tier: A (its tokens; the CSR list and bits_a), B (bits_ab & ~bits_a: its RM group
// means, bias log2(tokens of the group)) or C (~bits_ab: its block mean, bias log2(tokens)). The walk of a query block goes over
// units of 64 columns: the list's blocks, then 64 / RM tier-B blocks at a time, gathered, then 64 consecutive block means at a
// time, those of other tiers masked. (Gathering tier C would save tiles only where few blocks are left to it.) A masked column
// still takes part in the products, times 0, which keeps a NaN or an infinity of a block the query block attends to in another tier
// anyway. Where phases leaves out A or B the block might not be attended to at all, so there tier C is gathered too, four rows to an
// instruction (512 blocks x 12 heads, tier C alone with 480 blocks a list: 0.63 ms forward, 1.03 ms dQ; masked 0.33 and 0.46 ms).
constexpr int PH_A = 1, PH_B = 2, PH_C = 4;
constexpr int UNIT_RING = 8;                       // units whose column counts are staged at a time

struct TierMaps {
    const uint32_t *bits_a, *bits_ab;              // [BH, NB, W]
    int W, RM, mid_stride, tail_stride, phases;
    // Bias of a column that stands for n tokens, log2(n) over `unit`, rounded once; -inf for none. Lanes of a warp mostly ask for
    // one or two values, which the constant cache serves at once.
    float bias[65];
    void set_bias(double unit) {
        for (int n = 0; n <= 64; ++n) bias[n] = (float)(log2((double)n) / unit);
    }
    __host__ __device__ bool gather_tail() const { return (phases & (PH_A | PH_B)) != (PH_A | PH_B); }
    __host__ __device__ int tail_box() const { return gather_tail() ? 1 : 64; }
};

// One warp's walk over the tier-B (or, gathered, the tier-C) blocks of a query block: 32 words (1024 blocks) of its bitmap row at
// a time, a word per lane.
struct TierWalk {
    const uint32_t *ra, *rab;
    int NB, W, w0, before, total;                  // first word of the window, the tier's blocks before it and in it
    uint32_t word, pre;                            // this lane's word, the tier's blocks in the words below it
    bool tail;
    __device__ __forceinline__ uint32_t live(int w) const {
        const int left = NB - 32 * w;
        return left >= 32 ? 0xFFFFFFFFu : left > 0 ? (1u << left) - 1u : 0u;
    }
    __device__ __forceinline__ void fill(int lane) {
        const int w = w0 + lane;
        word = w < W ? (tail ? ~rab[w] : rab[w] & ~ra[w]) & live(w) : 0u;
        uint32_t incl = __popc(word);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
        }
        pre = incl - __popc(word);
        total = (int)__shfl_sync(0xffffffffu, incl, 31);
    }
    __device__ __forceinline__ void start(const TierMaps& t, int bh, int NB_, int qb, int lane, bool tail_ = false) {
        NB = NB_; W = t.W; tail = tail_;
        ra = t.bits_a + ((size_t)bh * NB + qb) * W;
        rab = t.bits_ab + ((size_t)bh * NB + qb) * W;
        w0 = before = 0;
        fill(lane);
    }
    // Lane l < per: number x0 + l of the tier's blocks, -1 past the last one. x0 never decreases.
    __device__ __forceinline__ int blocks(int x0, int per, int lane) {
        int id = -1;
        while (true) {
            const int rel = x0 + lane - before;
            int l = 0;                             // the last lane whose word starts at or before the entry
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                if ((int)__shfl_sync(0xffffffffu, pre, l + o) <= rel) l += o;
            uint32_t w = __shfl_sync(0xffffffffu, word, l);
            int k = rel - (int)__shfl_sync(0xffffffffu, pre, l), bit = 0;      // set bit number k of the word
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const int c = __popc(w & ((1u << o) - 1u));
                if (k >= c) { k -= c; w >>= o; bit += o; }
            }
            if (lane < per && rel >= 0 && rel < total) id = (w0 + l) * 32 + bit;
            if (x0 + per <= before + total || w0 + 32 >= W) return id;
            w0 += 32;
            before += total;
            fill(lane);
        }
    }
};

// Numbers of tier-B and of tier-C blocks of a query block (phases cleared are empty); one warp.
__device__ __forceinline__ int2 tier_sizes(const TierMaps& t, int bh, int NB, int qb, int lane) {
    TierWalk m;
    m.NB = NB;
    const uint32_t* ra = t.bits_a + ((size_t)bh * NB + qb) * t.W;
    const uint32_t* rab = t.bits_ab + ((size_t)bh * NB + qb) * t.W;
    int nB = 0, nC = 0;
    for (int w = lane; w < t.W; w += 32) {
        const uint32_t lv = m.live(w), wab = rab[w];
        nB += __popc(wab & ~ra[w] & lv);
        nC += __popc(~wab & lv);
    }
    nB = __reduce_add_sync(0xffffffffu, nB);
    nC = __reduce_add_sync(0xffffffffu, nC);
    return make_int2((t.phases & PH_B) ? nB : 0, (t.phases & PH_C) ? nC : 0);
}

// Units of a query block's tier C with nC blocks in it.
__device__ __forceinline__ int tail_units(const TierMaps& t, int NB, int nC) {
    return t.gather_tail() ? (nC + 63) / 64 : nC > 0 ? (NB + 63) / 64 : 0;
}
// The blocks of a gathered unit (number x among the tier's), -1 for none: one per lane and group of RM rows, or two per lane for
// single rows (lane, lane + 32). The walk starts again with the first unit of tier C.
__device__ __forceinline__ int2 unit_blocks(TierWalk& walk, const TierMaps& t, int bh, int NB, int qb, bool mid, int x, int lane) {
    int2 id = make_int2(-1, -1);
    if (!mid && !t.gather_tail()) return id;
    if (!mid && x == 0) walk.start(t, bh, NB, qb, lane, true);
    const int per = mid ? 64 / t.RM : 32;
#pragma unroll 1
    for (int h = 0; h < (mid ? 1 : 2); ++h) {
        const int got = walk.blocks((mid ? x : 2 * x + h) * per, per, lane);
        if (h) id.y = got; else id.x = got;
    }
    return id;
}

// Tokens behind the columns of a unit, 0 = masked, in two halves so that the loads can be on their way while the warp waits.
// Tier B: lane l has the tokens of its block and writes its RM groups; tier C: two blocks a lane.
__device__ __forceinline__ int2 unit_tokens(const int* blk_cnt, const TierMaps& t, int bh, int NB, int qb, bool mid, int2 id, int tile,
                                            int lane) {
    int n[2] = {0, 0};
    if (mid || t.gather_tail()) {
        if (id.x >= 0) n[0] = __ldg(blk_cnt + id.x);
        if (id.y >= 0) n[1] = __ldg(blk_cnt + id.y);
    } else {
        const uint32_t* rab = t.bits_ab + ((size_t)bh * NB + qb) * t.W;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = 64 * tile + 32 * h + lane;
            if (j < NB) {
                const int c = __ldg(blk_cnt + j);
                n[h] = (__ldg(rab + 2 * tile + h) >> lane) & 1u ? 0 : c;
            }
        }
    }
    return make_int2(n[0], n[1]);
}
__device__ __forceinline__ void write_counts(uint8_t* dst, int2 n, int RM, bool mid, int lane) {
    if (mid) {
        const int R = 64 / RM;
        if (lane < R)
            for (int g = 0; g < RM; ++g) dst[lane * RM + g] = (uint8_t)min(max(n.x - g * R, 0), R);
    } else {
        dst[lane] = (uint8_t)n.x;
        dst[32 + lane] = (uint8_t)n.y;
    }
}
// The TMA loads of a unit of means to dst, `half` bytes between the DH d halves; the whole warp. Where a gathered unit has no block
// any more its first one is read again (masked): nothing comes in that the query block does not attend to.
template <int DH>
__device__ __forceinline__ void load_means(uint32_t dst, uint32_t half, const CUtensorMap* mid_map, const CUtensorMap* tail_map,
                                           uint32_t bar, const TierMaps& t, int bh, bool mid, int2 id, int tile, int lane) {
    const int first = __shfl_sync(0xffffffffu, id.x, 0);
    if (mid) {
        const int row = bh * t.mid_stride + (id.x >= 0 ? id.x : first) * t.RM;
        if (lane < 64 / t.RM)
            for (int d = 0; d < DH; ++d) tma_load_2d(dst + d * half + lane * t.RM * 128, mid_map, bar, 64 * d, row);
    } else if (t.gather_tail()) {
        // lane 16 d + g: rows 4 g .. 4 g + 3 of d half d
        const int g = lane & 15, d = lane >> 4;
        int row[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int x = __shfl_sync(0xffffffffu, id.x, 4 * (g & 7) + i), y = __shfl_sync(0xffffffffu, id.y, 4 * (g & 7) + i);
            const int j = g < 8 ? x : y;
            row[i] = bh * t.tail_stride + (j >= 0 ? j : first);
        }
        if (d < DH) tma_gather4(dst + d * half + g * 512, tail_map, bar, 64 * d, row);
    } else if (lane < DH) {
        tma_load_2d(dst + lane * half, tail_map, bar, 64 * lane, bh * t.tail_stride + tile * 64);
    }
}

}  // namespace vsa
}  // namespace es
