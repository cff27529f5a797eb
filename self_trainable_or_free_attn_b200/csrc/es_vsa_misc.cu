// VSA2 stages around the attention kernels: pooling, the PSP router (pooled-row LSE, block scores), the exact global
// top-k with its CSR lists in both directions, gate fusion forward / backward and the final gradient assembly.
// Reference: csrc/vsa/vsa2_kernels.h:179-302 of shaoshitong/self_trainable_or_free_attn (parameter structs of the same
// stages) and tests/vsa_reference.py:28-87 (what they compute). Vectorised loads, warp shuffles and, for the two router
// passes, mma.sync tiles; integer stages (top-k, CSR) are exact and deterministic.
#include <cooperative_groups.h>

#include <atomic>
#include <string>

#include "es_api_internal.h"
#include "es_vsa_mma.cuh"

namespace es {
namespace vsa {

// ---------------------------------------------------------------------------------------------- pooling
// Means of the R-token router groups of q and k (optionally v) over their valid tokens, and the
// block means of q, k, v, fp32 sums rounded once to the element type. Empty groups and the padding rows of the pooled
// tensors are zero.
struct PoolArgs {
    const void *q, *k, *v;
    void *qr, *kr, *vr, *qc, *kc, *vc;
    const int* blk_cnt;
    int L, NB, R, G, Lr_pad, NBc_pad;
    int first;            // tensor of blockIdx.z = 0
};

//
// One CTA per (block, bh, tensor). RT = R for the group sizes in use (4 .. 32): all 64 rows are requested before the first is added;
// 0: any R, a row after the other. The sums are the same in both. 512 blocks x 12 heads, us: 49.8, three
// tensors one after the other and a few rows at a time 72.3; 100 blocks x 8 heads, D = 64: 3.2, 10.4.
template <typename T, int D, int RT>
__global__ void __launch_bounds__(D / 2) pool_kernel(const PoolArgs a) {
    const int blk = blockIdx.x, bh = blockIdx.y, t = a.first + blockIdx.z, c = 2 * threadIdx.x;
    const int tiles_c = a.NBc_pad, rows_r = a.Lr_pad, R = RT ? RT : a.R, G = TB / R;
    const void* src = t == 0 ? a.q : t == 1 ? a.k : a.v;
    T* dst_r = static_cast<T*>(t == 0 ? a.qr : t == 1 ? a.kr : a.vr);
    T* dst_c = static_cast<T*>(t == 0 ? a.qc : t == 1 ? a.kc : a.vc);
    auto put = [&](T* row, float x, float y) { *reinterpret_cast<uint32_t*>(row + c) = Elt<T>::pack(x, y); };
    if (blk >= a.NB) {                       // padding rows of the pooled tensors
        if (blk < tiles_c && dst_c) put(dst_c + ((size_t)bh * tiles_c + blk) * D, 0.f, 0.f);
        if (dst_r)
            for (int r = blk * G; r < min((blk + 1) * G, rows_r); ++r) put(dst_r + ((size_t)bh * rows_r + r) * D, 0.f, 0.f);
        return;
    }
    if (!src || !(dst_r || dst_c)) return;
    const int cnt = a.blk_cnt[blk];
    const T* x = static_cast<const T*>(src) + ((size_t)bh * a.L + (size_t)blk * TB) * D + c;
    auto row = [&](int r) { return __ldg(reinterpret_cast<const uint32_t*>(x + (size_t)r * D)); };
    float bx = 0.f, by = 0.f;
    auto group = [&](int g, float sx, float sy) {
        bx += sx; by += sy;
        const int n = min(cnt - g * R, R);
        const float inv = n > 0 ? 1.f / (float)n : 0.f;
        if (dst_r) put(dst_r + ((size_t)bh * rows_r + blk * G + g) * D, sx * inv, sy * inv);
    };
    if (RT) {
        uint32_t w[TB];
#pragma unroll
        for (int r = 0; r < TB; ++r) w[r] = r < cnt ? row(r) : 0u;
#pragma unroll
        for (int g = 0; g < TB / (RT ? RT : TB); ++g) {
            float sx = 0.f, sy = 0.f;
#pragma unroll
            for (int r = 0; r < RT; ++r) {
                const float2 f = Elt<T>::unpack(w[(g * RT + r) % TB]);
                sx += f.x; sy += f.y;
            }
            group(g, sx, sy);
        }
    } else {
        for (int g = 0; g < G; ++g) {
            float sx = 0.f, sy = 0.f;
            for (int r = g * R; r < min((g + 1) * R, cnt); ++r) {
                const float2 f = Elt<T>::unpack(row(r));
                sx += f.x; sy += f.y;
            }
            group(g, sx, sy);
        }
    }
    const float inv = 1.f / (float)cnt;
    if (dst_c) put(dst_c + ((size_t)bh * tiles_c + blk) * D, bx * inv, by * inv);
}

// ---------------------------------------------------------------------------------------------- router
// Pooled rows: row r = blk * G + g is valid when group g of block blk holds a token (g * R < blk_cnt[blk]).
struct RouterArgs {
    const void *qr, *kr;
    float* lse2;          // [BH, Lr_pad] log2-domain LSE over the valid pooled keys
    float* scores;        // [bh_count, NB, NB]
    const int* blk_cnt;
    int NB, R, G, Lr, Lr_pad, bh0, row_norm;
    float scale_log2;
};

// MODE 0: lse2 of 64 pooled query rows over all pooled keys. MODE 1: block scores of the 64 / G query blocks of the tile:
// score[i][j] = sum over the groups a of i and b of j of 2^(s - lse2), times the row normalisation; the G x G sums are
// taken from a shared-memory copy of the probabilities in a fixed order (reproducible). GT: G as a compile-time constant for
// R = 32, 16 and 8 (0: any power of two), so that the sums read 8 or 16 bytes at a time in the same order; the validity of a
// tile's 64 keys is found once by 64 threads and handed round as two words (with every thread testing its 16 columns, integer
// divisions were two thirds of the kernel). NB = 512, R = 16, 12 heads: LSE 55 us (137 before), scores
// 95 us (225); NB = 624: 86 us (191) and 130 us (537; 222 with three CTAs per SM). Rows of the probabilities are 68 floats apart; 64
// with chunks exchanged by the row was up to 23 % slower (R = 4, 24 blocks: 33 / 41 us), one to three percent faster at R = 16.
template <int D, int MODE> struct RouterSmem {
    static constexpr int SP = 68;                                        // MODE 1: row stride of the [64][SP] probabilities
    static constexpr uint32_t TILE = TB * D * 2, P_BYTES = 64 * SP * 4;
    static constexpr bool OVER_Q = MODE == 1 && D == 128;
    static constexpr uint32_t Q_ROOM = OVER_Q ? P_BYTES : TILE;
    static constexpr uint32_t VALID = Q_ROOM + 2 * TILE, P = OVER_Q ? 0 : VALID + 16;
    static constexpr uint32_t BYTES = VALID + 16 + (MODE == 1 && !OVER_Q ? P_BYTES : 0);
};
template <typename T, int D, int MODE, int GT, int CTAS>
__global__ void __launch_bounds__(128, CTAS) router_kernel(const RouterArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    using S = RouterSmem<D, MODE>;
    constexpr uint32_t TILE = S::TILE;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int qt = blockIdx.x, bh = a.bh0 + blockIdx.y;
    const uint32_t sQ = smem_addr(smem), sK = sQ + S::Q_ROOM;            // K: two stages
    uint32_t* sValid = reinterpret_cast<uint32_t*>(smem + S::VALID);     // [2 stages][2]: bit r = key r of the tile is valid
    // MODE 1: probabilities, at D = 128 in the place of the Q tile (its fragments are in registers), so that four CTAs fit an SM. At
    // 39 tiles x 12 heads three leave 24 of 468 CTAs to a second round.
    float* sP = reinterpret_cast<float*>(smem + S::P);
    constexpr int SP = S::SP;
    const int G = GT ? GT : a.G, lg = 31 - __clz(G);                     // R divides 64: G is a power of two
    auto valid_row = [&](int r) { return r < a.Lr && (r & (G - 1)) * a.R < a.blk_cnt[r >> lg]; };
    const T* q = static_cast<const T*>(a.qr) + ((size_t)bh * a.Lr_pad + (size_t)qt * TB) * D;
    const T* kbase = static_cast<const T*>(a.kr) + (size_t)bh * a.Lr_pad * D;
    const int nkt = a.Lr_pad / TB;
    load_tile<T, D>(sQ, q, D, tid);
    load_tile<T, D>(sK, kbase, D, tid);
    cp_commit();
    const int r0 = warp * 16 + (lane >> 2), r1 = r0 + 8;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f, ls0 = 0.f, ls1 = 0.f;
    if (MODE == 1) {
        const float* lse = a.lse2 + (size_t)bh * a.Lr_pad + (size_t)qt * TB;
        ls0 = lse[r0]; ls1 = lse[r1];
    }
    // validity of the thread's two query rows, found once, or in every tile where keeping it was slower (one to four percent)
    constexpr bool ONCE = D == 128 || GT == 2 || GT == 4;
    bool qv0 = MODE == 1 && ONCE && valid_row(qt * TB + r0), qv1 = MODE == 1 && ONCE && valid_row(qt * TB + r1);
    uint32_t qa[D / 16][4];
    for (int kt = 0; kt < nkt; ++kt) {
        const uint32_t sKt = sK + (uint32_t)(kt & 1) * TILE;
        if (kt + 1 < nkt) load_tile<T, D>(sK + (uint32_t)((kt + 1) & 1) * TILE, kbase + (size_t)(kt + 1) * TB * D, D, tid);
        cp_commit();
        if (warp < 2) {
            const unsigned w = __ballot_sync(0xffffffffu, valid_row(kt * TB + tid));
            if (lane == 0) sValid[(kt & 1) * 2 + warp] = w;
        }
        cp_wait<1>();
        __syncthreads();
        if (kt == 0) {
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) load_a<D>(sQ, warp * 16, ks, lane, qa[ks]);
            if (S::OVER_Q) __syncthreads();                               // the tile's room is the probabilities' from here on
        }
        float s[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
            for (int np = 0; np < 4; ++np) {
                uint32_t b[4];
                load_b_nk<D>(sKt, np, ks, lane, b);
                Elt<T>::mma(s[2 * np], qa[ks], b[0], b[1]);
                Elt<T>::mma(s[2 * np + 1], qa[ks], b[2], b[3]);
            }
        // validity of the pooled keys of this tile
        const uint32_t vw[2] = {sValid[(kt & 1) * 2] >> (2 * (lane & 3)), sValid[(kt & 1) * 2 + 1] >> (2 * (lane & 3))};
        bool kv[8][2];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int u = 0; u < 2; ++u) kv[i][u] = (vw[i >> 2] >> ((i & 3) * 8 + u)) & 1u;
        if (MODE == 0) {
            float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                s[i][0] = kv[i][0] ? s[i][0] * a.scale_log2 : -INFINITY;
                s[i][1] = kv[i][1] ? s[i][1] * a.scale_log2 : -INFINITY;
                s[i][2] = kv[i][0] ? s[i][2] * a.scale_log2 : -INFINITY;
                s[i][3] = kv[i][1] ? s[i][3] * a.scale_log2 : -INFINITY;
                mx0 = fmaxf(mx0, fmaxf(s[i][0], s[i][1]));
                mx1 = fmaxf(mx1, fmaxf(s[i][2], s[i][3]));
            }
            const float mn0 = fmaxf(m0, quad_max(mx0)), mn1 = fmaxf(m1, quad_max(mx1));
            const float ms0 = mn0 == -INFINITY ? 0.f : mn0, ms1 = mn1 == -INFINITY ? 0.f : mn1;
            float t0 = 0.f, t1 = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                t0 += exp2f(s[i][0] - ms0) + exp2f(s[i][1] - ms0);
                t1 += exp2f(s[i][2] - ms1) + exp2f(s[i][3] - ms1);
            }
            l0 = l0 * exp2f(m0 - ms0) + t0; l1 = l1 * exp2f(m1 - ms1) + t1;
            m0 = mn0; m1 = mn1;
        } else {
            // probabilities of this key tile -> shared memory, then fixed-order G x G sums
            if (!ONCE) { qv0 = valid_row(qt * TB + r0); qv1 = valid_row(qt * TB + r1); }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int c = i * 8 + 2 * (lane & 3);
                *reinterpret_cast<float2*>(sP + r0 * SP + c) =
                    make_float2((qv0 && kv[i][0]) ? exp2f(s[i][0] * a.scale_log2 - ls0) : 0.f,
                                (qv0 && kv[i][1]) ? exp2f(s[i][1] * a.scale_log2 - ls0) : 0.f);
                *reinterpret_cast<float2*>(sP + r1 * SP + c) =
                    make_float2((qv1 && kv[i][0]) ? exp2f(s[i][2] * a.scale_log2 - ls1) : 0.f,
                                (qv1 && kv[i][1]) ? exp2f(s[i][3] * a.scale_log2 - ls1) : 0.f);
            }
            __syncthreads();
            const int per = TB >> lg;                        // blocks per tile side
            for (int e = tid; e < per * per; e += 128) {
                const int bi = e >> (6 - lg), bj = e & (per - 1);
                const int qblk = qt * per + bi, kblk = kt * per + bj;
                if (qblk < a.NB && kblk < a.NB) {
                    const float* p0 = sP + bi * G * SP + bj * G;
                    float acc = 0.f;
                    if (GT >= 4) {
#pragma unroll
                        for (int x = 0; x < GT; ++x)
#pragma unroll
                            for (int y = 0; y < GT; y += 4) {
                                const float4 v = *reinterpret_cast<const float4*>(p0 + x * SP + y);
                                acc += v.x; acc += v.y; acc += v.z; acc += v.w;
                            }
                    } else if (GT == 2) {
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            const float2 v = *reinterpret_cast<const float2*>(p0 + x * SP);
                            acc += v.x; acc += v.y;
                        }
                    } else {
                        for (int x = 0; x < G; ++x)
                            for (int y = 0; y < G; ++y) acc += p0[x * SP + y];
                    }
                    float norm;
                    if (a.row_norm == 1) norm = 1.f / (float)(G * G);
                    else norm = 1.f / (float)((a.blk_cnt[qblk] + a.R - 1) / a.R);
                    a.scores[((size_t)blockIdx.y * a.NB + qblk) * a.NB + kblk] = acc * norm;
                }
            }
        }
        __syncthreads();
    }
    cp_wait<0>();
    if (MODE == 0) {
        l0 = quad_sum(l0); l1 = quad_sum(l1);
        if ((lane & 3) == 0) {
            float* lse = a.lse2 + (size_t)bh * a.Lr_pad + (size_t)qt * TB;
            lse[r0] = l0 > 0.f ? m0 + log2f(l0) : -INFINITY;
            lse[r1] = l1 > 0.f ? m1 + log2f(l1) : -INFINITY;
        }
    }
}

// ---------------------------------------------------------------------------------------------- exact global top-k
// Per (b, h): the `budget` largest of the NB x NB scores in the order (score descending, flat index ascending). Scores are
// non-negative, so their bit patterns order like the values. Stages: (1) 4-pass radix select of the threshold key and the
// number of entries equal to it that are taken; (2) per row, counts of larger and equal entries; (3) scans: equal-rank base
// of every row, row pointers; (4) per row, the ascending list and the selection bitmap; (5) per column, count, scan, list.
struct TopkArgs {
    const float* scores;    // [bh_count, NB, NB]
    int NB, W, bh0;
    long long budget;       // clamped to NB * NB
    int *q2k_ptr, *q2k_idx, *k2q_ptr, *k2q_idx;
    int* state;             // [bh_count, 4]: threshold key, equal entries to take (where stages are launches)
    int *gtcnt, *eqcnt, *eqbase, *colcnt;     // [bh_count, NB] each
    uint32_t* selbits;      // [bh_count, NB, W]
};

__device__ __forceinline__ uint32_t score_key(float x) {
    x += 0.0f;                                     // -0 -> +0
    const uint32_t u = __float_as_uint(x);
    return (u & 0x80000000u) ? 0u : u;             // negative values (never produced by the router) order as zero
}

// A cluster of eight CTAs per (b, h): each counts the digits of an eighth of the scores, reads the other seven histograms from
// their shared memory and finds the digit for itself. One CTA per (b, h) left 136 of 148 SMs idle at 12 heads, and its thread
// 0 walked the 256 bins; scores share their exponents, so the warps count into eight histograms. NB = 512, 12 heads:
// 23 us (129 before).
constexpr int SEL_CTAS = 8, SEL_COPIES = 8;
struct SelectShared {
    uint32_t part[SEL_COPIES][256], hist[2][256], warp_sum[8], prefix, need;
};
// The threshold key and how many entries equal to it are taken, for every thread of the cluster.
__device__ __forceinline__ void topk_select(const TopkArgs& a, SelectShared& sh, uint32_t& thr, int& take_equal) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    auto& part = sh.part;
    auto& hist = sh.hist;
    auto& warp_sum = sh.warp_sum;
    uint32_t &s_prefix = sh.prefix, &s_need = sh.need;
    const int b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, rank = (int)cluster.block_rank();
    const float* sc = a.scores + (size_t)b * a.NB * a.NB;
    const long long N = (long long)a.NB * a.NB, step = (N + SEL_CTAS - 1) / SEL_CTAS;
    const long long lo = min(rank * step, N), hi = min(lo + step, N);
    thr = 0xFFFFFFFFu;
    take_equal = 0;
    if (a.budget <= 0) return;                         // the same for every CTA of the cluster
    if (tid == 0) { s_prefix = 0; s_need = (uint32_t)a.budget; }
    uint32_t* mine = part[(tid >> 5) & (SEL_COPIES - 1)];
    for (int pass = 0; pass < 4; ++pass) {
        const int shift = 24 - 8 * pass;
        for (int i = tid; i < SEL_COPIES * 256; i += 1024) part[i >> 8][i & 255] = 0;
        __syncthreads();
        const uint32_t prefix = s_prefix, need = s_need, mask = pass == 0 ? 0u : (0xFFFFFFFFu << (shift + 8));
#pragma unroll 4
        for (long long i = lo + tid; i < hi; i += 1024) {
            const uint32_t key = score_key(sc[i]);
            if ((key & mask) == prefix) atomicAdd(&mine[(key >> shift) & 255], 1u);
        }
        __syncthreads();
        uint32_t* own = hist[pass & 1];                // the other buffer may still be read by a CTA that is one pass behind
        if (tid < 256) {
            uint32_t n = 0;
#pragma unroll
            for (int c = 0; c < SEL_COPIES; ++c) n += part[c][tid];
            own[tid] = n;
        }
        cluster.sync();
        // thread t holds digit 255 - t: the number of keys with a digit at least that large
        uint32_t n = 0, incl = 0;
        if (tid < 256) {
#pragma unroll
            for (int c = 0; c < SEL_CTAS; ++c) n += cluster.map_shared_rank(own, c)[255 - tid];
            incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += x;
            }
            if (lane == 31) warp_sum[tid >> 5] = incl;
        }
        __syncthreads();
        if (tid < 256) {
            for (int w = 0; w < (tid >> 5); ++w) incl += warp_sum[w];
            if (incl >= need && incl - n < need) {     // exactly one digit
                s_prefix = prefix | ((uint32_t)(255 - tid) << shift);
                s_need = need - (incl - n);
            }
        }
        __syncthreads();
    }
    thr = s_prefix;
    take_equal = (int)s_need;
}

// Exclusive prefix of v over the 1024 threads of a CTA.
__device__ __forceinline__ int scan_1024(int v, int* warp_total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) warp_total[warp] = incl;
    __syncthreads();
    const int before = incl - v + __reduce_add_sync(0xffffffffu, lane < warp ? warp_total[lane] : 0);
    __syncthreads();
    return before;
}

// Column counts -> k2q_ptr of one (b, h), by the 1024 threads of a CTA.
__device__ __forceinline__ void scan_columns(const TopkArgs& a, int b, int* warp_total) {
    const int tid = threadIdx.x, bh = a.bh0 + b, per = (a.NB + 1023) / 1024, lo = tid * per, hi = min(lo + per, a.NB);
    int n = 0;
    for (int r = lo; r < hi; ++r) n += __ldcg(a.colcnt + b * a.NB + r);
    int pos = scan_1024(n, warp_total) + (int)((long long)bh * a.budget);
    for (int r = lo; r < hi; ++r) {
        a.k2q_ptr[(size_t)bh * (a.NB + 1) + r] = pos;
        pos += __ldcg(a.colcnt + b * a.NB + r);
    }
    if (tid == 1023) a.k2q_ptr[(size_t)bh * (a.NB + 1) + a.NB] = pos;            // the last thread ends at the total
}
// Equal entries before a row and row pointers of one (b, h), by the 1024 threads of a CTA.
__device__ __forceinline__ void scan_rows(const TopkArgs& a, int b, int need, int* warp_total) {
    const int tid = threadIdx.x, bh = a.bh0 + b;
    const int per = (a.NB + 1023) / 1024, lo = min(tid * per, a.NB), hi = min(lo + per, a.NB);
    int equal = 0, n = 0;
    for (int r = lo; r < hi; ++r) equal += __ldcg(a.eqcnt + b * a.NB + r);
    const int eb0 = scan_1024(equal, warp_total);
    for (int r = lo, eb = eb0; r < hi; ++r) {
        const int e = __ldcg(a.eqcnt + b * a.NB + r);
        n += __ldcg(a.gtcnt + b * a.NB + r) + max(0, min(e, need - eb));
        eb += e;
    }
    int pos = scan_1024(n, warp_total) + (int)((long long)bh * a.budget);
    for (int r = lo, eb = eb0; r < hi; ++r) {
        const int e = __ldcg(a.eqcnt + b * a.NB + r);
        a.eqbase[b * a.NB + r] = eb;
        a.q2k_ptr[(size_t)bh * (a.NB + 1) + r] = pos;
        pos += __ldcg(a.gtcnt + b * a.NB + r) + max(0, min(e, need - eb));
        eb += e;
    }
    if (tid == 1023) a.q2k_ptr[(size_t)bh * (a.NB + 1) + a.NB] = pos;        // the last thread ends at the total
}

// One CTA per (b, h): kind 0 rows, kind 1 columns.
__global__ void __launch_bounds__(1024) topk_scan_kernel(const TopkArgs a, int kind) {
    __shared__ int warp_total[32];
    if (kind == 0) scan_rows(a, blockIdx.x, a.state[blockIdx.x * 4 + 1], warp_total);
    else scan_columns(a, blockIdx.x, warp_total);
}

// one warp per row
__global__ void __launch_bounds__(128) topk_count_kernel(const TopkArgs a) {
    const int b = blockIdx.y, row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= a.NB) return;
    const uint32_t thr = (uint32_t)a.state[b * 4];
    const float* sc = a.scores + ((size_t)b * a.NB + row) * a.NB;
    int gt = 0, eq = 0;
    for (int j = lane; j < a.NB; j += 32) {
        const uint32_t key = score_key(sc[j]);
        gt += key > thr; eq += key == thr;
    }
    for (int o = 16; o > 0; o >>= 1) {
        gt += __shfl_xor_sync(0xffffffffu, gt, o);
        eq += __shfl_xor_sync(0xffffffffu, eq, o);
    }
    if (lane == 0) { a.gtcnt[b * a.NB + row] = gt; a.eqcnt[b * a.NB + row] = eq; }
}

// one warp per row: the ascending kv list and the selection bits
__global__ void __launch_bounds__(128) topk_emit_rows_kernel(const TopkArgs a) {
    const int b = blockIdx.y, row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, bh = a.bh0 + b;
    if (row >= a.NB) return;
    const uint32_t thr = (uint32_t)a.state[b * 4];
    const int need = a.state[b * 4 + 1];
    const float* sc = a.scores + ((size_t)b * a.NB + row) * a.NB;
    int eqrank = a.eqbase[b * a.NB + row];
    int pos = a.q2k_ptr[(size_t)bh * (a.NB + 1) + row];
    for (int j0 = 0; j0 < a.NB; j0 += 32) {
        const int j = j0 + lane;
        const uint32_t key = j < a.NB ? score_key(sc[j]) : 0u;
        const bool gt = j < a.NB && key > thr, eq = j < a.NB && key == thr;
        const unsigned em = __ballot_sync(0xffffffffu, eq);
        const bool take = gt || (eq && eqrank + __popc(em & ((1u << lane) - 1)) < need);
        const unsigned tm = __ballot_sync(0xffffffffu, take);
        if (take) a.q2k_idx[pos + __popc(tm & ((1u << lane) - 1))] = j;
        if (lane == 0) a.selbits[((size_t)b * a.NB + row) * a.W + (j0 >> 5)] = tm;
        pos += __popc(tm);
        eqrank += __popc(em);
    }
}


// One CTA per word (32 columns) of the bitmap, its 8 warps an eighth of the rows each: count (pass 0) or emit the ascending
// query lists (pass 1). A warp takes 32 rows at a time, lane = row, and a vote per column turns them into that column's 32
// rows; lane j keeps column j's count. One thread per column walking the rows took 79 us per pass at NB = 512, 12 heads;
// this takes 7.
__device__ __forceinline__ int count_columns(const TopkArgs& a, int b, int w, int warp, int lane) {
    const uint32_t* bits = a.selbits + (size_t)b * a.NB * a.W + w;
    const int per = ((a.NB + 255) / 256) * 32, lo = warp * per, hi = min(lo + per, a.NB);
    int n = 0;
    for (int r0 = lo; r0 < hi; r0 += 32) {
        const uint32_t word = r0 + lane < hi ? __ldcg(bits + (size_t)(r0 + lane) * a.W) : 0u;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const int c = __popc(__ballot_sync(0xffffffffu, (word >> j) & 1u));
            n += lane == j ? c : 0;
        }
    }
    return n;
}
__device__ __forceinline__ void emit_columns(const TopkArgs& a, int b, int w, int warp, int lane, const int (&part)[8][32]) {
    const uint32_t* bits = a.selbits + (size_t)b * a.NB * a.W + w;
    const int per = ((a.NB + 255) / 256) * 32, lo = warp * per, hi = min(lo + per, a.NB), col = w * 32 + lane;
    int pos = col < a.NB ? __ldcg(a.k2q_ptr + (size_t)(a.bh0 + b) * (a.NB + 1) + col) : 0;
    for (int x = 0; x < warp; ++x) pos += part[x][lane];
    for (int r0 = lo; r0 < hi; r0 += 32) {
        const uint32_t word = r0 + lane < hi ? __ldcg(bits + (size_t)(r0 + lane) * a.W) : 0u;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const unsigned m = __ballot_sync(0xffffffffu, (word >> j) & 1u);
            if (m == 0) continue;                      // uniform
            const int at = __shfl_sync(0xffffffffu, pos, j);
            if ((word >> j) & 1u) a.k2q_idx[at + __popc(m & ((1u << lane) - 1))] = r0 + lane;
            pos += lane == j ? __popc(m) : 0;
        }
    }
}
__global__ void __launch_bounds__(256) topk_cols_kernel(const TopkArgs a, int pass) {
    __shared__ int part[8][32];
    const int b = blockIdx.y, w = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, col = w * 32 + lane;
    part[warp][lane] = count_columns(a, b, w, warp, lane);
    __syncthreads();
    if (pass == 0) {
        if (warp == 0 && col < a.NB) {
            int t = 0;
            for (int x = 0; x < 8; ++x) t += part[x][lane];
            a.colcnt[b * a.NB + col] = t;
        }
        return;
    }
    emit_columns(a, b, w, warp, lane, part);
}

// The selection alone, a cluster per (b, h).
__global__ void __cluster_dims__(SEL_CTAS, 1, 1) __launch_bounds__(1024) topk_select_kernel(const TopkArgs a) {
    __shared__ SelectShared sh;
    uint32_t thr;
    int need;
    topk_select(a, sh, thr, need);
    if (blockIdx.x == 0 && threadIdx.x == 0) { a.state[blockIdx.y * 4] = (int)thr; a.state[blockIdx.y * 4 + 1] = need; }
    cooperative_groups::this_cluster().sync();         // no CTA leaves while another reads its histogram
}

// The whole of the global top-k in one launch, a cluster per (b, h): threshold, counts per row, row pointers, lists and bitmap,
// and the lists of the columns. What one CTA leaves for the others of its cluster (counts, pointers, the bitmap) goes through
// global memory, written before a cluster barrier and read past it from L2. Where eight CTAs per head are enough (the rule is at
// es_vsa_global_topk) this saves six launches.
__global__ void __cluster_dims__(SEL_CTAS, 1, 1) __launch_bounds__(1024) topk_kernel(const TopkArgs a) {
    __shared__ SelectShared sh;
    __shared__ int warp_total[32];
    __shared__ int colpart[4][8][32];
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)cluster.block_rank(), bh = a.bh0 + b;
    uint32_t thr;
    int need;
    topk_select(a, sh, thr, need);
    const float* scores = a.scores + (size_t)b * a.NB * a.NB;
    const int row0 = rank * 32 + warp;                 // a warp's rows: row0, row0 + 256, ..
    for (int row = row0; row < a.NB; row += 32 * SEL_CTAS) {
        const float* sc = scores + (size_t)row * a.NB;
        int gt = 0, eq = 0;
#pragma unroll 4
        for (int j = lane; j < a.NB; j += 32) {
            const uint32_t key = score_key(sc[j]);
            gt += key > thr; eq += key == thr;
        }
        gt = __reduce_add_sync(0xffffffffu, gt);
        eq = __reduce_add_sync(0xffffffffu, eq);
        if (lane == 0) { a.gtcnt[b * a.NB + row] = gt; a.eqcnt[b * a.NB + row] = eq; }
    }
    cluster.sync();
    if (rank == 0) scan_rows(a, b, need, warp_total);
    cluster.sync();
    for (int row = row0; row < a.NB; row += 32 * SEL_CTAS) {
        const float* sc = scores + (size_t)row * a.NB;
        int eqrank = __ldcg(a.eqbase + b * a.NB + row), pos = __ldcg(a.q2k_ptr + (size_t)bh * (a.NB + 1) + row);
#pragma unroll 4
        for (int j0 = 0; j0 < a.NB; j0 += 32) {
            const int j = j0 + lane;
            const uint32_t key = j < a.NB ? score_key(sc[j]) : 0u;
            const bool gt = j < a.NB && key > thr, eq = j < a.NB && key == thr;
            const unsigned em = __ballot_sync(0xffffffffu, eq);
            const bool take = gt || (eq && eqrank + __popc(em & ((1u << lane) - 1)) < need);
            const unsigned tm = __ballot_sync(0xffffffffu, take);
            if (take) a.q2k_idx[pos + __popc(tm & ((1u << lane) - 1))] = j;
            if (lane == 0) a.selbits[((size_t)b * a.NB + row) * a.W + (j0 >> 5)] = tm;
            pos += __popc(tm);
            eqrank += __popc(em);
        }
    }
    cluster.sync();
    // columns: words rank, rank + 8, .. of the bitmap's rows, four at a time with eight warps each
    const int w8 = warp & 7, quarter = warp >> 3;
    for (int pass = 0; pass < 2; ++pass) {
        for (int w0 = rank; w0 < a.W; w0 += 4 * SEL_CTAS) {
            const int w = w0 + SEL_CTAS * quarter;
            if (w < a.W) colpart[quarter][w8][lane] = count_columns(a, b, w, w8, lane);
            __syncthreads();
            if (w < a.W && pass == 1) emit_columns(a, b, w, w8, lane, colpart[quarter]);
            const int col = w * 32 + lane;
            if (w < a.W && pass == 0 && w8 == 0 && col < a.NB) {
                int t = 0;
#pragma unroll
                for (int x = 0; x < 8; ++x) t += colpart[quarter][x][lane];
                a.colcnt[b * a.NB + col] = t;
            }
            __syncthreads();
        }
        if (pass == 1) break;
        cluster.sync();
        if (rank == 0) scan_columns(a, b, warp_total);
        cluster.sync();
    }
}

// ---------------------------------------------------------------------------------------------- original-VSA router
// Whole-block scores in the original's rounding (reference: BlockScoreParams, csrc/vsa/vsa2_kernels.h:243-253):
// S = rnd(rnd(qc . kc) * scale), rnd = round to the element type, scale = the fp32 reciprocal of sqrt(D): what Torch's
// `(q_c @ k_c^T) / sqrt(D)` computes in bf16 / fp16 (fp32-accumulated product rounded once, then multiplied by the fp32
// reciprocal of the scalar and rounded again). One thread per score; the means are small and stay in cache.
struct BlockScoreArgs {
    const void *qc, *kc;
    void* scores;            // [bh_count, NB, NB] element type
    int NB, NBc_pad, bh0;
    float inv_scale;
};
template <typename T, int D>
__global__ void __launch_bounds__(128) block_scores_kernel(const BlockScoreArgs a) {
    const int j = blockIdx.x * 128 + threadIdx.x, i = blockIdx.y, b = blockIdx.z, bh = a.bh0 + b;
    if (j >= a.NB) return;
    const T* q = static_cast<const T*>(a.qc) + ((size_t)bh * a.NBc_pad + i) * D;
    const T* k = static_cast<const T*>(a.kc) + ((size_t)bh * a.NBc_pad + j) * D;
    float acc = 0.f;
#pragma unroll 8
    for (int d = 0; d < D; d += 2) {
        const float2 x = Elt<T>::unpack(*reinterpret_cast<const uint32_t*>(q + d));
        const float2 y = Elt<T>::unpack(*reinterpret_cast<const uint32_t*>(k + d));
        acc = fmaf(x.x, y.x, acc);
        acc = fmaf(x.y, y.y, acc);
    }
    const float once = Elt<T>::to_float(Elt<T>::from_float(acc));
    static_cast<T*>(a.scores)[((size_t)b * a.NB + i) * a.NB + j] = Elt<T>::from_float(once * a.inv_scale);
}

// Per query row: exactly K = min(topk, NB) kv blocks, larger score first, ties to the smaller kv index, -0 == +0
// (reference: RowTopkParams, csrc/vsa/vsa2_kernels.h:255-270). One CTA per row: two-pass radix select of the K-th largest
// 16-bit key, then the ascending list and the selection bits. Row r of (b, h) owns idx[((b, h) * NB + r) * K ..).
struct RowTopkArgs {
    const uint16_t* scores;  // [bh_count, NB, NB]
    int NB, W, bh0, K, fp16;
    int *q2k_ptr, *q2k_idx;
    uint32_t* selbits;       // [bh_count, NB, W]
};
__device__ __forceinline__ uint32_t key16(uint16_t u, int fp16) {
    // bf16 and fp16 order like their bit patterns once the sign is handled; -0 becomes +0
    if ((u & 0x7FFFu) == 0) u = 0;
    (void)fp16;
    return (u & 0x8000u) ? (uint32_t)(uint16_t)~u : (uint32_t)(u | 0x8000u);
}
__global__ void __launch_bounds__(128) row_topk_kernel(const RowTopkArgs a) {
    __shared__ uint32_t hist[256];
    __shared__ uint32_t s_prefix, s_need;
    __shared__ int warp_gt[4], warp_eq[4];
    const int row = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, bh = a.bh0 + b;
    const uint16_t* sc = a.scores + ((size_t)b * a.NB + row) * a.NB;
    const long long base = ((long long)bh * a.NB + row) * a.K;
    if (tid == 0) {
        a.q2k_ptr[(size_t)bh * (a.NB + 1) + row] = (int)base;
        if (row == a.NB - 1) a.q2k_ptr[(size_t)bh * (a.NB + 1) + a.NB] = (int)(base + a.K);
        s_prefix = 0; s_need = (uint32_t)a.K;
    }
    __syncthreads();
    uint32_t thr = 0xFFFFFFFFu;
    int need = 0;
    if (a.K > 0) {
        for (int pass = 0; pass < 2; ++pass) {
            const int shift = 8 - 8 * pass;
            for (int x = tid; x < 256; x += 128) hist[x] = 0;
            __syncthreads();
            const uint32_t prefix = s_prefix, mask = pass == 0 ? 0u : 0xFF00u;
            for (int j = tid; j < a.NB; j += 128) {
                const uint32_t key = key16(sc[j], a.fp16);
                if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255], 1u);
            }
            __syncthreads();
            if (tid == 0) {
                uint32_t nd = s_need, d = 255;
                for (;; --d) {
                    if (hist[d] >= nd) break;
                    nd -= hist[d];
                    if (d == 0) break;
                }
                s_prefix = prefix | (d << shift);
                s_need = nd;
            }
            __syncthreads();
        }
        thr = s_prefix; need = (int)s_need;
    }
    // ascending emission, 128 columns at a time
    int pos = 0, eqrank = 0;
    for (int j0 = 0; j0 < a.NB; j0 += 128) {
        const int j = j0 + tid;
        const uint32_t key = j < a.NB ? key16(sc[j], a.fp16) : 0u;
        const bool gt = j < a.NB && a.K > 0 && key > thr, eq = j < a.NB && a.K > 0 && key == thr;
        const unsigned gm = __ballot_sync(0xffffffffu, gt), em = __ballot_sync(0xffffffffu, eq);
        if (lane == 0) { warp_gt[warp] = __popc(gm); warp_eq[warp] = __popc(em); }
        __syncthreads();
        int eq_before = eqrank, take_before = 0;
        for (int w = 0; w < warp; ++w) eq_before += warp_eq[w];
        const int my_eq = eq_before + __popc(em & ((1u << lane) - 1));
        const bool take = gt || (eq && my_eq < need);
        const unsigned tm = __ballot_sync(0xffffffffu, take);
        // positions: takes of the earlier warps of this chunk = their gt + their eq clipped to the remaining need
        int run_eq = eqrank;
        for (int w = 0; w < warp; ++w) {
            take_before += warp_gt[w] + max(0, min(warp_eq[w], need - run_eq));
            run_eq += warp_eq[w];
        }
        if (take) a.q2k_idx[base + pos + take_before + __popc(tm & ((1u << lane) - 1))] = j;
        if (lane == 0 && j0 + 32 * warp < a.W * 32) a.selbits[((size_t)b * a.NB + row) * a.W + (j0 >> 5) + warp] = tm;
        int chunk_take = 0, chunk_eq = 0, r2 = eqrank;
        for (int w = 0; w < 4; ++w) {
            chunk_take += warp_gt[w] + max(0, min(warp_eq[w], need - r2));
            r2 += warp_eq[w];
            chunk_eq += warp_eq[w];
        }
        pos += chunk_take; eqrank += chunk_eq;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------- gate fusion
// gate_mode: 0 none (weight 1), 1 one value per token [BH, L], 2 one per element [BH, L, D]; gate_act: 0 tanh, 1 identity.
struct FuseArgs {
    const void *of, *oc, *gate, *dout;
    void *o, *dout_f, *dout_c, *dgate;
    float *delta_f, *delta_c;
    const int* blk_cnt;
    int L, NB, NBc_pad, gate_mode, gate_act;
    int wide;             // every pointer is 16-byte aligned
};

// Eight 16-bit values from and to memory that is 16-byte aligned (wide), or 4-byte aligned.
__device__ __forceinline__ void load_piece(const void* p, uint32_t (&w)[4], int wide) {
    const uint32_t* q = static_cast<const uint32_t*>(p);
    if (wide) {
        const uint4 v = *reinterpret_cast<const uint4*>(q);
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = q[i];
    }
}
__device__ __forceinline__ void store_piece(void* p, const uint32_t (&w)[4], int wide) {
    uint32_t* q = static_cast<uint32_t*>(p);
    if (wide) {
        *reinterpret_cast<uint4*>(q) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = w[i];
    }
}

// One CTA per (block, bh), 16 bytes a thread and row, four rows of a thread in flight. Bound by HBM. A kernel per gate mode: none and
// per token need 32 registers, sixteen CTAs per SM; elementwise at D = 128 ten (48 registers: with twelve, 300 blocks x 5 heads 10.3 ->
// 12.5 us), at D = 64 twelve (ten: 27 -> 29). 32,768 tokens x 12 heads, D = 128, us, one kernel of twelve CTAs / here: per token 40.3 /
// 35.1, none 37.5 / 34.7, elementwise 55.4 / 54.7.
template <typename T, int D, int GATE>
__global__ void __launch_bounds__(128, GATE == 2 && D == 128 ? 10 : 12) fuse_fwd_kernel(const FuseArgs a) {
    constexpr int CH = D / 8, ROWS = 128 / CH;                 // 16-byte pieces per row, rows per pass
    const int blk = blockIdx.x, bh = blockIdx.y, c = 8 * (threadIdx.x % CH), r0 = threadIdx.x / CH;
    const int cnt = a.blk_cnt[blk];
    uint32_t ow[4];
    float oc[8];
    load_piece(static_cast<const T*>(a.oc) + ((size_t)bh * a.NBc_pad + blk) * D + c, ow, a.wide);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 v = Elt<T>::unpack(ow[i]);
        oc[2 * i] = v.x; oc[2 * i + 1] = v.y;
    }
#pragma unroll 4
    for (int r = r0; r < TB; r += ROWS) {
        const size_t row = (size_t)bh * a.L + (size_t)blk * TB + r;
        uint32_t out[4] = {0u, 0u, 0u, 0u};
        if (r < cnt) {
            uint32_t f[4], gw[4];
            load_piece(static_cast<const T*>(a.of) + row * D + c, f, a.wide);
            float gt = 1.f;
            if (GATE == 1) {
                gt = Elt<T>::to_float(static_cast<const T*>(a.gate)[row]);
                if (a.gate_act == 0) gt = tanhf(gt);
            } else if (GATE == 2) {
                load_piece(static_cast<const T*>(a.gate) + row * D + c, gw, a.wide);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 x = Elt<T>::unpack(f[i]);
                float gx = gt, gy = gt;
                if (GATE == 2) {
                    const float2 g = Elt<T>::unpack(gw[i]);
                    gx = g.x; gy = g.y;
                    if (a.gate_act == 0) { gx = tanhf(gx); gy = tanhf(gy); }
                }
                out[i] = Elt<T>::pack(x.x + gx * oc[2 * i], x.y + gy * oc[2 * i + 1]);
            }
        }
        store_piece(static_cast<T*>(a.o) + row * D + c, out, a.wide);
    }
}

// delta_f = rowsum(dO O_f); dO_c = sum over the block's valid rows of w dO; delta_c = rowsum(dO_c O_c); dgate = act'(g) * (dO .
// O_c) per token or per element; dout_f = dO on valid rows, else 0. One CTA per (block, bh), D / 8 lanes with 16 bytes each per
// row, all of a lane's rows loaded before the first is used; the row groups' shares of dO_c are added in their order. Blocks
// NB .. NBc_pad - 1 are the padding of dO_c and delta_c: zero. 32,768 tokens x 12 heads, D = 128, a gate per token: 63 us
// (149 us with a CTA-wide sum per row, 143 us with a warp per row and 8 bytes a lane: both bound by their instructions).
template <typename T, int D, int GATE>
__device__ __forceinline__ void fuse_bwd_rows(const FuseArgs& a, const int blk, const int bh, const int cnt, const uint32_t (&ow)[4],
                                              float (&sum)[8]) {
    constexpr int LR = D / 8, GROUPS = 256 / LR, ITER = TB / GROUPS;       // lanes per row, rows per pass, passes
    const int grp = threadIdx.x / LR, sub = threadIdx.x % LR, c = 8 * sub;
    const size_t first = (size_t)bh * a.L + (size_t)blk * TB;
    uint32_t dw[ITER][4], fw[ITER][4], gw[ITER][4];
    float g1[ITER];
#pragma unroll
    for (int it = 0; it < ITER; ++it) {
        const int r = it * GROUPS + grp;
        const size_t at = (first + r) * D + c;
#pragma unroll
        for (int i = 0; i < 4; ++i) dw[it][i] = fw[it][i] = gw[it][i] = 0u;
        g1[it] = 0.f;
        if (r < cnt) {
            load_piece(static_cast<const T*>(a.dout) + at, dw[it], a.wide);
            load_piece(static_cast<const T*>(a.of) + at, fw[it], a.wide);
            if (GATE == 1) g1[it] = Elt<T>::to_float(static_cast<const T*>(a.gate)[first + r]);
            if (GATE == 2) load_piece(static_cast<const T*>(a.gate) + at, gw[it], a.wide);
        }
    }
#pragma unroll
    for (int it = 0; it < ITER; ++it) {
        const int r = it * GROUPS + grp;
        const size_t row = first + r, at = row * D + c;
        if (a.dout_f) store_piece(static_cast<T*>(a.dout_f) + at, dw[it], a.wide);
        float gt = 1.f, rt = 1.f;                              // weight and its derivative factor
        if (GATE == 1) {
            gt = g1[it];
            if (a.gate_act == 0) { gt = tanhf(gt); rt = 1.f - gt * gt; }
        }
        float df = 0.f, dg = 0.f;
        uint32_t dgw[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 d = Elt<T>::unpack(dw[it][i]), f = Elt<T>::unpack(fw[it][i]), o = Elt<T>::unpack(ow[i]);
            df += d.x * f.x + d.y * f.y;
            float gx = gt, gy = gt;
            if (GATE == 1) dg += d.x * o.x + d.y * o.y;
            if (GATE == 2) {
                const float2 g = Elt<T>::unpack(gw[it][i]);
                float rx = 1.f, ry = 1.f;
                gx = g.x; gy = g.y;
                if (a.gate_act == 0) {
                    gx = tanhf(gx); gy = tanhf(gy);
                    rx = 1.f - gx * gx; ry = 1.f - gy * gy;
                }
                dgw[i] = r < cnt ? Elt<T>::pack(d.x * o.x * rx, d.y * o.y * ry) : 0u;
            }
            sum[2 * i] += gx * d.x; sum[2 * i + 1] += gy * d.y;
        }
#pragma unroll
        for (int o = LR / 2; o > 0; o >>= 1) {
            df += __shfl_xor_sync(0xffffffffu, df, o);
            if (GATE == 1) dg += __shfl_xor_sync(0xffffffffu, dg, o);
        }
        if (GATE == 2) store_piece(static_cast<T*>(a.dgate) + at, dgw, a.wide);
        if (sub == 0) {
            a.delta_f[row] = r < cnt ? df : 0.f;
            if (GATE == 1) static_cast<T*>(a.dgate)[row] = Elt<T>::from_float(r < cnt ? dg * rt : 0.f);
        }
    }
}

// Four CTAs per SM (64 registers), three with an elementwise gate at D = 128. 512 blocks x 12 heads, bf16, us, against one kernel for
// all modes (99 registers at D = 128, two CTAs per SM): token gate 96 -> 63, none 62 -> 42, elementwise 94 -> 85 (four CTAs: 99);
// at D = 64 39 -> 32 and, elementwise, 45 -> 43 (three: 48). bf16 at D = 128 spills 50 (token) and 68 bytes (elementwise) a thread for
// it.
template <typename T, int D, int GATE>
__global__ void __launch_bounds__(256, GATE == 2 && D == 128 ? 3 : 4) fuse_bwd_kernel(const FuseArgs a) {
    constexpr int LR = D / 8, GROUPS = 256 / LR;
    __shared__ __align__(16) float part[GROUPS][D];
    const int blk = blockIdx.x, bh = blockIdx.y, tid = threadIdx.x, grp = tid / LR, c = 8 * (tid % LR);
    T* dc_row = static_cast<T*>(a.dout_c) + ((size_t)bh * a.NBc_pad + blk) * D;
    float* delta_c = a.delta_c + (size_t)bh * a.NBc_pad + blk;
    if (blk >= a.NB) {
        if (tid < D / 2) reinterpret_cast<uint32_t*>(dc_row)[tid] = 0u;
        if (tid == 0) *delta_c = 0.f;
        return;
    }
    const int cnt = a.blk_cnt[blk];
    const T* oc_row = static_cast<const T*>(a.oc) + ((size_t)bh * a.NBc_pad + blk) * D;
    uint32_t ow[4];
    load_piece(oc_row + c, ow, a.wide);
    float sum[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) sum[i] = 0.f;
    fuse_bwd_rows<T, D, GATE>(a, blk, bh, cnt, ow, sum);
    *reinterpret_cast<float4*>(&part[grp][c]) = make_float4(sum[0], sum[1], sum[2], sum[3]);
    *reinterpret_cast<float4*>(&part[grp][c + 4]) = make_float4(sum[4], sum[5], sum[6], sum[7]);
    __syncthreads();
    __shared__ float red[D / 64];
    if (tid < D / 2) {
        float2 x = make_float2(0.f, 0.f);
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) { x.x += part[g][2 * tid]; x.y += part[g][2 * tid + 1]; }
        // the coarse branch sees dO_c rounded to the element type, like every tensor that crosses a kernel boundary
        const uint32_t packed = Elt<T>::pack(x.x, x.y);
        reinterpret_cast<uint32_t*>(dc_row)[tid] = packed;
        const float2 dc = Elt<T>::unpack(packed), o = Elt<T>::unpack(reinterpret_cast<const uint32_t*>(oc_row)[tid]);
        float t = dc.x * o.x + dc.y * o.y;
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) t += __shfl_xor_sync(0xffffffffu, t, k);
        if ((tid & 31) == 0) red[tid >> 5] = t;
    }
    __syncthreads();
    if (tid == 0) *delta_c = D == 128 ? red[0] + red[D / 64 - 1] : red[0];
}

// out = valid ? acc + add[block] / count : 0, cast to the element type (acc and add optional).
struct FinalArgs {
    const float *acc, *add;
    void* out;
    const int* blk_cnt;
    int L, add_nb;
};
template <typename T, int D>
__global__ void __launch_bounds__(D / 2) finalize_kernel(const FinalArgs a) {
    const int blk = blockIdx.x, bh = blockIdx.y, c = 2 * threadIdx.x;
    const int cnt = a.blk_cnt[blk];
    float ax = 0.f, ay = 0.f;
    if (a.add) {
        const float* p = a.add + ((size_t)bh * a.add_nb + blk) * D + c;
        ax = p[0] / (float)cnt; ay = p[1] / (float)cnt;
    }
    for (int r = 0; r < TB; ++r) {
        const size_t row = (size_t)bh * a.L + (size_t)blk * TB + r;
        uint32_t out = 0u;
        if (r < cnt) {
            float x = ax, y = ay;
            if (a.acc) { x += a.acc[row * D + c]; y += a.acc[row * D + c + 1]; }
            out = Elt<T>::pack(x, y);
        }
        *reinterpret_cast<uint32_t*>(static_cast<T*>(a.out) + row * D + c) = out;
    }
}

static int check_shape(const char* name, int BH, int L, int D, int dtype) {
    if (BH <= 0 || L <= 0 || L % TB != 0) return set_error(-1, (std::string(name) + ": BH > 0 and L a positive multiple of 64").c_str());
    if (D != 64 && D != 128) return set_error(-1, (std::string(name) + ": head dim must be 64 or 128").c_str());
    if (dtype != 0 && dtype != 1) return set_error(-1, (std::string(name) + ": dtype must be 0 (bf16) or 1 (fp16)").c_str());
    return 0;
}

#define VSA_LAUNCH(KERNEL, GRID, THREADS, SMEM, ARGS)                                              \
    do {                                                                                           \
        if (dtype == 0 && D == 128) KERNEL<__nv_bfloat16, 128><<<GRID, THREADS, SMEM, st>>>(ARGS);  \
        else if (dtype == 0) KERNEL<__nv_bfloat16, 64><<<GRID, THREADS, SMEM, st>>>(ARGS);          \
        else if (D == 128) KERNEL<__half, 128><<<GRID, THREADS, SMEM, st>>>(ARGS);                  \
        else KERNEL<__half, 64><<<GRID, THREADS, SMEM, st>>>(ARGS);                                 \
    } while (0)

}  // namespace vsa
}  // namespace es

using namespace es;
using namespace es::vsa;

extern "C" int es_vsa_pool(const void* q, const void* k, const void* v, void* qr, void* kr, void* vr, void* qc, void* kc,
                           void* vc, const int32_t* blk_cnt, int32_t BH, int32_t L, int32_t D, int32_t R, int32_t Lr_pad,
                           int32_t NBc_pad, int32_t dtype, void* stream) {
    if ((!q && !k && !v) || !blk_cnt) return set_error(-1, "es_vsa_pool: null pointer");
    if ((!q && (qr || qc)) || (!k && (kr || kc))) return set_error(-1, "es_vsa_pool: an output without its input");
    if (int rc = check_shape("es_vsa_pool", BH, L, D, dtype)) return rc;
    if (R < 1 || R > 64 || 64 % R != 0) return set_error(-1, "es_vsa_pool: R must divide 64");
    const int NB = L / TB, G = 64 / R;
    if (Lr_pad < NB * G || NBc_pad < NB) return set_error(-1, "es_vsa_pool: padded sizes smaller than the real ones");
    if ((vr || vc) && !v) return set_error(-1, "es_vsa_pool: v outputs without v");
    if (!aligned(4, q, k, v, qr, kr, vr, qc, kc, vc)) return set_error(-1, "es_vsa_pool: tensors must be 4-byte aligned");
    // tensors without outputs at either end have no CTAs (60,000 empty ones: 10 us)
    const bool out[3] = {qr || qc, kr || kc, vr || vc};
    const int first = out[0] ? 0 : out[1] ? 1 : 2, last = out[2] ? 2 : out[1] ? 1 : 0;
    if (first > last) return 0;
    PoolArgs a{q, k, v, qr, kr, vr, qc, kc, vc, blk_cnt, L, NB, R, G, Lr_pad, NBc_pad, first};
    cudaStream_t st = (cudaStream_t)stream;
    const int rows = max(max(NB, NBc_pad), (Lr_pad + G - 1) / G);
    const dim3 grid(rows, BH, last - first + 1);
#define POOL_CASE(TT, DD)                                                          \
    {                                                                              \
        if (R == 16) pool_kernel<TT, DD, 16><<<grid, DD / 2, 0, st>>>(a);          \
        else if (R == 8) pool_kernel<TT, DD, 8><<<grid, DD / 2, 0, st>>>(a);       \
        else if (R == 32) pool_kernel<TT, DD, 32><<<grid, DD / 2, 0, st>>>(a);     \
        else if (R == 4) pool_kernel<TT, DD, 4><<<grid, DD / 2, 0, st>>>(a);       \
        else pool_kernel<TT, DD, 0><<<grid, DD / 2, 0, st>>>(a);                   \
    }
    if (dtype == 0 && D == 128) POOL_CASE(__nv_bfloat16, 128)
    else if (dtype == 0) POOL_CASE(__nv_bfloat16, 64)
    else if (D == 128) POOL_CASE(__half, 128)
    else POOL_CASE(__half, 64)
#undef POOL_CASE
    ES_CHECK_LAUNCH("pool_kernel");
    return 0;
}

static int sm_count() {
    int dev = 0, sms = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess ? sms : 148;
}

// A kernel built for one CTA per SM fewer is a few percent faster (more registers), and so are fewer that run at once, but a round more
// costs far more: the larger number is taken where it saves a round. 12 heads, us, 3 / 4 CTAs per SM at D = 128: scores, 468 CTAs (NB =
// 624, R = 16) 222 / 130, 456 208 / 125, 768 (two rounds either way) 364 / 408, 600 (4 heads) 859 / 873; LSE, 468 113 / 86, 192 24.8 /
// 25.9. 4 / 5 at D = 64: scores, 600 761 / 446, 384 80 / 82; LSE, 600 327 / 279, 768 147 / 167.
template <typename T, int D, int MODE>
static int launch_router_as(const RouterArgs& a, int bh_count, cudaStream_t st) {
    constexpr int FEW = D == 128 ? 3 : 4, MANY = FEW + 1;
    constexpr bool BY_SMEM = D == 128 && MODE == 1;       // one kernel, and three of them where it asks for more shared memory
    const dim3 grid(a.Lr_pad / TB, bh_count);
    const long long n = (long long)grid.x * grid.y, sms = sm_count();
    const bool many = (n + MANY * sms - 1) / (MANY * sms) < (n + FEW * sms - 1) / (FEW * sms);
    const int smem = (int)RouterSmem<D, MODE>::BYTES + (BY_SMEM && !many ? 12 * 1024 : 0);
    auto launch = [&](auto few, auto more) -> int {
        auto kernel = many ? more : few;
        if (int rc = opt_in_shared_memory((const void*)kernel, smem)) return rc;
        kernel<<<grid, 128, smem, st>>>(a);
        ES_CHECK_LAUNCH("router_kernel");
        return 0;
    };
    constexpr int C0 = BY_SMEM ? MANY : FEW;
    if (a.G == 2) return launch(router_kernel<T, D, MODE, 2, C0>, router_kernel<T, D, MODE, 2, MANY>);
    if (a.G == 4) return launch(router_kernel<T, D, MODE, 4, C0>, router_kernel<T, D, MODE, 4, MANY>);
    if (a.G == 8) return launch(router_kernel<T, D, MODE, 8, C0>, router_kernel<T, D, MODE, 8, MANY>);
    return launch(router_kernel<T, D, MODE, 0, C0>, router_kernel<T, D, MODE, 0, MANY>);
}

template <int MODE>
static int launch_router(const RouterArgs& a, int D, int dtype, int bh_count, cudaStream_t st) {
    if (dtype == 0 && D == 128) return launch_router_as<__nv_bfloat16, 128, MODE>(a, bh_count, st);
    if (dtype == 0) return launch_router_as<__nv_bfloat16, 64, MODE>(a, bh_count, st);
    if (D == 128) return launch_router_as<__half, 128, MODE>(a, bh_count, st);
    return launch_router_as<__half, 64, MODE>(a, bh_count, st);
}

extern "C" int es_vsa_router_lse(const void* qr, const void* kr, float* lse2, const int32_t* blk_cnt, int32_t BH,
                                 int32_t NB, int32_t D, int32_t R, int32_t Lr_pad, int32_t dtype, void* stream) {
    if (!qr || !kr || !lse2 || !blk_cnt) return set_error(-1, "es_vsa_router_lse: null pointer");
    if (int rc = check_shape("es_vsa_router_lse", BH, NB * TB, D, dtype)) return rc;
    if (R < 1 || R > 64 || 64 % R != 0 || Lr_pad % TB != 0 || Lr_pad < NB * (64 / R))
        return set_error(-1, "es_vsa_router_lse: R must divide 64 and Lr_pad be a multiple of 64 covering NB * 64 / R");
    if (!aligned(16, qr, kr)) return set_error(-1, "es_vsa_router_lse: qr and kr must be 16-byte aligned");
    RouterArgs a{qr, kr, lse2, nullptr, blk_cnt, NB, R, 64 / R, NB * (64 / R), Lr_pad, 0, 1, LOG2E / sqrtf((float)D)};
    return launch_router<0>(a, D, dtype, BH, (cudaStream_t)stream);
}

extern "C" int es_vsa_router_scores(const void* qr, const void* kr, const float* lse2, float* scores,
                                    const int32_t* blk_cnt, int32_t BH, int32_t NB, int32_t D, int32_t R, int32_t Lr_pad,
                                    int32_t bh0, int32_t bh_count, int32_t row_norm, int32_t dtype, void* stream) {
    if (!qr || !kr || !lse2 || !scores || !blk_cnt) return set_error(-1, "es_vsa_router_scores: null pointer");
    if (int rc = check_shape("es_vsa_router_scores", BH, NB * TB, D, dtype)) return rc;
    if (R < 1 || R > 64 || 64 % R != 0 || Lr_pad % TB != 0 || Lr_pad < NB * (64 / R))
        return set_error(-1, "es_vsa_router_scores: R must divide 64 and Lr_pad be a multiple of 64 covering NB * 64 / R");
    if (bh0 < 0 || bh_count < 1 || bh0 + bh_count > BH) return set_error(-1, "es_vsa_router_scores: bad (b, h) range");
    if (row_norm != 0 && row_norm != 1) return set_error(-1, "es_vsa_router_scores: row_norm must be 0 or 1");
    if (!aligned(16, qr, kr)) return set_error(-1, "es_vsa_router_scores: qr and kr must be 16-byte aligned");
    RouterArgs a{qr, kr, const_cast<float*>(lse2), scores, blk_cnt, NB, R, 64 / R, NB * (64 / R), Lr_pad, bh0, row_norm,
                 LOG2E / sqrtf((float)D)};
    return launch_router<1>(a, D, dtype, bh_count, (cudaStream_t)stream);
}

// Clusters of topk_kernel that the current device runs at once (a cluster's CTAs share a GPC, so it is fewer than SMs / CTAs), asked
// for once per device; 0 where that fails.
static int topk_clusters_at_once() {
    static std::atomic<int> known[64];                   // 1 + the count
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int n = known[dev].load(std::memory_order_relaxed) - 1;
    if (n >= 0) return n;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = SEL_CTAS; attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(SEL_CTAS); cfg.blockDim = dim3(1024); cfg.attrs = &attr; cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, topk_kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();                              // the other path needs no clusters at once
        n = 0;
    }
    known[dev].store(n + 1, std::memory_order_relaxed);
    return n;
}

extern "C" long long es_vsa_topk_workspace_bytes(int32_t bh_count, int32_t NB) {
    if (bh_count <= 0 || NB <= 0) return 0;
    const long long W = (NB + 31) / 32;
    return (long long)bh_count * (4 + 4LL * NB + W * NB) * 4;
}

// Byte offset of the selection bitmap [bh_count, NB, ceil(NB / 32)] that es_vsa_global_topk leaves in its workspace.
extern "C" long long es_vsa_topk_bits_offset(int32_t bh_count, int32_t NB) {
    if (bh_count <= 0 || NB <= 0) return 0;
    return (long long)bh_count * (4 + 4LL * NB) * 4;
}

extern "C" int es_vsa_global_topk(const float* scores, int32_t NB, int32_t bh0, int32_t bh_count, long long budget,
                                  int32_t* q2k_ptr, int32_t* q2k_idx, int32_t* k2q_ptr, int32_t* k2q_idx, void* workspace,
                                  void* stream) {
    if (!scores || !q2k_ptr || !q2k_idx || !k2q_ptr || !k2q_idx || !workspace)
        return set_error(-1, "es_vsa_global_topk: null pointer");
    if (NB <= 0 || bh_count <= 0 || bh0 < 0) return set_error(-1, "es_vsa_global_topk: bad sizes");
    if (budget < 0 || budget > (long long)NB * NB) return set_error(-1, "es_vsa_global_topk: budget outside [0, NB * NB]");
    if ((long long)(bh0 + bh_count) * budget > 0x7FFFFFFFLL) return set_error(-1, "es_vsa_global_topk: offsets exceed int32");
    TopkArgs a{};
    a.scores = scores; a.NB = NB; a.W = (NB + 31) / 32; a.bh0 = bh0; a.budget = budget;
    a.q2k_ptr = q2k_ptr; a.q2k_idx = q2k_idx; a.k2q_ptr = k2q_ptr; a.k2q_idx = k2q_idx;
    int* w = static_cast<int*>(workspace);
    a.state = w; w += (size_t)bh_count * 4;
    a.gtcnt = w; w += (size_t)bh_count * NB;
    a.eqcnt = w; w += (size_t)bh_count * NB;
    a.eqbase = w; w += (size_t)bh_count * NB;
    a.colcnt = w; w += (size_t)bh_count * NB;
    a.selbits = reinterpret_cast<uint32_t*>(w);
    cudaStream_t st = (cudaStream_t)stream;
    // One launch where all clusters run at once (15 on a B200) and a warp has one row; beyond, the stages are launches of their own,
    // whose rows and columns go to all SMs. Device time of one call after the other in a graph, us, one launch / seven: 64 blocks x 15
    // heads 20.8 / 24.8, x 16 35.6 / 26.3 (a second round of clusters); 256 x 12 26.0 / 30.2, x 15 26.0 / 30.6, x 16 49.6 / 33.2;
    // 272 x 12 34.6 / 35.4, 288 x 12 36.1 / 35.8, 304 x 12 38.3 / 37.4, 384 x 12 42.0 / 40.6, 624 x 12 74.5 / 66.4, 1,600 x 1 324 / 171.
    if (NB <= 256 && bh_count <= topk_clusters_at_once()) {
        topk_kernel<<<dim3(SEL_CTAS, bh_count), 1024, 0, st>>>(a);
        ES_CHECK_LAUNCH("topk_kernel");
        return 0;
    }
    topk_select_kernel<<<dim3(SEL_CTAS, bh_count), 1024, 0, st>>>(a);
    ES_CHECK_LAUNCH("topk_select_kernel");
    const dim3 rows((NB + 3) / 4, bh_count), cols(a.W, bh_count);
    topk_count_kernel<<<rows, 128, 0, st>>>(a);
    ES_CHECK_LAUNCH("topk_count_kernel");
    topk_scan_kernel<<<bh_count, 1024, 0, st>>>(a, 0);
    ES_CHECK_LAUNCH("topk_scan_kernel");
    topk_emit_rows_kernel<<<rows, 128, 0, st>>>(a);
    ES_CHECK_LAUNCH("topk_emit_rows_kernel");
    topk_cols_kernel<<<cols, 256, 0, st>>>(a, 0);
    ES_CHECK_LAUNCH("topk_cols_kernel");
    topk_scan_kernel<<<bh_count, 1024, 0, st>>>(a, 1);
    ES_CHECK_LAUNCH("topk_scan_kernel");
    topk_cols_kernel<<<cols, 256, 0, st>>>(a, 1);
    ES_CHECK_LAUNCH("topk_cols_kernel");
    return 0;
}

extern "C" int es_vsa_fuse_fwd(const void* of, const void* oc, const void* gate, void* o, const int32_t* blk_cnt,
                               int32_t BH, int32_t L, int32_t D, int32_t NBc_pad, int32_t gate_mode, int32_t gate_act,
                               int32_t dtype, void* stream) {
    if (!of || !oc || !o || !blk_cnt) return set_error(-1, "es_vsa_fuse_fwd: null pointer");
    if (int rc = check_shape("es_vsa_fuse_fwd", BH, L, D, dtype)) return rc;
    if (gate_mode < 0 || gate_mode > 2 || (gate_mode != 0 && !gate)) return set_error(-1, "es_vsa_fuse_fwd: bad gate mode");
    if (gate_act < 0 || gate_act > 1 || NBc_pad < L / TB) return set_error(-1, "es_vsa_fuse_fwd: bad gate_act or NBc_pad");
    if (!aligned(4, of, oc, o, gate_mode == 2 ? gate : nullptr)) return set_error(-1, "es_vsa_fuse_fwd: tensors must be 4-byte aligned");
    FuseArgs a{};
    a.of = of; a.oc = oc; a.gate = gate; a.o = o; a.blk_cnt = blk_cnt; a.L = L; a.NB = L / TB; a.NBc_pad = NBc_pad;
    a.gate_mode = gate_mode; a.gate_act = gate_act;
    a.wide = (((uintptr_t)of | (uintptr_t)oc | (uintptr_t)o | (gate_mode == 2 ? (uintptr_t)gate : 0)) & 15) == 0;
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 grid(L / TB, BH);
#define FUSE_FWD_CASE(TT, DD)                                                              \
    {                                                                                      \
        if (gate_mode == 0) fuse_fwd_kernel<TT, DD, 0><<<grid, 128, 0, st>>>(a);           \
        else if (gate_mode == 1) fuse_fwd_kernel<TT, DD, 1><<<grid, 128, 0, st>>>(a);      \
        else fuse_fwd_kernel<TT, DD, 2><<<grid, 128, 0, st>>>(a);                          \
    }
    if (dtype == 0 && D == 128) FUSE_FWD_CASE(__nv_bfloat16, 128)
    else if (dtype == 0) FUSE_FWD_CASE(__nv_bfloat16, 64)
    else if (D == 128) FUSE_FWD_CASE(__half, 128)
    else FUSE_FWD_CASE(__half, 64)
#undef FUSE_FWD_CASE
    ES_CHECK_LAUNCH("fuse_fwd_kernel");
    return 0;
}

extern "C" int es_vsa_fuse_bwd(const void* dout, const void* of, const void* oc, const void* gate, void* dout_f,
                               float* delta_f, void* dout_c, float* delta_c, void* dgate, const int32_t* blk_cnt,
                               int32_t BH, int32_t L, int32_t D, int32_t NBc_pad, int32_t gate_mode, int32_t gate_act,
                               int32_t dtype, void* stream) {
    if (!dout || !of || !oc || !delta_f || !dout_c || !delta_c || !blk_cnt) return set_error(-1, "es_vsa_fuse_bwd: null pointer");
    if (int rc = check_shape("es_vsa_fuse_bwd", BH, L, D, dtype)) return rc;
    if (gate_mode < 0 || gate_mode > 2 || (gate_mode != 0 && (!gate || !dgate))) return set_error(-1, "es_vsa_fuse_bwd: bad gate mode");
    if (gate_act < 0 || gate_act > 1 || NBc_pad < L / TB) return set_error(-1, "es_vsa_fuse_bwd: bad gate_act or NBc_pad");
    if (!aligned(4, dout, of, oc, dout_f, dout_c, gate_mode == 2 ? gate : nullptr, gate_mode == 2 ? dgate : nullptr))
        return set_error(-1, "es_vsa_fuse_bwd: tensors must be 4-byte aligned");
    FuseArgs a{};
    a.dout = dout; a.of = of; a.oc = oc; a.gate = gate; a.dout_f = dout_f; a.delta_f = delta_f; a.dout_c = dout_c;
    a.delta_c = delta_c; a.dgate = dgate; a.blk_cnt = blk_cnt; a.L = L; a.NB = L / TB; a.NBc_pad = NBc_pad;
    a.gate_mode = gate_mode; a.gate_act = gate_act;
    a.wide = (((uintptr_t)dout | (uintptr_t)of | (uintptr_t)oc | (uintptr_t)dout_f | (uintptr_t)dout_c |
               (gate_mode == 2 ? (uintptr_t)gate | (uintptr_t)dgate : 0)) & 15) == 0;
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 grid(NBc_pad, BH);
#define FUSE_BWD_CASE(TT, DD)                                                              \
    {                                                                                      \
        if (gate_mode == 0) fuse_bwd_kernel<TT, DD, 0><<<grid, 256, 0, st>>>(a);           \
        else if (gate_mode == 1) fuse_bwd_kernel<TT, DD, 1><<<grid, 256, 0, st>>>(a);      \
        else fuse_bwd_kernel<TT, DD, 2><<<grid, 256, 0, st>>>(a);                          \
    }
    if (dtype == 0 && D == 128) FUSE_BWD_CASE(__nv_bfloat16, 128)
    else if (dtype == 0) FUSE_BWD_CASE(__nv_bfloat16, 64)
    else if (D == 128) FUSE_BWD_CASE(__half, 128)
    else FUSE_BWD_CASE(__half, 64)
#undef FUSE_BWD_CASE
    ES_CHECK_LAUNCH("fuse_bwd_kernel");
    return 0;
}

extern "C" int es_vsa_finalize(const float* acc, const float* add, void* out, const int32_t* blk_cnt, int32_t BH,
                               int32_t L, int32_t D, int32_t add_nb, int32_t dtype, void* stream) {
    if (!out || !blk_cnt) return set_error(-1, "es_vsa_finalize: null pointer");
    if (int rc = check_shape("es_vsa_finalize", BH, L, D, dtype)) return rc;
    if (add && add_nb < L / TB) return set_error(-1, "es_vsa_finalize: add_nb smaller than the block count");
    if (!aligned(4, out)) return set_error(-1, "es_vsa_finalize: out must be 4-byte aligned");
    FinalArgs a{acc, add, out, blk_cnt, L, add_nb};
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 grid(L / TB, BH);
    VSA_LAUNCH(finalize_kernel, grid, D / 2, 0, a);
    ES_CHECK_LAUNCH("finalize_kernel");
    return 0;
}

extern "C" int es_vsa_block_scores(const void* qc, const void* kc, void* scores, int32_t BH, int32_t NB, int32_t D,
                                   int32_t NBc_pad, int32_t bh0, int32_t bh_count, int32_t dtype, void* stream) {
    if (!qc || !kc || !scores) return set_error(-1, "es_vsa_block_scores: null pointer");
    if (int rc = check_shape("es_vsa_block_scores", BH, NB * TB, D, dtype)) return rc;
    if (NBc_pad < NB || bh0 < 0 || bh_count < 1 || bh0 + bh_count > BH) return set_error(-1, "es_vsa_block_scores: bad sizes");
    if (!aligned(4, qc, kc)) return set_error(-1, "es_vsa_block_scores: qc and kc must be 4-byte aligned");
    BlockScoreArgs a{qc, kc, scores, NB, NBc_pad, bh0, 1.0f / sqrtf((float)D)};
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 grid((NB + 127) / 128, NB, bh_count);
    VSA_LAUNCH(block_scores_kernel, grid, 128, 0, a);
    ES_CHECK_LAUNCH("block_scores_kernel");
    return 0;
}

extern "C" int es_vsa_row_topk(const void* scores, int32_t NB, int32_t bh0, int32_t bh_count, int32_t topk,
                               int32_t* q2k_ptr, int32_t* q2k_idx, int32_t* k2q_ptr, int32_t* k2q_idx, void* workspace,
                               int32_t dtype, void* stream) {
    if (!scores || !q2k_ptr || !q2k_idx || !k2q_ptr || !k2q_idx || !workspace) return set_error(-1, "es_vsa_row_topk: null pointer");
    if (NB <= 0 || bh_count <= 0 || bh0 < 0 || topk < 0) return set_error(-1, "es_vsa_row_topk: bad sizes");
    if (dtype != 0 && dtype != 1) return set_error(-1, "es_vsa_row_topk: dtype must be 0 (bf16) or 1 (fp16)");
    const int K = topk < NB ? topk : NB;
    if ((long long)(bh0 + bh_count) * NB * K > 0x7FFFFFFFLL) return set_error(-1, "es_vsa_row_topk: offsets exceed int32");
    // the workspace has the layout of es_vsa_global_topk's: the column stages are shared with it
    TopkArgs t{};
    t.NB = NB; t.W = (NB + 31) / 32; t.bh0 = bh0; t.budget = (long long)NB * K;
    t.q2k_ptr = q2k_ptr; t.q2k_idx = q2k_idx; t.k2q_ptr = k2q_ptr; t.k2q_idx = k2q_idx;
    int* w = static_cast<int*>(workspace);
    w += (size_t)bh_count * 4;                         // its thresholds, which rows here have none of
    t.gtcnt = w; w += (size_t)bh_count * NB;
    t.eqcnt = w; w += (size_t)bh_count * NB;
    t.eqbase = w; w += (size_t)bh_count * NB;
    t.colcnt = w; w += (size_t)bh_count * NB;
    t.selbits = reinterpret_cast<uint32_t*>(w);
    RowTopkArgs a{static_cast<const uint16_t*>(scores), NB, t.W, bh0, K, dtype, q2k_ptr, q2k_idx, t.selbits};
    cudaStream_t st = (cudaStream_t)stream;
    row_topk_kernel<<<dim3(NB, bh_count), 128, 0, st>>>(a);
    ES_CHECK_LAUNCH("row_topk_kernel");
    const dim3 cols(t.W, bh_count);
    topk_cols_kernel<<<cols, 256, 0, st>>>(t, 0);
    ES_CHECK_LAUNCH("topk_cols_kernel");
    topk_scan_kernel<<<bh_count, 1024, 0, st>>>(t, 1);
    ES_CHECK_LAUNCH("topk_scan_kernel");
    topk_cols_kernel<<<cols, 256, 0, st>>>(t, 1);
    ES_CHECK_LAUNCH("topk_cols_kernel");
    return 0;
}
