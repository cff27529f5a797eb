// VSA2 with 64 / RM / 1 representative tiers: every (query block, kv block) pair is attended at one of three resolutions,
// one online softmax over all of them.
//   tier A: the pair is in the CSR selection (and in bits_a): the block's valid tokens, bias 0;
//   tier B: bits_ab & ~bits_a: the block's RM group means (groups of 64 / RM tokens), each with bias log2(tokens in the group);
//   tier C: ~bits_ab: the block mean, bias log2(tokens in the block).
// Reference: experiments/vsa2_representative/vsa2_rep/reference.py:53-96 (the math) and csrc/rep/rep_api.cpp:90-505 of
// shaoshitong/self_trainable_or_free_attn (rep_attn_fwd, rep_attn_bwd_q, tier_a_bwd_kv, rep_unpool). The representative
// tables are the pooled means the router already needs (group means of K and V, block means of K and V).
//
// The attention runs in the tcgen05 kernels of es_vsa_tc_fwd.cu and es_vsa_tc_bwd.cu, as modes that walk all three tiers; the
// gradients of the representatives come from a pass of its own with one CTA per tile of 64 consecutive table rows: every
// table row has one owner, no atomics. Here: the entry points, and the spreading of the tables' gradients over the tokens.
#include <string>

#include "es_vsa_mma.cuh"
#include "es_vsa_tc.cuh"

namespace es {
namespace vsa {

// Token gradients from the three sources: out = valid ? tok[t] + mid[block * RM + group] / tokens in the group
// + (tail[block] + add[block]) / tokens in the block : 0. tok, mid, tail, add are fp32 and optional.
struct UnpoolArgs {
    const float *tok, *mid, *tail, *add;
    void* out;
    const int* blk_cnt;
    int L, RM, mid_stride, tail_stride, add_nb;
    int wide;                      // the fp32 tensors are 16-byte, out 8-byte aligned
};
// Four columns a lane, D / 4 lanes a row. A thread's rows follow one another, so that it loads and divides a group's gradient once or
// twice instead of once a row. TOK: with the tokens' own gradients, all rows of a thread requested before the first is needed;
// without them there is less to hold, and smaller CTAs write faster (256 threads: 27 instead of 25 us below, 62 instead of 48 where
// there is only `tail`, D = 64). Bound by HBM. D = 128, bf16, four groups a block, us, before (a row's division each) / here: 512 blocks
// x 12 heads, tok + mid + tail 59 / 45, mid + tail 55 / 25; 1,500 x 12 160 / 121 and 150 / 61.
template <bool TOK> constexpr int UNPOOL_THREADS = TOK ? 256 : 128;
template <typename T, int D, bool TOK>
__global__ void __launch_bounds__((UNPOOL_THREADS<TOK>), TOK ? (D == 128 ? 4 : 6) : 16) tier_unpool_kernel(const UnpoolArgs a) {
    constexpr int LR = D / 4, ROWS = TB / (UNPOOL_THREADS<TOK> / LR), QUADS = ROWS / 4;   // lanes per row, rows of a thread; groups have 4 rows or more
    const int blk = blockIdx.x, bh = blockIdx.y, c = 4 * (threadIdx.x % LR), r0 = threadIdx.x / LR * ROWS;
    const int cnt = a.blk_cnt[blk], R = TB / a.RM;
    auto load4 = [&](const float* p) { return a.wide ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]); };
    const size_t first = (size_t)bh * a.L + (size_t)blk * TB + r0;
    float4 tok[ROWS], m[QUADS];
    if (TOK) {
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
            if (r0 + i < cnt) tok[i] = load4(a.tok + (first + i) * D + c);
    }
    if (a.mid) {
#pragma unroll
        for (int x = 0; x < QUADS; ++x) m[x] = load4(a.mid + ((size_t)bh * a.mid_stride + (size_t)blk * a.RM + (r0 + 4 * x) / R) * D + c);
    }
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.tail) t = load4(a.tail + ((size_t)bh * a.tail_stride + blk) * D + c);
    if (a.add) {
        const float4 x = load4(a.add + ((size_t)bh * a.add_nb + blk) * D + c);
        t.x += x.x; t.y += x.y; t.z += x.z; t.w += x.w;
    }
    t.x /= (float)cnt; t.y /= (float)cnt; t.z /= (float)cnt; t.w /= (float)cnt;
#pragma unroll
    for (int x = 0; x < QUADS; ++x) {
        float4 base = t;
        if (a.mid) {
            const float cg = (float)min(cnt - (r0 + 4 * x) / R * R, R);    // (not positive: no row of the group is below cnt)
            base.x += m[x].x / cg; base.y += m[x].y / cg; base.z += m[x].z / cg; base.w += m[x].w / cg;
        }
#pragma unroll
        for (int i = 4 * x; i < 4 * x + 4; ++i) {
            uint32_t out[2] = {0u, 0u};
            if (r0 + i < cnt) {
                float4 y = base;
                if (TOK) { y.x += tok[i].x; y.y += tok[i].y; y.z += tok[i].z; y.w += tok[i].w; }
                out[0] = Elt<T>::pack(y.x, y.y);
                out[1] = Elt<T>::pack(y.z, y.w);
            }
            uint32_t* dst = reinterpret_cast<uint32_t*>(static_cast<T*>(a.out) + (first + i) * D + c);
            if (a.wide) *reinterpret_cast<uint2*>(dst) = make_uint2(out[0], out[1]);
            else { dst[0] = out[0]; dst[1] = out[1]; }
        }
    }
}

static int check_tier(const char* name, int BH, int L, int D, int dtype, int RM, int phases, int mid_stride, int tail_stride) {
    if (BH <= 0 || L <= 0 || L % TB != 0) return set_error(-1, (std::string(name) + ": BH > 0 and L a positive multiple of 64").c_str());
    if (D != 64 && D != 128) return set_error(-1, (std::string(name) + ": head dim must be 64 or 128").c_str());
    if (dtype != 0 && dtype != 1) return set_error(-1, (std::string(name) + ": dtype must be 0 (bf16) or 1 (fp16)").c_str());
    if (RM != 2 && RM != 4 && RM != 8 && RM != 16) return set_error(-1, (std::string(name) + ": mid_reps must be 2, 4, 8 or 16").c_str());
    if (phases < 0 || phases > 7) return set_error(-1, (std::string(name) + ": phases is a mask of 1 (A), 2 (B), 4 (C)").c_str());
    const int NB = L / TB;
    if (mid_stride < (NB * RM + TB - 1) / TB * TB || tail_stride < (NB + TB - 1) / TB * TB)
        return set_error(-1, (std::string(name) + ": the tables must be padded to multiples of 64 rows").c_str());
    if (NB > 4096) return set_error(-1, (std::string(name) + ": at most 4096 blocks").c_str());
    return 0;
}

// es_vsa_tc_fwd.cu, es_vsa_tc_bwd.cu
int tier_fwd_tc(const void* q, const void* k, const void* v, const void* k_mid, const void* v_mid, const void* k_tail,
                const void* v_tail, void* o, float* lse, const int* row_ptr, const int* col_idx, const TierMaps& tier,
                const int* blk_cnt, int BH, int L, int D, int dtype, cudaStream_t st);
int tier_bwd_q_tc(const void* q, const void* k, const void* v, const void* k_mid, const void* v_mid, const void* k_tail,
                  const void* v_tail, const void* dout, const float* lse, const float* delta, void* dq, const float* add, int add_nb,
                  const int* row_ptr, const int* col_idx, const TierMaps& tier, const int* blk_cnt, int BH, int L, int D, int dtype,
                  cudaStream_t st);
int tier_rep_bwd_tc(const void* q, const void* k_mid, const void* v_mid, const void* k_tail, const void* v_tail, const void* dout,
                    const float* lse, const float* delta, float* dk_mid, float* dv_mid, float* dk_tail, float* dv_tail,
                    const TierMaps& tier, const int* blk_cnt, int BH, int L, int D, int dtype, int tiles, cudaStream_t st);

}  // namespace vsa
}  // namespace es

using namespace es;
using namespace es::vsa;

// es_vsa_attn.cu
extern "C" int es_vsa_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const int32_t* row_ptr,
                               const int32_t* col_idx, const int32_t* blk_cnt, int32_t BH, int32_t L, int32_t D,
                               int32_t dtype, void* stream);
extern "C" int es_vsa_attn_bwd_q(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                                 const float* delta, void* dq, float* dq_f32, const float* add_dq, int32_t add_nb,
                                 const int32_t* q2k_ptr, const int32_t* q2k_idx, const int32_t* blk_cnt, int32_t BH,
                                 int32_t L, int32_t D, int32_t dtype, void* stream);

static TierMaps tier_maps(const int32_t* bits_a, const int32_t* bits_ab, int L, int RM, int mid_stride, int tail_stride, int phases) {
    return {(const uint32_t*)bits_a, (const uint32_t*)bits_ab, (L / TB + 31) / 32, RM, mid_stride, tail_stride, phases, {}};
}

extern "C" int es_vsa_tier_attn_fwd(const void* q, const void* k, const void* v, const void* k_mid, const void* v_mid,
                                    const void* k_tail, const void* v_tail, void* o, float* lse, const int32_t* q2k_ptr,
                                    const int32_t* q2k_idx, const int32_t* bits_a, const int32_t* bits_ab,
                                    const int32_t* blk_cnt, int32_t BH, int32_t L, int32_t D, int32_t mid_reps,
                                    int32_t mid_stride, int32_t tail_stride, int32_t phases, int32_t dtype, void* stream) {
    if (!q || !k || !v || !k_mid || !v_mid || !k_tail || !v_tail || !o || !lse || !q2k_ptr || !q2k_idx || !bits_a || !bits_ab || !blk_cnt)
        return set_error(-1, "es_vsa_tier_attn_fwd: null pointer");
    if (int rc = check_tier("es_vsa_tier_attn_fwd", BH, L, D, dtype, mid_reps, phases, mid_stride, tail_stride)) return rc;
    // tier A alone is the plain fine branch
    if (phases == PH_A) return es_vsa_attn_fwd(q, k, v, o, lse, q2k_ptr, q2k_idx, blk_cnt, BH, L, D, dtype, stream);
    return tier_fwd_tc(q, k, v, k_mid, v_mid, k_tail, v_tail, o, lse, q2k_ptr, q2k_idx,
                       tier_maps(bits_a, bits_ab, L, mid_reps, mid_stride, tail_stride, phases), blk_cnt, BH, L, D, dtype,
                       (cudaStream_t)stream);
}

extern "C" int es_vsa_tier_attn_bwd_q(const void* q, const void* k, const void* v, const void* k_mid, const void* v_mid,
                                      const void* k_tail, const void* v_tail, const void* dout, const float* lse,
                                      const float* delta, void* dq, const float* add_dq, int32_t add_nb,
                                      const int32_t* q2k_ptr, const int32_t* q2k_idx, const int32_t* bits_a,
                                      const int32_t* bits_ab, const int32_t* blk_cnt, int32_t BH, int32_t L, int32_t D,
                                      int32_t mid_reps, int32_t mid_stride, int32_t tail_stride, int32_t phases,
                                      int32_t dtype, void* stream) {
    if (!q || !k || !v || !k_mid || !v_mid || !k_tail || !v_tail || !dout || !lse || !delta || !dq || !q2k_ptr || !q2k_idx || !bits_a || !bits_ab || !blk_cnt)
        return set_error(-1, "es_vsa_tier_attn_bwd_q: null pointer");
    if (int rc = check_tier("es_vsa_tier_attn_bwd_q", BH, L, D, dtype, mid_reps, phases, mid_stride, tail_stride)) return rc;
    if (add_dq && add_nb < L / TB) return set_error(-1, "es_vsa_tier_attn_bwd_q: add_nb smaller than the block count");
    if (phases == PH_A)
        return es_vsa_attn_bwd_q(q, k, v, dout, lse, delta, dq, nullptr, add_dq, add_nb, q2k_ptr, q2k_idx, blk_cnt, BH, L, D, dtype,
                                 stream);
    return tier_bwd_q_tc(q, k, v, k_mid, v_mid, k_tail, v_tail, dout, lse, delta, dq, add_dq, add_nb, q2k_ptr, q2k_idx,
                         tier_maps(bits_a, bits_ab, L, mid_reps, mid_stride, tail_stride, phases), blk_cnt, BH, L, D, dtype,
                         (cudaStream_t)stream);
}

extern "C" int es_vsa_tier_rep_bwd(const void* q, const void* k_mid, const void* v_mid, const void* k_tail,
                                   const void* v_tail, const void* dout, const float* lse, const float* delta,
                                   float* dk_mid, float* dv_mid, float* dk_tail, float* dv_tail, const int32_t* bits_a,
                                   const int32_t* bits_ab, const int32_t* blk_cnt, int32_t BH, int32_t L, int32_t D,
                                   int32_t mid_reps, int32_t mid_stride, int32_t tail_stride, int32_t phases, int32_t dtype,
                                   void* stream) {
    if (!q || !k_mid || !v_mid || !k_tail || !v_tail || !dout || !lse || !delta || !dk_mid || !dv_mid || !dk_tail || !dv_tail || !bits_a || !bits_ab || !blk_cnt)
        return set_error(-1, "es_vsa_tier_rep_bwd: null pointer");
    if (int rc = check_tier("es_vsa_tier_rep_bwd", BH, L, D, dtype, mid_reps, phases, mid_stride, tail_stride)) return rc;
    const int NB = L / TB;
    const int tiles = ((phases & PH_B) ? (NB * mid_reps + TB - 1) / TB : 0) + ((phases & PH_C) ? (NB + TB - 1) / TB : 0);
    if (tiles == 0) return 0;
    return tier_rep_bwd_tc(q, k_mid, v_mid, k_tail, v_tail, dout, lse, delta, dk_mid, dv_mid, dk_tail, dv_tail,
                           tier_maps(bits_a, bits_ab, L, mid_reps, mid_stride, tail_stride, phases), blk_cnt, BH, L, D, dtype, tiles,
                           (cudaStream_t)stream);
}

extern "C" int es_vsa_tier_unpool(const float* tok, const float* mid, const float* tail, const float* add, int32_t add_nb,
                                  void* out, const int32_t* blk_cnt, int32_t BH, int32_t L, int32_t D, int32_t mid_reps,
                                  int32_t mid_stride, int32_t tail_stride, int32_t dtype, void* stream) {
    if (!out || !blk_cnt) return set_error(-1, "es_vsa_tier_unpool: null pointer");
    if (int rc = check_tier("es_vsa_tier_unpool", BH, L, D, dtype, mid_reps, 7, mid ? mid_stride : 1 << 30, tail ? tail_stride : 1 << 30)) return rc;
    if (add && add_nb < L / TB) return set_error(-1, "es_vsa_tier_unpool: add_nb smaller than the block count");
    if (!aligned(4, out)) return set_error(-1, "es_vsa_tier_unpool: out must be 4-byte aligned");
    const UnpoolArgs a{tok, mid, tail, add, out, blk_cnt, L, mid_reps, mid_stride, tail_stride, add_nb, aligned(16, tok, mid, tail, add) && aligned(8, out)};
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 grid(L / TB, BH);
    auto launch = [&](auto with, auto without) { (tok ? with : without)<<<grid, tok ? UNPOOL_THREADS<true> : UNPOOL_THREADS<false>, 0, st>>>(a); };
    if (dtype == 0 && D == 128) launch(tier_unpool_kernel<__nv_bfloat16, 128, true>, tier_unpool_kernel<__nv_bfloat16, 128, false>);
    else if (dtype == 0) launch(tier_unpool_kernel<__nv_bfloat16, 64, true>, tier_unpool_kernel<__nv_bfloat16, 64, false>);
    else if (D == 128) launch(tier_unpool_kernel<__half, 128, true>, tier_unpool_kernel<__half, 128, false>);
    else launch(tier_unpool_kernel<__half, 64, true>, tier_unpool_kernel<__half, 64, false>);
    ES_CHECK_LAUNCH("tier_unpool_kernel");
    return 0;
}
