// VSA2 split-KV scheduling: the task plan over a CSR list and the merges of the split rows.
//
// Contract (reference: csrc/vsa/split.cu:1-22 and the SplitPlanParams comment of csrc/vsa/vsa2_kernels.h:48-83 of
// shaoshitong/self_trainable_or_free_attn), for the NR = BH * NB rows of a q -> kv list (forward, dQ pass) or a kv -> q
// list (dK / dV pass):
//   a row of n blocks is eligible when n >= thr_h = max(min_len, ceil(tail_frac * W / resident),
//   ceil(rel_mean * nnz_h / NB)), W = all edges of the list, nnz_h = the edges of the row's (b, h); an eligible row has
//   ceil(n / chunk) chunks; with E = the number of eligible rows, row r is split when E <= budget and the running
//   (inclusive) chunk count of the eligible rows up to r stays <= max_slots. Split chunk j of a row covers the edges
//   [beg + j n / c, beg + (j + 1) n / c) and owns slot = its task index; the split chunks come first in the task list (in
//   row order), then one direct task {row, beg, end, -1} per remaining row. merges[m] = {row, first slot, chunks, 0} for the
//   m-th split row. info[8] = tasks, split rows, split slots, NR, E, E <= budget, thr without the per-head term, W.
// Everything stays on the device: one CTA computes the three prefix sums and writes the lists.
//
// Merges, one CTA per split row, chunks combined in their order (reproducible):
//   forward : o = sum_i 2^(lse_i - M) o_i / sum_i 2^(lse_i - M), lse = (M + log2 sum) ln 2; padded rows 0 and -inf
//   backward: out = valid ? sum_i part_i + add[block] / count : 0
#include <string>

#include "es_api_internal.h"
#include "es_vsa_mma.cuh"

namespace es {
namespace vsa {

struct PlanArgs {
    const int* ptr;
    int BH, NB, chunk, max_slots, min_len, resident, budget;
    double rel_mean, tail_frac;
    int *tasks, *merges, *info;
    int* work;            // [2 * NR] chunk counts, split flags (not used where rows are in registers)
};

// PER: rows of a thread that it keeps to itself (8 for up to 8,192 rows; all their loads are on their way together and nothing goes
// through `work`), or 0. 1,024 threads have 64 registers each, so part of the eight rows is in local memory (212 bytes stored, 568
// loaded a thread), which is still faster than `work`.
template <int PER>
__global__ void __launch_bounds__(1024) split_plan_kernel(const PlanArgs a) {
    __shared__ int warp_total[32];
    __shared__ int s_total;
    const int tid = threadIdx.x, NR = a.BH * a.NB;
    const int per = (NR + 1023) / 1024, lo = min(tid * per, NR), hi = min(lo + per, NR);
    int* cnt = a.work;
    int* flag = a.work + NR;
    // exclusive prefix over the threads, the total in s_total: shuffles and two barriers (20 barriers a scan in shared memory, five
    // scans: 20.5 us a plan of 6,144 rows, 16.2 with these, 12.8 with a thread's rows kept as well)
    auto scan = [&](int v) -> int {
        const int lane = tid & 31, warp = tid >> 5;
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
        }
        if (lane == 31) warp_total[warp] = incl;
        __syncthreads();
        const int r = incl - v + __reduce_add_sync(0xffffffffu, lane < warp ? warp_total[lane] : 0);
        if (tid == 1023) s_total = r + v;
        __syncthreads();
        return r;
    };
    const long long W = (long long)a.ptr[(size_t)a.BH * (a.NB + 1) - 1] - a.ptr[0];
    int gthr = a.min_len;
    if (a.tail_frac > 0.0) gthr = max(gthr, (int)ceil(a.tail_frac * (double)W / (double)a.resident));
    // chunks of the eligible rows, and how many rows are eligible
    int my_c = 0, my_e = 0;
    int r_beg[PER ? PER : 1], r_n[PER ? PER : 1], r_cnt[PER ? PER : 1], r_nnz[PER ? PER : 1];
    uint32_t r_split = 0;
    if (PER) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int r = lo + k, bh = r / a.NB, i = r - bh * a.NB;
            const int* hp = a.ptr + (size_t)bh * (a.NB + 1);
            r_beg[k] = r_n[k] = r_nnz[k] = 0;
            if (r < hi) {
                r_beg[k] = hp[i];
                r_n[k] = hp[i + 1];
                if (a.rel_mean > 0.0) r_nnz[k] = hp[a.NB] - hp[0];
            }
        }
    }
    auto row = [&](int n, int nnz) -> int {       // chunks of an eligible row, or 0
        int thr = gthr;
        if (a.rel_mean > 0.0) thr = max(thr, (int)ceil(a.rel_mean * (double)nnz / (double)a.NB));
        const int c = n >= thr ? (n + a.chunk - 1) / a.chunk : 0;
        my_c += c; my_e += n >= thr;
        return c;
    };
    if (PER) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            r_cnt[k] = 0;
            if (lo + k < hi) {
                r_n[k] -= r_beg[k];
                r_cnt[k] = row(r_n[k], r_nnz[k]);
            }
        }
    } else {
        for (int r = lo; r < hi; ++r) {
            const int bh = r / a.NB, i = r - bh * a.NB;
            const int* hp = a.ptr + (size_t)bh * (a.NB + 1);
            cnt[r] = row(hp[i + 1] - hp[i], a.rel_mean > 0.0 ? hp[a.NB] - hp[0] : 0);
        }
    }
    int run = scan(my_c);
    scan(my_e);
    const int E = s_total;
    const bool within = E <= a.budget;
    // split flags; slots of the split rows; number of direct rows before each row
    int my_slots = 0, my_split = 0, my_direct = 0;
    auto decide = [&](int c) -> bool {
        run += c;
        const bool split = within && c > 0 && run <= a.max_slots;
        my_slots += split ? c : 0; my_split += split; my_direct += !split;
        return split;
    };
    if (PER) {
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (lo + k < hi) r_split |= (uint32_t)decide(r_cnt[k]) << k;
    } else {
        for (int r = lo; r < hi; ++r) flag[r] = decide(cnt[r]);
    }
    int slot = scan(my_slots);
    const int t_split = s_total;
    int mrow = scan(my_split);
    const int n_split = s_total;
    int drow = scan(my_direct);
    const int n_direct = s_total;
    int4* tasks = reinterpret_cast<int4*>(a.tasks);
    int4* merges = reinterpret_cast<int4*>(a.merges);
    auto emit = [&](int r, int beg, int n, int c, bool split) {
        if (split) {
            for (int j = 0; j < c; ++j)
                tasks[slot + j] = make_int4(r, beg + (int)((long long)j * n / c), beg + (int)((long long)(j + 1) * n / c), slot + j);
            merges[mrow++] = make_int4(r, slot, c, 0);
            slot += c;
        } else {
            tasks[t_split + drow++] = make_int4(r, beg, beg + n, -1);
        }
    };
    if (PER) {
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (lo + k < hi) emit(lo + k, r_beg[k], r_n[k], r_cnt[k], (r_split >> k) & 1u);
    } else {
        for (int r = lo; r < hi; ++r) {
            const int bh = r / a.NB;
            const int* rp = a.ptr + (size_t)bh * (a.NB + 1) + (r - bh * a.NB);
            emit(r, rp[0], rp[1] - rp[0], cnt[r], flag[r]);
        }
    }
    if (tid == 0) {
        a.info[0] = t_split + n_direct; a.info[1] = n_split; a.info[2] = t_split; a.info[3] = NR;
        a.info[4] = E; a.info[5] = within ? 1 : 0; a.info[6] = gthr; a.info[7] = (int)W;
    }
}

struct MergeArgs {
    const int *merges, *info, *blk_cnt;
    const float *part, *part_lse, *add;
    void* out;
    float *out_f32, *lse;
    int L, NB, add_nb, mask_rows;
};

// FWD: weighted merge of normalised partials; otherwise the plain sum plus the per-block add.
template <typename T, int D, bool FWD>
__global__ void __launch_bounds__(128) split_merge_kernel(const MergeArgs a) {
    if ((int)blockIdx.x >= a.info[1]) return;
    const int4 mg = reinterpret_cast<const int4*>(a.merges)[blockIdx.x];
    const int bh = mg.x / a.NB, blk = mg.x - bh * a.NB, slot0 = mg.y, c = mg.z;
    const int cnt = a.blk_cnt[blk];
    constexpr int CH = D / 4;                       // float4 chunks per row
    for (int e = threadIdx.x; e < TB * CH; e += 128) {
        const int row = e / CH, ch = e % CH;
        const size_t tok = (size_t)bh * a.L + (size_t)blk * TB + row;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        float lse = -INFINITY;
        if (FWD) {
            if (row < cnt || !a.mask_rows) {
                float mx = -INFINITY;                          // NaN as soon as one partial is (fmaxf would drop it)
                for (int j = 0; j < c; ++j) {
                    const float x = a.part_lse[(size_t)(slot0 + j) * TB + row];
                    mx = x > mx || x != x ? x : mx;
                }
                if (mx != -INFINITY) {
                    float sum = 0.f;
                    for (int j = 0; j < c; ++j) {
                        const float w = exp2f(a.part_lse[(size_t)(slot0 + j) * TB + row] - mx);
                        const float4 x = *reinterpret_cast<const float4*>(a.part + ((size_t)(slot0 + j) * TB + row) * D + ch * 4);
                        sum += w;
                        acc.x += w * x.x; acc.y += w * x.y; acc.z += w * x.z; acc.w += w * x.w;
                    }
                    const float inv = 1.f / sum;
                    acc.x *= inv; acc.y *= inv; acc.z *= inv; acc.w *= inv;
                    lse = (mx + log2f(sum)) * LN2;
                }
            }
            if (ch == 0) a.lse[tok] = lse;
        } else if (row < cnt) {
            for (int j = 0; j < c; ++j) {
                const float4 x = *reinterpret_cast<const float4*>(a.part + ((size_t)(slot0 + j) * TB + row) * D + ch * 4);
                acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
            }
            if (a.add) {
                const float4 ad = *reinterpret_cast<const float4*>(a.add + ((size_t)bh * a.add_nb + blk) * D + ch * 4);
                const float inv = 1.f / (float)cnt;
                acc.x += ad.x * inv; acc.y += ad.y * inv; acc.z += ad.z * inv; acc.w += ad.w * inv;
            }
        }
        if (!FWD && a.out_f32) {
            *reinterpret_cast<float4*>(a.out_f32 + tok * D + ch * 4) = acc;
        } else {
            uint2 w;
            w.x = Elt<T>::pack(acc.x, acc.y);
            w.y = Elt<T>::pack(acc.z, acc.w);
            *reinterpret_cast<uint2*>(static_cast<T*>(a.out) + tok * D + ch * 4) = w;
        }
    }
}

template <bool FWD>
static int launch_merge(const MergeArgs& a, int n_merge_cap, int D, int dtype, cudaStream_t st) {
    if (dtype == 0 && D == 128) split_merge_kernel<__nv_bfloat16, 128, FWD><<<n_merge_cap, 128, 0, st>>>(a);
    else if (dtype == 0) split_merge_kernel<__nv_bfloat16, 64, FWD><<<n_merge_cap, 128, 0, st>>>(a);
    else if (D == 128) split_merge_kernel<__half, 128, FWD><<<n_merge_cap, 128, 0, st>>>(a);
    else split_merge_kernel<__half, 64, FWD><<<n_merge_cap, 128, 0, st>>>(a);
    ES_CHECK_LAUNCH("split_merge_kernel");
    return 0;
}

}  // namespace vsa
}  // namespace es

using namespace es;
using namespace es::vsa;

static bool plan_in_registers(int BH, int NB) { return (long long)BH * NB <= 8 * 1024; }

extern "C" long long es_vsa_split_plan_workspace_bytes(int32_t BH, int32_t NB) {
    return BH > 0 && NB > 0 && !plan_in_registers(BH, NB) ? 2LL * BH * NB * 4 : 0;
}

extern "C" int es_vsa_split_plan(const int32_t* ptr, int32_t BH, int32_t NB, int32_t chunk, int32_t max_slots,
                                 int32_t min_len, double rel_mean, double tail_frac, int32_t resident, int32_t budget,
                                 int32_t* tasks, int32_t* merges, int32_t* info, void* workspace, void* stream) {
    if (!ptr || !tasks || !merges || !info) return set_error(-1, "es_vsa_split_plan: null pointer");
    if (BH <= 0 || NB <= 0) return set_error(-1, "es_vsa_split_plan: BH and NB must be positive");
    if (!workspace && es_vsa_split_plan_workspace_bytes(BH, NB) > 0) return set_error(-1, "es_vsa_split_plan: null workspace");
    if (chunk < 1 || max_slots < 0) return set_error(-1, "es_vsa_split_plan: chunk >= 1 and max_slots >= 0");
    if (min_len < chunk + 1) return set_error(-1, "es_vsa_split_plan: min_len must be at least chunk + 1");
    if (resident < 1 || budget < 0 || rel_mean < 0.0 || tail_frac < 0.0)
        return set_error(-1, "es_vsa_split_plan: resident >= 1, budget >= 0, rel_mean >= 0, tail_frac >= 0");
    if (((uintptr_t)tasks | (uintptr_t)merges) & 15) return set_error(-1, "es_vsa_split_plan: tasks and merges must be 16-byte aligned");
    PlanArgs a{ptr, BH, NB, chunk, max_slots, min_len, resident, budget, rel_mean, tail_frac, tasks, merges, info,
               static_cast<int*>(workspace)};
    if (plan_in_registers(BH, NB)) split_plan_kernel<8><<<1, 1024, 0, (cudaStream_t)stream>>>(a);
    else split_plan_kernel<0><<<1, 1024, 0, (cudaStream_t)stream>>>(a);
    ES_CHECK_LAUNCH("split_plan_kernel");
    return 0;
}

extern "C" int es_vsa_split_merge_fwd(const float* part_o, const float* part_lse, const int32_t* merges,
                                      const int32_t* info, int32_t n_merge_cap, const int32_t* blk_cnt, void* o, float* lse,
                                      int32_t L, int32_t D, int32_t mask_rows, int32_t dtype, void* stream) {
    if (!merges || !info || !blk_cnt || !o || !lse) return set_error(-1, "es_vsa_split_merge_fwd: null pointer");
    if (n_merge_cap <= 0) return 0;
    if (!part_o || !part_lse) return set_error(-1, "es_vsa_split_merge_fwd: null partials");
    if (L <= 0 || L % TB != 0 || (D != 64 && D != 128) || (dtype != 0 && dtype != 1))
        return set_error(-1, "es_vsa_split_merge_fwd: bad L, D or dtype");
    if (!aligned(16, part_o, merges) || !aligned(8, o)) return set_error(-1, "es_vsa_split_merge_fwd: part_o and merges must be 16-byte, o 8-byte aligned");
    MergeArgs a{};
    a.merges = merges; a.info = info; a.blk_cnt = blk_cnt; a.part = part_o; a.part_lse = part_lse; a.out = o; a.lse = lse;
    a.L = L; a.NB = L / TB; a.mask_rows = mask_rows;
    return launch_merge<true>(a, n_merge_cap, D, dtype, (cudaStream_t)stream);
}

extern "C" int es_vsa_split_merge_sum(const float* part, const int32_t* merges, const int32_t* info, int32_t n_merge_cap,
                                      const float* add, int32_t add_nb, const int32_t* blk_cnt, void* out, float* out_f32,
                                      int32_t L, int32_t D, int32_t dtype, void* stream) {
    if (!merges || !info || !blk_cnt || (!out && !out_f32)) return set_error(-1, "es_vsa_split_merge_sum: null pointer");
    if (n_merge_cap <= 0) return 0;
    if (!part) return set_error(-1, "es_vsa_split_merge_sum: null partials");
    if (L <= 0 || L % TB != 0 || (D != 64 && D != 128) || (dtype != 0 && dtype != 1))
        return set_error(-1, "es_vsa_split_merge_sum: bad L, D or dtype");
    if (add && add_nb < L / TB) return set_error(-1, "es_vsa_split_merge_sum: add_nb smaller than the block count");
    if (!aligned(16, part, add, merges, out_f32) || !aligned(8, out))
        return set_error(-1, "es_vsa_split_merge_sum: part, add, merges and out_f32 must be 16-byte, out 8-byte aligned");
    MergeArgs a{};
    a.merges = merges; a.info = info; a.blk_cnt = blk_cnt; a.part = part; a.add = add; a.add_nb = add_nb; a.out = out;
    a.out_f32 = out_f32; a.L = L; a.NB = L / TB;
    return launch_merge<false>(a, n_merge_cap, D, dtype, (cudaStream_t)stream);
}
