// Entry points of the VSA2 block-sparse attention over CSR block lists: argument checks in front of the tcgen05 kernels of
// es_vsa_tc_fwd.cu and es_vsa_tc_bwd.cu.
#include <string>

#include "es_api_internal.h"

namespace es {
namespace vsa {

constexpr int TB = 64;                 // tokens per block

static int check_common(const char* name, int BH, int L, int D, int dtype) {
    if (BH <= 0 || L <= 0 || L % TB != 0) return set_error(-1, (std::string(name) + ": BH > 0 and L a positive multiple of 64").c_str());
    if (D != 64 && D != 128) return set_error(-1, (std::string(name) + ": head dim must be 64 or 128").c_str());
    if (dtype != 0 && dtype != 1) return set_error(-1, (std::string(name) + ": dtype must be 0 (bf16) or 1 (fp16)").c_str());
    return 0;
}

// es_vsa_tc_fwd.cu, es_vsa_tc_bwd.cu
int attn_fwd_tc(const void* q, const void* k, const void* v, void* o, float* lse, const int* row_ptr, const int* col_idx,
                const int* blk_cnt, int BH, int L, int rows, int D, int dtype, const int* tasks, const int* task_info, int n_tasks,
                float* part_o, float* part_lse, cudaStream_t st);
int attn_bwd_tc(bool kv, const void* q, const void* k, const void* v, const void* dout, const float* lse, const float* delta,
                void* out0, void* out1, float* f0, float* f1, const float* add0, const float* add1, int add_nb,
                const int* row_ptr, const int* col_idx, const int* blk_cnt, int BH, int L, int rows, int D, int dtype, const int* tasks,
                const int* task_info, int n_tasks, float* part0, float* part1, cudaStream_t st);

}  // namespace vsa
}  // namespace es

using namespace es;
using namespace es::vsa;

extern "C" int es_vsa_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const int32_t* row_ptr,
                               const int32_t* col_idx, const int32_t* blk_cnt, int32_t BH, int32_t L, int32_t D,
                               int32_t dtype, void* stream) {
    if (!q || !k || !v || !o || !lse || !row_ptr || !col_idx || !blk_cnt) return set_error(-1, "es_vsa_attn_fwd: null pointer");
    if (int rc = check_common("es_vsa_attn_fwd", BH, L, D, dtype)) return rc;
    return attn_fwd_tc(q, k, v, o, lse, row_ptr, col_idx, blk_cnt, BH, L, 0, D, dtype, nullptr, nullptr, 0, nullptr, nullptr,
                       (cudaStream_t)stream);
}

extern "C" int es_vsa_attn_bwd_kv(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                                  const float* delta, void* dk, void* dv, float* dk_f32, float* dv_f32,
                                  const float* add_dk, const float* add_dv, int32_t add_nb, const int32_t* k2q_ptr,
                                  const int32_t* k2q_idx, const int32_t* blk_cnt, int32_t BH, int32_t L, int32_t D,
                                  int32_t dtype, void* stream) {
    if (!q || !k || !v || !dout || !lse || !delta || !k2q_ptr || !k2q_idx || !blk_cnt)
        return set_error(-1, "es_vsa_attn_bwd_kv: null pointer");
    if ((!dk && !dk_f32) || (!dv && !dv_f32)) return set_error(-1, "es_vsa_attn_bwd_kv: no output for dK or dV");
    if ((add_dk || add_dv) && add_nb < L / TB) return set_error(-1, "es_vsa_attn_bwd_kv: add_nb smaller than the block count");
    if (int rc = check_common("es_vsa_attn_bwd_kv", BH, L, D, dtype)) return rc;
    return attn_bwd_tc(true, q, k, v, dout, lse, delta, dk, dv, dk_f32, dv_f32, add_dk, add_dv, add_nb, k2q_ptr, k2q_idx,
                       blk_cnt, BH, L, 0, D, dtype, nullptr, nullptr, 0, nullptr, nullptr, (cudaStream_t)stream);
}

extern "C" int es_vsa_attn_bwd_q(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                                 const float* delta, void* dq, float* dq_f32, const float* add_dq, int32_t add_nb,
                                 const int32_t* q2k_ptr, const int32_t* q2k_idx, const int32_t* blk_cnt, int32_t BH,
                                 int32_t L, int32_t D, int32_t dtype, void* stream) {
    if (!q || !k || !v || !dout || !lse || !delta || !q2k_ptr || !q2k_idx || !blk_cnt)
        return set_error(-1, "es_vsa_attn_bwd_q: null pointer");
    if (!dq && !dq_f32) return set_error(-1, "es_vsa_attn_bwd_q: no output for dQ");
    if (add_dq && add_nb < L / TB) return set_error(-1, "es_vsa_attn_bwd_q: add_nb smaller than the block count");
    if (int rc = check_common("es_vsa_attn_bwd_q", BH, L, D, dtype)) return rc;
    return attn_bwd_tc(false, q, k, v, dout, lse, delta, dq, nullptr, dq_f32, nullptr, add_dq, nullptr, add_nb, q2k_ptr,
                       q2k_idx, blk_cnt, BH, L, 0, D, dtype, nullptr, nullptr, 0, nullptr, nullptr, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------------------- coarse branch
static int check_coarse(const char* name, int BH, int L, int NB, int D, int dtype) {
    if (int rc = check_common(name, BH, L, D, dtype)) return rc;
    if (NB <= L - TB || NB > L) return set_error(-1, (std::string(name) + ": L must be NB rounded up to a multiple of 64").c_str());
    return 0;
}

extern "C" int es_vsa_coarse_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int32_t BH, int32_t L,
                                 int32_t NB, int32_t D, int32_t dtype, void* stream) {
    if (!q || !k || !v || !o || !lse) return set_error(-1, "es_vsa_coarse_fwd: null pointer");
    if (int rc = check_coarse("es_vsa_coarse_fwd", BH, L, NB, D, dtype)) return rc;
    return attn_fwd_tc(q, k, v, o, lse, nullptr, nullptr, nullptr, BH, L, NB, D, dtype, nullptr, nullptr, 0, nullptr, nullptr,
                       (cudaStream_t)stream);
}

extern "C" int es_vsa_coarse_bwd(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                                 const float* delta, float* dq, float* dk, float* dv, int32_t BH, int32_t L, int32_t NB,
                                 int32_t D, int32_t dtype, void* stream) {
    if (!q || !k || !v || !dout || !lse || !delta || !dq || !dk || !dv) return set_error(-1, "es_vsa_coarse_bwd: null pointer");
    if (int rc = check_coarse("es_vsa_coarse_bwd", BH, L, NB, D, dtype)) return rc;
    if (int rc = attn_bwd_tc(true, q, k, v, dout, lse, delta, nullptr, nullptr, dk, dv, nullptr, nullptr, 0, nullptr, nullptr,
                             nullptr, BH, L, NB, D, dtype, nullptr, nullptr, 0, nullptr, nullptr, (cudaStream_t)stream))
        return rc;
    return attn_bwd_tc(false, q, k, v, dout, lse, delta, nullptr, nullptr, dq, nullptr, nullptr, nullptr, 0, nullptr, nullptr,
                       nullptr, BH, L, NB, D, dtype, nullptr, nullptr, 0, nullptr, nullptr, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------------------- split-KV task launches
static int check_tasks(const char* name, const int32_t* tasks, const int32_t* info, int n_tasks_cap) {
    if (!tasks || !info) return set_error(-1, (std::string(name) + ": null task list").c_str());
    if (n_tasks_cap <= 0) return set_error(-1, (std::string(name) + ": the task grid is empty").c_str());
    if ((uintptr_t)tasks & 15) return set_error(-1, (std::string(name) + ": tasks must be 16-byte aligned").c_str());
    return 0;
}

extern "C" int es_vsa_attn_fwd_tasks(const void* q, const void* k, const void* v, void* o, float* lse,
                                     const int32_t* q2k_idx, const int32_t* blk_cnt, const int32_t* tasks,
                                     const int32_t* task_info, int32_t n_tasks_cap, float* part_o, float* part_lse,
                                     int32_t BH, int32_t L, int32_t D, int32_t dtype, void* stream) {
    if (!q || !k || !v || !o || !lse || !q2k_idx || !blk_cnt) return set_error(-1, "es_vsa_attn_fwd_tasks: null pointer");
    if (int rc = check_common("es_vsa_attn_fwd_tasks", BH, L, D, dtype)) return rc;
    if (int rc = check_tasks("es_vsa_attn_fwd_tasks", tasks, task_info, n_tasks_cap)) return rc;
    return attn_fwd_tc(q, k, v, o, lse, nullptr, q2k_idx, blk_cnt, BH, L, 0, D, dtype, tasks, task_info, n_tasks_cap, part_o,
                       part_lse, (cudaStream_t)stream);
}

extern "C" int es_vsa_attn_bwd_kv_tasks(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                                        const float* delta, void* dk, void* dv, float* dk_f32, float* dv_f32,
                                        const float* add_dk, const float* add_dv, int32_t add_nb, const int32_t* k2q_idx,
                                        const int32_t* blk_cnt, const int32_t* tasks, const int32_t* task_info,
                                        int32_t n_tasks_cap, float* part_dk, float* part_dv, int32_t BH, int32_t L,
                                        int32_t D, int32_t dtype, void* stream) {
    if (!q || !k || !v || !dout || !lse || !delta || !k2q_idx || !blk_cnt)
        return set_error(-1, "es_vsa_attn_bwd_kv_tasks: null pointer");
    if ((!dk && !dk_f32) || (!dv && !dv_f32)) return set_error(-1, "es_vsa_attn_bwd_kv_tasks: no output for dK or dV");
    if ((add_dk || add_dv) && add_nb < L / TB) return set_error(-1, "es_vsa_attn_bwd_kv_tasks: add_nb smaller than the block count");
    if (int rc = check_common("es_vsa_attn_bwd_kv_tasks", BH, L, D, dtype)) return rc;
    if (int rc = check_tasks("es_vsa_attn_bwd_kv_tasks", tasks, task_info, n_tasks_cap)) return rc;
    return attn_bwd_tc(true, q, k, v, dout, lse, delta, dk, dv, dk_f32, dv_f32, add_dk, add_dv, add_nb, nullptr, k2q_idx,
                       blk_cnt, BH, L, 0, D, dtype, tasks, task_info, n_tasks_cap, part_dk, part_dv, (cudaStream_t)stream);
}

extern "C" int es_vsa_attn_bwd_q_tasks(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                                       const float* delta, void* dq, float* dq_f32, const float* add_dq, int32_t add_nb,
                                       const int32_t* q2k_idx, const int32_t* blk_cnt, const int32_t* tasks,
                                       const int32_t* task_info, int32_t n_tasks_cap, float* part_dq, int32_t BH,
                                       int32_t L, int32_t D, int32_t dtype, void* stream) {
    if (!q || !k || !v || !dout || !lse || !delta || !q2k_idx || !blk_cnt)
        return set_error(-1, "es_vsa_attn_bwd_q_tasks: null pointer");
    if (!dq && !dq_f32) return set_error(-1, "es_vsa_attn_bwd_q_tasks: no output for dQ");
    if (add_dq && add_nb < L / TB) return set_error(-1, "es_vsa_attn_bwd_q_tasks: add_nb smaller than the block count");
    if (int rc = check_common("es_vsa_attn_bwd_q_tasks", BH, L, D, dtype)) return rc;
    if (int rc = check_tasks("es_vsa_attn_bwd_q_tasks", tasks, task_info, n_tasks_cap)) return rc;
    return attn_bwd_tc(false, q, k, v, dout, lse, delta, dq, nullptr, dq_f32, nullptr, add_dq, nullptr, add_nb, nullptr,
                       q2k_idx, blk_cnt, BH, L, 0, D, dtype, tasks, task_info, n_tasks_cap, part_dq, nullptr, (cudaStream_t)stream);
}
