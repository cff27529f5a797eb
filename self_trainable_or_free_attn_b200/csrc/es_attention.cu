// Fixed-offset block-sparse attention for sm_100a: one CTA per (128-row query tile, head), one CTA per SM.
//
// What it computes (reference: echosparse/kernels/block_attention.py:206-303, sparse_attention.py:1-13, 430-575,
// and the same formula in echosparse/kernels/sm120.py:27-96): for query row r with offset m_r (the previous step's
// log2 LSE), over three kinds of columns,
//     p = 2^(c * q_r.k_j - m_r + bias_j),   l_r = sum p,   O_r = sum bf16(p) v_j / l_r,   lse_r = m_r + log2 l_r
//   exact:  the tokens of the listed 64-token blocks (bias 0, tail tokens past L masked),
//   mean:   one column per block whose bit in skip_bits is clear: the block's mean key / value, bias log2(len),
//   refine: four representatives of every block of the tile's refine list, bias log2(cluster size).
// mass[h, tile, b] = sum over the tile's rows of the exact block b's p; flag[tile, h] = some valid row has
// log2 l_r outside [-th, th].  There is no running maximum and no rescaling.
//
// FALLBACK = true is the online-softmax recomputation of flagged tiles (triton_ops.py:203-234): a sweep of QK MMAs
// finds every row's maximum logit, then the same fixed-offset pipeline runs with that maximum as the offset, which is the
// online-softmax result without rescaling steps.
//
// Pipeline. An iteration covers 128 columns (two 64-token blocks, 128 block means, or 32 refine entries x 4).
//   warps 0-7  softmax: warp w owns rows 32 (w % 4) .. +31 of the tile and columns 64 (w / 4) .. +63 of the iteration
//   warp 8     issues the tcgen05 MMAs (one elected lane); warps 9 and 10 issue the TMA loads of the K and of the V
//              tiles (control code is one dependent chain per tile: two warps halve its length); warp 11 sums and
//              stores the block masses
// Tensor memory (512 columns): S of even iterations [0,128), S of odd iterations [128,256), O [256,384), Q [384,448).
// Q sits in tensor memory as the A operand of QK^T, so the only shared-memory traffic of the MMAs is K and V: with Q in
// shared memory a 128 x 64 x 16 MMA reads 6 KB in the 32 clocks it computes, more than the 128 B/clock an SM delivers.
// P (bf16 pairs) is written over the S columns it came from and is the A operand of PV. Two S buffers let QK of
// iteration i + 1 run while the softmax warps work on iteration i; PV(i) and QK(i + 2) follow as soon as P(i) is stored.
// K and V tiles (32 KB each, [d half][128 rows][128 B], four 8 KB TMA boxes; representative rows: 64 boxes of 512 B)
// travel through a ring of NSLOT shared-memory slots, about three iterations ahead of the MMAs. With one CTA per SM nothing hides
// a tile's start and end, so Q and O cross shared memory in whole lines: a tile of 32 iterations took 66,900 clocks with a row per
// thread on both sides, 60,300 now (the fused step of 32,760 tokens x 12 heads, 47 iterations a tile: 1.316 -> 1.301 ms).
#include "es_ptx.cuh"
#include "es_api_internal.h"
#include <algorithm>

namespace es {

constexpr int BM = 128;       // query rows per tile
constexpr int BK = 64;        // tokens per kv block
constexpr int HD = 128;       // head dim
constexpr int NSOFT = 256;    // softmax threads
constexpr int NTHREADS = NSOFT + 128;
constexpr int MMA_WARP = NSOFT / 32, LOADK_WARP = MMA_WARP + 1, LOADV_WARP = MMA_WARP + 2, MASS_WARP = MMA_WARP + 3;
constexpr int NMASS = 8;      // sets of partial block masses in flight between the softmax warps and the mass warp
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t O_COL = 256, Q_COL = 384;
constexpr int NSLOT = 6;      // K / V tiles in flight
constexpr int Q_SLOT = NSLOT - 1;    // Q passes through this slot before its first K / V tile
constexpr float kSeedLimit = 60.f;   // largest log2 row sum relative to a seeded offset (see dense_kernel)
constexpr int NBIAS = 8;      // refine iterations whose column biases are staged in shared memory at a time

constexpr uint32_t TILE_BYTES = 128 * HD * 2;    // 32 KB: [d half][128 rows][64 d], 128B-swizzled
constexpr uint32_t HALF_BYTES = TILE_BYTES / 2;  // one d half: 128 rows x 128 B
constexpr uint32_t BLK_BYTES = BK * 128;         // 64 rows of one d half: one TMA box
constexpr uint32_t SMEM_RING = 0;
constexpr uint32_t SMEM_CTL = SMEM_RING + NSLOT * TILE_BYTES;
constexpr uint32_t SMEM_BIAS = SMEM_CTL + 5632;                        // [NBIAS][128] floats
constexpr uint32_t SMEM_MASS = SMEM_BIAS + NBIAS * 128 * 4;            // [NMASS][2 column halves][128 rows] floats
constexpr uint32_t SMEM_ALLOC = SMEM_MASS + NMASS * 2 * BM * 4;        // 214,528 B: one CTA per SM

struct Ctl {
    uint64_t qload, qfull;             // Q in shared memory; Q in tensor memory (and its ring slot free)
    uint64_t full[NSLOT], empty[NSLOT];
    uint64_t sfull[2], pfull[2];
    uint64_t ofull, drain;
    uint64_t massbar[NMASS], flagbar, lbar;   // softmax warps -> the thread(s) that combine their partial results
    uint64_t massfree[NMASS];             // mass warp -> softmax warps: the set's partial sums have been read
    uint64_t sweepbar;                 // K load warp -> V load warp: the fallback sweep's tiles have all been issued
    uint32_t tmem_base;
    int abort;
    int flag_part[4];
    float l_part[2][BM];               // row sums of the two column halves
    float m_part[2][BM];               // row maxima of the two column halves (fallback sweep)
    float r_part[2][BM];               // dense: row sums of the rounded P
    float e_part[2][BM];               // dense: what rounding took from a half's largest P above the sample's; its key, or -1
    int key_part[2][BM];
    int redo;                          // some row left the range of the offset from a sample
    int stop;                          // the status word was set before the tile began
};
static_assert(sizeof(Ctl) <= 5632, "control block");

// Fallback modes: tiles whose flags a CTA looks at in one go, and the most of them that are its own.
constexpr int WALK_TILES = 64 * NTHREADS, WALK_MINE = 256;
static_assert(WALK_TILES / 8 + (WALK_MINE + 32) * 4 <= NMASS * 2 * BM * 4, "the walk's lists take the block masses' room");

struct AttnArgs {
    const __nv_bfloat16* q;      // (L, H, 128)
    const __nv_bfloat16* v;      // (L, H, 128), dense mode only (elsewhere V comes through its tensor map alone)
    const uint8_t* keep;         // (H, nq, nb), compensation mode only
    __nv_bfloat16* out;
    const int* counts;           // (nq, H)
    const int* blocks;           // (nq, H, nk) ascending block ids
    int nk;
    const float* offset;         // (nq*128, H) log2
    float* lse;                  // (nq*128, H) log2
    int* flags;                  // (nq, H)
    float* mass;                 // (H, nq, nb) or null
    const int* skip_bits;        // (H, nq, nw)
    int nw;
    const int* refine;           // (nq, H, rw) padded with nb
    int rw;
    const __nv_bfloat16* k_rep;  // (H, nb4, 128)
    const __nv_bfloat16* v_rep;
    const float* log_counts;     // (H, nb4)
    int nb4;
    int L, H, nq, nb;
    float scale_log2, th;
    int tail_valid;              // tokens of the last block
    float tail_log2;             // log2(tail_valid)
    int nvirt, nref;             // mean iterations (128 blocks each), refine iterations (32 list entries each)
    int walk;                    // fallback modes: CTAs find the flagged tiles and share them; 0: one CTA per tile tests its flag
    int* status;
};

// How dense_kernel shares out its tiles (plan_dense chooses). CTA c takes the whole tiles c, c + grid, .. below `whole`; the
// iterations of the tiles from there on are one line, of which it takes [edge(c), edge(c + 1)) (c < ctas). dense_merge_kernel
// puts together the tiles that more than one CTA worked on.
struct DenseSplit {
    int n;                       // iterations of a tile
    int whole, ctas;
    int line;                    // iterations of the tiles that are cut
    float* part;                 // [2 ctas] partial results; null: every tile is whole, one CTA per tile
    __host__ __device__ int edge(int c) const { return (int)((unsigned)line * (unsigned)c / (unsigned)ctas); }   // line * ctas < 2^32
};
constexpr int PART_ROWS = 3;                                  // a partial result: m, l and the sum of the rounded P of every row,
constexpr int PART_FLOATS = BM * (HD + PART_ROWS);            // then O as [d / 4][row][4]

__device__ __forceinline__ float2 exp2_pair(float2 x) { return make_float2(ex2_approx(x.x), ex2_approx(x.y)); }

// Order of a tile's iterations. The refine iterations (64 small TMA boxes per tile, slow to fill) are spread evenly among
// the others instead of coming last, so that the ring refills during the cheap iterations in between: iteration i is the
// refine iteration i / p when i % p == p - 1 and i / p < nref (p = nt / nref); the other iterations are the exact ones,
// then the block-mean ones, in their order. kind: 0 exact, 1 block means, 2 refine; idx counts within the kind.
struct Sched {
    int n, nvirt, nref, p;
    __device__ __forceinline__ void decode(int i, int& kind, int& idx) const {
        if (nref > 0) {
            const int q = i / p;
            if (i - q * p == p - 1 && q < nref) { kind = 2; idx = q; return; }
            i -= min(q, nref);
        }
        if (i < n) { kind = 0; idx = i; }
        else { kind = 1; idx = i - n; }
    }
};

// The same order walked one iteration at a time, without the division: ph = i % p, q = i / p, o = iterations before i
// that are not refine iterations.
struct SchedIter {
    int ph = 0, q = 0, o = 0;
    __device__ __forceinline__ void get(const Sched& s, int& kind, int& idx) const {
        if (s.nref > 0 && ph == s.p - 1 && q < s.nref) { kind = 2; idx = q; }
        else if (o < s.n) { kind = 0; idx = o; }
        else { kind = 1; idx = o - s.n; }
    }
    __device__ __forceinline__ void advance(const Sched& s) {
        if (!(s.nref > 0 && ph == s.p - 1 && q < s.nref)) ++o;
        if (++ph == s.p) { ph = 0; ++q; }
    }
};

// How a tile ended, the same for every thread of the CTA: done; dense mode, to be done again since `sample` did not do (dense_kernel);
// or stopped by a wait that gave up, in this CTA or another, after which the CTA does no other tile.
enum TileEnd { TILE_DONE, TILE_AGAIN, TILE_STOP };

// One (query tile, head): `tile` = head * nq + query tile. `again`: the CTA has run a tile before (its barriers exist).
// Dense mode: `sample` takes the offset from a sample of the columns.
// The CTA runs iterations first .. last - 1 of the tile and leaves a partial result in `part`, or with null the outputs.
template <int MODE>
__device__ __forceinline__ TileEnd attention_tile(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmKm,
                                                  const CUtensorMap& tmVm, const CUtensorMap& tmKr, const CUtensorMap& tmVr,
                                                  const AttnArgs& a, const int tile, const bool again, const bool sample,
                                                  const int first = 0, const int last = 0, float* const part = nullptr) {
    constexpr bool COMPENSATE = MODE == 2;     // block-mean compensation of flagged tiles, added to out / lse in place
    constexpr bool DENSE = MODE == 3;          // online softmax over every block: no list, no flags
    constexpr bool FALLBACK = MODE == 1 || DENSE;    // the offset comes from a sweep; MODE 1: of flagged tiles, over their lists
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // adjacent tile numbers are adjacent query tiles of one head: their kv lists overlap in L2
    const int qb = tile % a.nq, h = tile / a.nq;
    const int th_idx = qb * a.H + h;
    if ((MODE == 1 || COMPENSATE) && !a.walk) {
        if (a.flags[th_idx] == 0) return TILE_DONE;    // uniform over the CTA, before anything is allocated
    }
    // The tile's first global loads do not depend on one another: the list length, the first window of block ids (load
    // warps) and this row's offset (softmax warps) are requested here (in the fallback modes: once the tile is known to be
    // flagged), before the barrier set-up and the tensor-memory allocation, whose latencies they then share instead of
    // following them.
    const int n64_early = COMPENSATE ? 0 : DENSE ? a.nb : __ldg(a.counts + th_idx);
    int win_early = 0;
    float m_early = 0.f;
    if (warp == LOADK_WARP || warp == LOADV_WARP) {
        if (!COMPENSATE && !DENSE && lane < a.nk) win_early = __ldg(a.blocks + (size_t)th_idx * a.nk + lane);
        if (lane == 0) {
            const bool is_v = warp == LOADV_WARP;
            if (!COMPENSATE) tma_prefetch_desc(is_v ? &tmV : &tmK);
            if (MODE == 0 || COMPENSATE) tma_prefetch_desc(is_v ? &tmVm : &tmKm);
            if (MODE == 0) tma_prefetch_desc(is_v ? &tmVr : &tmKr);
        }
    } else if (warp < NSOFT / 32) {
        if (!FALLBACK) m_early = a.offset[((size_t)qb * BM + 32 * (warp & 3) + lane) * a.H + h];
    }

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t base = smem_u32(smem_raw);
    Ctl* ctl = reinterpret_cast<Ctl*>(smem_raw + SMEM_CTL);
    const uint32_t sRing = base + SMEM_RING;
    volatile int* abort_flag = &ctl->abort;
    float* bias_ring = reinterpret_cast<float*>(smem_raw + SMEM_BIAS);
    float* mass_rows = reinterpret_cast<float*>(smem_raw + SMEM_MASS);

    if (tid == 0) {
        const int earlier = *reinterpret_cast<volatile int*>(a.status);      // (on its way during the set-up)
        if (base & 1023u) atomicCAS(a.status, 0, 901);   // the swizzled tiles need a 1024-byte aligned base
        if (again) {
            // a CTA that walks a list of tiles makes its barriers anew for every tile
            for (uint64_t* b = &ctl->qload; b <= &ctl->sweepbar; ++b) mbar_inval(smem_u32(b));
        }
        mbar_init(smem_u32(&ctl->qload), 1);
        mbar_init(smem_u32(&ctl->qfull), NSOFT);
        for (int i = 0; i < NSLOT; ++i) {
            mbar_init(smem_u32(&ctl->full[i]), 1);
            mbar_init(smem_u32(&ctl->empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&ctl->sfull[i]), 1);
            mbar_init(smem_u32(&ctl->pfull[i]), NSOFT);
        }
        mbar_init(smem_u32(&ctl->ofull), 1);
        mbar_init(smem_u32(&ctl->drain), 1);
        for (int i = 0; i < NMASS; ++i) {
            mbar_init(smem_u32(&ctl->massbar[i]), 8);
            mbar_init(smem_u32(&ctl->massfree[i]), 1);
        }
        mbar_init(smem_u32(&ctl->flagbar), 4);
        mbar_init(smem_u32(&ctl->lbar), NSOFT);
        mbar_init(smem_u32(&ctl->sweepbar), 1);
        ctl->abort = (base & 1023u) || earlier ? 1 : 0;
        ctl->redo = 0;
        ctl->stop = ctl->abort;
        mbar_fence_init();
        fence_proxy_async_smem();
    }
    if (warp == MMA_WARP) {
        tmem_alloc(smem_u32(&ctl->tmem_base), TMEM_COLS);
        // a CTA that may allocate again (for its next tile, or for the same one in two sweeps) keeps its permit
        if ((MODE == 0 || (MODE != 3 && !a.walk)) && !again) tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    if (ctl->stop) {
        // A wait has given up earlier (the status word is set until the host reads it): no more work is started. One thread reads
        // the word, which may change at any time: threads that read it each for themselves could part here.
        if (warp == MMA_WARP) tmem_dealloc(tmem, TMEM_COLS);
        return TILE_STOP;
    }

    const int n64 = n64_early;
    const int n = DENSE ? last - first : (n64 + 1) >> 1;      // exact iterations: pairs of 64-token blocks
    // iterations of the fallback sweep: all, or for a sample one in 32 (1 to 8 of them) spread over the list
    const int nsample = min(n, min(max(n >> 5, 1), 8));
    // a sample of one iteration needs no sweep: it is a look at the logits of iteration 0, which stay for their own softmax
    const bool first_is_sample = DENSE && sample && nsample == 1;
    const int nsweep = first_is_sample ? 0 : DENSE && sample ? nsample : n;
    const bool find_top = DENSE && sample && n > nsample;
    auto sweep_iter = [&](int i) { return DENSE && sample ? i * n / nsweep : i; };
    const int nvirt = FALLBACK ? 0 : a.nvirt;
    const int nref = (FALLBACK || COMPENSATE) ? 0 : a.nref;
    const int nt = n + nvirt + nref;
    const int* list = a.blocks + (size_t)th_idx * a.nk;
    const Sched sched{n, nvirt, nref, nref > 0 ? max(nt / nref, 1) : 1};

    // K and V tiles travel through one ring of NSLOT slots in the order the MMA warp consumes them:
    //   [fallback sweep: K(0) K(1) ... K(nsweep-1)]  K(0) K(1)  { V(i) K(i+2) } for i = 0 .. nt-1
    // tile number `seq` lives in slot seq % NSLOT; its barriers are in phase (seq / NSLOT) & 1.
    uint32_t pseq = 0;                                // load warps: one past the last tile issued (used again at teardown)

    if (warp == LOADK_WARP || warp == LOADV_WARP) {
        // ------------------------------------------------------------ loads: one warp walks the K tiles, one the V tiles
        const bool is_v = warp == LOADV_WARP;
        bool ok = true;
        const CUtensorMap* map_x = is_v ? &tmV : &tmK;       // exact blocks
        const CUtensorMap* map_m = is_v ? &tmVm : &tmKm;     // block means
        const CUtensorMap* map_r = is_v ? &tmVr : &tmKr;     // representative tables
        const int* rl = a.refine + (size_t)th_idx * a.rw;
        const uint32_t full0 = smem_u32(&ctl->full[0]), empty0 = smem_u32(&ctl->empty[0]);
        const uint32_t box_off = (uint32_t)(lane >> 1) * HALF_BYTES + (uint32_t)(lane & 1) * BLK_BYTES;   // lanes 0..3
        const int box_x = (lane >> 1) * 64;
        // block ids: a 32-entry window of the list held across the lanes, one coalesced load per 16 iterations
        int win = lane < n64 ? win_early : 0, wbase = 0;       // the first window was requested at the top of the kernel
        // tile number `seq` of the ring: K or V tile of iteration i (i < 0: K tile -i-1 of the fallback sweep)
        auto put = [&](uint32_t seq, int i) {
            if (!ok) return;
            int ra = 0, rb = 64;
            const CUtensorMap* m = map_m;
            int kind, idx;
            if (i < 0) { kind = 0; idx = -i - 1; }        // a K tile of the fallback sweep
            else sched.decode(i, kind, idx);
            if (kind == 0) {
                const int e = DENSE ? 2 * (first + idx) : 2 * idx;
                if (DENSE) {
                    ra = e * BK;
                    rb = ra + BK;
                } else {
                    if ((e & ~31) != wbase) {
                        wbase = e & ~31;
                        win = (wbase + lane < n64) ? list[wbase + lane] : 0;
                    }
                    ra = __shfl_sync(0xffffffffu, win, e & 31) * BK;
                    rb = __shfl_sync(0xffffffffu, win, (e + 1) & 31) * BK;
                }
                if (e + 1 >= n64) rb = ra;                     // odd list: block a again, masked in the softmax
                m = map_x;
            } else {
                ra = idx * 128;                                // rows of the block-mean tables
                rb = ra + 64;
            }
            const uint32_t slot = seq % NSLOT, par = ((seq / NSLOT) & 1) ^ 1;
            if (lane == 0) {
                ok = mbar_wait(empty0 + 8 * slot, par, abort_flag, a.status, 101);
                if (seq == Q_SLOT) ok = ok && mbar_wait(smem_u32(&ctl->qfull), 0, abort_flag, a.status, 103);
            }
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;     // the other lanes sleep at the shuffle instead of polling
            if (!ok) return;
            const uint32_t dst = sRing + slot * TILE_BYTES, bar = full0 + 8 * slot;
            if (kind != 2) {
                if (lane == 0) mbar_arrive_expect_tx(bar, TILE_BYTES);
                __syncwarp();
                if (lane < 4) tma_load_3d(dst + box_off, m, bar, box_x, (lane & 1) ? rb : ra, h);
            } else {
                // refine iteration: list entry 32 c + e (held by lane e) fills rows 4e .. 4e+3 of the tile: the block's four
                // representatives are contiguous rows of the table, one 512-byte TMA box per d half
                const int cr = idx;
                const int my = rl[32 * cr + lane];
                if (!is_v) {
                    // the 128 column biases (log2 cluster sizes) of this iteration, for the softmax warps. Slot cr % NBIAS is
                    // free again: this tile's ring slot was released by QK(i - 3), which was issued after the softmax warps
                    // had handed over iteration i - 5.
                    *reinterpret_cast<float4*>(bias_ring + (cr % NBIAS) * 128 + 4 * lane) =
                        __ldg(reinterpret_cast<const float4*>(a.log_counts + (size_t)h * a.nb4 + 4 * my));
                    __syncwarp();
                }
                if (lane == 0) mbar_arrive_expect_tx(bar, TILE_BYTES);
                __syncwarp();
                tma_load_3d(dst + (uint32_t)lane * 512u, map_r, bar, 0, 4 * my, h);
                tma_load_3d(dst + HALF_BYTES + (uint32_t)lane * 512u, map_r, bar, 64, 4 * my, h);
            }
            pseq = seq + 1;
        };
        if (is_v) {
            // Q through the ring's last slot. A thread's own row by plain loads is 32 lines to an instruction, 3,000 clocks a tile.
            if (lane == 0) mbar_arrive_expect_tx(smem_u32(&ctl->qload), TILE_BYTES);
            __syncwarp();
            if (lane < 4) tma_load_3d(sRing + Q_SLOT * TILE_BYTES + box_off, &tmQ, smem_u32(&ctl->qload), box_x, qb * BM + (lane & 1) * BK, h);
        }
        // K: the sweep's tiles come first in the ring, then K(0), K(1) and K(i + 2) after every V(i). V(i) comes after the K tiles
        // 0 .. min(i + 2, nt) - 1 and the V tiles before it. A wait on a slot's `empty` barrier can only tell two consecutive
        // rounds apart (one parity bit), so the V warp must not start polling while the ring is still rounds behind its first
        // tile: it starts once the K warp has issued the last sweep tile.
        if (is_v && FALLBACK) {
            if (lane == 0) ok = mbar_wait(smem_u32(&ctl->sweepbar), 0, abort_flag, a.status, 102);
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        }
        const int sweeps = FALLBACK ? nsweep : 0, lead = is_v ? 0 : sweeps;
#pragma unroll 1
        for (int j = 0; j <= lead + nt; ++j) {
            if (FALLBACK && !is_v && j == lead) {
                if (lane == 0) mbar_arrive(smem_u32(&ctl->sweepbar));
                wbase = -1;
            }
            if (j == lead + nt) break;
            const int i = j - lead;
            put((uint32_t)(i < 0 ? j : sweeps + (is_v ? min(i + 2, nt) + i : i < 2 ? i : 2 * i - 1)), i < 0 ? -sweep_iter(j) - 1 : i);
        }
    } else if (warp == MMA_WARP) {
        // ------------------------------------------------------------ MMAs: the warp runs uniformly, one elected lane issues
        constexpr uint32_t IDESC = umma_idesc_bf16(BM, 128, 0);        // S = Q K^T: A (Q) from tensor memory, B K-major
        constexpr uint32_t IDESC_PV = umma_idesc_bf16(BM, HD, 1);      // O += P V: A (P) from tensor memory, B MN-major
        // Shared-memory descriptors: everything but the start address is a constant of the layout, so the words are built
        // once and an MMA costs one add. K-major (K): LBO 16, SBO 1024; MN-major (V): LBO = one d half, SBO 1024.
        const uint64_t dk0 = umma_desc_sw128(0, 16, 1024), dv0 = umma_desc_sw128(0, HALF_BYTES, 1024);
        const uint32_t k_hi = (uint32_t)(dk0 >> 32), k_lo0 = (uint32_t)dk0;
        const uint32_t v_hi = (uint32_t)(dv0 >> 32), v_lo0 = (uint32_t)dv0;
        uint32_t cslot = 0, cpar = 0, nQK[2] = {0, 0}, wP[2] = {0, 0};
        const uint32_t full0 = smem_u32(&ctl->full[0]), empty0 = smem_u32(&ctl->empty[0]);
        const uint32_t sfull0 = smem_u32(&ctl->sfull[0]), pfull0 = smem_u32(&ctl->pfull[0]);
        bool ok = mbar_wait_warp(smem_u32(&ctl->qfull), 0, abort_flag, a.status, 201);     // Q is in tensor memory
        // next tile of the ring: returns its slot
        auto take = [&]() -> uint32_t {
            const uint32_t slot = cslot;
            ok = ok && mbar_wait_warp(full0 + 8 * slot, cpar, abort_flag, a.status, 202);
            if (++cslot == NSLOT) { cslot = 0; cpar ^= 1; }
            return slot;
        };
        // S[buf] <- Q K^T. The S columns also hold the previous P of that buffer: every earlier use must have been handed
        // back by the softmax warps (pfull) before they are overwritten; the PV that read it was issued before (in order).
        auto issue_qk = [&](int buf) {
            const uint32_t slot = take();
            while (ok && wP[buf] < nQK[buf]) {
                ok = mbar_wait_warp(pfull0 + 8 * buf, wP[buf] & 1, abort_flag, a.status, 203);
                ++wP[buf];
            }
            if (!ok) return;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t d = tmem + (uint32_t)buf * 128;
                const uint32_t kb_lo = k_lo0 + ((sRing + slot * TILE_BYTES) >> 4);
#pragma unroll
                for (int ks = 0; ks < HD / 16; ++ks)
                    umma_ts_lohi(d, tmem + Q_COL + ks * 8, kb_lo + (uint32_t)(((ks >> 2) * HALF_BYTES + (ks & 3) * 32) >> 4),
                                 k_hi, IDESC, ks > 0);
                umma_commit(sfull0 + 8 * buf);
                umma_commit(empty0 + 8 * slot);
            }
            __syncwarp();
            ++nQK[buf];
        };
        if (FALLBACK) {
            for (int i = 0; i < nsweep && ok; ++i) issue_qk(i & 1);
        }
        if (nt > 0) issue_qk(0);
        if (nt > 1) issue_qk(1);
        for (int i = 0; i < nt && ok; ++i) {
            const int buf = i & 1;
            const uint32_t slot = take();
            ok = ok && mbar_wait_warp(pfull0 + 8 * buf, wP[buf] & 1, abort_flag, a.status, 205);   // P(i) stored
            if (!ok) break;
            ++wP[buf];
            tc_fence_after();
            if (elect_one()) {
                const uint32_t p = tmem + (uint32_t)buf * 128;     // bf16 pairs: keys 0-63 in columns [0,32), 64-127 in [64,96)
                const uint32_t vb_lo = v_lo0 + ((sRing + slot * TILE_BYTES) >> 4);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                    umma_ts_lohi(tmem + O_COL, p + (ks < 4 ? ks * 8 : 64 + (ks - 4) * 8),
                                 vb_lo + (uint32_t)((ks * 2048) >> 4), v_hi, IDESC_PV,
                                 (i > 0 || ks > 0) ? 1u : 0u);
                umma_commit(empty0 + 8 * slot);
                if (i + 1 == nt) umma_commit(smem_u32(&ctl->ofull));
            }
            __syncwarp();
            if (i + 2 < nt) issue_qk(buf);
        }
        // every MMA issued above has finished before tensor memory is freed
        if (elect_one()) umma_commit(smem_u32(&ctl->drain));
        __syncwarp();
        mbar_wait(smem_u32(&ctl->drain), 0, abort_flag, a.status, 206);
    } else if (warp == MASS_WARP) {
        // ------------------------------------------------------------ block masses: lane 0 / 1 = first / second block of a pair
        if (!FALLBACK && !COMPENSATE && a.mass != nullptr) {
            float* mrow = a.mass + ((size_t)h * a.nq + qb) * a.nb;
            bool ok = true;
            for (int e = 0; e < n && ok; ++e) {
                const int set = e % NMASS, c = lane & 1;
                const bool mine = lane < 2 && 2 * e + c < n64;
                const int blk = mine ? __ldg(list + 2 * e + c) : 0;           // fetched before the wait
                ok = mbar_wait_warp(smem_u32(&ctl->massbar[set]), (e / NMASS) & 1, abort_flag, a.status, 308);
                if (!ok) break;
                // rows lane, lane + 32, lane + 64, lane + 96 of both column halves, then the 32 lanes: always the same order
                const float* mp = mass_rows + set * 2 * BM;
                float m0 = (mp[lane] + mp[lane + 32]) + (mp[lane + 64] + mp[lane + 96]);
                float m1 = (mp[BM + lane] + mp[BM + lane + 32]) + (mp[BM + lane + 64] + mp[BM + lane + 96]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    m0 += __shfl_xor_sync(0xffffffffu, m0, o);
                    m1 += __shfl_xor_sync(0xffffffffu, m1, o);
                }
                if (mine) mrow[blk] = c ? m1 : m0;
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&ctl->massfree[set]));
            }
        }
    } else {
        // ------------------------------------------------------------ softmax and epilogue
        const int rq = warp & 3, ch = warp >> 2;             // row quarter, column half
        const int trow = 32 * rq + lane, row = qb * BM + trow;
        const bool valid = row < a.L;
        const uint32_t lane_base = tmem + ((uint32_t)(32 * rq) << 16);
        uint32_t s[64];
        bool ok = true;

        // this thread's half of its Q row -> tensor memory (bf16 pairs, 32 columns), the A operand of every QK^T
        ok = mbar_wait_warp(smem_u32(&ctl->qload), 0, abort_flag, a.status, 309);
        {
            const uint8_t* src = smem_raw + SMEM_RING + Q_SLOT * TILE_BYTES + ch * HALF_BYTES + trow * 128;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint4 w = *reinterpret_cast<const uint4*>(src + ((i ^ (trow & 7)) << 4));
                s[4 * i] = w.x; s[4 * i + 1] = w.y; s[4 * i + 2] = w.z; s[4 * i + 3] = w.w;
            }
            tmem_st32(lane_base + Q_COL + 32 * ch, s);
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(smem_u32(&ctl->qfull));
        }
        float m = FALLBACK ? 0.f : m_early;
        float best = 0.f;                          // dense: the largest logit found so far (at first the sample's) and its key
        int best_key = -1;
        float p_best = 1.f;                        // its P, rounded (1 for the sample's maximum, the offset)
        uint32_t uS[2] = {0, 0};

        if (FALLBACK) {
            float mx = -INFINITY;
            for (int i = 0; i < (first_is_sample ? 1 : nsweep) && ok; ++i) {
                const int buf = i & 1, e = 2 * (first + sweep_iter(i)) + ch;
                const bool has = e < n64;
                const int blk = DENSE ? e : list[has ? e : e - 1];
                ok = ok && mbar_wait_warp(smem_u32(&ctl->sfull[buf]), uS[buf] & 1, abort_flag, a.status, 301);
                if (!ok) break;
                if (!first_is_sample) ++uS[buf];
                tc_fence_after();
                tmem_ld32(lane_base + buf * 128 + 64 * ch, &s[0]);
                tmem_ld32(lane_base + buf * 128 + 64 * ch + 32, &s[32]);
                tmem_wait_ld_regs(&s[0]);
                tmem_wait_ld_regs(&s[32]);
                if (!first_is_sample) {
                    tc_fence_before();
                    mbar_arrive(smem_u32(&ctl->pfull[buf]));
                }
                int lim = (blk == a.nb - 1) ? a.tail_valid : BK;
                if (!has) lim = 0;
#pragma unroll
                for (int c = 0; c < 64; ++c)
                    if (c < lim) mx = fmaxf(mx, __uint_as_float(s[c]));
            }
            // the row maximum over both column halves
            ctl->m_part[ch][trow] = mx;
            mbar_arrive(smem_u32(&ctl->lbar));
            ok = mbar_wait_warp(smem_u32(&ctl->lbar), 0, abort_flag, a.status, 306) && ok;
            best = fmaxf(ctl->m_part[0][trow], ctl->m_part[1][trow]);
            m = (best == -INFINITY) ? 0.f : best * a.scale_log2;
        }

        float2 lsum = make_float2(0.f, 0.f);
        // dense: the row sum of P as rounded for PV, in rounded float32 adds. Taken by the tensor core along with PV (a product with
        // ones, no faster: 6.93 ms for 32,760 tokens x 12 heads, 6.89 so) it was cut off at every add: the sum of 65,536 terms 1e-5
        // short, of 119,056 2e-5, in every row on the same side.
        float2 rsum = make_float2(0.f, 0.f);
        const int* bits = a.skip_bits + ((size_t)h * a.nq + qb) * a.nw;
        const bool want_mass = !FALLBACK && !COMPENSATE && a.mass != nullptr;
        const float2 sc2 = make_float2(a.scale_log2, a.scale_log2);
        // kind, index and block id of an iteration are found one iteration ahead, so that the list entry (a global load)
        // has arrived long before it is needed
        SchedIter walk;
        int kind = 0, idx = 0, blk = 0;
        auto block_of = [&](int kd, int ix) -> int {
            if (kd != 0) return 0;
            const int e = 2 * (first + ix) + ch;
            return DENSE ? e : __ldg(list + (e < n64 ? e : e - 1));
        };
        if (nt > 0) {
            walk.get(sched, kind, idx);
            blk = block_of(kind, idx);
        }
        for (int i = 0; i < nt && ok; ++i) {
            const int buf = i & 1;
            const bool exact = kind == 0, pooled = kind == 1;
            const bool has = !exact || 2 * (first + idx) + ch < n64;
            const int cur_idx = idx, cur_blk = blk;
            int nkind = 0, nidx = 0, nblk = 0;
            walk.advance(sched);
            if (i + 1 < nt) {
                walk.get(sched, nkind, nidx);
                nblk = block_of(nkind, nidx);
            }
            // the skip words of a block-mean iteration are fetched before the wait, so that their latency is hidden by it
            uint32_t w0 = 0, w1 = 0;
            if (pooled && !COMPENSATE) {
                w0 = (uint32_t)__ldg(bits + 4 * cur_idx + 2 * ch);
                w1 = (uint32_t)__ldg(bits + 4 * cur_idx + 2 * ch + 1);
            }
            ok = ok && mbar_wait_warp(smem_u32(&ctl->sfull[buf]), uS[buf] & 1, abort_flag, a.status, 302);
            if (!ok) break;
            ++uS[buf];
            tc_fence_after();
            const uint32_t scol = lane_base + buf * 128 + 64 * ch;
            tmem_ld32(scol, &s[0]);
            tmem_ld32(scol + 32, &s[32]);
            tmem_wait_ld();                            // (naming the registers: 4.07 against 4.03 ms of a Wan-1.3B step)
            float2 acc = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
            uint32_t pk[32];
            if (exact) {
                int lim = (cur_blk == a.nb - 1) ? a.tail_valid : BK;
                if (!has) lim = 0;
                const float2 off2 = make_float2(-m, -m);
                if (lim == BK) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float2 xv = __ffma2_rn(make_float2(__uint_as_float(s[2 * j]), __uint_as_float(s[2 * j + 1])), sc2, off2);
                        const float2 p = exp2_pair(xv);
                        if (j & 1) acc1 = __fadd2_rn(acc1, p); else acc = __fadd2_rn(acc, p);
                        pk[j] = pack_bf16x2(p.x, p.y);
                        if (DENSE) rsum = __fadd2_rn(rsum, make_float2(__uint_as_float(pk[j] << 16), __uint_as_float(pk[j] & 0xFFFF0000u)));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float2 xv = __ffma2_rn(make_float2(__uint_as_float(s[2 * j]), __uint_as_float(s[2 * j + 1])), sc2, off2);
                        float2 p = exp2_pair(xv);
                        p.x = 2 * j < lim ? p.x : 0.f;
                        p.y = 2 * j + 1 < lim ? p.y : 0.f;
                        acc = __fadd2_rn(acc, p);
                        pk[j] = pack_bf16x2(p.x, p.y);
                        if (DENSE) rsum = __fadd2_rn(rsum, make_float2(__uint_as_float(pk[j] << 16), __uint_as_float(pk[j] & 0xFFFF0000u)));
                    }
                }
            } else if (pooled) {
                // block-mean columns: column c of this half is block 128 cv + 64 ch + c; a set bit masks it
                const int cv = cur_idx;
                if (COMPENSATE) {
                    // every block that was not kept (refined ones included) is compensated: bits from the keep mask
                    const int b0 = 128 * cv + 64 * ch;
                    const uint8_t* kp = a.keep + ((size_t)h * a.nq + qb) * a.nb + b0;
                    w0 = 0; w1 = 0;
#pragma unroll
                    for (int c = 0; c < 32; ++c) {
                        w0 |= (uint32_t)(b0 + c >= a.nb ? 1 : kp[c] != 0) << c;
                        w1 |= (uint32_t)(b0 + 32 + c >= a.nb ? 1 : kp[32 + c] != 0) << c;
                    }
                }
                const float2 off2 = make_float2(-m + 6.0f, -m + 6.0f);   // log2(64): a mean stands for its block's tokens
                const int last_c = (a.nb - 1) - (128 * cv + 64 * ch);    // column of the (maybe shorter) last block
                const float fix = a.tail_log2 - 6.0f;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    float2 xv = __ffma2_rn(make_float2(__uint_as_float(s[2 * j]), __uint_as_float(s[2 * j + 1])), sc2, off2);
                    if (2 * j == last_c) xv.x += fix;
                    if (2 * j + 1 == last_c) xv.y += fix;
                    if (COMPENSATE) { xv.x = fminf(xv.x, 100.0f); xv.y = fminf(xv.y, 100.0f); }   // triton_ops.py:275
                    float2 p = exp2_pair(xv);
                    const uint32_t w = j < 16 ? w0 : w1;
                    p.x = ((w >> ((2 * j) & 31)) & 1u) ? 0.f : p.x;
                    p.y = ((w >> ((2 * j + 1) & 31)) & 1u) ? 0.f : p.y;
                    acc = __fadd2_rn(acc, p);
                    pk[j] = pack_bf16x2(p.x, p.y);
                }
            } else {
                // representatives: column c of this half has the bias that the K load warp staged for this iteration
                const int cr = cur_idx;
                const float4* bb = reinterpret_cast<const float4*>(bias_ring + (cr % NBIAS) * 128 + 64 * ch);
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float4 b4 = bb[e];
                    const int c = 4 * e;
                    const float2 x0 = __ffma2_rn(make_float2(__uint_as_float(s[c]), __uint_as_float(s[c + 1])), sc2,
                                                 make_float2(b4.x - m, b4.y - m));
                    const float2 x1 = __ffma2_rn(make_float2(__uint_as_float(s[c + 2]), __uint_as_float(s[c + 3])), sc2,
                                                 make_float2(b4.z - m, b4.w - m));
                    const float2 p0 = exp2_pair(x0), p1 = exp2_pair(x1);
                    acc = __fadd2_rn(acc, p0);
                    acc1 = __fadd2_rn(acc1, p1);
                    pk[c / 2] = pack_bf16x2(p0.x, p0.y);
                    pk[c / 2 + 1] = pack_bf16x2(p1.x, p1.y);
                }
            }
            tmem_st32(scol, pk);                       // P over the first 32 of this thread's own 64 S columns
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(smem_u32(&ctl->pfull[buf]));
            acc = __fadd2_rn(acc, acc1);
            lsum = __fadd2_rn(lsum, acc);
            if (DENSE && find_top) {
                // a logit above the row's largest so far, and its key (P has left already: this is off the chain to PV)
                // rounding keeps the order: a larger logit has a P that rounds to no less than the best one's, and P is packed already
                uint32_t pm[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    pm[x] = max_bf16x2(pk[8 * x], pk[8 * x + 1]);
#pragma unroll
                    for (int y = 2; y < 8; ++y) pm[x] = max_bf16x2(pm[x], pk[8 * x + y]);
                }
                pm[0] = max_bf16x2(max_bf16x2(pm[0], pm[1]), max_bf16x2(pm[2], pm[3]));
                const float p_top = fmaxf(__uint_as_float(pm[0] << 16), __uint_as_float(pm[0] & 0xFFFF0000u));
                if (__any_sync(0xffffffffu, p_top >= p_best)) {
                    const int lim = !has ? 0 : cur_blk == a.nb - 1 ? a.tail_valid : BK;
                    if (lim != BK) {
#pragma unroll
                        for (int c = 0; c < 64; ++c)
                            if (c >= lim) s[c] = 0xff800000u;
                    }
                    float mx[8];
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
                        const float* x = reinterpret_cast<const float*>(s) + 8 * g;
                        mx[g] = fmaxf(fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3])), fmaxf(fmaxf(x[4], x[5]), fmaxf(x[6], x[7])));
                    }
                    const float top = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), fmaxf(fmaxf(mx[4], mx[5]), fmaxf(mx[6], mx[7])));
                    const bool better = top > best;
                    if (__any_sync(0xffffffffu, better)) {
                        // its column by halving: each level keeps the half of the candidates that holds the maximum
                        const bool h5 = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) < top;
                        const bool h4 = fmaxf(h5 ? mx[4] : mx[0], h5 ? mx[5] : mx[1]) < top;
                        const float m0 = h5 ? mx[4] : mx[0], m2 = h5 ? mx[6] : mx[2];
                        const bool h3 = (h4 ? m2 : m0) < top;
                        uint32_t t[32];
#pragma unroll
                        for (int c = 0; c < 32; ++c) t[c] = h5 ? s[32 + c] : s[c];
#pragma unroll
                        for (int c = 0; c < 16; ++c) t[c] = h4 ? t[16 + c] : t[c];
                        int at = 0;
#pragma unroll
                        for (int c = 0; c < 8; ++c) at = __uint_as_float(h3 ? t[8 + c] : t[c]) == top ? c : at;
                        best = better ? top : best;
                        best_key = better ? cur_blk * BK + 32 * h5 + 16 * h4 + 8 * h3 + at : best_key;
                        p_best = better ? __uint_as_float(pack_bf16x2(ex2_approx(fmaf(top, a.scale_log2, -m)), 0.f) << 16) : p_best;
                    }
                }
            }
            if (want_mass && exact) {
                // per-block mass: every row leaves its sum over the block's columns in shared memory; the mass warp adds
                // the 128 rows in a fixed order and stores the result (no atomics: the map is reproducible bit for bit). A
                // set of row sums is written again NMASS exact iterations later, once the mass warp has handed it back.
                const int set = cur_idx % NMASS, round = cur_idx / NMASS;
                if (round > 0) {
                    ok = mbar_wait_warp(smem_u32(&ctl->massfree[set]), (round - 1) & 1, abort_flag, a.status, 304);
                    if (!ok) break;
                }
                mass_rows[(set * 2 + ch) * BM + trow] = acc.x + acc.y;      // this row's sum over the block's 64 columns
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&ctl->massbar[set]));
            }
            kind = nkind; idx = nidx; blk = nblk;
        }

        // ---- epilogue: row sums of both column halves, then this thread's 64 columns of O
        ctl->l_part[ch][trow] = lsum.x + lsum.y;
        // (not in m_part: with one or two iterations nothing keeps the other half's warp from still reading its maxima)
        if (DENSE) {
            const float top = ex2_approx(fmaf(best, a.scale_log2, -m));      // the bits of the loop
            ctl->r_part[ch][trow] = rsum.x + rsum.y;
            ctl->e_part[ch][trow] = best_key < 0 ? 0.f : top - __uint_as_float(pack_bf16x2(top, 0.f) << 16);
            ctl->key_part[ch][trow] = best_key;
        }
        mbar_arrive(smem_u32(&ctl->lbar));
        ok = mbar_wait_warp(smem_u32(&ctl->lbar), FALLBACK ? 1 : 0, abort_flag, a.status, 307) && ok;
        const float l = ctl->l_part[0][trow] + ctl->l_part[1][trow];
        // compensation: out = (out + sum e v) / (1 + sum e), lse += log2(1 + sum e) (triton_ops.py:280-282)
        const float lg = COMPENSATE ? log2f(1.0f + l) : log2f(l);
        // dense: the V rows of the remembered keys, on their way while the last PV runs
        int top_key[2];
        float e_top[2];
        uint4 vtop[2][8];
#pragma unroll
        for (int x = 0; x < (DENSE ? 2 : 0); ++x) {
            e_top[x] = ctl->e_part[x][trow];
            top_key[x] = ctl->key_part[x][trow];
            const uint4* src = reinterpret_cast<const uint4*>(a.v + ((size_t)max(top_key[x], 0) * a.H + h) * HD + 64 * ch);
#pragma unroll
            for (int c = 0; c < 8; ++c) vtop[x][c] = top_key[x] >= 0 ? __ldg(src + c) : make_uint4(0, 0, 0, 0);
        }
        if (nt > 0) ok = mbar_wait_warp(smem_u32(&ctl->ofull), 0, abort_flag, a.status, 303) && ok;
        if (ok) {
            tc_fence_after();
            const float rounded = DENSE ? (ctl->r_part[0][trow] + ctl->r_part[1][trow]) + (e_top[0] + e_top[1]) : 0.f;
            const float inv = COMPENSATE ? 1.0f / (1.0f + l) : DENSE ? 1.0f / rounded : 1.0f / l;
            bool finite = true;
            // The outputs are turned in shared memory, 32 rows of a column half per warp, in the ring (every K / V tile has been
            // consumed): four whole lines to a store. A thread's own row at a time is 16 bytes of 32 lines, 4,000 clocks a tile; a
            // TMA store keeps the CTA 1,000 clocks longer, until it has read its source.
            uint8_t* stage = smem_raw + SMEM_RING + warp * (32 * 128);
            auto chunk = [&](int r, int c) { return reinterpret_cast<uint4*>(stage + r * 128 + ((c ^ (r & 7)) << 4)); };
            if (COMPENSATE) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {              // the old outputs, four rows to a load
                    const int r = 4 * i + (lane >> 3), grow = qb * BM + 32 * rq + r;
                    if (grow < a.L) *chunk(r, lane & 7) = *reinterpret_cast<const uint4*>(a.out + ((size_t)grow * a.H + h) * HD + 64 * ch + 8 * (lane & 7));
                }
                __syncwarp();
            }
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t* o = &s[0];
                if (nt > 0) {
                    tmem_ld32(lane_base + O_COL + 64 * ch + 32 * half, o);
                    tmem_wait_ld_regs(o);
                }
                if (DENSE) {
#pragma unroll
                    for (int x = 0; x < 2; ++x)
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            const uint4 w4 = vtop[x][4 * half + c / 4];
                            const uint32_t w = (c & 3) == 0 ? w4.x : (c & 3) == 1 ? w4.y : (c & 3) == 2 ? w4.z : w4.w;
                            o[2 * c] = __float_as_uint(fmaf(e_top[x], __uint_as_float(w << 16), __uint_as_float(o[2 * c])));
                            o[2 * c + 1] = __float_as_uint(fmaf(e_top[x], __uint_as_float(w & 0xFFFF0000u), __uint_as_float(o[2 * c + 1])));
                        }
#pragma unroll
                    for (int c = 0; c < 32; ++c) finite = finite && fabsf(__uint_as_float(o[c])) <= 3.0e38f;
                }
                if (DENSE && part != nullptr) {
                    if (valid) {
#pragma unroll
                        for (int c = 0; c < 32; c += 4)
                            *reinterpret_cast<uint4*>(part + PART_ROWS * BM + (16 * ch + 8 * half + c / 4) * (4 * BM) + 4 * trow) =
                                make_uint4(o[c], o[c + 1], o[c + 2], o[c + 3]);
                    }
                    continue;
                }
#pragma unroll
                for (int c = 0; c < 32; c += 8) {
                    uint4 w;
                    uint4* dst = chunk(lane, 4 * half + c / 8);
                    if (COMPENSATE) {
                        const uint4 old = *dst;
                        const uint32_t ow[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            o[c + 2 * e] = __float_as_uint(__uint_as_float(o[c + 2 * e]) + __uint_as_float(ow[e] << 16));
                            o[c + 2 * e + 1] = __float_as_uint(__uint_as_float(o[c + 2 * e + 1]) + __uint_as_float(ow[e] & 0xFFFF0000u));
                        }
                    }
                    w.x = pack_bf16x2(__uint_as_float(o[c]) * inv, __uint_as_float(o[c + 1]) * inv);
                    w.y = pack_bf16x2(__uint_as_float(o[c + 2]) * inv, __uint_as_float(o[c + 3]) * inv);
                    w.z = pack_bf16x2(__uint_as_float(o[c + 4]) * inv, __uint_as_float(o[c + 5]) * inv);
                    w.w = pack_bf16x2(__uint_as_float(o[c + 6]) * inv, __uint_as_float(o[c + 7]) * inv);
                    if (nt == 0) w = make_uint4(0, 0, 0, 0);
                    *dst = w;
                }
            }
            if (!(DENSE && part != nullptr)) {
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = 4 * i + (lane >> 3), grow = qb * BM + 32 * rq + r;
                    if (grow < a.L) *reinterpret_cast<uint4*>(a.out + ((size_t)grow * a.H + h) * HD + 64 * ch + 8 * (lane & 7)) = *chunk(r, lane & 7);
                }
            }
            tc_fence_before();
            if (ch == 0) {
                // rows past L keep the "no offset" value, as echosparse/kernels/sm120.py:96
                if (DENSE && part != nullptr) {
                    part[trow] = m;
                    part[BM + trow] = l;
                    part[2 * BM + trow] = rounded;
                } else {
                    a.lse[(size_t)row * a.H + h] = valid ? m + lg : 1e30f;
                }
            }
            if (DENSE && sample) {
                // the maximum of the sample was no usable offset for some row: the tile is done again in two sweeps
                const bool bad = valid && !(lg <= kSeedLimit && lg >= -1.f && finite);
                if (__any_sync(0xffffffffu, bad) && lane == 0) ctl->redo = 1;
            }
            if (ch == 0) {
                if (!FALLBACK && !COMPENSATE) {
                    // a tile whose row sums leave 2^[-th, th] is flagged and recomputed with online softmax
                    const bool bad = valid && !(lg >= -a.th && lg <= a.th);
                    const unsigned ballot = __ballot_sync(0xffffffffu, bad);
                    if (lane == 0) {
                        ctl->flag_part[rq] = ballot != 0;
                        mbar_arrive(smem_u32(&ctl->flagbar));
                    }
                    if (tid == 0 && mbar_wait(smem_u32(&ctl->flagbar), 0, abort_flag, a.status, 305))
                        a.flags[th_idx] = ctl->flag_part[0] | ctl->flag_part[1] | ctl->flag_part[2] | ctl->flag_part[3];
                }
            }
        }
    }

    // ---------------------------------------------------------------- teardown
    __syncwarp();
    if (warp == LOADV_WARP && lane == 0 && *abort_flag) {            // Q may still be on its way
        const uint64_t t_end = global_timer_ns() + 100000ull;
        while (!mbar_try_wait(smem_u32(&ctl->qload), 0) && global_timer_ns() < t_end) {}
    }
    if ((warp == LOADK_WARP || warp == LOADV_WARP) && lane == 0 && *abort_flag) {
        // a wait gave up somewhere: give the loads this warp issued a moment (100 us in all) to land before the CTA's
        // shared memory goes away; a tile that was never issued cannot hold the CTA back
        const uint64_t t_end = global_timer_ns() + 100000ull;
        for (uint32_t back = 1; back <= 2 * NSLOT && back <= pseq; ++back) {
            const uint32_t sq = pseq - back;
            while (!mbar_try_wait(smem_u32(&ctl->full[sq % NSLOT]), (sq / NSLOT) & 1) && global_timer_ns() < t_end) {}
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
    // (past the barrier nothing of this tile writes them, and the next tile's set-up comes after another one)
    return *abort_flag ? TILE_STOP : DENSE && sample && ctl->redo != 0 ? TILE_AGAIN : TILE_DONE;
}

template <int MODE>
__global__ void __launch_bounds__(NTHREADS, 1)
attention_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV,
                 const __grid_constant__ CUtensorMap tmKm, const __grid_constant__ CUtensorMap tmVm,
                 const __grid_constant__ CUtensorMap tmKr, const __grid_constant__ CUtensorMap tmVr, const AttnArgs a) {
    if (MODE == 0 || !a.walk) {
        attention_tile<MODE>(tmQ, tmK, tmV, tmKm, tmVm, tmKr, tmVr, a, (int)blockIdx.x, false, false);
        return;
    }
    // Fallback modes, one CTA per SM: every CTA finds the flagged tiles (a fraction of a percent of all, as a rule) and takes every
    // gridDim-th, counted in the order of the tile numbers so that the CTAs at work share a head's K and V in L2. All read all
    // flags (of a range's heads), 94 KB at 591 tiles x 40 heads, in coalesced loads, into a bit per tile in tile order: 2 us. A kernel of its own that made
    // the list took 25 us there, 0.10 ms of a Wan-14B step, and 2.3 us and a launch at 4,152 tokens x 2 heads.
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint32_t* bits = reinterpret_cast<uint32_t*>(smem_raw + SMEM_MASS);       // the block masses' room: these modes have none
    int* mine = reinterpret_cast<int*>(bits + WALK_TILES / 32);
    int* warp_sum = mine + WALK_MINE;
    constexpr int PER = WALK_TILES / 32 / NTHREADS;                          // words of a thread
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, total = a.nq * a.H;
    const int step = min(WALK_TILES, (WALK_MINE - 1) * (int)gridDim.x);
    int found = 0;                                                           // flagged tiles before this range
    bool again = false;
    for (int e0 = 0; e0 < total; e0 += step) {
        for (int w = tid; w < WALK_TILES / 32; w += NTHREADS) bits[w] = 0;
        __syncthreads();
        const int h0 = e0 / a.nq, heads = (min(e0 + step, total) - 1) / a.nq - h0 + 1;     // the range's heads: one range, all of them
#pragma unroll 8
        for (int f = tid; f < heads * a.nq; f += NTHREADS) {
            const int qb = f / heads, h = h0 + f % heads, e = h * a.nq + qb - e0;          // flags are (tile, head), tile numbers head * nq + tile
            if (__ldg(a.flags + (heads == a.H ? f : qb * a.H + h)) != 0 && e >= 0 && e < step) atomicOr(bits + (e >> 5), 1u << (e & 31));
        }
        __syncthreads();
        uint32_t w[PER];
        int n = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            w[i] = bits[tid * PER + i];
            n += __popc(w[i]);
        }
        int incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        int rank = found + incl - n, count = 0;
        for (int i = 0; i < NTHREADS / 32; ++i) {
            if (i < warp) rank += warp_sum[i];
            count += warp_sum[i];
        }
        // ranks blockIdx, blockIdx + grid, .. are this CTA's; the first of the range goes to mine[0]
        const int grid = gridDim.x, lead = ((int)blockIdx.x - found % grid + grid) % grid;
        // (found by their rank: a division for every flagged tile was 3 us where all tiles of a short sequence are flagged)
        if (n > 0) {
            int skip = lead - (rank - found);                               // flagged tiles of this thread before the first of this CTA's
            if (skip < 0) skip = (skip % grid + grid) % grid;
            int slot = skip < n ? (rank - found + skip - lead) / grid : 0;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                uint32_t m = w[i];
                for (int left = __popc(m); left > skip; skip = grid - 1) {
                    for (left -= skip + 1; skip > 0; --skip) m &= m - 1;
                    mine[slot++] = e0 + 32 * (tid * PER + i) + __ffs(m) - 1;
                    m &= m - 1;
                }
                skip -= __popc(m);
            }
        }
        __syncthreads();
        for (int t = 0; lead + t * grid < count; ++t) {
            if (attention_tile<MODE>(tmQ, tmK, tmV, tmKm, tmVm, tmKr, tmVr, a, mine[t], again, false) == TILE_STOP) return;
            again = true;
            __syncthreads();
        }
        found += count;
    }
}

// Online softmax over every block, one CTA per tile. A first sweep of QK MMAs over all columns, only to find the row maxima,
// costs half as much tensor work again as the attention itself, and no offset has to be that exact: P is bf16 and the sums are
// fp32, both as precise relative to any offset, as long as nothing leaves their exponent range. So the offset is the row's
// maximum over a sample of the columns: the row sum then contains that maximum's own term 1, and the tile stands unless a row
// sum passed 2^kSeedLimit or an output is not finite; only then is it done again with the maximum over all columns.
// What an exact maximum gives besides is that the row's largest term is 1, so that its rounding costs nothing; a sample's maximum
// rarely is the row's, and where few keys hold most of a row that is most of P's error. So the outputs are divided by the sum of the
// rounded P, which cancels the rounding of a dominant term, and every half of a row remembers its largest logit above the sample's
// and the key: the epilogue adds (P - rounded P) V[key]. Relative error against fp64, two sweeps / as here / without the remembered
// terms: 32,760 tokens x 12 heads 1.716e-3 / 1.682e-3 / 1.726e-3; 9,360 tokens of random q, k with logits of deviation 3.2
// 1.821e-3 / 1.763e-3 / 2.017e-3. Time of the first shape, when this was chosen, 9.7 / 6.2 / 5.6 ms, of 1,560 tokens 95 / 56 / 46 us (one iteration in four
// searched: 6.1 ms, but 1.95e-3 on the random rows).
// Every half keeps its term however small its share. Leaving those below 1 / 256 of the row rounded was no faster on the first shape
// (6.89 ms, 6.84 so), on rows of logits with deviation 1, whose largest grows often, by 5 % (12,000 x 24 1.72 ms, 1.82 so).
// (Flagged tiles, MODE 1, are those whose offset was far off, where a sample's maximum often is too: 0.81 ms of a Wan-14B step with
// a sample first, 0.47 ms in two sweeps.)
//
// Few tiles, or a few more than the SMs, leave most SMs idle: 1,560 tokens of 12 heads are 156 tiles on 148 SMs, two waves of which
// the second is nearly empty. So the last tiles are cut by iterations (plan_dense): each piece takes its own offset from its own
// columns and leaves m, the row sums and O in fp32, and a second kernel adds the pieces of a tile in their order. The error against fp64 is never larger than
// that of whole tiles (897 to 9,360 tokens, 1 to 24 heads: 0.96 to 1.00 of it; every piece remembers its own largest terms). One launch after
// the other, us, whole tiles / cut: 1,560 tokens x 12 heads 44.5 / 36.1, x 1 head 23.0 / 14.1, 4,096 x 1 44.2 / 20.9, 6,000 x 4
// 120 / 91, 8,000 x 12 485 / 422; 4,096 tokens x 8 heads (1.73 waves of 32 iterations) stay whole: 87.7 / 93.0.
__global__ void __launch_bounds__(NTHREADS, 1)
dense_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
             const __grid_constant__ CUtensorMap tmV, const AttnArgs a, const DenseSplit d) {
    const int c = blockIdx.x, whole = d.part ? d.whole : (int)gridDim.x;
    int x = 0, end = 0;                                   // this CTA's stretch of the cut tiles' iterations
    if (d.part && c < d.ctas) { x = d.edge(c); end = d.edge(c + 1); }
    int next = c, tile = 0, first = 0, last = d.n;
    float* part = nullptr;
    bool redo = false;
    for (bool again = false;; again = true) {
        if (!redo) {
            if (next < whole) {
                tile = next;
                next += gridDim.x;
            } else if (x < end) {
                const int t = x / d.n;
                tile = d.whole + t;
                first = x - t * d.n;
                last = min(d.n, end - t * d.n);
                x = t * d.n + last;
                // a piece that ends a tile goes to the CTA's first slot, one that only starts it to its second
                part = last - first == d.n ? nullptr : d.part + (size_t)(2 * c + (first == 0)) * PART_FLOATS;
            } else {
                break;
            }
        }
        if (again) __syncthreads();
        const TileEnd end_of_tile = attention_tile<3>(tmQ, tmK, tmV, tmK, tmV, tmK, tmV, a, tile, again, !redo, first, last, part);
        if (end_of_tile == TILE_STOP) break;
        redo = end_of_tile == TILE_AGAIN;
    }
    launch_dependents();
}

// The pieces of a cut tile, added in their order: block (t, y) does MERGE_COLS columns of the t-th cut tile, one row per thread.
constexpr int MERGE_COLS = 8;
__global__ void __launch_bounds__(BM)
dense_merge_kernel(const AttnArgs a, const DenseSplit d) {
    constexpr int N4 = MERGE_COLS / 4, AT_ONCE = 4;
    const int t = blockIdx.x, x0 = t * d.n, x1 = x0 + d.n, trow = threadIdx.x;
    wait_prerequisites();
    // a wait has given up: pieces may be missing, and what the scratch holds in their place is nothing (needed before the stores only)
    const int stopped = *reinterpret_cast<volatile int*>(a.status);
    const int tile = d.whole + t, qb = tile % a.nq, h = tile / a.nq, row = qb * BM + trow;
    int c = (int)((unsigned)x0 * (unsigned)d.ctas / (unsigned)d.line);        // the first CTA with a piece of the tile
    while (c > 0 && d.edge(c) > x0) --c;
    while (d.edge(c + 1) <= x0) ++c;
    const int next = d.edge(c + 1);
    if (next >= x1) return;                               // one CTA did the whole tile
    // pieces c, c + 1, ..: the first, which starts the tile, is in its CTA's second slot, the others are in the first
    const float* p = d.part + (size_t)(2 * c + 1) * PART_FLOATS;
    float M = -INFINITY, l = 0.f, r = 0.f;
    float4 o[N4];
#pragma unroll
    for (int i = 0; i < N4; ++i) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    bool more = true;
    while (more) {
        float mp[AT_ONCE], lp[AT_ONCE], rp[AT_ONCE];
        float4 v[AT_ONCE][N4];
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) {
            mp[u] = lp[u] = rp[u] = 0.f;
#pragma unroll
            for (int i = 0; i < N4; ++i) v[u][i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (more) {
                mp[u] = p[trow]; lp[u] = p[BM + trow]; rp[u] = p[2 * BM + trow];
                const float4* po = reinterpret_cast<const float4*>(p + PART_ROWS * BM) + (size_t)N4 * blockIdx.y * BM + trow;
#pragma unroll
                for (int i = 0; i < N4; ++i) v[u][i] = po[i * BM];
                ++c;
                p = d.part + (size_t)(2 * c) * PART_FLOATS;
                more = c < d.ctas && d.edge(c) < x1;
            }
        }
        float Mn = M;
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u)
            if (lp[u] != 0.f) Mn = fmaxf(Mn, mp[u]);      // a piece whose logits are all -inf has no maximum
        const float w0 = l != 0.f ? exp2f(M - Mn) : 0.f;
        l *= w0; r *= w0;
#pragma unroll
        for (int i = 0; i < N4; ++i) o[i] = make_float4(o[i].x * w0, o[i].y * w0, o[i].z * w0, o[i].w * w0);
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) {
            const float w = lp[u] != 0.f ? exp2f(mp[u] - Mn) : 0.f;
            l = fmaf(w, lp[u], l);
            r = fmaf(w, rp[u], r);
#pragma unroll
            for (int i = 0; i < N4; ++i)
                o[i] = make_float4(fmaf(w, v[u][i].x, o[i].x), fmaf(w, v[u][i].y, o[i].y), fmaf(w, v[u][i].z, o[i].z), fmaf(w, v[u][i].w, o[i].w));
        }
        M = Mn;
    }
    if (stopped != 0) return;
    if (M == -INFINITY) M = 0.f;
    const bool valid = row < a.L;
    if (blockIdx.y == 0) a.lse[(size_t)row * a.H + h] = valid ? M + log2f(l) : 1e30f;
    if (!valid) return;
    const float inv = 1.0f / r;
    uint4* dst = reinterpret_cast<uint4*>(a.out + ((size_t)row * a.H + h) * HD + MERGE_COLS * blockIdx.y);
#pragma unroll
    for (int i = 0; i < MERGE_COLS / 8; ++i)
        dst[i] = make_uint4(pack_bf16x2(o[2 * i].x * inv, o[2 * i].y * inv), pack_bf16x2(o[2 * i].z * inv, o[2 * i].w * inv),
                            pack_bf16x2(o[2 * i + 1].x * inv, o[2 * i + 1].y * inv),
                            pack_bf16x2(o[2 * i + 1].z * inv, o[2 * i + 1].w * inv));
}

// ---------------------------------------------------------------------------------------------- host side
// Representative tables (H, rows, 128) bf16 viewed as dims {128 d, rows, H}; a box is 64 d x 4 rows (one block's four rows).
static int make_rep_map(CUtensorMap* m, const void* ptr, int rows, int H) {
    cuuint64_t dims[3] = {(cuuint64_t)HD, (cuuint64_t)rows, (cuuint64_t)H};
    cuuint64_t strides[2] = {(cuuint64_t)HD * 2, (cuuint64_t)rows * HD * 2};
    cuuint32_t box[3] = {64, 4, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return encode_tensor_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                             CU_TENSOR_MAP_SWIZZLE_128B);
}

static int make_map(CUtensorMap* m, const void* ptr, int rows, int H, int box_rows) {
    // (rows, H, 128) bf16 viewed as dims {128 d, rows, H}; a box is 64 d x box_rows rows, 128-byte swizzled
    cuuint64_t dims[3] = {(cuuint64_t)HD, (cuuint64_t)rows, (cuuint64_t)H};
    cuuint64_t strides[2] = {(cuuint64_t)H * HD * 2, (cuuint64_t)HD * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return encode_tensor_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                             CU_TENSOR_MAP_SWIZZLE_128B);
}

struct AttnCall {
    const void *q, *k, *v, *k_mean, *v_mean;
    AttnArgs a;
    DenseSplit split;            // dense mode
    int sms;
};

// Times in iterations of a dense tile (1.17 us at 12 heads of 1,560 tokens): what a piece costs besides its own, and a merging
// launch where the cut tiles are fewer than a wave (3 us) and where they are one or two waves (7 us).
constexpr int PIECE_COST = 5, MERGE_FEW = 3, MERGE_MANY = 7;

// One wave of whole tiles after the other, or the tiles of the last wave cut into the same number of pieces each, or those of the
// last two waves cut without regard to their ends, so that a CTA works on two or three tiles: whichever these counts say is shortest.
static DenseSplit plan_dense(int tiles, int nb, int sms) {
    DenseSplit d{};
    d.n = (nb + 1) / 2;
    const int waves = tiles / sms, rest = tiles % sms;
    long long best = 19ll * (waves + (rest > 0)) * (d.n + PIECE_COST) / 20;       // cut only where that saves a twentieth
    if (rest == 0 || 2ll * sms * sms * d.n >= 1ll << 32) return d;
    const int pieces = std::min(sms / rest, d.n);
    if (pieces > 1) {
        const long long t = (long long)waves * (d.n + PIECE_COST) + (d.n + pieces - 1) / pieces + PIECE_COST + MERGE_FEW;
        if (t < best) {
            best = t;
            d.whole = waves * sms; d.line = rest * d.n; d.ctas = rest * pieces;
        }
    }
    const int lead = std::max(waves - 1, 0), cut = tiles - lead * sms, ctas = std::min(sms, cut * d.n);
    const long long t = (long long)lead * (d.n + PIECE_COST) + (cut * d.n + ctas - 1) / ctas + 2 * PIECE_COST + MERGE_MANY;
    if (t < best) { d.whole = lead * sms; d.line = cut * d.n; d.ctas = ctas; }
    return d;
}

static int launch_attention(const AttnCall& c, int mode, cudaStream_t stream) {
    const AttnArgs& a = c.a;
    if (a.L <= 0 || a.H <= 0) return set_error(-1, "attention: L and H must be positive");
    if (a.status == nullptr) return set_error(-2, "attention: the device status word is not available on this device");
    if (((uintptr_t)c.q | (uintptr_t)c.k | (uintptr_t)c.v | (uintptr_t)a.out) & 15)
        return set_error(-1, "attention: q, k, v, out must be 16-byte aligned");
    CUtensorMap tq, tk, tv, tkm, tvm, tkr, tvr;
    int rc;
    if ((rc = make_map(&tq, c.q, a.L, a.H, BK))) return rc;
    if ((rc = make_map(&tk, c.k, a.L, a.H, BK))) return rc;
    if ((rc = make_map(&tv, c.v, a.L, a.H, BK))) return rc;
    if (c.k_mean) {
        if ((rc = make_map(&tkm, c.k_mean, a.nb, a.H, BK))) return rc;
        if ((rc = make_map(&tvm, c.v_mean, a.nb, a.H, BK))) return rc;
    } else {
        tkm = tk; tvm = tv;
    }
    if (a.nref > 0) {
        if (((uintptr_t)a.k_rep | (uintptr_t)a.v_rep) & 15) return set_error(-1, "attention: k_rep, v_rep must be 16-byte aligned");
        if ((rc = make_rep_map(&tkr, a.k_rep, a.nb4, a.H))) return rc;
        if ((rc = make_rep_map(&tvr, a.v_rep, a.nb4, a.H))) return rc;
    } else {
        tkr = tk; tvr = tv;
    }
    if (mode == 3) {
        if ((rc = opt_in_shared_memory((const void*)dense_kernel, (int)SMEM_ALLOC))) return rc;
        const DenseSplit& d = c.split;
        dense_kernel<<<!d.part ? a.nq * a.H : d.whole ? c.sms : d.ctas, NTHREADS, SMEM_ALLOC, stream>>>(tq, tk, tv, a, d);
        cudaError_t e3 = cudaGetLastError();
        if (e3 != cudaSuccess) return set_error(-2, cudaGetErrorString(e3));
        count_launch();
        if (d.part) {
            if ((rc = prefer_shared_memory((const void*)dense_merge_kernel))) return rc;
            if ((e3 = launch_dependent(dense_merge_kernel, dim3(d.line / d.n, HD / MERGE_COLS), dim3(BM), 0, stream, a, d)) != cudaSuccess)
                return set_error(-2, cudaGetErrorString(e3));
            count_launch();
        }
        return 0;
    }
    auto kern = mode == 0 ? attention_kernel<0> : mode == 1 ? attention_kernel<1> : attention_kernel<2>;
    if ((rc = opt_in_shared_memory((const void*)kern, (int)SMEM_ALLOC))) return rc;
    int grid = a.nq * a.H;
    if (mode != 0 && a.walk) {
        int dev = 0, sms = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return set_error(-2, "attention: cannot read the SM count");
        grid = sms < grid ? sms : grid;
    }
    kern<<<grid, NTHREADS, SMEM_ALLOC, stream>>>(tq, tk, tv, tkm, tvm, tkr, tvr, a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(-2, cudaGetErrorString(e));
    count_launch();
    return 0;
}

static void fill_common(AttnArgs& a, int L, int H, float threshold) {
    a.L = L; a.H = H;
    a.nq = (L + BM - 1) / BM;
    a.nb = (L + BK - 1) / BK;
    a.scale_log2 = 1.4426950408889634f / sqrtf((float)HD);
    a.th = threshold;
    a.tail_valid = L - (a.nb - 1) * BK;
    a.tail_log2 = log2f((float)a.tail_valid);
    a.status = device_status_ptr();
}

static void fill_q(AttnCall& c) { c.a.q = static_cast<const __nv_bfloat16*>(c.q); }

}  // namespace es

using namespace es;

extern "C" int es_block_attention(const void* q, const void* k, const void* v, void* out, const int32_t* counts,
                                  const int32_t* blocks, int32_t nk, const float* offset, float* lse, int32_t* flags,
                                  float* mass, int32_t L, int32_t H, float threshold, void* stream) {
    if (!q || !k || !v || !out || !counts || !blocks || !offset || !lse || !flags)
        return set_error(-1, "es_block_attention: null pointer");
    AttnCall c{};
    c.q = q; c.k = k; c.v = v; c.k_mean = nullptr; c.v_mean = nullptr;
    fill_common(c.a, L, H, threshold);
    c.a.out = (__nv_bfloat16*)out; c.a.counts = counts; c.a.blocks = blocks; c.a.nk = nk;
    c.a.offset = offset; c.a.lse = lse; c.a.flags = flags; c.a.mass = mass;
    c.a.nvirt = 0; c.a.nref = 0;
    fill_q(c);
    return launch_attention(c, 0, (cudaStream_t)stream);
}

extern "C" int es_sparse_attention(const void* q, const void* k, const void* v, const void* k_mean, const void* v_mean,
                                   const int32_t* skip_bits, int32_t nw, void* out, const int32_t* counts,
                                   const int32_t* blocks, int32_t nk, const float* offset, float* lse, int32_t* flags,
                                   const int32_t* refine, int32_t rw, const void* k_rep, const void* v_rep,
                                   const float* log_counts, float* mass, int32_t L, int32_t H, float threshold,
                                   void* stream) {
    if (!q || !k || !v || !out || !counts || !blocks || !offset || !lse || !flags || !k_mean || !v_mean || !skip_bits)
        return set_error(-1, "es_sparse_attention: null pointer");
    AttnCall c{};
    c.q = q; c.k = k; c.v = v; c.k_mean = k_mean; c.v_mean = v_mean;
    fill_common(c.a, L, H, threshold);
    c.a.out = (__nv_bfloat16*)out; c.a.counts = counts; c.a.blocks = blocks; c.a.nk = nk;
    c.a.offset = offset; c.a.lse = lse; c.a.flags = flags; c.a.mass = mass;
    c.a.skip_bits = skip_bits; c.a.nw = nw;
    c.a.nvirt = (c.a.nb + 127) / 128;
    if (nw < 4 * c.a.nvirt) return set_error(-1, "es_sparse_attention: skip_bits needs 4 * ceil(nb / 128) words per tile");
    if (rw % 32 != 0) return set_error(-1, "es_sparse_attention: refine width must be a multiple of 32");
    if (rw > 0 && (!refine || !k_rep || !v_rep || !log_counts))
        return set_error(-1, "es_sparse_attention: refine list without representative tables");
    if (rw > 0 && !aligned(16, refine, log_counts)) return set_error(-1, "es_sparse_attention: refine and log_counts must be 16-byte aligned");
    c.a.refine = refine; c.a.rw = rw; c.a.nref = rw / 32;
    c.a.k_rep = (const __nv_bfloat16*)k_rep; c.a.v_rep = (const __nv_bfloat16*)v_rep; c.a.log_counts = log_counts;
    c.a.nb4 = (c.a.nb + 1) * 4;
    fill_q(c);
    return launch_attention(c, 0, (cudaStream_t)stream);
}

extern "C" int es_exact_fallback(const void* q, const void* k, const void* v, void* out, const int32_t* counts,
                                 const int32_t* blocks, int32_t nk, float* lse, const int32_t* flags, int32_t L,
                                 int32_t H, int32_t* tile_scratch, void* stream) {
    if (!q || !k || !v || !out || !counts || !blocks || !lse || !flags)
        return set_error(-1, "es_exact_fallback: null pointer");
    AttnCall c{};
    c.q = q; c.k = k; c.v = v; c.k_mean = nullptr; c.v_mean = nullptr;
    fill_common(c.a, L, H, 0.f);
    c.a.out = (__nv_bfloat16*)out; c.a.counts = counts; c.a.blocks = blocks; c.a.nk = nk;
    c.a.offset = lse; c.a.lse = lse; c.a.flags = const_cast<int32_t*>(flags); c.a.mass = nullptr;
    c.a.nvirt = 0; c.a.nref = 0;
    c.a.walk = tile_scratch != nullptr;
    fill_q(c);
    return launch_attention(c, 1, (cudaStream_t)stream);
}

extern "C" int es_compensate_fallback(const void* q, const void* k_mean, const void* v_mean, const uint8_t* keep,
                                      float* lse, void* out, const int32_t* flags, int32_t L, int32_t H,
                                      int32_t* tile_scratch, void* stream) {
    if (!q || !k_mean || !v_mean || !keep || !lse || !out || !flags)
        return set_error(-1, "es_compensate_fallback: null pointer");
    AttnCall c{};
    // no exact blocks in this pass: the K / V maps are only placeholders and point at the mean tables
    c.q = q; c.k = k_mean; c.v = v_mean; c.k_mean = k_mean; c.v_mean = v_mean;
    fill_common(c.a, L, H, 0.f);
    c.a.out = (__nv_bfloat16*)out; c.a.counts = nullptr; c.a.blocks = nullptr; c.a.nk = 0;
    c.a.offset = lse; c.a.lse = lse; c.a.flags = const_cast<int32_t*>(flags); c.a.mass = nullptr;
    c.a.keep = keep;
    c.a.nvirt = (c.a.nb + 127) / 128; c.a.nref = 0;
    c.a.walk = tile_scratch != nullptr;
    fill_q(c);
    return launch_attention(c, 2, (cudaStream_t)stream);
}

static int dense_sms(int* sms) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return set_error(-2, "es_dense_attention: cannot read the SM count");
    return 0;
}

extern "C" long long es_dense_scratch_bytes(int32_t L, int32_t H) {
    int sms = 0;
    if (L <= 0 || H <= 0 || dense_sms(&sms)) return 0;
    return 2ll * plan_dense((L + BM - 1) / BM * H, (L + BK - 1) / BK, sms).ctas * PART_FLOATS * (long long)sizeof(float);
}

static int dense_call(const char* who, const void* q, const void* k, const void* v, void* out, float* lse, void* scratch,
                      long long scratch_bytes, int32_t L, int32_t H, void* stream) {
    if (!q || !k || !v || !out || !lse) return set_error(-1, who);
    if (!aligned(16, scratch)) return set_error(-1, "es_dense_attention_split: scratch must be 16-byte aligned");
    AttnCall c{};
    c.q = q; c.k = k; c.v = v;
    fill_common(c.a, L, H, 0.f);
    c.a.out = (__nv_bfloat16*)out; c.a.lse = lse; c.a.v = (const __nv_bfloat16*)v;
    fill_q(c);
    c.split.n = (c.a.nb + 1) / 2;
    if (scratch && L > 0 && H > 0) {
        if (int rc = dense_sms(&c.sms)) return rc;
        const DenseSplit d = plan_dense(c.a.nq * H, c.a.nb, c.sms);
        if (2ll * d.ctas * PART_FLOATS * (long long)sizeof(float) > scratch_bytes)
            return set_error(-1, "es_dense_attention_split: scratch is smaller than es_dense_scratch_bytes says");
        if (d.ctas > 0) { c.split = d; c.split.part = static_cast<float*>(scratch); }
    }
    return launch_attention(c, 3, (cudaStream_t)stream);
}

extern "C" int es_dense_attention(const void* q, const void* k, const void* v, void* out, float* lse, int32_t L, int32_t H,
                                  void* stream) {
    return dense_call("es_dense_attention: null pointer", q, k, v, out, lse, nullptr, 0, L, H, stream);
}

extern "C" int es_dense_attention_split(const void* q, const void* k, const void* v, void* out, float* lse, void* scratch,
                                        int64_t scratch_bytes, int32_t L, int32_t H, void* stream) {
    return dense_call("es_dense_attention_split: null pointer", q, k, v, out, lse, scratch, scratch_bytes, L, H, stream);
}
