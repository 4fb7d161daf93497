// Sampled decoding on the device: LM head + per-group top-k with repeat penalty
// (map_matvec_topk_t_xq4[_ex]_dev: adamah-MAIN/adamah/adamah.c:9727-9832 and
// shaders/src/f32/map_matvec_topk_t_xq4.comp), and the decoder's own sampling step that keeps
// non-greedy generation on the GPU (role of the reference engine's fused top-k branch,
// adam/models/engine.py:3403-3512, and of its host-side rule `_sample`, :3711-3729).
//
// Design.  The logits of one LM-head product (1 MB at a 262144-row vocabulary) are written once by the
// dequant GEMV and stay in L2; selection then works on them in two short parallel stages instead of a
// serial insertion list per work group as in the shader:
//   stage 1  one CTA per group of rows keeps each thread's values in registers and extracts the group's k
//            best: every warp its own, then one warp merges the warps' lists (no barrier per candidate);
//   stage 2  (decoder only) one CTA per sequence merges the groups' sorted candidates: k rounds of a warp's arg-max
//            over the heads of the groups, which leaves the k best sorted; then soft-max with temperature,
//            nucleus cut and the draw run on one warp.
// Ties go to the lower row index everywhere (map_argmax.comp `better`), NaN counts as -FLT_MAX.
#include "common.cuh"
#include "gemv.cuh"
#include "token.cuh"

#include <cstdlib>

namespace ab {

int weight_ref(const Map* m, uint64_t off, uint64_t n_elems, int* wtype, WeightRef* w);
int run_gemv(uint32_t map_id, uint64_t off, int wtype, GemvArgs& ga);
void launch_gemv_q4map(const float* x, const Map* w, uint64_t w_off, float* y, uint32_t K, uint32_t N);

constexpr float SNEG = -3.402823466e+38f;
constexpr int SEL_T = 256;                 // threads of a selection CTA
constexpr int SEL_V = 8;                   // values a thread keeps in registers (a group has at most SEL_T * SEL_V rows)
constexpr uint32_t TOPK_MAX = 64;

// A value as an unsigned number in the order of `better` (both zeros are one number; nothing is 0).
__device__ __forceinline__ uint32_t rank_of(float v) {
    const uint32_t u = __float_as_uint(v + 0.0f);
    return u & 0x80000000u ? ~u : u | 0x80000000u;
}
// The warp's best of (rank, row), ties to the lower row; rank 0: there is none.  True on the lane that holds it.
__device__ __forceinline__ bool warp_best(uint32_t o, uint32_t row, uint32_t& best, uint32_t& best_row) {
    best = __reduce_max_sync(0xffffffffu, o);
    best_row = __reduce_min_sync(0xffffffffu, o == best ? row : 0xffffffffu);
    return best != 0u && o == best && row == best_row;
}

// The k best of this CTA's values, sorted: thread t holds values val[j] of rows key[j], ascending with j (key < 0 = empty slot).
// Every warp sorts out its own k best (a round is two warp reductions and, on the winner's lane, a look at its eight values; no
// barrier), then one warp merges the warps' lists the same way.  As k rounds of an arg-max over the CTA it took 1 us per round.
struct TopkLists { float v[SEL_T / 32][TOPK_MAX]; int i[SEL_T / 32][TOPK_MAX]; };
__device__ __forceinline__ void block_topk(float (&val)[SEL_V], int (&key)[SEL_V], uint32_t k, float* out_v, int* out_i, TopkLists& l) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t rank[SEL_V];
#pragma unroll
    for (int j = 0; j < SEL_V; ++j) rank[j] = key[j] >= 0 ? rank_of(val[j]) : 0u;
    uint32_t o = 0u, best, row;
    int at = 0;
    auto look = [&]() {
        o = 0u;
#pragma unroll
        for (int j = 0; j < SEL_V; ++j) if (rank[j] > o) { o = rank[j]; at = key[j]; }
    };
    look();
    for (uint32_t r = 0; r < k; ++r) {
        const bool mine = warp_best(o, (uint32_t)at, best, row);
        if (mine) {
            float v = 0.f;
#pragma unroll
            for (int j = 0; j < SEL_V; ++j) if (key[j] == at) { v = val[j]; rank[j] = 0u; }
            l.v[warp][r] = v; l.i[warp][r] = at;
            look();
        }
        if (best == 0u && lane == 0) { l.v[warp][r] = SNEG; l.i[warp][r] = -1; }
    }
    __syncthreads();
    if (warp == 0) {
        uint32_t next = 0;
        auto head = [&]() {
            const bool in = lane < SEL_T / 32 && next < k && l.i[lane][next] >= 0;
            o = in ? rank_of(l.v[lane][next]) : 0u;
            at = in ? l.i[lane][next] : 0;
        };
        head();
        for (uint32_t r = 0; r < k; ++r) {
            const bool mine = warp_best(o, (uint32_t)at, best, row);
            if (mine) { out_v[r] = l.v[lane][next]; out_i[r] = at; ++next; head(); }
            if (best == 0u && lane == 0) { out_v[r] = SNEG; out_i[r] = -1; }
        }
    }
    __syncthreads();
}

__device__ __forceinline__ float penalised(float v, int row, const uint32_t* __restrict__ pen, uint32_t n_pen, float penalty) {
    if (!(v == v)) v = SNEG;
    for (uint32_t i = 0; i < n_pen; ++i)
        if (pen[i] == (uint32_t)row) return v > 0.f ? __fdiv_rn(v, penalty) : v * penalty;
    return v;
}

// Stage 1.  Group g = rows [g * rpg, min(N, (g + 1) * rpg)); candidates land at cand_v / cand_i [g * k + r]
// (decoder) or, through locs, in the activation map with the row index stored as float32 (operator).
__global__ void __launch_bounds__(SEL_T) k_group_topk(const float* __restrict__ logits, uint32_t N, uint32_t rpg, uint32_t k,
                                                      const uint32_t* __restrict__ pen, uint32_t n_pen, float penalty,
                                                      float* __restrict__ cand_v, int* __restrict__ cand_i,
                                                      float* __restrict__ map, uint64_t n_el, const uint32_t* __restrict__ li,
                                                      const uint32_t* __restrict__ lv, uint32_t* err) {
    __shared__ TopkLists lists;
    __shared__ float out_v[TOPK_MAX]; __shared__ int out_i[TOPK_MAX];
    const uint32_t g = blockIdx.x, r0 = g * rpg, r1 = min(N, r0 + rpg);
    float val[SEL_V]; int key[SEL_V];
#pragma unroll
    for (int j = 0; j < SEL_V; ++j) {
        const uint32_t row = r0 + threadIdx.x + j * SEL_T;
        key[j] = row < r1 ? (int)row : -1;
        val[j] = row < r1 ? penalised(logits[row], (int)row, pen, n_pen, penalty) : SNEG;
    }
    block_topk(val, key, k, out_v, out_i, lists);
    if (threadIdx.x < k) {
        const uint32_t o = g * k + threadIdx.x;
        if (map) {
            const uint64_t di = li[o], dv = lv[o];
            if (di >= n_el || dv >= n_el) atomicOr(err, DEVERR_OOB_MAP);
            else { map[di] = (float)(out_i[threadIdx.x] < 0 ? 0 : out_i[threadIdx.x]); map[dv] = out_v[threadIdx.x]; }
        } else { cand_v[o] = out_v[threadIdx.x]; cand_i[o] = out_i[threadIdx.x]; }
    }
}

// ---- decoder sampling step ------------------------------------------------------------------------------
// uniform in [0, 1) from (seed, sequence, position): splitmix64 of the three, top 24 bits
__host__ __device__ inline float sample_uniform(uint64_t seed, uint32_t seq, uint32_t pos) {
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * (((uint64_t)seq << 32 | pos) + 1ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z = z ^ (z >> 31);
    return (float)(z >> 40) * (1.0f / 16777216.0f);
}

// The ids whose logits get the repeat penalty: the tokens among the last 64 of the history (prompt included with on_prompt, else
// generated tokens only), as the reference's `set(prev[-64:])` (engine.py:3713): a thread each, an id may stand there twice.
// Position q of sequence b holds prompt_tok[q] for q < prompt_len and the logged sample otherwise.
__device__ __forceinline__ uint32_t history_ids(const int32_t* prompt_tok, const int32_t* gen_log, int32_t plen, int32_t pos_new,
                                                int on_prompt, uint32_t* ids) {
    const int32_t lo = max(on_prompt ? 0 : plen, pos_new - 64), q = lo + (int32_t)threadIdx.x;
    if (q < pos_new) ids[threadIdx.x] = (uint32_t)(q < plen ? prompt_tok[q] : gen_log[q]);      // none: negative, no row's number
    return (uint32_t)max(pos_new - lo, 0);
}

// Stage 1 for the decoder: grid (groups, batch); every CTA reads the history for itself.
__global__ void __launch_bounds__(SEL_T) k_sample_stage1(const float* __restrict__ logits, uint32_t V, uint32_t k,
                                                         const int32_t* __restrict__ pos, const int32_t* __restrict__ prompt_len,
                                                         const int32_t* __restrict__ prompt_tok, const int32_t* __restrict__ gen_log, uint32_t ld,
                                                         float penalty, int on_prompt, float* __restrict__ cand_v, int* __restrict__ cand_i) {
    __shared__ TopkLists lists;
    __shared__ float out_v[TOPK_MAX]; __shared__ int out_i[TOPK_MAX];
    __shared__ uint32_t s_pen[64];
    const uint32_t g = blockIdx.x, b = blockIdx.y, groups = gridDim.x;
    const uint32_t n_pen = penalty != 1.0f ? history_ids(prompt_tok + (size_t)b * ld, gen_log + (size_t)b * ld, prompt_len[b], pos[b], on_prompt, s_pen) : 0u;
    const float* lg = logits + (size_t)b * V;
    const uint32_t rpg = SEL_T * SEL_V, r0 = g * rpg, r1 = min(V, r0 + rpg);
    float val[SEL_V]; int key[SEL_V];
#pragma unroll
    for (int j = 0; j < SEL_V; ++j) {
        const uint32_t row = r0 + threadIdx.x + j * SEL_T;
        key[j] = row < r1 ? (int)row : -1;
        val[j] = row < r1 ? lg[row] : SNEG;
        if (!(val[j] == val[j])) val[j] = SNEG;
    }
    __syncthreads();
    uint32_t seen = 0;                                  // this thread's values that have had their penalty
    for (uint32_t i = 0; i < n_pen; ++i) {
        const uint32_t d = s_pen[i] - r0;
        if (d < rpg && (d & (SEL_T - 1)) == threadIdx.x) {
#pragma unroll
            for (int j = 0; j < SEL_V; ++j)
                if ((d / SEL_T) == (uint32_t)j && !(seen >> j & 1u)) { seen |= 1u << j; val[j] = val[j] > 0.f ? __fdiv_rn(val[j], penalty) : val[j] * penalty; }
        }
    }
    block_topk(val, key, k, out_v, out_i, lists);
    if (threadIdx.x < k) {
        const size_t o = ((size_t)b * groups + g) * k + threadIdx.x;
        cand_v[o] = out_v[threadIdx.x]; cand_i[o] = out_i[threadIdx.x];
    }
}

// Stage 2: one CTA per sequence.  The k best of all groups' candidates (`groups` lists of k, each sorted, copied to shared
// memory where they fit), then on warp 0:
// p_i = exp((l_i - l_0) / T) / sum, nucleus = the shortest prefix whose probability reaches top_p
// (np.searchsorted(cumsum, top_p) + 1, engine.py:3724-3726), renormalise, inverse-CDF draw with the uniform u.
// temperature <= 0 takes the best candidate (engine.py:3719).  Writes the token where the next step reads it and
// into the log at the sequence's (already advanced) position.
__global__ void __launch_bounds__(SEL_T) k_sample_stage2(const float* __restrict__ cand_v, const int* __restrict__ cand_i, uint32_t groups, uint32_t k, int in_shared,
                                                         float temperature, float top_p, uint64_t seed,
                                                         const int32_t* __restrict__ pos, int32_t* __restrict__ cur_tok, float* __restrict__ cur_val,
                                                         int32_t* __restrict__ gen_log, uint32_t ld, uint2* __restrict__ far_heads, float* __restrict__ dbg) {
    __shared__ float out_v[TOPK_MAX]; __shared__ int out_i[TOPK_MAX];
    const uint32_t b = blockIdx.x;
    const uint32_t n_cand = groups * k;
    const float* cv = cand_v + (size_t)b * n_cand;
    const int* ci = cand_i + (size_t)b * n_cand;
    extern __shared__ unsigned char sel_sm[];
    // [groups] the rank and row of a group's head (in `far_heads` where there are too many), [groups] candidates of it that are taken;
    // then the candidates
    uint2* hd = far_heads ? far_heads + (size_t)b * groups : reinterpret_cast<uint2*>(sel_sm);
    unsigned char* head = sel_sm + (far_heads ? 0 : (size_t)groups * 8);
    if (in_shared) {
        float* v = reinterpret_cast<float*>(sel_sm + (((size_t)groups * 9 + 15) & ~(size_t)15));
        int* i = reinterpret_cast<int*>(v + n_cand);
#pragma unroll 8
        for (uint32_t c = threadIdx.x; c < n_cand; c += SEL_T) { v[c] = cv[c]; i[c] = ci[c]; }
        cv = v; ci = i;
        __syncthreads();
    }
    auto head_of = [&](uint32_t q, uint32_t taken) {
        const uint32_t c = q * k + taken;
        return taken < k && ci[c] >= 0 ? make_uint2(rank_of(cv[c]), (uint32_t)ci[c]) : make_uint2(0u, 0u);
    };
    for (uint32_t q = threadIdx.x; q < groups; q += SEL_T) { head[q] = 0; hd[q] = head_of(q, 0u); }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const uint32_t lane = threadIdx.x;
    // one warp: a lane's groups by their heads
    uint32_t o = 0u, at = 0u, mg = 0u, best, row;
    auto look = [&]() {
        o = 0u;
#pragma unroll 4
        for (uint32_t q = lane; q < groups; q += 32) {
            const uint2 h = hd[q];
            if (h.x > o || (h.x == o && h.y < at)) { o = h.x; at = h.y; mg = q; }
        }
    };
    look();
    for (uint32_t r = 0; r < k; ++r) {
        if (warp_best(o, at, best, row)) {
            out_v[r] = cv[mg * k + head[mg]]; out_i[r] = (int)at;
            hd[mg] = head_of(mg, ++head[mg]);
            look();
        }
        if (best == 0u && lane == 0) { out_v[r] = SNEG; out_i[r] = -1; }
    }
    __syncwarp();
    uint32_t n = 0;
    for (uint32_t r = 0; r < k; ++r) if (out_i[r] >= 0) n = r + 1;
    int chosen = 0;
    if (n > 1 && temperature > 0.f) {
        // two candidates per lane; every sum in candidate order, as a sequential cumulative sum
        __shared__ float s_p[TOPK_MAX], s_q[TOPK_MAX];
        const float l0 = out_v[0];
#pragma unroll
        for (int h = 0; h < 2; ++h) { const uint32_t r = lane + 32 * h; s_p[r] = r < n ? expf(__fdiv_rn(out_v[r] - l0, temperature)) : 0.f; }
        __syncwarp();
        float sum = 0.f;
#pragma unroll 8
        for (uint32_t r = 0; r < n; ++r) sum += s_p[r];
        uint32_t keep = n;
        if (top_p < 1.0f) {
#pragma unroll
            for (int h = 0; h < 2; ++h) { const uint32_t r = lane + 32 * h; s_q[r] = __fdiv_rn(s_p[r], sum); }
            __syncwarp();
            float cs = 0.f;
            for (uint32_t r = 0; r < n; ++r) {
                cs += s_q[r];
                if (cs >= top_p) { keep = r + 1; break; }
            }
        }
        float ks = 0.f;
#pragma unroll 8
        for (uint32_t r = 0; r < keep; ++r) ks += s_p[r];
        const float u = sample_uniform(seed, b, (uint32_t)pos[b]);
        const float target = u * ks;
        float acc = 0.f;
        chosen = (int)keep - 1;
        for (uint32_t r = 0; r < keep; ++r) {
            acc += s_p[r];
            if (target < acc) { chosen = (int)r; break; }
        }
        if (dbg && lane == 0) { dbg[b * 4] = (float)keep; dbg[b * 4 + 1] = u; dbg[b * 4 + 2] = sum; dbg[b * 4 + 3] = (float)n; }
    }
    if (lane == 0) {
        const int tok = out_i[chosen] < 0 ? 0 : out_i[chosen];
        cur_tok[b] = tok;
        cur_val[b] = out_v[chosen];
        const int32_t q = pos[b];
        if ((uint32_t)q < ld) gen_log[(size_t)b * ld + q] = tok;
    }
}

static float* s_cand_v = nullptr; static int* s_cand_i = nullptr; static size_t s_cand_n = 0;
static uint2* s_heads = nullptr; static size_t s_heads_n = 0;

// Enqueue the sampling step for `batch` sequences whose soft-capped logits lie at logits[b * V .. ) and whose
// positions were already advanced.  k = 1..64.
int launch_sample(const float* logits, uint32_t V, uint32_t batch, uint32_t k, float temperature, float top_p, float penalty, int on_prompt,
                  uint64_t seed, const int32_t* pos, const int32_t* prompt_len, const int32_t* prompt_tok, int32_t* gen_log, uint32_t ld,
                  int32_t* cur_tok, float* cur_val) {
    if (k == 0 || k > TOPK_MAX) return fail(ADAMAH_ERR_INVALID, "sampling: top_k must be 1..64 on the device");
    const uint32_t groups = (V + SEL_T * SEL_V - 1) / (SEL_T * SEL_V);
    // Heads, candidates taken and the candidates in shared memory where they fit (82 KB at a vocabulary of 262144 and k = 64); the heads
    // alone as far as 37 million rows, beyond which they are in global memory, too.
    constexpr size_t LIMIT = 160 * 1024;
    const size_t near = ((size_t)groups * 9 + 15) & ~(size_t)15, all = near + (size_t)groups * k * 8;
    const bool in_shared = all <= LIMIT, far = near > LIMIT;
    const size_t need = (size_t)batch * groups * k, need_heads = far ? (size_t)batch * groups : 0;
    if (s_cand_n < need || s_heads_n < need_heads) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(g.stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
            return fail(ADAMAH_ERR_INVALID, "sampling: the first sampled step must run outside a graph capture");
        cudaStreamSynchronize(g.stream);
        if (s_cand_n < need) {
            cudaFree(s_cand_v); cudaFree(s_cand_i); s_cand_v = nullptr; s_cand_i = nullptr; s_cand_n = 0;
            if (cudaMalloc((void**)&s_cand_v, need * 4) != cudaSuccess || cudaMalloc((void**)&s_cand_i, need * 4) != cudaSuccess) {
                cudaGetLastError();
                return fail(ADAMAH_ERR_MEMORY, "sampling: out of device memory");
            }
            s_cand_n = need;
        }
        if (s_heads_n < need_heads) {
            cudaFree(s_heads); s_heads = nullptr; s_heads_n = 0;
            if (cudaMalloc((void**)&s_heads, need_heads * sizeof(uint2)) != cudaSuccess) { cudaGetLastError(); return fail(ADAMAH_ERR_MEMORY, "sampling: out of device memory"); }
            s_heads_n = need_heads;
        }
    }
    k_sample_stage1<<<dim3(groups, batch), SEL_T, 0, g.stream>>>(logits, V, k, pos, prompt_len, prompt_tok, gen_log, ld, penalty, on_prompt, s_cand_v, s_cand_i);
    if (cudaFuncSetAttribute(k_sample_stage2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LIMIT) != cudaSuccess)
        return fail(ADAMAH_ERR_BACKEND, "sampling: cannot raise the shared-memory limit");
    k_sample_stage2<<<batch, SEL_T, in_shared ? all : far ? (size_t)groups : near, g.stream>>>(s_cand_v, s_cand_i, groups, k, in_shared ? 1 : 0, temperature, top_p, seed, pos, cur_tok, cur_val, gen_log, ld,
                                                                                              far ? s_heads : nullptr, nullptr);
    count_launch(2);
    return check_launch("decoder sampling");
}

static float* s_logits = nullptr; static size_t s_logits_n = 0;
int logits_scratch(size_t n, float** out) {
    if (s_logits_n < n) {
        if (s_logits) { cudaStreamSynchronize(g.stream); cudaFree(s_logits); s_logits = nullptr; s_logits_n = 0; }
        if (cudaMalloc((void**)&s_logits, n * 4) != cudaSuccess) { cudaGetLastError(); return fail(ADAMAH_ERR_MEMORY, "out of device memory for %zu logits", n); }
        s_logits_n = n;
    }
    *out = s_logits;
    return ADAMAH_OK;
}
void sample_free_all() {
    cudaFree(s_logits); s_logits = nullptr; s_logits_n = 0;
    cudaFree(s_cand_v); cudaFree(s_cand_i); cudaFree(s_heads);
    s_cand_v = nullptr; s_cand_i = nullptr; s_heads = nullptr; s_cand_n = s_heads_n = 0;
}

}  // namespace ab

using namespace ab;

// Reference signature and results (adamah.c:9727-9822): for every group of rows_per_group rows of W the k
// largest of W[n,:] . x after the repeat penalty, as (row index as float32, value) pairs stored at
// locs_idx_dst / locs_val_dst [group * k + r] of the activation map; unfilled entries are (0, -FLT_MAX).
// W may be a Q4 map (the reference's storage) or a GGUF-block map.
extern "C" int map_matvec_topk_t_xq4_ex_dev(uint32_t map_act, uint32_t map_wt, uint32_t a_h, uint32_t b_h, uint32_t penalty_ids_h,
                                            uint32_t idx_dst_h, uint32_t val_dst_h, uint32_t K, uint32_t N, uint32_t k,
                                            uint32_t n_penalty, float repeat_penalty, uint32_t rows_per_group) {
    if (!ready()) return ADAMAH_ERR_INVALID;
    Map* a = get_map(map_act);
    Map* w = get_map(map_wt);
    if (!a || !w) return ADAMAH_ERR_NOT_FOUND;
    if (a->dtype != ADAMAH_DTYPE_F32 || a->pack_size != 1) return fail(ADAMAH_ERR_INVALID, "matvec_topk: map %u must be float32 with pack_size 1", map_act);
    if (N == 0 || k == 0) return ADAMAH_OK;                                  // adamah.c:9737
    if (k > TOPK_MAX || n_penalty > 64) return fail(ADAMAH_ERR_INVALID, "matvec_topk: k and n_penalty are limited to 64");
    if (rows_per_group == 0 || !K) return fail(ADAMAH_ERR_INVALID, "matvec_topk: rows_per_group and K must not be 0");
    if (rows_per_group > (uint32_t)(SEL_T * SEL_V)) return fail(ADAMAH_ERR_INVALID, "matvec_topk: rows_per_group is limited to %d", SEL_T * SEL_V);
    const uint32_t groups = (N + rows_per_group - 1) / rows_per_group;
    if (!handle_ok(idx_dst_h, groups * k * 4) || !handle_ok(val_dst_h, groups * k * 4) || !handle_ok(penalty_ids_h, n_penalty * 4)) return ADAMAH_ERR_NOT_FOUND;
    uint32_t ab_, bb;
    if (!hfirst(a_h, &ab_) || !hfirst(b_h, &bb)) return ADAMAH_ERR_NOT_FOUND;
    if ((uint64_t)ab_ + K > a->n_elems) return fail(ADAMAH_ERR_INVALID, "matvec_topk: activation range beyond map %u", map_act);
    float* lg = nullptr;
    int rc = logits_scratch(N, &lg);
    if (rc) return rc;
    const float* x = (const float*)a->buf + ab_;
    if (w->dtype == ADAMAH_DTYPE_Q4) {
        if ((uint64_t)bb + (uint64_t)N * K > w->n_elems) return fail(ADAMAH_ERR_INVALID, "matvec_topk: weight range beyond map %u", map_wt);
        launch_gemv_q4map(x, w, bb, lg, K, N);
    } else {
        int wtype; GemvArgs ga = {};
        if ((rc = weight_ref(w, bb, (uint64_t)N * K, &wtype, &ga.w0))) return rc;
        if (ab_ % 4 || K % 4) return fail(ADAMAH_ERR_INVALID, "matvec_topk: activation offset must be a multiple of 4 elements");
        ga.x = x; ga.ldx = (int)K; ga.y = lg; ga.ldy = (int)N; ga.N = (int)N; ga.K = (int)K; ga.B = 1; ga.epi = EPI_STORE;
        if ((rc = run_gemv(map_wt, bb, wtype, ga))) return rc;
    }
    k_group_topk<<<groups, SEL_T, 0, g.stream>>>(lg, N, rows_per_group, k, hlocs(penalty_ids_h), n_penalty, repeat_penalty, nullptr, nullptr,
                                                 (float*)a->buf, a->n_elems, hlocs(idx_dst_h), hlocs(val_dst_h), g.dev_err);
    count_launch();
    rc = check_launch("map_matvec_topk_t_xq4");
    end_of_op();
    return rc;
}

extern "C" int map_matvec_topk_t_xq4_dev(uint32_t map_act, uint32_t map_wt, uint32_t a_h, uint32_t b_h, uint32_t penalty_ids_h,
                                         uint32_t idx_dst_h, uint32_t val_dst_h, uint32_t K, uint32_t N, uint32_t k,
                                         uint32_t n_penalty, float repeat_penalty) {
    return map_matvec_topk_t_xq4_ex_dev(map_act, map_wt, a_h, b_h, penalty_ids_h, idx_dst_h, val_dst_h, K, N, k, n_penalty, repeat_penalty, 256);
}
