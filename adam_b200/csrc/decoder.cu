// Fused decoder: one decoded token for a batch of sequences as a fixed sequence
// of kernels (captured once into a CUDA graph and replayed), with positions and
// token ids living in device memory so that consecutive tokens need no host work.
//
// It computes what the reference engine's per-token loop computes
// (adam/models/engine.py:2971-3706 `_forward`: embed, per layer RMSNorm -> QKV ->
// QK-norm + RoPE -> KV append -> attention -> o-proj -> post-norm + residual ->
// RMSNorm -> gate/up -> GeGLU -> down -> post-norm + residual, final norm, LM head
// + arg-max), with the arithmetic of the reference's numpy decoder
// (tests/diagnostics/diag_inference.py:973-1037).  Differences from the reference
// runtime, all additive: B independent sequences per step, a paged KV cache in
// fp16 or fp32, an optional sliding-window mask on non-global layers, rotary angles
// read from a table the host supplies, chunked prefill (many prompt positions per
// pass), prefix reuse, and a part-wise step for tensor-parallel callers.
#include "common.cuh"
#include "gemv.cuh"
#include "gemv_mma.cuh"
#include "gemm_tc.cuh"
#include "token.cuh"
#include "blocks8.cuh"
#include "attn_prefill.cuh"

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

namespace ab {

int weight_ref(const Map* m, uint64_t off, uint64_t n_elems, int* wtype, WeightRef* w);
int argmax_scratch(float** pv, int** pi, unsigned int** tk);
int launch_sample(const float* logits, uint32_t V, uint32_t batch, uint32_t k, float temperature, float top_p, float penalty, int on_prompt,
                  uint64_t seed, const int32_t* pos, const int32_t* prompt_len, const int32_t* prompt_tok, int32_t* gen_log, uint32_t ld,
                  int32_t* cur_tok, float* cur_val);
bool capturing();

enum { MAT_Q = 0, MAT_K, MAT_V, MAT_O, MAT_GATE, MAT_UP, MAT_DOWN, MAT_EMBD, MAT_OUTPUT, MAT_KINDS };
enum { NORM_ATTN = 0, NORM_POST_ATTN, NORM_FFN, NORM_POST_FFW, NORM_Q, NORM_K, NORM_OUTPUT, NORM_KINDS };

struct Mat { bool bound; int wtype; WeightRef w; uint32_t rows, cols; uint32_t map_id; uint64_t elem_off; const uint8_t* tiled; };

struct Layer {
    Mat m[7];
    const float* norm[6];       // NORM_ATTN .. NORM_K (NULL = absent)
    bool qkv_contiguous, gateup_pairable;
    const uint8_t* qkv_tiled;   // row-tiled copy of the q,k,v rows as one tensor
};

// One pass of prefill: rows (sequence, position) of the plan and the attention tiles they are cut into.
struct PrefillChunk { uint32_t n_rows, n_tiles, tile_rows; const int32_t *row_seq, *row_pos; const AttnTile* tiles; };

struct Decoder {
    bool used;
    adam_b200_decoder_desc d;
    std::vector<Layer> layers;
    Mat embd, output;
    const float* output_norm;
    float* rope_cos[2]; float* rope_sin[2]; uint32_t rope_pos[2];
    // device state
    int32_t* pos;  int32_t* cur_tok;  float* cur_val;  int32_t* prompt_len;  int32_t* prompt_tok;  int32_t* gen_log;
    int32_t* block_table; uint32_t max_pages_per_seq, n_pages;
    void* kv_pool; size_t page_elems;
    float *hbuf[2], *qkv, *attn_out, *proj, *act, *logits; int h_final;
    float *part_o, *part_ml; unsigned int* attn_ticket; uint32_t n_splits;
    // chunked prefill: what the rows of all chunks are (device copy and pinned source of one call; see PrefillPlan)
    uint8_t *plan, *plan_pin; size_t plan_cap; cudaEvent_t plan_read;
    std::vector<PrefillChunk> chunks; const int32_t* plan_n; std::vector<int32_t> plan_pos;     // chunks of a call, its tokens and first positions
    int32_t* even_plan;         // the plan of a chunk with the same number of tokens for all, made on the device: row_seq, row_pos, tiles
    bool pos_shared;            // positions may move without the host's doing: recorded graphs, a caller that has their address
    // adam_b200_decoder_score: two groups of score_rows rows of logits (NULL: none fit, D->logits takes one at a time), the
    // winners of a group, and the copies to the host
    float* score_logits; int32_t* score_tok; uint32_t score_rows; cudaEvent_t score_ev[4]; cudaStream_t score_copy;
    uint32_t rows_cap;          // rows the activation buffers hold
    std::vector<uint32_t> hpos, hplen, hres;   // host mirror of positions, prompt lengths and reserved tokens (argument checks)
    std::vector<int32_t> hbt;            // host mirror of the block table
    int32_t* tok_ring[4]; cudaEvent_t tok_event[4]; uint32_t tok_next;   // pinned slots for asynchronous token reads
    uint32_t batch;             // active sequences
    bool use_tiles;             // build row-tiled weight copies for the tensor-core GEMV
    // device-side sampling (adam_b200_decoder_set_sampling; used by steps with flag bit4)
    uint32_t smp_k; float smp_temp, smp_top_p, smp_penalty; int smp_on_prompt; uint64_t smp_seed;
    std::vector<uint32_t> free_pages;
    cudaGraphExec_t graph[2]; cudaGraph_t graph_src[2]; uint32_t graph_batch[2]; uint64_t graph_kernels[2];
    // single-launch token kernel (token.cuh): 0 = not examined yet, 1 = ready, -1 = this model does not qualify
    int tk_state; TkArgs tk; int tk_grid; int tk_wt; void* tk_mem[9];
    cudaGraphExec_t tk_graph[2]; cudaGraph_t tk_graph_src[2]; int tk_graph_state[2];   // TK_GRAPH_N token kernels per replay (index = LM head or not); state -1 = capture refused
};

constexpr uint32_t MAX_DECODERS = 8;
constexpr uint32_t ATTN_SPLIT = 64;        // fewest tokens an attention CTA takes before another CTA is added
constexpr uint32_t ATTN_MAX_SPLITS = 64;   // attention CTAs per (sequence, kv head)
// Rows (sequences x tokens) of one prefill chunk: 1024, or 2048 where the tiles of an n_embd-wide product (128 x 128) do not
// give every SM one at 1024.  Prompts and one step, ms with 1024 and with 2048 rows: 1B shape (n_embd 1152, 72 tiles at 1024)
// 32 prompts x 512 105.4 and 90.8, 8 x 160 12.5 and 8.7, one of 1500 tokens 13.5 and 10.6; 27B shape (8 layers, 336 tiles)
// 64 x 128 175.6 and 178.0, 16 x 128 45.0 and 45.8, 4 x 900 83.8 and 86.9, one of 900 tokens 22.2 and 22.2.
static uint32_t prefill_rows(uint32_t n_embd) { return (uint64_t)((n_embd + 127) / 128) * (1024 / 128) < (uint64_t)g.sm_count ? 2048u : 1024u; }
static Decoder* g_dec[MAX_DECODERS];

static Decoder* get_dec(uint32_t id) {
    if (!ready()) return nullptr;
    if (id >= MAX_DECODERS || !g_dec[id]) { fail(ADAMAH_ERR_NOT_FOUND, "decoder %u does not exist", id); return nullptr; }
    return g_dec[id];
}

// ---- kernels ---------------------------------------------------------------
#ifdef ADAM_B200_STEP_TRACE
// step trace: [4 products][8 CTAs][8 stamps] then [32 attention CTAs][8 stamps] of layer g_step_trace_layer
static long long* g_step_trace = nullptr; static uint32_t g_step_trace_layer = 0; static int g_step_trace_slot = -1;
#endif

// h[b] = dequant(token_embd[row tok]) * emb_scale   (diag_inference.py:975-977)
template <int WT>
__global__ void k_embed(const WeightRef w, uint32_t n_embd, uint32_t n_vocab, float emb_scale,
                        const int32_t* __restrict__ pos, const int32_t* __restrict__ prompt_len, const int32_t* __restrict__ prompt_tok,
                        uint32_t prompt_ld, const int32_t* __restrict__ cur_tok, float* __restrict__ h,
                        const int32_t* __restrict__ row_seq, const int32_t* __restrict__ row_pos, uint32_t* err) {
    pdl_launch_dependents();
    pdl_wait();
    // decode: row = sequence at its own position; prefill: row r = (sequence row_seq[r], position row_pos[r])
    const uint32_t r = blockIdx.x;
    const uint32_t b = row_seq ? (uint32_t)row_seq[r] : r;
    const int32_t p = row_pos ? row_pos[r] : pos[b];
    int32_t tok = (p < prompt_len[b]) ? prompt_tok[(size_t)b * prompt_ld + p] : cur_tok[b];
    if (tok < 0 || (uint32_t)tok >= n_vocab) { if (threadIdx.x == 0) atomicOr(err, DEVERR_BAD_TOKEN); tok = 0; }
    float* out = h + (size_t)r * n_embd;
    if (WT == WT_Q8_0 || WT == WT_Q5_0) {
        // code * fp16 scale is exact in float32; the embedding multiplier rounds once (map_row_gather_xq8.comp)
        const size_t b0 = (size_t)tok * (n_embd / 32);
        for (uint32_t i = threadIdx.x; i < n_embd; i += blockDim.x) {
            const size_t blk = b0 + (i >> 5);
            const uint32_t j = i & 31;
            int q;
            if (WT == WT_Q8_0) q = (int)reinterpret_cast<const int8_t*>(w.q)[blk * 32 + j];
            else {
                const uint32_t byte = reinterpret_cast<const uint8_t*>(w.q)[blk * 16 + (j & 15)];
                q = (int)((j < 16 ? (byte & 15u) : (byte >> 4)) | (((w.h[blk] >> j) & 1u) << 4)) - 16;
            }
            out[i] = __fmul_rn(__fmul_rn((float)q, __half2float(w.d[blk])), emb_scale);
        }
    } else if (WT == WT_Q4_0) {
        const uint32_t nblk = n_embd / 32;
        const uint8_t* q = reinterpret_cast<const uint8_t*>(w.q + (size_t)tok * nblk);
        const __half* d = w.d + (size_t)tok * nblk;
        for (uint32_t i = threadIdx.x; i < nblk * 16; i += blockDim.x) {
            const uint32_t blk = i >> 4, j = i & 15;
            const float s = __half2float(d[blk]);
            const uint32_t byte = q[blk * 16 + j];
            out[blk * 32 + j]      = __fmul_rn(__fmul_rn((float)(int)(byte & 15) - 8.f, s), emb_scale);
            out[blk * 32 + 16 + j] = __fmul_rn(__fmul_rn((float)(int)(byte >> 4) - 8.f, s), emb_scale);
        }
    } else {
        const uint32_t nsb = n_embd / 256;
        const uint8_t* base = reinterpret_cast<const uint8_t*>(w.q) + (size_t)tok * nsb * 144;
        for (uint32_t i = threadIdx.x; i < nsb * 128; i += blockDim.x) {
            const uint32_t sb = i >> 7, bi = i & 127, grp = bi >> 5, j = bi & 31;
            const uint8_t* blk = base + (size_t)sb * 144;
            const uint4 hdr = *reinterpret_cast<const uint4*>(blk);
            float s0, m0, s1, m1;
            // same products as the loader: (d*sc), (dmin*m), each rounded once
            {
                const int sh = (grp & 1) * 16;
                const uint32_t s16 = (hdr.y >> sh) & 0xFFFFu, m16 = (hdr.z >> sh) & 0xFFFFu, t16 = (hdr.w >> sh) & 0xFFFFu;
                uint32_t sp, mp;
                if (grp < 2) { sp = s16 & 0x3F3Fu; mp = m16 & 0x3F3Fu; }
                else { sp = (t16 & 0x0F0Fu) | ((s16 >> 2) & 0x3030u); mp = ((t16 >> 4) & 0x0F0Fu) | ((m16 >> 2) & 0x3030u); }
                const float dd = __half2float(__ushort_as_half((unsigned short)(hdr.x & 0xFFFFu)));
                const float dm = __half2float(__ushort_as_half((unsigned short)(hdr.x >> 16)));
                s0 = __fmul_rn(dd, (float)(sp & 0xFFu)); s1 = __fmul_rn(dd, (float)(sp >> 8));
                m0 = __fmul_rn(dm, (float)(mp & 0xFFu)); m1 = __fmul_rn(dm, (float)(mp >> 8));
            }
            const uint32_t byte = blk[16 + bi];
            float* o = out + sb * 256 + grp * 64;
            o[j]      = __fmul_rn(__fsub_rn(__fmul_rn((float)(byte & 15), s0), m0), emb_scale);
            o[32 + j] = __fmul_rn(__fsub_rn(__fmul_rn((float)(byte >> 4), s1), m1), emb_scale);
        }
    }
}

// Cluster primitives of the attention launch whose position splits form one thread-block cluster: the splits'
// partial results go to the first CTA's shared memory.  The hardware cluster barrier only says that every CTA has started
// (every thread of every CTA arrives and waits exactly once); CTA 0 leaves last, when the results it waits for are there.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t dsmem_addr_rank0(const void* p) {          // address of `p` in the cluster's CTA 0
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(0));
    return r;
}
// Stores that count their bytes on a barrier next to where they go: whoever waits for the barrier sees the data, no fence and
// no second cluster barrier.
__device__ __forceinline__ void st_async4(uint32_t addr, float4 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 :: "r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async2(uint32_t addr, float2 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" :: "r"(addr), "f"(v.x), "f"(v.y), "r"(bar) : "memory");
}

// Decode attention for one (split, kv head, sequence), all query heads that share
// the kv head, with the steps that precede it folded in:
//   * per-head RMSNorm + half-split RoPE of the query rows (map_qk_norm_rope_x.comp),
//     angles read from the host-made table;
//   * the CTA whose range holds the newest position does the same for the key row
//     and appends key and value to the paged cache (map_row_copy.comp);
//   * p = softmax(cap*tanh(q.k*scale/cap)) over positions [start, seq), o = p @ V
//     (map_matmul_t.comp + map_attn_softmax_value.comp; diag_inference.py:989-1012).
// Work split.  Positions are walked in chunks of ATTN_CP = 8 (aligned to absolute
// multiples of 8, so a chunk never straddles a page whose size is a multiple of 8).
// The active CTAs (at most gridDim.x, at least one per 8 chunks) take contiguous
// runs of chunks; inside a CTA the 8 warps take chunks round-robin.  A lane owns
// head_dim/32 consecutive dims of every K and V row.  The rows of a warp's chunk
// come by bulk copy (mbarrier completion) into shared memory of its own (8 KB, 16 KB fp32), ahead of the dependency wait for the first chunk; the next chunk's K rows
// are requested as soon as the scores are done and its V rows after the P@V
// accumulation.  (Rows in registers, two chunks in flight, took 211 registers: a
// cluster of 8 such CTAs found no place beside the kernels around it and started
// late.)  The 8 x heads partial dot products of a chunk are
// summed over the lanes with a reduce-scatter (one shuffle per value) that leaves
// score (position j, head g) on one lane; the soft-max runs online per warp, and
// (max, sum, o) are merged across warps in shared memory, then across CTAs by the
// CTA that finishes last.
constexpr int ATTN_CP = 8;
constexpr int ATTN_SMEM_LIMIT = 220 * 1024;    // 16 slots of fp16 or 12 of fp32 rows of 256, queries, the cluster's partial results
constexpr uint32_t ATTN_CHUNKS_PER_CTA = 32;   // chunks a CTA takes (4 per warp) before another CTA joins, when the grid is already large;
                                               // launches with few (sequence, head) pairs pass a smaller number in the upper half of `hpc`

template <typename T, int GS_MAX, int HD>
__global__ void __launch_bounds__(256) k_attention(const float* __restrict__ qkv, uint32_t qkv_ld,
                                                   const float* __restrict__ q_norm, const float* __restrict__ k_norm, float eps,
                                                   const float* __restrict__ cos_t, const float* __restrict__ sin_t, uint32_t n_pos,
                                                   void* __restrict__ kv_pool_v, KvGeom geo,
                                                   const int32_t* __restrict__ block_table, const int32_t* __restrict__ pos,
                                                   uint32_t n_head, uint32_t layer, uint32_t window, float scale, float cap,
                                                   float* __restrict__ out, float* __restrict__ part_o, float* __restrict__ part_ml,
                                                   unsigned int* __restrict__ ticket, uint32_t n_splits_max, uint32_t hpc, uint32_t n_slots, uint32_t* err STEP_TRACE_PARAM) {
#ifdef ADAM_B200_STEP_TRACE
#define AT_STAMP(slot) do { if (threadIdx.x == 0 && blockIdx.z == 0 && (blockIdx.y * gridDim.x + blockIdx.x) < 32) STEP_STAMP(trace, (blockIdx.y * gridDim.x + blockIdx.x) * 8 + (slot)); } while (0)
#else
#define AT_STAMP(slot) do { } while (0)
#endif
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ float s_m[8][GS_MAX], s_l[8][GS_MAX];
    __shared__ float s_w[8][GS_MAX], s_M[GS_MAX];
    __shared__ bool s_last;
    __shared__ __align__(8) uint64_t s_bar[16][2], s_mb;                // a slot's keys and values; the cluster's partial results
    AT_STAMP(0);
    // In a cluster asked for at once, by the CTAs without positions too: the next kernel starts when every CTA has asked (one that
    // leaves a cluster early counts only when the whole cluster is done, which held the o-proj back until the merge).  Large
    // grids of independent splits ask late and keep their own shared-memory split: the kernels around them fill the SMs (64
    // sequences of the 27B shape, 8 layers: 3.30 ms per step, 3.42 when asked at once, 3.57 with the largest split, too).
    if (n_splits_max == 0) pdl_launch_dependents();
    // n_splits_max == 0: the gridDim.x splits of a (sequence, head group) are one thread-block cluster and merge
    // through CTA 0's shared memory instead of global memory, a ticket and the last CTA to arrive.
    const bool cmerge = n_splits_max == 0;
    // (the barriers first: the fences would wait for loads in flight)
    if (threadIdx.x < 32) mbar_init(&s_bar[0][0] + threadIdx.x, 1);
    if (threadIdx.x == 0) mbar_init(&s_mb, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (cmerge) cluster_arrive();               // "this CTA runs": waited for before the first store into CTA 0
    const uint32_t cpc_min = (hpc >> 16) ? (hpc >> 16) : ATTN_CHUNKS_PER_CTA;     // chunks per CTA before another CTA joins
    hpc &= 0xFFFFu;
    T* __restrict__ kv_pool = reinterpret_cast<T*>(kv_pool_v);
    constexpr int DPL = HD / 32;                // dims per lane
    constexpr int CP = ATTN_CP, ROWB = HD * (int)sizeof(T);   // positions per chunk, bytes of a row
    constexpr int NV = CP * GS_MAX;             // scores per chunk
    constexpr int VPL = NV >= 32 ? NV / 32 : 1; // scores a lane holds after the reduce-scatter
    constexpr int LPV = NV >= 32 ? 1 : 32 / NV; // lanes that hold the same score
    constexpr float NEG = -1.0e30f;
    static_assert(DPL >= 1 && (GS_MAX == 1 || GS_MAX == 2 || GS_MAX == 4 || GS_MAX == 8), "unsupported attention shape");
    // blockIdx.y = (kv head, group of `hpc` query heads that share it)
    const uint32_t hgn = (n_head / geo.n_kv) / hpc;
    const uint32_t split = blockIdx.x, kvh = blockIdx.y / hgn, hg = blockIdx.y % hgn, b = blockIdx.z;
    const uint32_t head0 = kvh * (n_head / geo.n_kv) + hg * hpc;
    const uint32_t slot_y = b * gridDim.y + blockIdx.y;        // scratch slot of this (sequence, head group)
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // The block table is written by the host before the step's first kernel, so it can be
    // read ahead of the dependency wait: up to 128 entries sit in registers across the warp.
    const int32_t* bt = block_table + (size_t)b * geo.max_pages;
    const bool bt_regs = geo.max_pages <= 128;
    int32_t btr[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) { const uint32_t i = lane + 32 * k; btr[k] = (bt_regs && i < geo.max_pages) ? bt[i] : -1; }
    auto page_of = [&](uint32_t pn) -> int32_t {        // called by whole warps
        if (!bt_regs) return pn < geo.max_pages ? bt[pn] : -1;
        int32_t v = __shfl_sync(0xffffffffu, btr[0], pn & 31);
        if (geo.max_pages > 32) {
            const int32_t v1 = __shfl_sync(0xffffffffu, btr[1], pn & 31), v2 = __shfl_sync(0xffffffffu, btr[2], pn & 31), v3 = __shfl_sync(0xffffffffu, btr[3], pn & 31);
            v = pn < 32 ? v : pn < 64 ? v1 : pn < 96 ? v2 : v3;
        }
        return pn < geo.max_pages ? v : -1;
    };
    // QK-norm weights are read-only too.
    constexpr int NP = (HD / 2 + 31) / 32;          // rotation pairs per lane
    // Up to four query heads a warp has one row at most (query, key or value): its weights; eight heads fetch them per row.
    constexpr bool W1 = GS_MAX <= 4;
    float w0[NP], w1[NP];
    auto load_norm = [&](const float* w) {
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const uint32_t i = lane + 32 * j;
            const bool in = w && i < HD / 2;
            w0[j] = in ? w[i] : 1.f; w1[j] = in ? w[i + HD / 2] : 1.f;
        }
    };
    if constexpr (W1) load_norm(warp < hpc ? q_norm : k_norm);
    // Positions only change in the step's last kernel, and the step's first kernel is
    // launched with a full dependency on it, so the position, and everything in the cache
    // older than this step, can be read ahead of the wait as well.
    const uint32_t hd = HD, half = HD / 2, gs = hpc;
    const int32_t p = pos[b];
    const uint32_t seq = (uint32_t)p + 1;
    const uint32_t start = (window > 0 && seq > window) ? seq - window : 0;
    const uint32_t c_first = start / CP, n_chunks = (seq - 1) / CP - c_first + 1;
    const uint32_t n_act = min((uint32_t)gridDim.x, (n_chunks + cpc_min - 1) / cpc_min);
    if (split >= n_act) { if (cmerge) cluster_wait(); return; }
    const uint32_t cpc = (n_chunks + n_act - 1) / n_act;
    const uint32_t c0 = min(c_first + split * cpc, c_first + n_chunks), c1 = min(c_first + n_chunks, c0 + cpc);
    const uint32_t c_new = (uint32_t)p / CP;      // chunk whose newest row comes from this step's q/k/v
    const bool owner = c_new >= c0 && c_new < c1;
    // Slots of a chunk each, CP key rows and CP value rows: the first n_slots (8 to 16) chunks of the CTA are requested at once,
    // slot i chunk i; warp w's chunks behind them go through slot w.  A warp's partial result ends up in its slot.
    constexpr uint32_t SLOT = 2 * CP * ROWB;
    float* s_q = reinterpret_cast<float*>(sm + n_slots * SLOT);         // [gs][hd]
    float* s_kn = s_q + gs * hd;                // [hd] newest key (as stored)
    float* s_vn = s_kn + hd;                    // [hd] newest value (as stored)
    float* s_cp = s_vn + hd;                    // cluster merge, CTA 0 only: [split][gs * hd + 4 * gs] (16-byte aligned rows)
    // Rows of chunk c: keys (kv = 0), values (1) or both (2).  A chunk whose rows are all there and consecutive is one copy,
    // otherwise a lane fetches a row each.  Positions outside [start, seq) then read the nearest row inside; their scores and value
    // rows are masked later.
    const bool whole = geo.page % CP == 0;
    auto request = [&](uint32_t c, uint32_t kv, uint32_t slot) {
        const uint32_t j = lane % CP, k = kv == 2 ? lane / CP : kv;
        const uint32_t tp = min(max(c * CP + j, start), seq - 1);
        const uint32_t pn = tp / geo.page;
        const uint32_t pg = (uint32_t)max(page_of(pn), 0);
        if (lane < 2 && (kv == 2 || lane == kv)) mbar_expect_tx(&s_bar[slot][lane], CP * ROWB);
        __syncwarp();
        const bool one = whole && c * CP >= start && c * CP + CP <= seq;
        if (lane < (kv == 2 ? 2 * CP : CP) && (!one || j == 0))
            bulk_g2s(sm + slot * SLOT + (k * CP + j) * ROWB, kv_pool + kv_index(geo, pg, layer, k, kvh, tp - pn * geo.page), one ? CP * ROWB : ROWB, &s_bar[slot][k]);
    };
    uint32_t c = c0 + warp;
    for (uint32_t i = warp; i < n_slots && c0 + i < c1; i += 8) request(c0 + i, 2, i);
    uint32_t c_late = c0 + warp + ((n_slots - warp + 7) & ~7u);         // the warp's first chunk behind those
    // Rows of this warp's later chunks: asked into L2 now, one request each for keys and values where they are consecutive.
    if (whole && lane < 2) {
        for (uint32_t c2 = c_late; c2 < c1; c2 += 8) {
            const uint32_t pn = c2 * CP / geo.page;
            const int32_t pg = bt[pn < geo.max_pages ? pn : 0];
            if (pg >= 0)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;"
                             :: "l"(kv_pool + kv_index(geo, (uint32_t)pg, layer, lane, kvh, c2 * CP - pn * geo.page)), "r"(CP * ROWB) : "memory");
        }
    }

    // ---- a warp per row: query heads, and (owner only) the newest key and value rows ----
    const uint32_t pp = (uint32_t)p < n_pos ? (uint32_t)p : n_pos - 1;
    if ((uint32_t)p >= n_pos && tid == 0) atomicOr(err, DEVERR_OOB_MAP);
    const float* ct = cos_t + (size_t)pp * half;
    const float* st = sin_t + (size_t)pp * half;
    float cs[NP], sn[NP];
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        const uint32_t i = lane + 32 * j;
        cs[j] = i < half ? ct[i] : 1.f;
        sn[j] = i < half ? st[i] : 0.f;
    }
    AT_STAMP(1);
    if (n_splits_max != 0) pdl_launch_dependents();
    pdl_wait();                                 // this step's q/k/v rows come from the previous kernel
    AT_STAMP(2);
    const float* row_q = qkv + (size_t)b * qkv_ld + (size_t)head0 * hd;
    const float* row_k = qkv + (size_t)b * qkv_ld + (size_t)n_head * hd + (size_t)kvh * hd;
    const float* row_v = row_k + (size_t)geo.n_kv * hd;
    const uint32_t n_rows = gs + (owner ? 2u : 0u);
    for (uint32_t r = warp; r < n_rows; r += 8) {
        const bool is_q = r < gs, is_k = (r == gs);
        const float* src = is_q ? row_q + (size_t)r * hd : (is_k ? row_k : row_v);
        size_t kv_off = 0;
        bool ok = true;
        if (!is_q) {
            const uint32_t page_no = (uint32_t)p / geo.page;
            const int32_t page_id = page_of(page_no);
            if (page_id < 0) { ok = false; if (lane == 0) atomicOr(err, DEVERR_OOB_MAP); }
            else if (hg != 0) ok = false;               // one head group appends to the cache; the others only need the rows
            if (ok) kv_off = kv_index(geo, (uint32_t)page_id, layer, is_k ? 0u : 1u, kvh, (uint32_t)p % geo.page);
        }
        if (!is_q && !is_k) {
            for (uint32_t i = lane; i < hd; i += 32) {
                const float v = src[i];
                s_vn[i] = kv_round<T>(v);
                if (ok) st_kv(kv_pool + kv_off + i, v);
            }
            continue;
        }
        const float* w = is_q ? q_norm : k_norm;
        float x0[NP], x1[NP];
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const uint32_t i = lane + 32 * j;
            const bool in = i < half;
            x0[j] = in ? src[i] : 0.f;
            x1[j] = in ? src[i + half] : 0.f;
        }
        if constexpr (!W1) load_norm(w);
        float rinv = 1.f;
        if (w) {
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int j = 0; j < NP; ++j) { s0 = fmaf(x0[j], x0[j], s0); s1 = fmaf(x1[j], x1[j], s1); }
            rinv = rsqrt_newton(fmaf(warp_sum(s0 + s1), 1.0f / (float)HD, eps));
        }
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const uint32_t i = lane + 32 * j;
            if (i < half) {
                float a0 = x0[j], a1 = x1[j];
                if (w) { a0 = a0 * rinv * w0[j]; a1 = a1 * rinv * w1[j]; }
                const float y0 = __fsub_rn(__fmul_rn(a0, cs[j]), __fmul_rn(a1, sn[j]));
                const float y1 = __fadd_rn(__fmul_rn(a0, sn[j]), __fmul_rn(a1, cs[j]));
                if (is_q) { s_q[r * hd + i] = y0; s_q[r * hd + i + half] = y1; }
                else {
                    s_kn[i] = kv_round<T>(y0); s_kn[i + half] = kv_round<T>(y1);
                    if (ok) { st_kv(kv_pool + kv_off + i, y0); st_kv(kv_pool + kv_off + i + half, y1); }
                }
            }
        }
    }
    __syncthreads();
    AT_STAMP(3);

    // ---- this warp's chunks: scores, online soft-max, P@V ----
    float q[GS_MAX][DPL], o[GS_MAX][DPL], m_run[VPL], l_run[VPL];
#pragma unroll
    for (int g = 0; g < GS_MAX; ++g)
#pragma unroll
        for (int d = 0; d < DPL; ++d) { q[g][d] = g < (int)gs ? s_q[g * hd + lane * DPL + d] : 0.f; o[g][d] = 0.f; }
#pragma unroll
    for (int r = 0; r < VPL; ++r) { m_run[r] = NEG; l_run[r] = 0.f; }
    bool timed_out = false;
    auto landed = [&](uint32_t slot, uint32_t k, uint32_t ph) {         // bounded; a warp that gives up keeps meeting the CTA's barriers
        const bool ok = __all_sync(0xffffffffu, mbar_wait(&s_bar[slot][k], ph));
        if (!ok && lane == 0) atomicOr(err, DEVERR_WAIT);
        timed_out |= !ok;
        return ok;
    };
    const int jn = (int)((uint32_t)p % CP);
    uint32_t ph = 0;                                        // parity of the warp's own slot
    for (; c < c1 && !timed_out; c += 8) {
        KvRow<T, DPL> row;
        float sc[NV];
        const bool extra = c - c0 >= 8 && c - c0 < n_slots;
        const uint32_t slot = extra ? c - c0 : warp;
        unsigned char* s_kv = sm + slot * SLOT;
        const bool late = !extra && c_late < c1;            // the slot has another chunk to take when its rows are read
        if (!landed(slot, 0, extra ? 0u : ph)) break;
        // the newest position's rows come from this step's q/k/v, not from the cache (a lane writes and reads its own dims)
        if (c == c_new) { row.from_float(s_kn + lane * DPL); row.store(reinterpret_cast<T*>(s_kv + jn * ROWB) + lane * DPL); }
#pragma unroll
        for (int j = 0; j < CP; ++j) {
            float kf[DPL];
            row.load(reinterpret_cast<const T*>(s_kv + j * ROWB) + lane * DPL);
            row.to_float(kf);
#pragma unroll
            for (int g = 0; g < GS_MAX; ++g) {
                if constexpr (DPL >= 2) {
                    float a0 = 0.f, a1 = 0.f;
#pragma unroll
                    for (int d = 0; d < DPL; d += 2) fma2(a0, a1, q[g][d], q[g][d + 1], kf[d], kf[d + 1]);
                    sc[j * GS_MAX + g] = a0 + a1;
                } else {
                    sc[j * GS_MAX + g] = q[g][0] * kf[0];
                }
            }
        }
        if (late) { __syncwarp(); request(c_late, 0, warp); }
        warp_reduce_scatter<NV>(sc, lane);
        float pz[VPL], alpha[VPL];
#pragma unroll
        for (int r = 0; r < VPL; ++r) {
            const uint32_t v = NV >= 32 ? lane * VPL + r : lane / LPV;
            const uint32_t j = v / GS_MAX, g = v % GS_MAX;
            const uint32_t tp = c * CP + j;
            const bool valid = tp >= start && tp < seq && g < gs;
            float sv = sc[r] * scale;
            if (cap > 0.f) sv = tanhf(sv / cap) * cap;
            sv = valid ? sv : NEG;
            float cm = sv;
#pragma unroll
            for (int off = 32 / CP; off < 32; off <<= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, off));
            const float m_new = fmaxf(m_run[r], cm);
            alpha[r] = expf(m_run[r] - m_new);
            pz[r] = valid ? expf(sv - m_new) : 0.f;
            float ps = pz[r];
#pragma unroll
            for (int off = 32 / CP; off < 32; off <<= 1) ps += __shfl_xor_sync(0xffffffffu, ps, off);
            l_run[r] = fmaf(l_run[r], alpha[r], ps);
            m_run[r] = m_new;
        }
#pragma unroll
        for (int g = 0; g < GS_MAX; ++g) {
            // lane and slot that hold (position 0, head g)
            const float al = __shfl_sync(0xffffffffu, alpha[g % VPL], NV >= 32 ? g / VPL : g * LPV);
#pragma unroll
            for (int d = 0; d < DPL; ++d) o[g][d] *= al;
        }
        if (!landed(slot, 1, extra ? 0u : ph)) break;
        if (c == c_new) { row.from_float(s_vn + lane * DPL); row.store(reinterpret_cast<T*>(s_kv + (CP + jn) * ROWB) + lane * DPL); }
        // Value rows outside [start, seq) count with probability 0, and 0 times what stands there (an earlier sequence's infinities) need
        // not be 0.  The fence: a bulk copy writes the slot next.
        if (c * CP < start || c * CP + CP > seq) {
            row.zero();
#pragma unroll
            for (int j = 0; j < CP; ++j)
                if (c * CP + j < start || c * CP + j >= seq) row.store(reinterpret_cast<T*>(s_kv + (CP + j) * ROWB) + lane * DPL);
            if (late) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
#pragma unroll
        for (int j = 0; j < CP; ++j) {
            float vf[DPL];
            row.load(reinterpret_cast<const T*>(s_kv + (CP + j) * ROWB) + lane * DPL);
            row.to_float(vf);
#pragma unroll
            for (int g = 0; g < GS_MAX; ++g) {
                const int v = j * GS_MAX + g;
                const float pv = __shfl_sync(0xffffffffu, pz[v % VPL], NV >= 32 ? v / VPL : v * LPV);
                if constexpr (DPL >= 2) {
#pragma unroll
                    for (int d = 0; d < DPL; d += 2) fma2(o[g][d], o[g][d + 1], pv, pv, vf[d], vf[d + 1]);
                } else {
                    o[g][0] = fmaf(pv, vf[0], o[g][0]);
                }
            }
        }
        if (late) { __syncwarp(); request(c_late, 1, warp); c_late += 8; }
        if (!extra) ph ^= 1u;
    }
    AT_STAMP(4);
    if (timed_out) { for (uint32_t i = warp; i < n_slots; i += 8) for (int k = 0; k < 2; ++k) { mbar_wait(&s_bar[i][k], 0u); mbar_wait(&s_bar[i][k], 1u); } }     // a bounded chance for copies in flight
    // ---- merge the warps: a warp's partial result goes where its rows were ----
    __syncwarp();
    {
        float* so = reinterpret_cast<float*>(sm + warp * SLOT) + lane * DPL;
#pragma unroll
        for (int g = 0; g < GS_MAX; ++g) {
            if (g < (int)gs) {
                if constexpr (DPL % 4 == 0) {
#pragma unroll
                    for (int d = 0; d < DPL; d += 4) *reinterpret_cast<float4*>(so + g * hd + d) = make_float4(o[g][d], o[g][d + 1], o[g][d + 2], o[g][d + 3]);
                } else {
#pragma unroll
                    for (int d = 0; d < DPL; ++d) so[g * hd + d] = o[g][d];
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < VPL; ++r) {
        const uint32_t v = NV >= 32 ? lane * VPL + r : lane / LPV;
        if (v < GS_MAX && (NV >= 32 || (lane % LPV) == 0)) { s_m[warp][v] = m_run[r]; s_l[warp][v] = l_run[r]; }
    }
    __syncthreads();
    if (cmerge) AT_STAMP(5);
    // One head per CTA: every thread forms the eight warps' weights itself, which takes no second barrier (and eight
    // exponentials in a row of latencies instead of one).  More heads: the weights are shared.
    if constexpr (GS_MAX > 1) {
    if (tid < 8 * GS_MAX) {                     // weight of warp w for head g
        const uint32_t w = tid / GS_MAX, g = tid % GS_MAX;
        float M = NEG;
#pragma unroll
        for (int w2 = 0; w2 < 8; ++w2) M = fmaxf(M, s_m[w2][g]);
        s_w[w][g] = expf(s_m[w][g] - M);
        if (w == 0) s_M[g] = M;
    }
    __syncthreads();
    }
    // thread -> 4 consecutive outputs (all of one head)
    const uint32_t n_out4 = gs * hd / 4;
    float* po = part_o + ((size_t)slot_y * n_splits_max + split) * gs * hd;
    float* pml = part_ml + ((size_t)slot_y * n_splits_max + split) * gs * 2;
    float* orow = out + ((size_t)b * n_head + head0) * hd;
    const uint32_t pstride = gs * hd + 4 * gs;
    bool joined = false;
    if (cmerge) {
        cluster_wait();                         // every CTA of the cluster has started: CTA 0's shared memory can be written
        if (split == 0 && tid == 0) mbar_expect_tx(&s_mb, (n_act - 1) * (gs * hd * 4 + gs * 8));
    }
    for (uint32_t i4 = tid; i4 < n_out4; i4 += blockDim.x) {
        const uint32_t g = (i4 * 4) / hd;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        float L = 0.f, M = NEG, wt[8];
        if constexpr (GS_MAX == 1) {
#pragma unroll
            for (int w = 0; w < 8; ++w) { wt[w] = s_m[w][0]; M = fmaxf(M, wt[w]); }
#pragma unroll
            for (int w = 0; w < 8; ++w) wt[w] = expf(wt[w] - M);
        } else M = s_M[g];
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const float ww = GS_MAX == 1 ? wt[w] : s_w[w][g];
            const float4 x = reinterpret_cast<const float4*>(sm + w * SLOT)[i4];
            v.x = fmaf(ww, x.x, v.x); v.y = fmaf(ww, x.y, v.y); v.z = fmaf(ww, x.z, v.z); v.w = fmaf(ww, x.w, v.w);
            L = fmaf(ww, s_l[w][g], L);
        }
        if (n_act == 1) {
            reinterpret_cast<float4*>(orow)[i4] = quotient4(v, L);
        }
        else if (cmerge) {
            if (split != 0) {
                float* mine = s_cp + (size_t)split * pstride;
                st_async4(dsmem_addr_rank0(mine + i4 * 4), v, dsmem_addr_rank0(&s_mb));
                if ((i4 * 4) % hd == 0) st_async2(dsmem_addr_rank0(mine + gs * hd + g * 2), make_float2(M, L), dsmem_addr_rank0(&s_mb));
            } else {
                AT_STAMP(6);
                if (!joined) {                  // every split's partial result is in this CTA's shared memory
                    if (!mbar_wait(&s_mb, 0u)) { atomicOr(err, DEVERR_WAIT); mbar_wait(&s_mb, 0u); }
                    joined = true;
                }
                // this CTA's own and up to seven more (one cluster of the usual size) at a time, loads and exponentials side by side
                float4 num = v;
                float den = L;
                for (uint32_t s0 = 1; s0 < n_act; s0 += 7) {
                    float2 ml[7]; float4 x[7];
                    float Mn = M;
#pragma unroll
                    for (int k = 0; k < 7; ++k) {
                        const float* ps = s_cp + (size_t)min(s0 + k, n_act - 1) * pstride;
                        ml[k] = *reinterpret_cast<const float2*>(ps + gs * hd + g * 2);
                        x[k] = reinterpret_cast<const float4*>(ps)[i4];
                        Mn = fmaxf(Mn, ml[k].x);
                    }
                    const float a0 = expf(M - Mn);
                    num.x *= a0; num.y *= a0; num.z *= a0; num.w *= a0; den *= a0;
#pragma unroll
                    for (int k = 0; k < 7; ++k) {
                        // (a weight of 0 for the repeated ones would make NaN of an infinity)
                        const bool in = s0 + k < n_act;
                        const float w = expf(ml[k].x - Mn);
                        num.x = in ? fmaf(w, x[k].x, num.x) : num.x; num.y = in ? fmaf(w, x[k].y, num.y) : num.y;
                        num.z = in ? fmaf(w, x[k].z, num.z) : num.z; num.w = in ? fmaf(w, x[k].w, num.w) : num.w;
                        den = in ? fmaf(w, ml[k].y, den) : den;
                    }
                    M = Mn;
                }
                reinterpret_cast<float4*>(orow)[i4] = quotient4(num, den);
            }
        } else {
            reinterpret_cast<float4*>(po)[i4] = v;
            if ((i4 * 4) % hd == 0) *reinterpret_cast<float2*>(pml + g * 2) = make_float2(M, L);
        }
    }
    if (cmerge) { AT_STAMP(7); return; }
    if (n_act == 1) return;
    AT_STAMP(5);
    __threadfence();
    __syncthreads();
    unsigned int* tkt = ticket + slot_y;
    if (tid == 0) s_last = (atomicAdd(tkt, 1u) == n_act - 1);
    __syncthreads();
    AT_STAMP(6);
    if (!s_last) return;
    __threadfence();
    // ---- merge the splits (last CTA to arrive): all loads of a batch of 4 splits are
    // issued together, then folded in with a running maximum ----
    const float* po0 = part_o + ((size_t)slot_y * n_splits_max) * gs * hd;
    const float* pml0 = part_ml + ((size_t)slot_y * n_splits_max) * gs * 2;
    for (uint32_t i4 = tid; i4 < n_out4; i4 += blockDim.x) {
        const uint32_t g = (i4 * 4) / hd;
        float M = NEG, den = 0.f;
        float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t s0 = 0; s0 < n_act; s0 += 4) {
            float2 ml[4]; float4 x[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t sidx = min(s0 + k, n_act - 1);
                ml[k] = __ldcg(reinterpret_cast<const float2*>(pml0 + ((size_t)sidx * gs + g) * 2));
                x[k] = __ldcg(reinterpret_cast<const float4*>(po0 + (size_t)sidx * gs * hd) + i4);
            }
            float Mn = M;
#pragma unroll
            for (int k = 0; k < 4; ++k) if (s0 + k < n_act) Mn = fmaxf(Mn, ml[k].x);
            const float a0 = expf(M - Mn);
            num.x *= a0; num.y *= a0; num.z *= a0; num.w *= a0; den *= a0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (s0 + k < n_act) {
                    const float w = expf(ml[k].x - Mn);
                    num.x = fmaf(w, x[k].x, num.x); num.y = fmaf(w, x[k].y, num.y);
                    num.z = fmaf(w, x[k].z, num.z); num.w = fmaf(w, x[k].w, num.w);
                    den = fmaf(w, ml[k].y, den);
                }
            }
            M = Mn;
        }
        reinterpret_cast<float4*>(orow)[i4] = quotient4(num, den);
    }
    AT_STAMP(7);
    if (tid == 0) *tkt = 0u;
}

// End of a prefill: every sequence moves on by its own number of tokens, or all by `even`.
__global__ void k_advance_by(int32_t* __restrict__ pos, const int32_t* __restrict__ n, int32_t even, uint32_t batch) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < batch) pos[b] += n ? n[b] : even;
}
// The plan of a chunk of T tokens for each of `batch` sequences, from where they are now: row r = (sequence r / T, position
// pos + r % T), and attention tiles of up to `step` positions, those with the longest reach first.
__global__ void k_even_plan(const int32_t* __restrict__ pos, uint32_t batch, uint32_t T, uint32_t step, int32_t* __restrict__ row_seq,
                            int32_t* __restrict__ row_pos, AttnTile* __restrict__ tiles) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x, per = (T + step - 1) / step;
    if (r >= batch * T) return;
    row_seq[r] = (int32_t)(r / T);
    row_pos[r] = pos[r / T] + (int32_t)(r % T);
    if (r >= batch * per) return;
    const uint32_t s = r % batch, first = (per - 1 - r / batch) * step;
    tiles[r] = AttnTile{(int32_t)(s * T + first), (int32_t)s, pos[s] + (int32_t)first, (int32_t)min(step, T - first)};
}

// End of a step: advance positions; when the LM head ran, log the sampled token.
__global__ void k_advance(int32_t* __restrict__ pos, const int32_t* __restrict__ cur_tok, int32_t* __restrict__ gen_log,
                          uint32_t log_ld, uint32_t batch, int with_lm) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= batch) return;
    const int32_t p = pos[b] + 1;
    pos[b] = p;
    if (with_lm && (uint32_t)p < log_ld) gen_log[(size_t)b * log_ld + p] = cur_tok[b];
}

__global__ void k_fill_i32(int32_t* p, int32_t v, size_t n) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

// ---- host side ---------------------------------------------------------------

constexpr uint32_t TK_GRAPH_N = 8;
static void free_token_kernel(Decoder* D) {
    if (D->tk_state == 1) cudaStreamSynchronize(g.stream);
    for (int i = 0; i < 2; ++i) {
        if (D->tk_graph[i]) { cudaGraphExecDestroy(D->tk_graph[i]); cudaGraphDestroy(D->tk_graph_src[i]); D->tk_graph[i] = nullptr; D->tk_graph_src[i] = nullptr; }
        D->tk_graph_state[i] = 0;
    }
    for (void*& m : D->tk_mem) { if (m) cudaFree(m); m = nullptr; }
    D->tk_state = 0;
}

static void free_graphs(Decoder* D) {
    for (int i = 0; i < 2; ++i) {
        if (D->graph[i]) { cudaGraphExecDestroy(D->graph[i]); cudaGraphDestroy(D->graph_src[i]); D->graph[i] = nullptr; D->graph_src[i] = nullptr; }
    }
    free_token_kernel(D);
}

static void score_release(Decoder* D) {
    cudaFree(D->score_logits); cudaFree(D->score_tok);
    for (cudaEvent_t& e : D->score_ev) if (e) { cudaEventDestroy(e); e = nullptr; }
    if (D->score_copy) cudaStreamDestroy(D->score_copy);
    D->score_logits = nullptr; D->score_tok = nullptr; D->score_copy = nullptr; D->score_rows = 0;
}
static void destroy(Decoder* D) {
    cudaStreamSynchronize(g.stream);
    free_graphs(D);
    free_token_kernel(D);
    for (int i = 0; i < 4; ++i) { if (D->tok_ring[i]) cudaFreeHost(D->tok_ring[i]); if (D->tok_event[i]) cudaEventDestroy(D->tok_event[i]); }
    void* ptrs[] = {D->pos, D->cur_tok, D->cur_val, D->prompt_len, D->prompt_tok, D->gen_log, D->block_table, D->kv_pool, D->hbuf[0], D->hbuf[1], D->qkv,
                    D->attn_out, D->proj, D->act, D->logits, D->part_o, D->part_ml, D->attn_ticket, D->plan, D->even_plan,
                    D->rope_cos[0], D->rope_sin[0], D->rope_cos[1], D->rope_sin[1]};
    for (void* p : ptrs) cudaFree(p);
    cudaFreeHost(D->plan_pin);
    if (D->plan_read) cudaEventDestroy(D->plan_read);
    score_release(D);
    delete D;
}

void decoder_destroy_all() {
    for (uint32_t i = 0; i < MAX_DECODERS; ++i) if (g_dec[i]) { destroy(g_dec[i]); g_dec[i] = nullptr; }
}

#define DCU(x) do { cudaError_t e__ = (x); if (e__ != cudaSuccess) return fail(e__ == cudaErrorMemoryAllocation ? ADAMAH_ERR_MEMORY : ADAMAH_ERR_BACKEND, "%s: %s", #x, cudaGetErrorString(e__)); } while (0)

static bool is_global_layer(const adam_b200_decoder_desc& d, uint32_t L) { return d.global_every == 0 || (L + 1) % d.global_every == 0; }

static size_t kv_elem_size(const adam_b200_decoder_desc& d) { return d.kv_dtype == 1 ? 2 : 4; }

typedef void (*AttnKernel)(const float*, uint32_t, const float*, const float*, float, const float*, const float*, uint32_t, void*, KvGeom,
                           const int32_t*, const int32_t*, uint32_t, uint32_t, uint32_t, float, float, float*, float*, float*,
                           unsigned int*, uint32_t, uint32_t, uint32_t, uint32_t* STEP_TRACE_PARAM);

template <typename T, int GS>
static AttnKernel pick_attn_hd(uint32_t hd) {
    switch (hd) {
    case 32: return k_attention<T, GS, 32>;
    case 64: return k_attention<T, GS, 64>;
    case 128: return k_attention<T, GS, 128>;
    default: return k_attention<T, GS, 256>;
    }
}

// Launch shape of a decode attention.
struct AttnShape {
    uint32_t gs, hpc, work, pairs;      // query heads per kv head and per CTA; (sequence, head), (sequence, head group) pairs
    uint32_t cluster;                   // CTAs of a cluster of position splits; 0: independent splits, 8 slots each
    uint32_t slots;                     // chunks in flight per CTA of a cluster
    size_t smem, smem_cluster;          // of a CTA of independent splits, of a cluster
};
static AttnShape attn_shape(uint32_t n_head, uint32_t n_kv, uint32_t head_dim, uint32_t kv_bytes, uint32_t batch, uint32_t reach, uint32_t most = 16) {
    AttnShape s = {};
    s.gs = n_head / n_kv;
    // Query heads per CTA: one while that still leaves SMs idle (lowest latency; the CTAs
    // of a kv head re-read its rows from L2), the whole group once the grid is large.
    // Measured at the 1B shape (4 query heads on 1 kv head): up to three sequences are fastest with a CTA per query head, eight
    // sequences with two heads per CTA, 16 or more sequences and prefill chunks with the whole group per CTA (the rows of a kv
    // head are then read once instead of once per query head).
    static const uint32_t hpc_env = getenv("ADAM_B200_ATTN_HPC") ? (uint32_t)atoi(getenv("ADAM_B200_ATTN_HPC")) : 0u;
    s.work = batch * n_head;
    const uint32_t hpc_auto = s.work <= 12u ? 1u : (s.work <= 32u ? (s.gs % 2u == 0u ? 2u : 1u) : s.gs);      // a divisor of the group
    s.hpc = (hpc_env && s.gs % hpc_env == 0 && hpc_env <= 8u) ? hpc_env : hpc_auto;
    s.pairs = n_kv * (s.gs / s.hpc) * batch;
    // Few pairs in flight: the position splits of a pair form one thread-block cluster -- of 8 CTAs up to 16 pairs, of 4 up to 32, of 2
    // up to 64: one CTA per SM -- and merge through shared memory (no partial results in global memory, no ticket, no last-CTA pass:
    // 3 us less per launch at the 1B shape).  The lines at 32 and 56 rest on 48 sequences (clusters of 2 slower), 56 and 64 (faster)
    // of that shape at a context of 512.  With an fp32 cache 9 sequences take 1.14 ms per step as clusters of 8 with 11 slots and 1.17
    // as independent splits, 12 take 1.17 and 1.19, 16 the same.  A cluster covers any context, its CTAs taking more chunks each, so
    // layers that may attend to more than 2048 positions keep the wider grid of independent splits.  (Clusters of 16 were measured
    // slower: they start later, and so does every kernel behind them.)  ADAM_B200_ATTN_CLUSTER=0 turns the path off, =16 allows
    // clusters of 16.
    static const int cluster_env = getenv("ADAM_B200_ATTN_CLUSTER") ? atoi(getenv("ADAM_B200_ATTN_CLUSTER")) : 8;
    static const uint32_t cluster_pairs = getenv("ADAM_B200_ATTN_CLUSTER_WORK") ? (uint32_t)atoi(getenv("ADAM_B200_ATTN_CLUSTER_WORK")) : 64u;
    if (cluster_env != 0 && s.pairs <= cluster_pairs && (s.pairs <= 32u || s.pairs >= 56u) && reach <= 2048u)
        s.cluster = s.pairs > 32u ? 2u : s.pairs > 16u ? 4u : cluster_env == 16 ? std::min(most, 16u) : 8u;
    // Chunks in flight per CTA: one per warp; up to two in a cluster of splits, where a context just beyond 8 chunks per CTA (a window
    // of 512) would have a warp wait for memory a second time: as many as fit beside the queries and, in the first CTA, the splits'
    // partial results.  (Elsewhere CTAs without positions would hold that much, too.)
    const size_t slot = (size_t)2 * ATTN_CP * head_dim * kv_bytes, rows = ((size_t)s.hpc + 2) * head_dim * 4, merge = (size_t)s.cluster * s.hpc * (head_dim + 4) * 4;
    s.smem = 8 * slot + rows;
    if (s.cluster) {
        const size_t fit = rows + merge < (size_t)ATTN_SMEM_LIMIT ? (ATTN_SMEM_LIMIT - rows - merge) / slot : 0;
        s.slots = (uint32_t)std::min<size_t>(16, std::min<size_t>((192u << 10) / slot, fit));
        if (s.slots < 8u) s.cluster = 0;
        s.smem_cluster = s.slots * slot + rows + merge;
    }
    return s;
}

template <typename T>
static int launch_attn_t(Decoder* D, uint32_t L, uint32_t batch) {
    const adam_b200_decoder_desc& d = D->d;
    KvGeom geo{d.n_layer, d.n_head_kv, d.head_dim, d.page_size, D->max_pages_per_seq, D->page_elems};
    const uint32_t window = ((d.flags & 1u) && d.sliding_window > 0 && !is_global_layer(d, L)) ? d.sliding_window : 0;
    const uint32_t reach = window ? (window < d.kv_cap ? window : d.kv_cap) : d.kv_cap;
    AttnShape s = attn_shape(d.n_head, d.n_head_kv, d.head_dim, sizeof(T), batch, reach);
    const int which = is_global_layer(d, L) ? 1 : 0;
    const Layer& ly = D->layers[L];
    const uint32_t qkv_ld = (d.n_head + 2 * d.n_head_kv) * d.head_dim;
    AttnKernel kern = s.hpc <= 1 ? pick_attn_hd<T, 1>(d.head_dim) : s.hpc <= 2 ? pick_attn_hd<T, 2>(d.head_dim)
                    : s.hpc <= 4 ? pick_attn_hd<T, 4>(d.head_dim) : pick_attn_hd<T, 8>(d.head_dim);
    // Chunks of 8 positions a CTA takes before another CTA joins: with few (sequence, head) pairs the SMs are idle and a
    // CTA's chain of dependent chunk loads is the attention's whole time, so the positions are spread thinly (one chunk
    // per warp); with many pairs the grid is full anyway and every extra CTA only repeats the query prologue.
    static const uint32_t cpc_env = getenv("ADAM_B200_ATTN_CPC") ? (uint32_t)atoi(getenv("ADAM_B200_ATTN_CPC")) : 0u;
    const uint32_t cpc = cpc_env ? cpc_env : (s.work <= 64u ? 8u : ATTN_CHUNKS_PER_CTA);
    // Position splits launched: no more than this layer can reach (a split without positions still costs a CTA its start and the
    // read of the position: 15 of 16 CTAs of the 27B shape's 64 sequences, 60 of the launch's 75 us), and no more than four
    // CTAs per SM in all -- beyond that the pairs alone fill the GPU and a CTA takes more chunks instead.
    const uint32_t useful = ((reach + ATTN_CP - 1) / ATTN_CP + 1 + cpc - 1) / cpc, fill = (4u * (uint32_t)g.sm_count + s.pairs - 1) / s.pairs;
    dim3 grid(std::min(D->n_splits, std::min(useful, fill)), d.n_head_kv * (s.gs / s.hpc), batch);
    // Per kernel: whether its limit is raised, and how many clusters of a size run at once (which the heads per CTA change, too).
    struct Known { AttnKernel k; size_t smem; uint32_t cs; int n; };
    static std::mutex lock;
    static Known known[64]; static int n_known = 0;
    const auto at_once = [&](uint32_t cs, size_t smem) -> int {          // clusters, or 0 for independent splits; negative: no launch
        std::lock_guard<std::mutex> hold(lock);
        bool raised = false;
        for (int i = 0; i < n_known; ++i) {
            if (known[i].k != kern) continue;
            if (known[i].cs == cs && known[i].smem == smem) return known[i].n;
            raised = true;
        }
        if (!raised && cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, ATTN_SMEM_LIMIT) != cudaSuccess) return -1;
        int n = 0;
        if (cs) {
            if (cs > 8 && cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) cudaGetLastError();
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(cs, grid.y, 1); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = cs; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
            cfg.attrs = at; cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, (const void*)kern, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
        }
        if (n_known == 64) n_known = 0;
        known[n_known++] = Known{kern, smem, cs, n};
        return n;
    };
    int n = at_once(s.cluster, s.smem_cluster);
    if (s.cluster == 16 && n >= 0 && n < (int)s.pairs) {
        s = attn_shape(d.n_head, d.n_head_kv, d.head_dim, sizeof(T), batch, reach, 8);
        n = at_once(s.cluster, s.smem_cluster);
    }
    if (n < 0) return fail(ADAMAH_ERR_BACKEND, "attention: cannot raise the shared-memory limit");
    const uint32_t cs = n >= (int)s.pairs ? s.cluster : 0u;
    cudaError_t e;
    const auto args = [&](auto launch, uint32_t n_splits, uint32_t per_cta, uint32_t slots) {
        return launch(D->qkv, qkv_ld, ly.norm[NORM_Q], ly.norm[NORM_K], d.norm_eps, D->rope_cos[which], D->rope_sin[which], D->rope_pos[which],
                      D->kv_pool, geo, D->block_table, D->pos, d.n_head, L, window, d.attn_scale, d.attn_softcap, D->attn_out, D->part_o, D->part_ml,
                      D->attn_ticket, n_splits, s.hpc | (per_cta << 16), slots, g.dev_err STEP_TRACE_ARG((g_step_trace && L == g_step_trace_layer) ? g_step_trace + 4 * 64 : nullptr));
    };
    if (cs) {
        grid.x = cs;
        e = args([&](auto... a) -> cudaError_t { return launch_k_cluster(kern, grid, dim3(256), s.smem_cluster, g.stream, g.pdl, cs, true, a...); }, 0u, cpc_env ? cpc_env : 8u, s.slots);
    } else {
        e = args([&](auto... a) -> cudaError_t { return launch_k(kern, grid, dim3(256), s.smem, g.stream, g.pdl, a...); }, D->n_splits, cpc, 8u);
    }
    if (e != cudaSuccess) return fail(ADAMAH_ERR_BACKEND, "attention: launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    count_ran(!cs ? RAN_ATTN_SPLITS : cs == 2 ? RAN_ATTN_CLUSTER_2 : cs == 4 ? RAN_ATTN_CLUSTER_4 : cs == 8 ? RAN_ATTN_CLUSTER_8 : RAN_ATTN_CLUSTER_16);
    return ADAMAH_OK;
}

// The embedding kernel takes a full dependency on everything before it (no programmatic launch): later kernels
// of the step rely on the previous step's position update and cache writes being complete before any of them starts.
// Is the stream being recorded, by adam_b200_capture_begin or by a caller that lent it?
static bool stream_recorded() {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(g.stream, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone;
}
static bool pdl_allowed() {
    static const bool allow = !(getenv("ADAM_B200_PDL") && atoi(getenv("ADAM_B200_PDL")) == 0);
    return allow;
}

template <int WT>
static void launch_embed_t(Decoder* D, uint32_t rows, const int32_t* row_seq, const int32_t* row_pos) {
    const adam_b200_decoder_desc& d = D->d;
    static const bool set = carveout_max((const void*)k_embed<WT>, 0);        // once for each of the kernels
    (void)set;
    launch_k(k_embed<WT>, dim3(rows), dim3(256), 0, g.stream, false, D->embd.w, d.n_embd, D->embd.rows, d.emb_scale, D->pos, D->prompt_len, D->prompt_tok,
             d.kv_cap, D->cur_tok, D->hbuf[0], row_seq, row_pos, g.dev_err);
}
static void launch_embed(Decoder* D, uint32_t rows, const int32_t* row_seq, const int32_t* row_pos) {
    switch (D->embd.wtype) {
    case WT_Q4_0: launch_embed_t<WT_Q4_0>(D, rows, row_seq, row_pos); break;
    case WT_Q4_K: launch_embed_t<WT_Q4_K>(D, rows, row_seq, row_pos); break;
    case WT_Q8_0: launch_embed_t<WT_Q8_0>(D, rows, row_seq, row_pos); break;
    default:      launch_embed_t<WT_Q5_0>(D, rows, row_seq, row_pos); break;
    }
    count_launch();
}

static int gemv(const Mat& m, const Mat* m2, GemvArgs a, int B, int epi) {
#ifdef ADAM_B200_STEP_TRACE
    if (g_step_trace && g_step_trace_slot >= 0) { a.trace = g_step_trace + 64 * g_step_trace_slot; g_step_trace_slot = -1; }
#endif
    a.w0 = m.w; if (m2) a.w1 = m2->w;
    a.N = (int)m.rows; a.K = (int)m.cols; a.B = B; a.epi = epi;
    if (B >= TC_MIN_ROWS && (!m2 || m2->wtype == m.wtype)) {
        const uint8_t* t1 = m2 ? m2->tiled : nullptr;
        const GemmRoute route = gemm_route(m.wtype, a, m.tiled, t1, g.maps[m.map_id].wide || (m2 && g.maps[m2->map_id].wide));
        if (route != GEMM_NONE) return launch_gemm(route, m.wtype, m.tiled, t1, a, g.stream);
    }
    if (m.tiled && (!m2 || (m2->tiled && m2->wtype == m.wtype)) && gemv_mma_supports(m.wtype, a))
        return launch_gemv_mma(m.wtype, m.tiled, m2 ? m2->tiled : nullptr, a, g.stream);
    return launch_gemv(m.wtype, a, g.stream);
}

// Enqueue one token step for `batch` sequences on the context stream.  Five
// kernels per layer: QKV GEMV (input RMSNorm and, past layer 0, the previous
// layer's post-FFN norm + residual folded into its prologue), attention (QK-norm,
// RoPE, KV append folded in), o-proj GEMV, gate/up GEMV (post-attention norm +
// residual + FFN norm in the prologue, GeGLU in the epilogue), down GEMV.  The
// residual stream alternates between two buffers because a prologue's CTA 0
// writes the updated stream while the other CTAs still read the old one.
static int enqueue_step_impl(Decoder* D, uint32_t batch, bool with_lm, bool want_logits);
static int enqueue_step(Decoder* D, uint32_t batch, bool with_lm, bool want_logits) {
    static const bool allow = !(getenv("ADAM_B200_PDL") && atoi(getenv("ADAM_B200_PDL")) == 0);
    g.pdl = allow;
    const int rc = enqueue_step_impl(D, batch, with_lm, want_logits);
    g.pdl = false;
    return rc;
}
// One part of a token step.  Parts 2L and 2L+1 are the attention half (embedding for L = 0,
// QKV, attention, o-proj) and the FFN half (gate/up, down) of layer L; part 2*n_layer is the
// LM head, part 2*n_layer + 1 advances the positions.  A tensor-parallel caller all-reduces
// `proj` after every layer part and merges the arg-max pairs after the LM-head part.
// The LM head over rows r0 .. r0 + rows of the step's or chunk's residual stream: winners to tok / val ([rows]), the
// soft-capped logits to `logits` ([rows][n_vocab]) where it is given.
static int enqueue_head(Decoder* D, uint32_t r0, uint32_t rows, float* logits, int32_t* tok, float* val) {
    const adam_b200_decoder_desc& d = D->d;
    const uint32_t E = d.n_embd;
    const Mat& lm = D->output.bound ? D->output : D->embd;
    int rc;
    GemvArgs a = {};
    a.ldx = (int)E; a.eps = d.norm_eps; a.h_in = D->hbuf[1] + (size_t)r0 * E; a.add_src = D->proj + (size_t)r0 * E;
    a.w_post = D->layers[d.n_layer - 1].norm[NORM_POST_FFW]; a.w_pre = D->output_norm; a.h_out = D->hbuf[0] + (size_t)r0 * E;
    a.y = logits; a.ldy = (int)lm.rows; a.softcap = d.final_softcap;
    a.out_tok = tok; a.out_val = val;
    a.w0 = lm.w; a.N = (int)lm.rows; a.K = (int)lm.cols; a.B = (int)rows; a.epi = EPI_ARGMAX;
    D->h_final = 0;
    if (const GemmRoute route = gemm_route(lm.wtype, a, lm.tiled, nullptr, g.maps[lm.map_id].wide)) return launch_gemm(route, lm.wtype, lm.tiled, nullptr, a, g.stream);
    if (wt_is_b8(lm.wtype)) {
        // Q8_0 / Q5_0 LM head: the norm chain, the products and the arg-max as three kernels; the products land in the
        // logits buffer (soft-capped afterwards only when the caller wants them)
        float* y = logits ? logits : D->logits;
        if ((rc = launch_chain_rows(a.h_in, a.add_src, a.w_post, a.w_pre, a.h_out, D->act, (int)E, (int)rows, d.norm_eps, g.stream, g.pdl))) return rc;
        if ((rc = launch_gemv_b8(lm.wtype, lm.w, D->act, (int)E, y, (int)lm.rows, (int)lm.rows, (int)E, (int)rows, g.stream))) return rc;
        return launch_argmax_rows(y, (int)lm.rows, (int)rows, d.final_softcap, logits != nullptr, tok, val, nullptr, g.stream, false);
    }
    if ((rc = argmax_scratch(&a.part_val, &a.part_idx, &a.ticket))) return rc;
    return gemv(lm, nullptr, a, (int)rows, EPI_ARGMAX);
}
// One sequence: matrix `i` that a launch asks into L2 for a kernel that runs two or three launches later.  The layers' products
// are then bound by latency and not by HBM (0.435 -> 0.431 ms per step at the 1B shape); larger matrices stream at its rate anyway.
static void ask_ahead(GemvArgs& a, int i, const Mat& m, const uint8_t* tiled, uint32_t rows) {
    if (!tiled || (m.wtype != WT_Q4_0 && m.wtype != WT_Q4_K)) return;
    const size_t bytes = (size_t)rows / 16 * (m.cols / 64) * mma_tile_bytes(m.wtype);
    if (bytes > (8u << 20)) return;
    a.pf[i] = tiled; a.pf_bytes[i] = (uint32_t)bytes;
}
static uint32_t n_parts(const Decoder* D) { return 2 * D->d.n_layer + 2; }
static int enqueue_part(Decoder* D, uint32_t batch, uint32_t part, bool with_lm, bool want_logits) {
    const adam_b200_decoder_desc& d = D->d;
    const uint32_t E = d.n_embd, q_dim = d.n_head * d.head_dim, k_dim = d.n_head_kv * d.head_dim, qkv_ld = q_dim + 2 * k_dim;
    int rc;
    if (part < 2 * d.n_layer && !(part & 1u)) {
        const uint32_t L = part / 2;
        const Layer& ly = D->layers[L];
        if (L == 0) launch_embed(D, batch, nullptr, nullptr);
        const int cur = L == 0 ? 0 : 1;             // residual stream buffer on entry
        GemvArgs in = {};
        in.ldx = (int)E; in.eps = d.norm_eps; in.h_in = D->hbuf[cur]; in.w_pre = ly.norm[NORM_ATTN];
        if (L > 0) { in.add_src = D->proj; in.w_post = D->layers[L - 1].norm[NORM_POST_FFW]; in.h_out = D->hbuf[cur ^ 1]; }
        in.y = D->qkv; in.ldy = (int)qkv_ld;
        if (batch == 1) {
            ask_ahead(in, 0, ly.m[MAT_GATE], ly.m[MAT_GATE].tiled, d.n_ff);
            ask_ahead(in, 1, ly.m[MAT_UP], ly.m[MAT_UP].tiled, d.n_ff);
            ask_ahead(in, 2, ly.m[MAT_O], ly.m[MAT_O].tiled, E);
        }
        if (ly.qkv_contiguous) {
            Mat qkv = ly.m[MAT_Q]; qkv.rows = qkv_ld; qkv.tiled = ly.qkv_tiled;
#ifdef ADAM_B200_STEP_TRACE
            if (L == g_step_trace_layer) g_step_trace_slot = 0;
#endif
            if ((rc = gemv(qkv, nullptr, in, batch, EPI_STORE))) return rc;
        } else {
            if ((rc = gemv(ly.m[MAT_Q], nullptr, in, batch, EPI_STORE))) return rc;
            GemvArgs in2 = in; in2.h_out = nullptr;
            in2.y = D->qkv + q_dim;
            if ((rc = gemv(ly.m[MAT_K], nullptr, in2, batch, EPI_STORE))) return rc;
            in2.y = D->qkv + q_dim + k_dim;
            if ((rc = gemv(ly.m[MAT_V], nullptr, in2, batch, EPI_STORE))) return rc;
        }
        rc = d.kv_dtype == 1 ? launch_attn_t<__half>(D, L, batch) : launch_attn_t<float>(D, L, batch);
        if (rc) return rc;
        GemvArgs o = {};
        o.x = D->attn_out; o.ldx = (int)q_dim; o.y = D->proj; o.ldy = (int)E;
        if (batch == 1) {
            ask_ahead(o, 0, ly.m[MAT_DOWN], ly.m[MAT_DOWN].tiled, E);
            if (L + 1 < d.n_layer) ask_ahead(o, 1, D->layers[L + 1].m[MAT_Q], D->layers[L + 1].qkv_tiled, qkv_ld);
        }
#ifdef ADAM_B200_STEP_TRACE
        if (L == g_step_trace_layer) g_step_trace_slot = 1;
#endif
        if ((rc = gemv(ly.m[MAT_O], nullptr, o, batch, EPI_STORE))) return rc;
    } else if (part < 2 * d.n_layer) {
        const Layer& ly = D->layers[part / 2];
        // the stream is in buffer 0 here for every layer (layer 0 never flipped, the others flipped in their QKV)
        GemvArgs gu = {};
        gu.ldx = (int)E; gu.eps = d.norm_eps; gu.h_in = D->hbuf[0]; gu.add_src = D->proj; gu.w_post = ly.norm[NORM_POST_ATTN];
        gu.w_pre = ly.norm[NORM_FFN]; gu.h_out = D->hbuf[1]; gu.y = D->act; gu.ldy = (int)d.n_ff;
#ifdef ADAM_B200_STEP_TRACE
        if (part / 2 == g_step_trace_layer) g_step_trace_slot = 2;
#endif
        if ((rc = gemv(ly.m[MAT_GATE], &ly.m[MAT_UP], gu, batch, d.ffn_act == 0 ? EPI_GEGLU : EPI_SWIGLU))) return rc;
        GemvArgs dn = {};
        dn.x = D->act; dn.ldx = (int)d.n_ff; dn.y = D->proj; dn.ldy = (int)E;
#ifdef ADAM_B200_STEP_TRACE
        if (part / 2 == g_step_trace_layer) g_step_trace_slot = 3;
#endif
        if ((rc = gemv(ly.m[MAT_DOWN], nullptr, dn, batch, EPI_STORE))) return rc;
    } else if (part == 2 * d.n_layer) {
        if (with_lm) {
            if ((rc = enqueue_head(D, 0, batch, want_logits ? D->logits : nullptr, D->cur_tok, D->cur_val))) return rc;
        }
    } else {
        static bool set = false;
        if (!set) { carveout_max((const void*)k_advance, 0); set = true; }
        launch_k(k_advance, dim3((batch + 63) / 64), dim3(64), 0, g.stream, g.pdl, D->pos, D->cur_tok, D->gen_log, d.kv_cap, batch, with_lm ? 1 : 0);
        count_launch();
    }
    return check_launch("decoder step");
}

static int enqueue_step_impl(Decoder* D, uint32_t batch, bool with_lm, bool want_logits) {
    for (uint32_t part = 0; part < n_parts(D); ++part) {
        const int rc = enqueue_part(D, batch, part, with_lm, want_logits);
        if (rc) return rc;
    }
    return ADAMAH_OK;
}

static int validate_bound(Decoder* D) {
    const adam_b200_decoder_desc& d = D->d;
    if (!D->embd.bound) return fail(ADAMAH_ERR_INVALID, "decoder: token_embd is not bound");
    if (!D->output_norm) return fail(ADAMAH_ERR_INVALID, "decoder: output_norm is not bound");
    if (!D->rope_cos[0] || !D->rope_cos[1]) return fail(ADAMAH_ERR_INVALID, "decoder: rotary tables are not set");
    for (uint32_t L = 0; L < d.n_layer; ++L) {
        Layer& ly = D->layers[L];
        for (int k = 0; k < 7; ++k) if (!ly.m[k].bound) return fail(ADAMAH_ERR_INVALID, "decoder: layer %u matrix %d is not bound", L, k);
        if (!ly.norm[NORM_ATTN] || !ly.norm[NORM_FFN]) return fail(ADAMAH_ERR_INVALID, "decoder: layer %u pre-norms are not bound", L);
        // q, k, v stored back to back -> one wider GEMV (adam/models/engine.py:1612-1661)
        const Mat &q = ly.m[MAT_Q], &k = ly.m[MAT_K], &v = ly.m[MAT_V];
        const size_t ipr = q.cols / (q.wtype == WT_Q4_0 ? 32 : 256) * (q.wtype == WT_Q4_0 ? 1 : 9);   // uint4 per row
        ly.qkv_contiguous = q.wtype == k.wtype && k.wtype == v.wtype && k.w.q == q.w.q + (size_t)q.rows * ipr &&
                            v.w.q == k.w.q + (size_t)k.rows * ipr;
        if (ly.qkv_contiguous && D->use_tiles && !ly.qkv_tiled) {
            const uint32_t rows = q.rows + k.rows + v.rows;
            if (rows % 16 == 0 && q.cols % 64 == 0 && tile_tensor(q.map_id, q.elem_off, rows, q.cols) == ADAMAH_OK)
                ly.qkv_tiled = (const uint8_t*)find_tiled(q.map_id, q.elem_off, rows, q.cols);
        }
    }
    return ADAMAH_OK;
}

// ---- single-launch token kernel: eligibility, work split, buffers -----------------------------

// Spread one product over the grid (see TkPhase): the estimate is the number of tile pairs the busiest
// warp walks plus fixed costs per row group, per K split inside the CTA and per K split across CTAs.
static bool tk_pick_phase(TkPhase& P, int n_rg, int pairs, int nm, int grid, int max_cpr) {
    double best = 1e300;
    bool found = false;
    for (int cpr = 1; cpr <= max_cpr; ++cpr) {
        for (int KS = 1; KS <= TK_NW; ++KS) {
            const int RG = TK_NW / KS;
            if (RG < 1 || KS * cpr > pairs) continue;
            if (KS > 1 && RG > 15) continue;                   // named barriers 1..15
            const int n_sets = (n_rg + RG - 1) / RG;
            int G = grid / cpr;
            if (G > n_sets) G = n_sets;
            if (G < 1) continue;
            const int sets_per_cta = (n_sets + G - 1) / G;
            const int per_warp = (pairs + KS * cpr - 1) / (KS * cpr);
            const double cost = (double)sets_per_cta * (per_warp * nm + 2.0) + (KS > 1 ? 1.0 : 0.0) + (cpr > 1 ? 1.0 : 0.0) + 0.01 * KS;
            if (cost < best) { best = cost; P.n_rg = n_rg; P.pairs = pairs; P.RG = RG; P.KS = KS; P.cpr = cpr; P.G = G; found = true; }
        }
    }
    return found;
}

static int prepare_token_kernel(Decoder* D) {
    const adam_b200_decoder_desc& d = D->d;
    D->tk_state = -1;
    static const bool allow = !(getenv("ADAM_B200_TOKEN_KERNEL") && atoi(getenv("ADAM_B200_TOKEN_KERNEL")) == 0);
    if (!allow || !D->use_tiles || d.tp_size > 1) return ADAMAH_OK;
    int coop = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, g.device);
    if (!coop) return ADAMAH_OK;
    const uint32_t E = d.n_embd, q_dim = d.n_head * d.head_dim, k_dim = d.n_head_kv * d.head_dim, FF = d.n_ff;
    if (!token_supported_hd((int)d.head_dim) || d.n_layer > (uint32_t)TK_MAX_LAYERS || d.page_size % 8) return ADAMAH_OK;
    if (E % 64 || q_dim % 64 || FF % 64 || E > (uint32_t)TK_MAX_E || q_dim > 2u * TK_THREADS * 4u) return ADAMAH_OK;
    const Mat& lm = D->output.bound ? D->output : D->embd;
    if (!lm.tiled || lm.rows % 16) return ADAMAH_OK;
    if (wt_is_b8(D->embd.wtype) || wt_is_b8(lm.wtype)) return ADAMAH_OK;     // Q8_0 / Q5_0 tables run on the chain of kernels
    const int wt = lm.wtype;
    if (wt == WT_Q4_K && (E % 256 || q_dim % 256 || FF % 256)) return ADAMAH_OK;
    auto al16 = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
    if (!al16(D->output_norm)) return ADAMAH_OK;
    for (uint32_t L = 0; L < d.n_layer; ++L) {
        const Layer& ly = D->layers[L];
        if (!ly.qkv_contiguous || !ly.qkv_tiled || !ly.m[MAT_O].tiled || !ly.m[MAT_GATE].tiled || !ly.m[MAT_UP].tiled || !ly.m[MAT_DOWN].tiled) return ADAMAH_OK;
        for (int k : {MAT_Q, MAT_O, MAT_GATE, MAT_UP, MAT_DOWN}) if (ly.m[k].wtype != wt) return ADAMAH_OK;
        for (int k : {NORM_ATTN, NORM_POST_ATTN, NORM_FFN, NORM_POST_FFW}) if (!al16(ly.norm[k])) return ADAMAH_OK;
    }
    TkArgs a = {};
    // the gate/up product decides the grid: every CTA must take part in it (it is what makes each CTA's
    // reads a precondition of the next layer, see token_kernel.cuh), so a product with fewer sets than SMs
    // shrinks the grid instead
    int grid = g.sm_count;
    {
        TkPhase best = {}; double best_cost = 1e300; int best_grid = 0;
        for (int KS = 1; KS <= TK_NW; ++KS) {
            const int RG = TK_NW / KS, pairs = (int)E / 64, n_rg = (int)FF / 16;
            if (KS > pairs || (KS > 1 && RG > 15)) continue;
            const int n_sets = (n_rg + RG - 1) / RG;
            const int gr = n_sets < g.sm_count ? n_sets : g.sm_count;
            const int sets_per_cta = (n_sets + gr - 1) / gr;
            const int per_warp = (pairs + KS - 1) / KS;
            // idle SMs cost LM-head bandwidth: weigh them in
            const double cost = ((double)sets_per_cta * (per_warp * 2 + 2.0) + (KS > 1 ? 1.0 : 0.0) + 0.01 * KS) * (1.0 + 2.0 * (g.sm_count - gr) / (double)g.sm_count);
            if (cost < best_cost) { best_cost = cost; best_grid = gr; best.n_rg = n_rg; best.pairs = pairs; best.RG = RG; best.KS = KS; best.cpr = 1; best.G = gr; }
        }
        if (best_grid < 1) return ADAMAH_OK;
        grid = best_grid;
        a.ph[TK_GU] = best;
    }
    if (grid < (int)d.n_head) return ADAMAH_OK;
    if (!tk_pick_phase(a.ph[TK_QKV], (int)(q_dim + 2 * k_dim) / 16, (int)E / 64, 1, grid, 1)) return ADAMAH_OK;
    if (!tk_pick_phase(a.ph[TK_O], (int)E / 16, (int)q_dim / 64, 1, grid, 1)) return ADAMAH_OK;
    if (!tk_pick_phase(a.ph[TK_DOWN], (int)E / 16, (int)FF / 64, 1, grid, 2)) return ADAMAH_OK;
    if (!tk_pick_phase(a.ph[TK_LM], (int)lm.rows / 16, (int)E / 64, 1, grid, 1)) return ADAMAH_OK;
    // attention CTAs per query head: what the grid offers, at most 8192 gathered values per o-proj CTA
    a.s_max = grid / (int)d.n_head;
    if (a.s_max > TK_MAX_SPLITS) a.s_max = TK_MAX_SPLITS;
    if (a.s_max > 4) a.s_max = 4;                         // the o-proj merges up to four splits in one poll
    {   // per-warp staging regions of the o-proj and down-proj inputs: the widest K slice of a warp
        int np = 0;
        for (int ph : {TK_O, TK_DOWN}) {
            const TkPhase& P = a.ph[ph];
            const int n = (P.pairs + P.KS * P.cpr - 1) / (P.KS * P.cpr);
            if (n > np) np = n;
        }
        if (np > 8) return ADAMAH_OK;                     // a warp's slice must fit sixteen loads per lane
        a.wu_cap = 2 * np;
    }
    a.n_layer = (int)d.n_layer; a.E = (int)E; a.q_dim = (int)q_dim; a.k_dim = (int)k_dim; a.FF = (int)FF; a.V = (int)lm.rows;
    a.H = (int)d.n_head; a.KV = (int)d.n_head_kv;
    a.embd = D->embd.w; a.embd_wt = D->embd.wtype; a.emb_scale = d.emb_scale;
    a.lm_tiled = lm.tiled; a.out_norm = D->output_norm;
    a.eps = d.norm_eps; a.attn_scale = d.attn_scale; a.attn_cap = d.attn_softcap; a.final_cap = d.final_softcap; a.act = (int)d.ffn_act;
    a.pos = D->pos; a.cur_tok = D->cur_tok; a.cur_val = D->cur_val; a.prompt_len = D->prompt_len; a.prompt_tok = D->prompt_tok;
    a.gen_log = D->gen_log; a.log_ld = d.kv_cap;
    a.block_table = D->block_table;
    a.geo = KvGeom{d.n_layer, d.n_head_kv, d.head_dim, d.page_size, D->max_pages_per_seq, D->page_elems};
    a.kv_pool = D->kv_pool;
    for (int w = 0; w < 2; ++w) { a.cos_t[w] = D->rope_cos[w]; a.sin_t[w] = D->rope_sin[w]; }
    a.n_pos = D->rope_pos[0] < D->rope_pos[1] ? D->rope_pos[0] : D->rope_pos[1];
    a.h_out = D->hbuf[0];
    a.err = g.dev_err;
    if (token_smem_bytes(wt, a, (int)d.head_dim) > 220 * 1024) return ADAMAH_OK;
    // device memory: layer table, exchange buffers (two halves each), step counter and the sticky word
    std::vector<TkLayer> hl(d.n_layer);
    for (uint32_t L = 0; L < d.n_layer; ++L) {
        const Layer& ly = D->layers[L];
        TkLayer& t = hl[L];
        t.w[0] = ly.qkv_tiled; t.w[1] = ly.m[MAT_O].tiled; t.w[2] = ly.m[MAT_GATE].tiled; t.w[3] = ly.m[MAT_UP].tiled; t.w[4] = ly.m[MAT_DOWN].tiled;
        t.norm[TKN_ATTN] = ly.norm[NORM_ATTN]; t.norm[TKN_POST_ATTN] = ly.norm[NORM_POST_ATTN]; t.norm[TKN_FFN] = ly.norm[NORM_FFN];
        t.norm[TKN_POST_FFW] = ly.norm[NORM_POST_FFW]; t.norm[TKN_Q] = ly.norm[NORM_Q]; t.norm[TKN_K] = ly.norm[NORM_K];
        t.window = ((d.flags & 1u) && d.sliding_window > 0 && !is_global_layer(d, L)) ? d.sliding_window : 0;
        t.rope = is_global_layer(d, L) ? 1u : 0u;
    }
    const size_t sizes[9] = {
        hl.size() * sizeof(TkLayer),
        2 * (size_t)(q_dim + 2 * k_dim) * 8,
        2 * (size_t)d.n_head * a.s_max * (d.head_dim + 2) * 8,
        2 * (size_t)a.ph[TK_O].cpr * E * 8,
        2 * (size_t)FF * 8,
        2 * (size_t)a.ph[TK_DOWN].cpr * E * 8,
        2 * (size_t)grid * 8,
        4, 4};
    for (int i = 0; i < 9; ++i) {
        if (cudaMalloc(&D->tk_mem[i], sizes[i]) != cudaSuccess) {
            cudaGetLastError();
            for (void*& m : D->tk_mem) { if (m) cudaFree(m); m = nullptr; }
            return fail(ADAMAH_ERR_MEMORY, "decoder: out of device memory for the token kernel's buffers");
        }
        cudaMemsetAsync(D->tk_mem[i], 0, sizes[i], g.stream);
    }
    cudaMemcpyAsync(D->tk_mem[0], hl.data(), sizes[0], cudaMemcpyHostToDevice, g.stream);
    cudaStreamSynchronize(g.stream);
    a.layers = (const TkLayer*)D->tk_mem[0];
    a.x_qkv = (uint2*)D->tk_mem[1]; a.x_att = (uint2*)D->tk_mem[2]; a.x_po = (uint2*)D->tk_mem[3]; a.x_act = (uint2*)D->tk_mem[4];
    a.x_pd = (uint2*)D->tk_mem[5]; a.x_amax = (uint2*)D->tk_mem[6]; a.seq = (uint32_t*)D->tk_mem[7]; a.dead = (uint32_t*)D->tk_mem[8];
    D->tk = a; D->tk_grid = grid; D->tk_wt = wt;
    D->tk_state = 1;
    return ADAMAH_OK;
}

static long long* g_tk_trace = nullptr;     // diagnostics buffer (device), see adam_b200_decoder_token_trace
static int g_tk_trace_layer = 0, g_tk_trace_phase = 2;

// One token of the single active sequence as one launch.
static int enqueue_token(Decoder* D, bool with_lm, bool want_logits) {
    TkArgs a = D->tk;
    a.trace = g_tk_trace; a.trace_layer = g_tk_trace_layer; a.trace_phase = g_tk_trace_phase;
    a.with_lm = with_lm ? 1 : 0;
    a.logits = want_logits ? D->logits : nullptr;
    const int rc = launch_token(D->tk_wt, D->d.kv_dtype == 1, (int)D->d.head_dim, a, D->tk_grid, g.stream);
    if (rc == ADAMAH_OK && with_lm) D->h_final = 0;
    return rc;
}

}  // namespace ab

using namespace ab;

extern "C" int adam_b200_decoder_create(const adam_b200_decoder_desc* desc, uint32_t* id_out) {
    if (!ready()) return ADAMAH_ERR_INVALID;
    if (!desc || !id_out) return fail(ADAMAH_ERR_INVALID, "decoder_create: null argument");
    adam_b200_decoder_desc d = *desc;
    if (!d.n_layer || !d.n_embd || !d.n_head || !d.n_head_kv || !d.head_dim || !d.n_ff || !d.n_vocab || !d.max_batch || !d.kv_cap)
        return fail(ADAMAH_ERR_INVALID, "decoder_create: zero dimension");
    if (d.n_head % d.n_head_kv || d.n_head / d.n_head_kv > 8) return fail(ADAMAH_ERR_INVALID, "decoder_create: unsupported GQA group");
    if (d.head_dim != 32 && d.head_dim != 64 && d.head_dim != 128 && d.head_dim != 256)
        return fail(ADAMAH_ERR_INVALID, "decoder_create: head_dim must be 32, 64, 128 or 256");
    if (d.n_embd % 32 || d.n_ff % 32) return fail(ADAMAH_ERR_INVALID, "decoder_create: widths must be multiples of 32");
    if (d.kv_dtype > 1) return fail(ADAMAH_ERR_INVALID, "decoder_create: kv_dtype must be 0 (f32) or 1 (f16)");
    if (d.page_size == 0) d.page_size = 64;
    if (d.attn_scale == 0.f) d.attn_scale = 1.0f / sqrtf((float)d.head_dim);
    uint32_t id = MAX_DECODERS;
    for (uint32_t i = 0; i < MAX_DECODERS; ++i) if (!g_dec[i]) { id = i; break; }
    if (id == MAX_DECODERS) return fail(ADAMAH_ERR_MEMORY, "decoder table full");
    Decoder* D = new Decoder();
    D->d = d;
    D->use_tiles = !(d.flags & 2u);
    D->layers.resize(d.n_layer);
    D->max_pages_per_seq = (d.kv_cap + d.page_size - 1) / d.page_size;
    D->n_pages = d.n_pages ? d.n_pages : D->max_pages_per_seq * d.max_batch;
    D->d.n_pages = D->n_pages;
    D->page_elems = (size_t)d.n_layer * 2 * d.n_head_kv * d.page_size * d.head_dim;
    D->n_splits = (d.kv_cap + ATTN_SPLIT - 1) / ATTN_SPLIT;      // ATTN_SPLIT = ATTN_CP * ATTN_CHUNKS_PER_CTA
    if (D->n_splits > ATTN_MAX_SPLITS) D->n_splits = ATTN_MAX_SPLITS;
    const uint64_t most = (uint64_t)d.max_batch * d.kv_cap;     // no more prompt rows than that exist
    const uint32_t chunk = prefill_rows(d.n_embd);
    D->rows_cap = (uint32_t)(most < chunk ? (most > 64 ? most : 64) : chunk);
    if (D->rows_cap < d.max_batch) D->rows_cap = d.max_batch;
    const size_t B = d.max_batch, E = d.n_embd, q_dim = (size_t)d.n_head * d.head_dim, k_dim = (size_t)d.n_head_kv * d.head_dim;
    const uint32_t gs = d.n_head / d.n_head_kv;
    g_dec[id] = D;
#define DALLOC(p, bytes) do { cudaError_t e__ = cudaMalloc((void**)&(p), (bytes)); if (e__ != cudaSuccess) { destroy(D); g_dec[id] = nullptr; \
        return fail(ADAMAH_ERR_MEMORY, "decoder_create: cudaMalloc(%zu) failed: %s", (size_t)(bytes), cudaGetErrorString(e__)); } } while (0)
    DALLOC(D->pos, B * 4); DALLOC(D->cur_tok, B * 4); DALLOC(D->cur_val, B * 4); DALLOC(D->prompt_len, B * 4);
    DALLOC(D->prompt_tok, B * d.kv_cap * 4); DALLOC(D->gen_log, B * d.kv_cap * 4);
    DALLOC(D->block_table, B * D->max_pages_per_seq * 4);
    DALLOC(D->kv_pool, (size_t)D->n_pages * D->page_elems * kv_elem_size(d));
    DALLOC(D->logits, B * (size_t)d.n_vocab * 4);
    DALLOC(D->part_o, B * d.n_head_kv * D->n_splits * gs * d.head_dim * 4);
    DALLOC(D->part_ml, B * d.n_head_kv * D->n_splits * gs * 2 * 4);
    DALLOC(D->attn_ticket, B * d.n_head * 4);
    // Buffers of a chunk's rows: 205 MB at the 27B shape and 1024 rows, fewer rows where that much is not left.
    struct { void** p; size_t row; } const bufs[7] = {{(void**)&D->hbuf[0], E * 4}, {(void**)&D->hbuf[1], E * 4}, {(void**)&D->qkv, (q_dim + 2 * k_dim) * 4},
        {(void**)&D->attn_out, q_dim * 4}, {(void**)&D->proj, E * 4}, {(void**)&D->act, (size_t)d.n_ff * 4}, {(void**)&D->even_plan, 8 + sizeof(AttnTile)}};
    const uint32_t fewest = std::max(64u, d.max_batch);
    for (;;) {
        int n = 0;
        while (n < 7 && cudaMalloc(bufs[n].p, bufs[n].row * D->rows_cap) == cudaSuccess) ++n;
        if (n == 7) break;
        cudaGetLastError();
        for (int i = 0; i < 7; ++i) { if (i < n) cudaFree(*bufs[i].p); *bufs[i].p = nullptr; }
        if (D->rows_cap == fewest) {
            const uint32_t rows = D->rows_cap;
            destroy(D); g_dec[id] = nullptr;
            return fail(ADAMAH_ERR_MEMORY, "decoder_create: out of device memory for %u rows of activations", rows);
        }
        D->rows_cap = std::max(fewest, D->rows_cap / 2);
    }
#undef DALLOC
    // workspace of the many-row GEMM (without it those rows run on the GEMV kernels)
    gemm_tc_prepare((int)D->rows_cap, (int)std::max(std::max((size_t)d.n_ff, E), q_dim));
    cudaMemsetAsync(D->attn_ticket, 0, B * d.n_head * 4, g.stream);
    cudaMemsetAsync(D->even_plan, 0, D->rows_cap * (8 + sizeof(AttnTile)), g.stream);
    cudaMemsetAsync(D->pos, 0, B * 4, g.stream);
    cudaMemsetAsync(D->cur_tok, 0, B * 4, g.stream);
    cudaMemsetAsync(D->cur_val, 0, B * 4, g.stream);
    cudaMemsetAsync(D->prompt_len, 0, B * 4, g.stream);
    cudaMemsetAsync(D->kv_pool, 0, (size_t)D->n_pages * D->page_elems * kv_elem_size(d), g.stream);
    k_fill_i32<<<(unsigned)((B * D->max_pages_per_seq + 255) / 256), 256, 0, g.stream>>>(D->block_table, -1, B * D->max_pages_per_seq);
    cudaStreamSynchronize(g.stream);
    for (uint32_t p = 0; p < D->n_pages; ++p) D->free_pages.push_back(D->n_pages - 1 - p);
    *id_out = id;
    return ADAMAH_OK;
}

extern "C" int adam_b200_decoder_destroy(uint32_t id) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    destroy(D);
    g_dec[id] = nullptr;
    return ADAMAH_OK;
}

extern "C" int adam_b200_decoder_bind_matrix(uint32_t id, uint32_t layer, uint32_t kind, uint32_t map_wt, uint64_t elem_off,
                                             uint32_t rows, uint32_t cols) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    Map* m = get_map(map_wt);
    if (!m) return ADAMAH_ERR_NOT_FOUND;
    if (kind >= MAT_KINDS || (kind < MAT_EMBD && layer >= D->d.n_layer)) return fail(ADAMAH_ERR_INVALID, "bind_matrix: bad layer/kind");
    const adam_b200_decoder_desc& d = D->d;
    const uint32_t q_dim = d.n_head * d.head_dim, k_dim = d.n_head_kv * d.head_dim;
    const uint32_t want_r[MAT_KINDS] = {q_dim, k_dim, k_dim, d.n_embd, d.n_ff, d.n_ff, d.n_embd, d.n_vocab, d.n_vocab};
    const uint32_t want_c[MAT_KINDS] = {d.n_embd, d.n_embd, d.n_embd, q_dim, d.n_embd, d.n_embd, d.n_ff, d.n_embd, d.n_embd};
    // A tensor-parallel shard looks tokens up in the whole embedding table while its LM head
    // (n_vocab) covers only the shard's vocabulary rows.
    const bool full_embd = kind == MAT_EMBD && d.tp_size > 1 && rows >= d.n_vocab && cols == d.n_embd;
    if (!full_embd && (rows != want_r[kind] || cols != want_c[kind]))
        return fail(ADAMAH_ERR_INVALID, "bind_matrix: kind %u expects [%u,%u], got [%u,%u]", kind, want_r[kind], want_c[kind], rows, cols);
    Mat mt = {};
    int rc = weight_ref(m, elem_off, (uint64_t)rows * cols, &mt.wtype, &mt.w);
    if (rc) return rc;
    if (mt.wtype == WT_Q4_K && cols % 256) return fail(ADAMAH_ERR_INVALID, "bind_matrix: Q4_K needs cols %% 256 == 0");
    if (wt_is_b8(mt.wtype) && ((kind != MAT_EMBD && kind != MAT_OUTPUT) || d.tp_size > 1 || d.n_ff < d.n_embd))
        return fail(ADAMAH_ERR_INVALID, "bind_matrix: Q8_0 / Q5_0 blocks are accepted for token_embd and output, on one GPU, with n_ff >= n_embd");
    mt.rows = rows; mt.cols = cols; mt.bound = true; mt.map_id = map_wt; mt.elem_off = elem_off; mt.tiled = nullptr;
    // q, k, v get one combined tiled copy later (validate_bound); token_embd is tiled only as the LM head
    const bool solo = kind == MAT_O || kind == MAT_GATE || kind == MAT_UP || kind == MAT_DOWN || kind == MAT_OUTPUT || kind == MAT_EMBD;
    if (D->use_tiles && solo && !wt_is_b8(mt.wtype) && rows % 16 == 0 && cols % 64 == 0) {
        if (tile_tensor(map_wt, elem_off, rows, cols) == ADAMAH_OK) mt.tiled = (const uint8_t*)find_tiled(map_wt, elem_off, rows, cols);
    }
    if (kind == MAT_EMBD) D->embd = mt; else if (kind == MAT_OUTPUT) D->output = mt; else D->layers[layer].m[kind] = mt;
    free_graphs(D);
    return ADAMAH_OK;
}

extern "C" int adam_b200_decoder_bind_norm(uint32_t id, uint32_t layer, uint32_t kind, uint32_t map_f32, uint64_t elem_off, uint32_t n) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    Map* m = get_map(map_f32);
    if (!m) return ADAMAH_ERR_NOT_FOUND;
    if (m->dtype != ADAMAH_DTYPE_F32) return fail(ADAMAH_ERR_INVALID, "bind_norm: map %u is not float32", map_f32);
    if (kind >= NORM_KINDS || (kind != NORM_OUTPUT && layer >= D->d.n_layer)) return fail(ADAMAH_ERR_INVALID, "bind_norm: bad layer/kind");
    const uint32_t want = (kind == NORM_Q || kind == NORM_K) ? D->d.head_dim : D->d.n_embd;
    if (n != want) return fail(ADAMAH_ERR_INVALID, "bind_norm: kind %u expects %u weights, got %u", kind, want, n);
    if (elem_off + n > m->n_elems) return fail(ADAMAH_ERR_INVALID, "bind_norm: range beyond map %u", map_f32);
    const float* p = (const float*)m->buf + elem_off;
    if (kind == NORM_OUTPUT) D->output_norm = p; else D->layers[layer].norm[kind] = p;
    free_graphs(D);
    return ADAMAH_OK;
}

extern "C" int adam_b200_decoder_set_rope(uint32_t id, uint32_t which, const float* cos_t, const float* sin_t, uint32_t n_pos, uint32_t half) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (which > 1 || !cos_t || !sin_t || half != D->d.head_dim / 2 || n_pos < D->d.kv_cap)
        return fail(ADAMAH_ERR_INVALID, "set_rope: need which in {0,1}, half == head_dim/2 and n_pos >= kv_cap");
    cudaStreamSynchronize(g.stream);
    cudaFree(D->rope_cos[which]); cudaFree(D->rope_sin[which]);
    D->rope_cos[which] = D->rope_sin[which] = nullptr;
    const size_t bytes = (size_t)n_pos * half * 4;
    DCU(cudaMalloc((void**)&D->rope_cos[which], bytes));
    DCU(cudaMalloc((void**)&D->rope_sin[which], bytes));
    DCU(cudaMemcpy(D->rope_cos[which], cos_t, bytes, cudaMemcpyHostToDevice));
    DCU(cudaMemcpy(D->rope_sin[which], sin_t, bytes, cudaMemcpyHostToDevice));
    D->rope_pos[which] = n_pos;
    free_graphs(D);
    return ADAMAH_OK;
}

// Start `batch` sequences: prompts (ragged, concatenated) are copied to the
// device, positions reset to 0, and pages reserved for `reserve[b]` tokens each.
extern "C" int adam_b200_decoder_begin(uint32_t id, uint32_t batch, const int32_t* prompt_tokens, const uint32_t* prompt_lens,
                                       const uint32_t* reserve) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    const adam_b200_decoder_desc& d = D->d;
    if (batch == 0 || batch > d.max_batch || !prompt_lens || !reserve) return fail(ADAMAH_ERR_INVALID, "decoder_begin: bad batch");
    if (capturing()) return fail(ADAMAH_ERR_INVALID, "decoder_begin: not allowed while a graph is being captured");
    int rc = validate_bound(D);
    if (rc) return rc;
    DCU(cudaStreamSynchronize(g.stream));
    // return all pages, then reserve
    D->free_pages.clear();
    for (uint32_t p = 0; p < D->n_pages; ++p) D->free_pages.push_back(D->n_pages - 1 - p);
    std::vector<int32_t> bt((size_t)d.max_batch * D->max_pages_per_seq, -1), plen(d.max_batch, 0), ptok((size_t)batch * d.kv_cap, 0);
    size_t off = 0;
    for (uint32_t b = 0; b < batch; ++b) {
        if (prompt_lens[b] == 0 || prompt_lens[b] > d.kv_cap || reserve[b] < prompt_lens[b] || reserve[b] > d.kv_cap)
            return fail(ADAMAH_ERR_INVALID, "decoder_begin: sequence %u needs 1 <= prompt <= reserve <= kv_cap (%u)", b, d.kv_cap);
        const uint32_t need = (reserve[b] + d.page_size - 1) / d.page_size;
        if (need > D->free_pages.size()) return fail(ADAMAH_ERR_MEMORY, "decoder_begin: KV page pool exhausted (%u pages)", D->n_pages);
        for (uint32_t p = 0; p < need; ++p) { bt[(size_t)b * D->max_pages_per_seq + p] = (int32_t)D->free_pages.back(); D->free_pages.pop_back(); }
        plen[b] = (int32_t)prompt_lens[b];
        if (!prompt_tokens) return fail(ADAMAH_ERR_INVALID, "decoder_begin: null prompt");
        for (uint32_t t = 0; t < prompt_lens[b]; ++t) {
            const int32_t tk = prompt_tokens[off + t];
            if (tk < 0 || (uint32_t)tk >= D->embd.rows) return fail(ADAMAH_ERR_INVALID, "decoder_begin: token id %d outside the vocabulary", tk);
            ptok[(size_t)b * d.kv_cap + t] = tk;
        }
        off += prompt_lens[b];
    }
    DCU(cudaMemcpyAsync(D->block_table, bt.data(), bt.size() * 4, cudaMemcpyHostToDevice, g.stream));
    DCU(cudaMemcpyAsync(D->prompt_len, plen.data(), plen.size() * 4, cudaMemcpyHostToDevice, g.stream));
    DCU(cudaMemcpyAsync(D->prompt_tok, ptok.data(), ptok.size() * 4, cudaMemcpyHostToDevice, g.stream));
    DCU(cudaMemsetAsync(D->pos, 0, (size_t)d.max_batch * 4, g.stream));
    DCU(cudaMemsetAsync(D->cur_tok, 0, (size_t)d.max_batch * 4, g.stream));
    DCU(cudaMemsetAsync(D->gen_log, 0xFF, (size_t)d.max_batch * d.kv_cap * 4, g.stream));
    if (D->tk_state == 1) DCU(cudaMemsetAsync(D->tk_mem[8], 0, 4, g.stream));
    DCU(cudaStreamSynchronize(g.stream));
    D->batch = batch;
    D->hpos.assign(batch, 0);
    D->hplen.assign(prompt_lens, prompt_lens + batch);
    D->hres.assign(reserve, reserve + batch);
    D->hbt = bt;
    return ADAMAH_OK;
}

// Continue the single active sequence with a new prompt whose first n_reuse tokens are the ones
// whose keys and values are already in the cache (role of generate(reuse_prefix=..),
// adam/models/engine.py:3815-3833): positions restart at n_reuse, the cache pages are kept and
// extended to `reserve` tokens.  n_reuse must not exceed the positions computed so far.
extern "C" int adam_b200_decoder_continue(uint32_t id, const int32_t* prompt_tokens, uint32_t prompt_len, uint32_t reserve, uint32_t n_reuse) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    const adam_b200_decoder_desc& d = D->d;
    if (D->batch != 1) return fail(ADAMAH_ERR_INVALID, "decoder_continue: needs one active sequence");
    if (capturing()) return fail(ADAMAH_ERR_INVALID, "decoder_continue: not allowed while a graph is being captured");
    if (!prompt_tokens || prompt_len == 0 || prompt_len > d.kv_cap || reserve < prompt_len || reserve > d.kv_cap)
        return fail(ADAMAH_ERR_INVALID, "decoder_continue: needs 1 <= prompt <= reserve <= kv_cap (%u)", d.kv_cap);
    if (n_reuse >= prompt_len || n_reuse > D->hpos[0])
        return fail(ADAMAH_ERR_INVALID, "decoder_continue: %u reused positions, but %u are cached and the prompt has %u tokens", n_reuse, D->hpos[0], prompt_len);
    DCU(cudaStreamSynchronize(g.stream));
    std::vector<int32_t> ptok(prompt_len);
    for (uint32_t t = 0; t < prompt_len; ++t) {
        if (prompt_tokens[t] < 0 || (uint32_t)prompt_tokens[t] >= D->embd.rows) return fail(ADAMAH_ERR_INVALID, "decoder_continue: token id %d outside the vocabulary", prompt_tokens[t]);
        ptok[t] = prompt_tokens[t];
    }
    uint32_t have = 0;
    while (have < D->max_pages_per_seq && D->hbt[have] >= 0) ++have;
    const uint32_t need = (reserve + d.page_size - 1) / d.page_size;
    if (need > have) {
        if (need - have > D->free_pages.size()) return fail(ADAMAH_ERR_MEMORY, "decoder_continue: KV page pool exhausted (%u pages)", D->n_pages);
        for (uint32_t p = have; p < need; ++p) { D->hbt[p] = (int32_t)D->free_pages.back(); D->free_pages.pop_back(); }
        DCU(cudaMemcpyAsync(D->block_table, D->hbt.data(), (size_t)D->max_pages_per_seq * 4, cudaMemcpyHostToDevice, g.stream));
    }
    const int32_t plen = (int32_t)prompt_len, p0 = (int32_t)n_reuse;
    DCU(cudaMemcpyAsync(D->prompt_len, &plen, 4, cudaMemcpyHostToDevice, g.stream));
    DCU(cudaMemcpyAsync(D->prompt_tok, ptok.data(), (size_t)prompt_len * 4, cudaMemcpyHostToDevice, g.stream));
    DCU(cudaMemcpyAsync(D->pos, &p0, 4, cudaMemcpyHostToDevice, g.stream));
    DCU(cudaMemsetAsync(D->cur_tok, 0, 4, g.stream));
    DCU(cudaMemsetAsync(D->gen_log, 0xFF, (size_t)d.kv_cap * 4, g.stream));
    if (D->tk_state == 1) DCU(cudaMemsetAsync(D->tk_mem[8], 0, 4, g.stream));
    DCU(cudaStreamSynchronize(g.stream));
    D->hpos[0] = n_reuse;
    D->hplen[0] = prompt_len;
    D->hres[0] = reserve;
    return ADAMAH_OK;
}

// Run `n_steps` token steps.  flags bit0: run the LM head + arg-max (the sampled
// id feeds the next step once the prompt is consumed); bit1: also store the
// soft-capped logits; bit2: launch kernels directly instead of replaying a graph;
// bit4: draw the token with the rule of adam_b200_decoder_set_sampling instead of the arg-max;
// bit3: use the chain of per-operation kernels even where the single-launch token
// kernel (one sequence, row-tiled weights) would run.
// Returns without waiting unless called outside batch_begin/batch_end.
extern "C" int adam_b200_decoder_step(uint32_t id, uint32_t n_steps, uint32_t flags) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (D->batch == 0) return fail(ADAMAH_ERR_INVALID, "decoder_step: call decoder_begin first");
    const bool sample = (flags & 16u) != 0;
    const bool with_lm = flags & 1u, want_logits = (flags & 2u) != 0 || sample, direct = (flags & 4u) != 0, chain = (flags & 8u) != 0;
    if (want_logits && !with_lm) return fail(ADAMAH_ERR_INVALID, "decoder_step: logits need the LM head flag");
    if (sample && D->smp_k == 0) return fail(ADAMAH_ERR_INVALID, "decoder_step: call adam_b200_decoder_set_sampling before a sampled step");
    // the sampled token replaces the arg-max one right after every step (positions are already advanced)
    auto sample_step = [&]() -> int {
        if (!sample) return ADAMAH_OK;
        const Mat& lm = D->output.bound ? D->output : D->embd;
        return launch_sample(D->logits, lm.rows, D->batch, D->smp_k, D->smp_temp, D->smp_top_p, D->smp_penalty, D->smp_on_prompt, D->smp_seed,
                             D->pos, D->prompt_len, D->prompt_tok, D->gen_log, D->d.kv_cap, D->cur_tok, D->cur_val);
    };
    int rc = ADAMAH_OK;
    // a step past the reserved pages would only set a device error bit and return ids that look valid
    for (uint32_t b = 0; b < D->batch; ++b)
        if ((uint64_t)D->hpos[b] + n_steps > D->hres[b])
            return fail(ADAMAH_ERR_INVALID, "decoder_step: sequence %u is at position %u of %u reserved, cannot take %u more steps", b, D->hpos[b], D->hres[b], n_steps);
    for (uint32_t& hp : D->hpos) hp += n_steps;
    if (stream_recorded()) D->pos_shared = true;
    if (D->batch == 1 && !chain && D->tk_state == 0 && !capturing()) { if ((rc = prepare_token_kernel(D))) return rc; }
    if (D->batch == 1 && !chain && D->tk_state == 1 && !capturing()) {
        uint32_t s = 0;
        // Several steps at once replay a graph of TK_GRAPH_N launches: a cooperative launch costs the host
        // more than the kernel's start-up on the device, and back-to-back graph nodes close that gap.
        static const bool use_graph = !(getenv("ADAM_B200_TOKEN_GRAPH") && atoi(getenv("ADAM_B200_TOKEN_GRAPH")) == 0);
        const int gi = with_lm ? 1 : 0;
        if (use_graph && !want_logits && !direct && n_steps >= TK_GRAPH_N && D->tk_graph_state[gi] >= 0) {
            if (!D->tk_graph[gi]) {
                const uint64_t l0 = g.launches;
                DCU(cudaStreamSynchronize(g.stream));
                cudaGraph_t graph = nullptr;
                bool ok = cudaStreamBeginCapture(g.stream, cudaStreamCaptureModeRelaxed) == cudaSuccess;
                for (uint32_t k = 0; ok && k < TK_GRAPH_N; ++k) ok = enqueue_token(D, with_lm, false) == ADAMAH_OK;
                if (cudaStreamEndCapture(g.stream, &graph) != cudaSuccess) ok = false;
                if (ok && cudaGraphInstantiate(&D->tk_graph[gi], graph, 0) != cudaSuccess) ok = false;
                g.launches = l0;
                if (ok) { D->tk_graph_src[gi] = graph; D->tk_graph_state[gi] = 1; }
                else { cudaGetLastError(); if (graph) cudaGraphDestroy(graph); D->tk_graph[gi] = nullptr; D->tk_graph_state[gi] = -1; }
            }
            if (D->tk_graph[gi]) {
                for (; s + TK_GRAPH_N <= n_steps; s += TK_GRAPH_N) DCU(cudaGraphLaunch(D->tk_graph[gi], g.stream));
                count_launch(s);
            }
        }
        for (; s < n_steps && rc == ADAMAH_OK; ++s) { rc = enqueue_token(D, with_lm, want_logits); if (rc == ADAMAH_OK) rc = sample_step(); }
        end_of_op();
        return rc;
    }
    if (direct || want_logits || capturing()) {
        for (uint32_t s = 0; s < n_steps && rc == ADAMAH_OK; ++s) { rc = enqueue_step(D, D->batch, with_lm, want_logits); if (rc == ADAMAH_OK) rc = sample_step(); }
    } else {
        const int gi = with_lm ? 1 : 0;
        if (!D->graph[gi] || D->graph_batch[gi] != D->batch) {
            if (D->graph[gi]) { cudaGraphExecDestroy(D->graph[gi]); cudaGraphDestroy(D->graph_src[gi]); D->graph[gi] = nullptr; }
            {   // scratch must exist before the capture starts (no allocation inside it)
                float* pv; int* pi; unsigned int* tk;
                if ((rc = argmax_scratch(&pv, &pi, &tk))) return rc;
            }
            const uint64_t l0 = g.launches;
            DCU(cudaStreamSynchronize(g.stream));
            DCU(cudaStreamBeginCapture(g.stream, cudaStreamCaptureModeRelaxed));
            rc = enqueue_step(D, D->batch, with_lm, false);
            cudaGraph_t graph = nullptr;
            cudaError_t e = cudaStreamEndCapture(g.stream, &graph);
            if (rc) { if (graph) cudaGraphDestroy(graph); return rc; }
            if (e != cudaSuccess) return fail(ADAMAH_ERR_BACKEND, "decoder_step: capture failed: %s", cudaGetErrorString(e));
            DCU(cudaGraphInstantiate(&D->graph[gi], graph, 0));
            D->graph_src[gi] = graph;
            D->graph_batch[gi] = D->batch;
            D->graph_kernels[gi] = g.launches - l0;
            g.launches = l0;
        }
        for (uint32_t s = 0; s < n_steps; ++s) DCU(cudaGraphLaunch(D->graph[gi], g.stream));
        count_launch(D->graph_kernels[gi] * n_steps);
    }
    end_of_op();
    return rc;
}

// Sampling rule of steps that carry flag bit4 (role of GenerationConfig, adam/models/engine.py:24-29, applied as
// `_sample` does, :3711-3729): repeat penalty on the distinct ids among the last 64 of the history (generated
// tokens, plus the prompt with repeat_on_prompt), temperature, the top_k (1..64) best, soft-max, nucleus top_p,
// one draw per step from a counter-based generator keyed by (seed, sequence, position).  temperature <= 0 or
// top_k == 1 picks the best penalised logit.
extern "C" int adam_b200_decoder_set_sampling(uint32_t id, uint32_t top_k, float top_p, float temperature, float repeat_penalty,
                                              uint32_t repeat_on_prompt, uint64_t seed) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (top_k == 0 || top_k > 64) return fail(ADAMAH_ERR_INVALID, "decoder_set_sampling: top_k must be 1..64");
    if (!(repeat_penalty > 0.f)) return fail(ADAMAH_ERR_INVALID, "decoder_set_sampling: repeat_penalty must be positive");
    D->smp_k = top_k; D->smp_top_p = top_p; D->smp_temp = temperature; D->smp_penalty = repeat_penalty;
    D->smp_on_prompt = repeat_on_prompt ? 1 : 0; D->smp_seed = seed;
    return ADAMAH_OK;
}

// Asynchronous read of the current tokens: tokens_async enqueues, behind everything issued so
// far, a copy of the current token ids into one of four pinned slots and returns the slot;
// tokens_wait blocks until that copy has landed (later work on the stream keeps running) and
// hands the ids out.  Lets a caller keep the next step queued while it looks at the last ids.
extern "C" int adam_b200_decoder_tokens_async(uint32_t id, uint32_t* slot_out) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (!slot_out || D->batch == 0) return fail(ADAMAH_ERR_INVALID, "decoder_tokens_async: no active sequences or null argument");
    if (capturing()) return fail(ADAMAH_ERR_INVALID, "decoder_tokens_async: not allowed while a graph is being captured");
    const uint32_t slot = D->tok_next;
    D->tok_next = (slot + 1) & 3u;
    if (!D->tok_ring[slot]) {
        DCU(cudaMallocHost((void**)&D->tok_ring[slot], (size_t)D->d.max_batch * 4));
        DCU(cudaEventCreateWithFlags(&D->tok_event[slot], cudaEventDisableTiming));
    }
    DCU(cudaMemcpyAsync(D->tok_ring[slot], D->cur_tok, (size_t)D->batch * 4, cudaMemcpyDeviceToHost, g.stream));
    DCU(cudaEventRecord(D->tok_event[slot], g.stream));
    *slot_out = slot;
    return ADAMAH_OK;
}
extern "C" int adam_b200_decoder_tokens_wait(uint32_t id, uint32_t slot, int32_t* out) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (slot > 3 || !out || !D->tok_ring[slot]) return fail(ADAMAH_ERR_INVALID, "decoder_tokens_wait: bad slot");
    DCU(cudaEventSynchronize(D->tok_event[slot]));
    memcpy(out, D->tok_ring[slot], (size_t)D->batch * 4);
    return ADAMAH_OK;
}

// Overwrite the current token of every active sequence (host-side sampling: the caller read the
// logits of the last step and drew its own tokens; they feed the next step).
extern "C" int adam_b200_decoder_set_tokens(uint32_t id, const int32_t* tokens) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (!tokens || D->batch == 0) return fail(ADAMAH_ERR_INVALID, "decoder_set_tokens: no active sequences or null argument");
    if (capturing()) return fail(ADAMAH_ERR_INVALID, "decoder_set_tokens: not allowed while a graph is being captured");
    for (uint32_t b = 0; b < D->batch; ++b)
        if (tokens[b] < 0 || (uint32_t)tokens[b] >= D->embd.rows) return fail(ADAMAH_ERR_INVALID, "decoder_set_tokens: token id %d outside the vocabulary", tokens[b]);
    DCU(cudaMemcpyAsync(D->cur_tok, tokens, (size_t)D->batch * 4, cudaMemcpyHostToDevice, g.stream));
    DCU(cudaStreamSynchronize(g.stream));
    return ADAMAH_OK;
}

// Chunked prefill: consume the next n_tokens[b] prompt tokens of every active sequence, many rows (sequence, position)
// per pass: the rows of a chunk go through the products together, their keys and values are appended first and attention
// then reads the whole chunk from the cache (causal by position).  No LM head: the token after a prompt's last one comes
// from a normal step.  Same results as single steps (the reference consumes prompts token by token, engine.py:3838-3847).
//
// The plan of a call lists its rows sequence by sequence, cut into chunks of equal size, and each sequence's run inside a
// chunk is cut into attention tiles; one copy takes it to the device.
static int plan_prefill(Decoder* D, const uint32_t* n_tokens) {
    const adam_b200_decoder_desc& d = D->d;
    const uint32_t group = d.n_head / d.n_head_kv;
    uint64_t total = 0;
    for (uint32_t b = 0; b < D->batch; ++b) total += n_tokens[b];
    D->chunks.clear();
    D->plan_pos.assign(D->hpos.begin(), D->hpos.end());
    if (!total) return ADAMAH_OK;
    if (D->pos_shared) {
        DCU(cudaMemcpyAsync(D->plan_pos.data(), D->pos, (size_t)D->batch * 4, cudaMemcpyDeviceToHost, g.stream));
        DCU(cudaStreamSynchronize(g.stream));
        for (uint32_t b = 0; b < D->batch; ++b)
            if (D->plan_pos[b] < 0 || (uint64_t)D->plan_pos[b] + n_tokens[b] > d.kv_cap)
                return fail(ADAMAH_ERR_INVALID, "decoder_prefill: sequence %u is at position %d of %u", b, D->plan_pos[b], d.kv_cap);
    }
    const uint64_t n_chunks = (total + D->rows_cap - 1) / D->rows_cap;
    uint64_t size = ((total + n_chunks - 1) / n_chunks + 63) / 64 * 64;
    if (size > D->rows_cap) size = D->rows_cap;
    std::vector<int32_t> seq, pos;
    std::vector<AttnTile> tiles;
    seq.reserve(total); pos.reserve(total);
    struct Cut { uint32_t row, rows, tile, n_tiles, tile_rows; };
    std::vector<Cut> cuts;
    uint32_t b = 0, at = 0;                             // sequence and how many of its tokens are placed
    while (seq.size() < total) {
        Cut c = {(uint32_t)seq.size(), 0, (uint32_t)tiles.size(), 0, 0};
        struct Run { uint32_t row, b, pos, n; };
        std::vector<Run> runs;
        while (c.rows < size && b < D->batch) {
            const uint32_t n = std::min<uint32_t>(n_tokens[b] - at, (uint32_t)size - c.rows);
            const uint32_t from = (uint32_t)D->plan_pos[b] + at;
            if (n) runs.push_back(Run{c.rows, b, from, n});
            for (uint32_t i = 0; i < n; ++i) { seq.push_back((int32_t)b); pos.push_back((int32_t)(from + i)); }
            c.rows += n; at += n;
            if (at == n_tokens[b]) { ++b; at = 0; }
        }
        c.tile_rows = attn_prefill_rows(c.rows, group, d.n_head_kv, d.head_dim, (uint32_t)g.sm_count);
        const uint32_t step = attn_prefill_tokens(group, c.tile_rows);
        for (const Run& r : runs)
            for (uint32_t i = 0; i < r.n; i += step)
                tiles.push_back(AttnTile{(int32_t)(r.row + i), (int32_t)r.b, (int32_t)(r.pos + i), (int32_t)std::min(step, r.n - i)});
        c.n_tiles = (uint32_t)tiles.size() - c.tile;
        // the tiles with the longest reach first: they end last otherwise
        std::sort(tiles.begin() + c.tile, tiles.end(), [](const AttnTile& x, const AttnTile& y) { return x.pos > y.pos; });
        cuts.push_back(c);
    }
    const size_t o_pos = seq.size() * 4, o_tiles = (2 * seq.size() * 4 + 15) & ~(size_t)15, o_n = o_tiles + tiles.size() * sizeof(AttnTile), bytes = o_n + (size_t)D->batch * 4;
    if (bytes > D->plan_cap) {
        DCU(cudaStreamSynchronize(g.stream));
        cudaFree(D->plan); cudaFreeHost(D->plan_pin);
        D->plan = D->plan_pin = nullptr; D->plan_cap = 0;
        const size_t cap = bytes * 2;
        DCU(cudaMalloc((void**)&D->plan, cap));
        DCU(cudaMallocHost((void**)&D->plan_pin, cap));
        D->plan_cap = cap;
    } else if (D->plan_read) DCU(cudaEventSynchronize(D->plan_read));       // the copy of the call before has left the pinned source
    if (!D->plan_read) DCU(cudaEventCreateWithFlags(&D->plan_read, cudaEventDisableTiming));
    memcpy(D->plan_pin, seq.data(), seq.size() * 4);
    memcpy(D->plan_pin + o_pos, pos.data(), pos.size() * 4);
    memcpy(D->plan_pin + o_tiles, tiles.data(), tiles.size() * sizeof(AttnTile));
    memcpy(D->plan_pin + o_n, n_tokens, (size_t)D->batch * 4);
    DCU(cudaMemcpyAsync(D->plan, D->plan_pin, bytes, cudaMemcpyHostToDevice, g.stream));
    DCU(cudaEventRecord(D->plan_read, g.stream));
    for (const Cut& c : cuts)
        D->chunks.push_back(PrefillChunk{c.rows, c.n_tiles, c.tile_rows, (const int32_t*)D->plan + c.row, (const int32_t*)(D->plan + o_pos) + c.row,
                                         (const AttnTile*)(D->plan + o_tiles) + c.tile});
    D->plan_n = (const int32_t*)(D->plan + o_n);
    return ADAMAH_OK;
}

// Part 2L / 2L+1 of one chunk: the attention half of layer L (preceded by the embedding for L = 0) / its FFN half.
static int enqueue_prefill_part(Decoder* D, const PrefillChunk& c, uint32_t part) {
    const adam_b200_decoder_desc& d = D->d;
    const uint32_t rows = c.n_rows;
    const uint32_t E = d.n_embd, q_dim = d.n_head * d.head_dim, k_dim = d.n_head_kv * d.head_dim, qkv_ld = q_dim + 2 * k_dim;
    int rc;
    const uint32_t L = part / 2;
    const Layer& ly = D->layers[L];
    if (!(part & 1u)) {
        if (L == 0) launch_embed(D, rows, c.row_seq, c.row_pos);
        const int cur = L == 0 ? 0 : 1;
        GemvArgs in = {};
        in.ldx = (int)E; in.eps = d.norm_eps; in.h_in = D->hbuf[cur]; in.w_pre = ly.norm[NORM_ATTN];
        if (L > 0) { in.add_src = D->proj; in.w_post = D->layers[L - 1].norm[NORM_POST_FFW]; in.h_out = D->hbuf[cur ^ 1]; }
        in.y = D->qkv; in.ldy = (int)qkv_ld;
        if (ly.qkv_contiguous) {
            Mat qkv = ly.m[MAT_Q]; qkv.rows = qkv_ld; qkv.tiled = ly.qkv_tiled;
            if ((rc = gemv(qkv, nullptr, in, rows, EPI_STORE))) return rc;
        } else {
            if ((rc = gemv(ly.m[MAT_Q], nullptr, in, rows, EPI_STORE))) return rc;
            GemvArgs in2 = in; in2.h_out = nullptr;
            in2.y = D->qkv + q_dim;
            if ((rc = gemv(ly.m[MAT_K], nullptr, in2, rows, EPI_STORE))) return rc;
            in2.y = D->qkv + q_dim + k_dim;
            if ((rc = gemv(ly.m[MAT_V], nullptr, in2, rows, EPI_STORE))) return rc;
        }
        const int which = is_global_layer(d, L) ? 1 : 0;
        AttnPrefillArgs a = {};
        a.qkv = D->qkv; a.qkv_ld = qkv_ld; a.q_norm = ly.norm[NORM_Q]; a.k_norm = ly.norm[NORM_K]; a.eps = d.norm_eps;
        a.cos_t = D->rope_cos[which]; a.sin_t = D->rope_sin[which]; a.n_pos = D->rope_pos[which];
        a.kv_pool = D->kv_pool; a.geo = KvGeom{d.n_layer, d.n_head_kv, d.head_dim, d.page_size, D->max_pages_per_seq, D->page_elems};
        a.block_table = D->block_table; a.row_seq = c.row_seq; a.row_pos = c.row_pos; a.tiles = c.tiles; a.n_tiles = c.n_tiles;
        a.n_rows = rows; a.n_head = d.n_head; a.head_dim = d.head_dim; a.layer = L;
        a.window = ((d.flags & 1u) && d.sliding_window > 0 && !which) ? d.sliding_window : 0;
        a.scale = d.attn_scale; a.cap = d.attn_softcap; a.out = D->attn_out; a.err = g.dev_err;
        if ((rc = launch_qkv_prep(a, d.kv_dtype == 1, g.stream, g.pdl))) return rc;
        if ((rc = launch_attn_prefill(a, d.kv_dtype == 1, c.tile_rows, g.stream, g.pdl))) return rc;
        GemvArgs o = {};
        o.x = D->attn_out; o.ldx = (int)q_dim; o.y = D->proj; o.ldy = (int)E;
        if ((rc = gemv(ly.m[MAT_O], nullptr, o, rows, EPI_STORE))) return rc;
    } else {
        GemvArgs gu = {};
        gu.ldx = (int)E; gu.eps = d.norm_eps; gu.h_in = D->hbuf[0]; gu.add_src = D->proj; gu.w_post = ly.norm[NORM_POST_ATTN];
        gu.w_pre = ly.norm[NORM_FFN]; gu.h_out = D->hbuf[1]; gu.y = D->act; gu.ldy = (int)d.n_ff;
        if ((rc = gemv(ly.m[MAT_GATE], &ly.m[MAT_UP], gu, rows, d.ffn_act == 0 ? EPI_GEGLU : EPI_SWIGLU))) return rc;
        GemvArgs dn = {};
        dn.x = D->act; dn.ldx = (int)d.n_ff; dn.y = D->proj; dn.ldy = (int)E;
        if ((rc = gemv(ly.m[MAT_DOWN], nullptr, dn, rows, EPI_STORE))) return rc;
    }
    return check_launch("decoder prefill");
}

static void enqueue_prefill_end(Decoder* D, uint32_t even) {       // 0: the plan's numbers of tokens
    launch_k(k_advance_by, dim3((D->batch + 63) / 64), dim3(64), 0, g.stream, g.pdl, D->pos, even ? (const int32_t*)nullptr : D->plan_n, (int32_t)even, D->batch);
    count_launch();
}
// A chunk of T tokens of every sequence, planned on the device: it can be recorded and replayed from wherever the sequences are.
// What reads the plan comes behind the embedding, which is launched with a full dependency.
static PrefillChunk even_chunk(const Decoder* D, uint32_t T, uint32_t* step) {
    const adam_b200_decoder_desc& d = D->d;
    const uint32_t group = d.n_head / d.n_head_kv, rows = D->batch * T, tile_rows = attn_prefill_rows(rows, group, d.n_head_kv, d.head_dim, (uint32_t)g.sm_count);
    *step = attn_prefill_tokens(group, tile_rows);
    return PrefillChunk{rows, D->batch * ((T + *step - 1) / *step), tile_rows, D->even_plan, D->even_plan + D->rows_cap, (const AttnTile*)(D->even_plan + 2 * (size_t)D->rows_cap)};
}
static int enqueue_even_part(Decoder* D, uint32_t T, uint32_t part) {
    uint32_t step;
    const PrefillChunk c = even_chunk(D, T, &step);
    if (part == 0) {
        k_even_plan<<<(c.n_rows + 127) / 128, 128, 0, g.stream>>>(D->pos, D->batch, T, step, D->even_plan, D->even_plan + D->rows_cap, (AttnTile*)(D->even_plan + 2 * (size_t)D->rows_cap));
        count_launch();
    }
    if (part < 2 * D->d.n_layer) return enqueue_prefill_part(D, c, part);
    enqueue_prefill_end(D, T);
    return check_launch("decoder prefill");
}
static int check_prefill(Decoder* D, const uint32_t* n_tokens, const char* name) {
    if (D->batch == 0) return fail(ADAMAH_ERR_INVALID, "%s: call decoder_begin first", name);
    for (uint32_t b = 0; b < D->batch; ++b)
        if ((uint64_t)D->hpos[b] + n_tokens[b] > D->hplen[b])
            return fail(ADAMAH_ERR_INVALID, "%s: sequence %u has only %u prompt tokens left", name, b, D->hplen[b] - D->hpos[b]);
    return ADAMAH_OK;
}

// One part of one prefill chunk of n_tokens (n_tokens * batch rows, at most what buffer 0 of
// adam_b200_decoder_buffer_ptr holds) tokens per sequence, for tensor-parallel callers: parts 0 .. 2*n_layer-1 as in
// adam_b200_decoder_step_part (all-reduce the projection buffer, batch * n_tokens rows, after each), part 2*n_layer
// advances the positions.
extern "C" int adam_b200_decoder_prefill_part(uint32_t id, uint32_t n_tokens, uint32_t part) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (part > 2 * D->d.n_layer) return fail(ADAMAH_ERR_INVALID, "decoder_prefill_part: part %u of %u", part, 2 * D->d.n_layer + 1);
    if (D->batch && (n_tokens == 0 || (uint64_t)n_tokens * D->batch > D->rows_cap)) return fail(ADAMAH_ERR_INVALID, "decoder_prefill_part: a chunk holds at most %u rows", D->rows_cap);
    int rc = ADAMAH_OK;
    const std::vector<uint32_t> n(D->batch, n_tokens);
    if ((part == 0 || !D->batch) && (rc = check_prefill(D, n.data(), "decoder_prefill_part"))) return rc;
    if (stream_recorded()) D->pos_shared = true;
    g.pdl = pdl_allowed();
    rc = enqueue_even_part(D, n_tokens, part);
    g.pdl = false;
    if (rc == ADAMAH_OK && part == 2 * D->d.n_layer) for (uint32_t& hp : D->hpos) hp += n_tokens;
    end_of_op();
    return rc;
}

// n_tokens[b] prompt tokens of every active sequence b; none for a sequence is fine.
extern "C" int adam_b200_decoder_prefill_ragged(uint32_t id, const uint32_t* n_tokens) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (!n_tokens) return fail(ADAMAH_ERR_INVALID, "decoder_prefill: null argument");
    if (capturing()) return fail(ADAMAH_ERR_INVALID, "decoder_prefill: not allowed while a graph is being captured");
    int rc = check_prefill(D, n_tokens, "decoder_prefill");
    if (rc) return rc;
    if (stream_recorded()) {                    // a caller's own capture of the stream that it lent
        for (uint32_t b = 1; b < D->batch; ++b) if (n_tokens[b] != n_tokens[0]) return fail(ADAMAH_ERR_INVALID, "decoder_prefill: only equal numbers of tokens can be recorded");
        D->pos_shared = true;
        g.pdl = pdl_allowed();
        const uint32_t most = D->rows_cap / D->batch;
        for (uint32_t left = n_tokens[0], T; left && rc == ADAMAH_OK; left -= T) {
            T = std::min(left, most);
            for (uint32_t part = 0; part <= 2 * D->d.n_layer && rc == ADAMAH_OK; ++part) rc = enqueue_even_part(D, T, part);
        }
        g.pdl = false;
    } else if ((rc = plan_prefill(D, n_tokens))) return rc;
    if (!D->chunks.empty()) {
        g.pdl = pdl_allowed();
        for (const PrefillChunk& c : D->chunks)
            for (uint32_t part = 0; part < 2 * D->d.n_layer && rc == ADAMAH_OK; ++part) rc = enqueue_prefill_part(D, c, part);
        if (rc == ADAMAH_OK) { enqueue_prefill_end(D, 0); rc = check_launch("decoder prefill"); }
        g.pdl = false;
        D->chunks.clear();
    }
    if (rc == ADAMAH_OK) for (uint32_t b = 0; b < D->batch; ++b) D->hpos[b] += n_tokens[b];
    end_of_op();
    return rc;
}

// What scoring needs besides the decoder's buffers.  Where two groups of 64 rows of logits (134 MB at the 1B shape) would leave
// less than 64 MB on the device, smaller groups, and at last the logits buffer that every decoder has.
static int score_prepare(Decoder* D) {
    const adam_b200_decoder_desc& d = D->d;
    constexpr uint32_t ROWS = 64;                       // rows per LM-head call: one arg-max scratch
    DCU(cudaMalloc((void**)&D->score_tok, ROWS * 8));
    for (cudaEvent_t& e : D->score_ev) DCU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    DCU(cudaStreamCreateWithFlags(&D->score_copy, cudaStreamNonBlocking));
    uint32_t rows = ROWS;
    for (; rows; rows /= 2) {
        const size_t need = (size_t)2 * rows * d.n_vocab * 4;
        size_t left = 0, total = 0;
        DCU(cudaMemGetInfo(&left, &total));
        if (left < need + (64u << 20)) continue;
        if (cudaMalloc((void**)&D->score_logits, need) == cudaSuccess) break;
        cudaGetLastError();
        D->score_logits = nullptr;
    }
    D->score_rows = rows ? rows : std::min(ROWS, d.max_batch);
    return ADAMAH_OK;
}

// Logits after every one of the next n_tokens prompt tokens of the single active sequence (a text under evaluation): the
// positions go through the layers together like a prompt, then the LM head runs over the chunk's rows, and the logits of
// one group of rows travel to the host while the next is computed.  Bound by the copy (1 MB per position at the 1B shape)
// and the latency of the layers' kernels.
// Leaves the decoder as n_tokens steps with logits would: positions, log, current token, and the last position's logits and
// rows where adam_b200_decoder_read_logits and adam_b200_decoder_read_buffer read them.
extern "C" int adam_b200_decoder_score(uint32_t id, uint32_t n_tokens, float* out) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (stream_recorded()) return fail(ADAMAH_ERR_INVALID, "decoder_score: not allowed while a graph is being captured");
    if (!out || n_tokens == 0 || D->batch != 1) return fail(ADAMAH_ERR_INVALID, "decoder_score: needs one active sequence, tokens and a destination");
    const adam_b200_decoder_desc& d = D->d;
    if (d.tp_size > 1) return fail(ADAMAH_ERR_INVALID, "decoder_score: not available with tensor parallelism");
    int rc = check_prefill(D, &n_tokens, "decoder_score");
    if (rc || (rc = plan_prefill(D, &n_tokens))) return rc;
    { float* pv; int* pi; unsigned int* tk; if ((rc = argmax_scratch(&pv, &pi, &tk))) return rc; }
    if (!D->score_rows && (rc = score_prepare(D))) { score_release(D); return rc; }
    const uint32_t GROUP = D->score_rows, halves = D->score_logits ? 2 : 1;
    float* const base = D->score_logits ? D->score_logits : D->logits;
    int32_t* tok = D->score_tok;
    float* val = (float*)(tok + GROUP);
    cudaError_t err = cudaSuccess;
    auto ok = [&](cudaError_t e) { if (err == cudaSuccess) err = e; };
    uint32_t done = 0, n_group = 0, last_row = 0, in_group = 0;
    const uint32_t p0 = (uint32_t)D->plan_pos[0];
    g.pdl = pdl_allowed();
    for (const PrefillChunk& c : D->chunks) {
        for (uint32_t part = 0; part < 2 * d.n_layer && rc == ADAMAH_OK; ++part) rc = enqueue_prefill_part(D, c, part);
        for (uint32_t r0 = 0; r0 < c.n_rows && rc == ADAMAH_OK; r0 += GROUP, ++n_group) {
            const uint32_t m = std::min(GROUP, c.n_rows - r0), half = n_group % halves;
            float* lg = base + (size_t)half * GROUP * d.n_vocab;
            if (n_group >= halves) ok(cudaStreamWaitEvent(g.stream, D->score_ev[2 + half], 0));     // the half's copy has left
            if ((rc = enqueue_head(D, r0, m, lg, tok, val))) break;
            // logged as the token of the position behind, as a step's
            const uint32_t fits = p0 + done + 1 < d.kv_cap ? std::min(m, d.kv_cap - p0 - done - 1) : 0;
            if (fits) ok(cudaMemcpyAsync(D->gen_log + p0 + done + 1, tok, (size_t)fits * 4, cudaMemcpyDeviceToDevice, g.stream));
            ok(cudaEventRecord(D->score_ev[half], g.stream));
            ok(cudaStreamWaitEvent(D->score_copy, D->score_ev[half], 0));
            ok(cudaMemcpyAsync(out + (size_t)done * d.n_vocab, lg, (size_t)m * d.n_vocab * 4, cudaMemcpyDeviceToHost, D->score_copy));
            ok(cudaEventRecord(D->score_ev[2 + half], D->score_copy));
            done += m; last_row = r0 + m - 1; in_group = m - 1;
        }
        if (rc || err != cudaSuccess) break;
    }
    if (rc == ADAMAH_OK && err == cudaSuccess) {
        enqueue_prefill_end(D, 0);
        const float* last = base + ((size_t)((n_group - 1) % halves) * GROUP + in_group) * d.n_vocab;
        if (halves == 1) ok(cudaStreamWaitEvent(g.stream, D->score_ev[2], 0));      // the row is overwritten in place
        if (last != D->logits) ok(cudaMemcpyAsync(D->logits, last, (size_t)d.n_vocab * 4, cudaMemcpyDeviceToDevice, g.stream));
        ok(cudaMemcpyAsync(D->cur_tok, tok + in_group, 4, cudaMemcpyDeviceToDevice, g.stream));
        ok(cudaMemcpyAsync(D->cur_val, val + in_group, 4, cudaMemcpyDeviceToDevice, g.stream));
        const uint32_t q_dim = d.n_head * d.head_dim, qkv_ld = q_dim + 2 * d.n_head_kv * d.head_dim;
        float* bufs[5] = {D->hbuf[0], D->qkv, D->attn_out, D->proj, D->act};
        const uint32_t lds[5] = {d.n_embd, qkv_ld, q_dim, d.n_embd, d.n_ff};
        if (last_row) for (int i = 0; i < 5; ++i) ok(cudaMemcpyAsync(bufs[i], bufs[i] + (size_t)last_row * lds[i], (size_t)lds[i] * 4, cudaMemcpyDeviceToDevice, g.stream));
        rc = check_launch("decoder score");
    }
    g.pdl = false;
    D->chunks.clear();
    ok(cudaStreamSynchronize(D->score_copy));
    ok(cudaStreamSynchronize(g.stream));                // the caller reads `out` on return
    g.submits++;
    if (rc == ADAMAH_OK && err != cudaSuccess) rc = fail(ADAMAH_ERR_BACKEND, "decoder_score: %s", cudaGetErrorString(err));
    if (rc == ADAMAH_OK) D->hpos[0] += n_tokens;
    return rc;
}

extern "C" int adam_b200_decoder_prefill(uint32_t id, uint32_t n_tokens) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    const std::vector<uint32_t> n(D->batch ? D->batch : 1, n_tokens);
    return adam_b200_decoder_prefill_ragged(id, n.data());
}

// Where the time of a one-sequence step on the graph of per-operation kernels goes (diagnostics build only):
// out == NULL arms the trace for `layer` (the step graphs are recorded again with the trace buffer attached);
// a later call with a buffer waits for the stream and copies 512 stamps of the most recent step: the four
// products of the layer (QKV, o-proj, gate/up, down) as [product][CTA 0..7][8] and its attention launch as
// [CTA 0..31][8], nanoseconds of the GPU's global timer (slot meanings: adam_b200.h).
extern "C" int adam_b200_decoder_step_trace(uint32_t id, uint32_t layer, long long* out, uint32_t n_words) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
#ifdef ADAM_B200_STEP_TRACE
    const size_t words = 4 * 64 + 32 * 8;
    if (!out) {
        if (layer >= D->d.n_layer) return fail(ADAMAH_ERR_INVALID, "decoder_step_trace: layer %u of %u", layer, D->d.n_layer);
        DCU(cudaStreamSynchronize(g.stream));
        if (!g_step_trace) DCU(cudaMalloc(&g_step_trace, words * 8));
        DCU(cudaMemset(g_step_trace, 0, words * 8));
        g_step_trace_layer = layer;
        free_graphs(D);
        return ADAMAH_OK;
    }
    if (!g_step_trace) return fail(ADAMAH_ERR_INVALID, "decoder_step_trace: not armed");
    DCU(cudaStreamSynchronize(g.stream));
    DCU(cudaMemcpy(out, g_step_trace, (n_words < words ? n_words : words) * 8, cudaMemcpyDeviceToHost));
    return ADAMAH_OK;
#else
    (void)layer; (void)out; (void)n_words;
    return fail(ADAMAH_ERR_INVALID, "decoder_step_trace: this library was built without ADAM_B200_STEP_TRACE (python -m adam_b200.build --step-trace)");
#endif
}

// One part of a token step, enqueued directly on the stream (no graph): see enqueue_part.
// For callers that interleave their own work between parts (tensor parallelism: an
// all-reduce of the projection buffer after every layer part, a merge of the arg-max
// pairs after the LM-head part).  flags as in adam_b200_decoder_step.
extern "C" int adam_b200_decoder_n_parts(uint32_t id) {
    Decoder* D = get_dec(id);
    return D ? (int)n_parts(D) : ADAMAH_ERR_NOT_FOUND;
}
extern "C" int adam_b200_decoder_step_part(uint32_t id, uint32_t part, uint32_t flags) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (!D->batch) return fail(ADAMAH_ERR_INVALID, "decoder_step_part: call decoder_begin first");
    if (part >= n_parts(D)) return fail(ADAMAH_ERR_INVALID, "decoder_step_part: part %u of %u", part, n_parts(D));
    const bool with_lm = flags & 1u, want_logits = (flags & 2u) != 0;
    if (part == 0)
        for (uint32_t b = 0; b < D->batch; ++b)
            if (D->hpos[b] + 1u > D->hres[b]) return fail(ADAMAH_ERR_INVALID, "decoder_step_part: sequence %u has used all %u reserved positions", b, D->hres[b]);
    if (part + 1 == n_parts(D) && stream_recorded()) D->pos_shared = true;
    g.pdl = pdl_allowed();
    const int rc = enqueue_part(D, D->batch, part, with_lm, want_logits);
    g.pdl = false;
    if (rc == ADAMAH_OK && part + 1 == n_parts(D)) for (uint32_t& hp : D->hpos) hp += 1;
    end_of_op();
    return rc;
}
// Diagnostics of the single-launch token kernel: run ONE token step (LM head included) of the active
// sequence with per-phase SM clock stamps of layer `layer` and of the LM head recorded by every CTA, and
// return them: out[cta * 16 + slot] (clock64 values of that CTA's SM; slots 0..9 = layer phases, 10..13 = LM
// head), n_cta_out = CTAs launched.  out must hold 16 * 256 values.
extern "C" int adam_b200_decoder_token_trace(uint32_t id, uint32_t layer, long long* out, uint32_t* n_cta_out) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (!out || !n_cta_out || D->batch != 1) return fail(ADAMAH_ERR_INVALID, "decoder_token_trace: needs one active sequence");
    if (D->tk_state == 0) { const int rc0 = prepare_token_kernel(D); if (rc0) return rc0; }
    if (D->tk_state != 1) return fail(ADAMAH_ERR_INVALID, "decoder_token_trace: this model does not run on the token kernel");
    if (D->hpos[0] + 1u > D->hres[0]) return fail(ADAMAH_ERR_INVALID, "decoder_token_trace: no reserved position left");
    const size_t bytes = (size_t)TK_TRACE_SLOTS * 256 * sizeof(long long);
    DCU(cudaMalloc((void**)&g_tk_trace, bytes));
    DCU(cudaMemsetAsync(g_tk_trace, 0, bytes, g.stream));
    g_tk_trace_layer = (int)(layer & 0xFFFFu); g_tk_trace_phase = (int)(layer >> 16);
    D->hpos[0] += 1;
    const int rc = enqueue_token(D, true, false);
    cudaMemcpyAsync(out, g_tk_trace, bytes, cudaMemcpyDeviceToHost, g.stream);
    cudaStreamSynchronize(g.stream);
    cudaFree(g_tk_trace);
    g_tk_trace = nullptr;
    *n_cta_out = (uint32_t)D->tk_grid;
    return rc;
}

// Exercises the bounded waits of the single-launch token kernel without any fault: ONE token step is launched
// with its last CTA left out and every wait limited to `wait_us` microseconds.  The packets that CTA would have
// produced never arrive, so the waits of the others run out; they record DEVERR_WAIT in the device error word,
// set the decoder's sticky word and return.  Later steps return at once until decoder_begin / decoder_continue
// clears the word.  Returns after the launch has finished.
extern "C" int adam_b200_decoder_test_wait_expiry(uint32_t id, uint32_t wait_us) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (D->batch != 1) return fail(ADAMAH_ERR_INVALID, "decoder_test_wait_expiry: needs one active sequence");
    if (D->tk_state == 0) { const int rc0 = prepare_token_kernel(D); if (rc0) return rc0; }
    if (D->tk_state != 1 || D->tk_grid < 2) return fail(ADAMAH_ERR_INVALID, "decoder_test_wait_expiry: this model does not run on the token kernel");
    if (wait_us == 0 || wait_us > 1000000u) return fail(ADAMAH_ERR_INVALID, "decoder_test_wait_expiry: wait_us must be 1 .. 1000000");
    TkArgs a = D->tk;
    a.with_lm = 1; a.logits = nullptr; a.trace = nullptr;
    a.wait_cycles = (long long)wait_us * 2000;              // SM clocks at about 2 GHz
    const int rc = launch_token(D->tk_wt, D->d.kv_dtype == 1, (int)D->d.head_dim, a, D->tk_grid - 1, g.stream);
    DCU(cudaStreamSynchronize(g.stream));
    return rc;
}

// Device address and size of one of the decoder's buffers, for callers that run their own
// kernels or collectives on them (same stream, see adam_b200_set_stream):
//   0 = projection output [rows][n_embd] f32 (what a tensor-parallel caller all-reduces; rows =
//       batch in a decode step, batch * n_tokens in a prefill chunk; at least max(max_batch, 64) rows)
//   1 = current token ids [max_batch] i32     2 = their logit values [max_batch] f32
//   3 = positions [max_batch] i32
extern "C" int adam_b200_decoder_buffer_ptr(uint32_t id, uint32_t which, uint64_t* ptr_out, uint64_t* bytes_out) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (!ptr_out || !bytes_out) return fail(ADAMAH_ERR_INVALID, "decoder_buffer_ptr: null argument");
    const size_t B = D->d.max_batch;
    switch (which) {
    case 0: *ptr_out = (uint64_t)(uintptr_t)D->proj; *bytes_out = (size_t)D->rows_cap * D->d.n_embd * 4; break;
    case 1: *ptr_out = (uint64_t)(uintptr_t)D->cur_tok; *bytes_out = B * 4; break;
    case 2: *ptr_out = (uint64_t)(uintptr_t)D->cur_val; *bytes_out = B * 4; break;
    case 3: *ptr_out = (uint64_t)(uintptr_t)D->pos; *bytes_out = B * 4; D->pos_shared = true; break;
    default: return fail(ADAMAH_ERR_INVALID, "decoder_buffer_ptr: unknown buffer %u", which);
    }
    return ADAMAH_OK;
}

// Reads (after synchronising): positions, current sampled tokens, and the log of
// sampled tokens: out_log[b][p] = id sampled for position p (-1 where none).
extern "C" int adam_b200_decoder_read_state(uint32_t id, int32_t* pos_out, int32_t* cur_tok_out) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (pos_out) DCU(cudaMemcpyAsync(pos_out, D->pos, (size_t)D->d.max_batch * 4, cudaMemcpyDeviceToHost, g.stream));
    if (cur_tok_out) DCU(cudaMemcpyAsync(cur_tok_out, D->cur_tok, (size_t)D->d.max_batch * 4, cudaMemcpyDeviceToHost, g.stream));
    DCU(cudaStreamSynchronize(g.stream));
    return ADAMAH_OK;
}
extern "C" int adam_b200_decoder_read_log(uint32_t id, uint32_t seq, uint32_t first_pos, uint32_t n, int32_t* out) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (!out || seq >= D->d.max_batch || (uint64_t)first_pos + n > D->d.kv_cap) return fail(ADAMAH_ERR_INVALID, "decoder_read_log: bad range");
    DCU(cudaMemcpyAsync(out, D->gen_log + (size_t)seq * D->d.kv_cap + first_pos, (size_t)n * 4, cudaMemcpyDeviceToHost, g.stream));
    DCU(cudaStreamSynchronize(g.stream));
    return ADAMAH_OK;
}
extern "C" int adam_b200_decoder_read_logits(uint32_t id, uint32_t seq, float* out) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    if (!out || seq >= D->d.max_batch) return fail(ADAMAH_ERR_INVALID, "decoder_read_logits: bad sequence");
    DCU(cudaMemcpyAsync(out, D->logits + (size_t)seq * D->d.n_vocab, (size_t)D->d.n_vocab * 4, cudaMemcpyDeviceToHost, g.stream));
    DCU(cudaStreamSynchronize(g.stream));
    return ADAMAH_OK;
}
// The launch shape that a step's attention asks for (the device may not run that many clusters at once): heads per CTA, (sequence,
// head group) pairs, CTAs per cluster or 0, a cluster's slots and bytes of shared memory, bytes of a CTA of independent splits.
extern "C" int adam_b200_attention_shape(uint32_t n_head, uint32_t n_head_kv, uint32_t head_dim, uint32_t kv_dtype, uint32_t batch, uint32_t reach, uint32_t* out) {
    if (!out || !n_head_kv || n_head < n_head_kv || n_head % n_head_kv || n_head / n_head_kv > 8 || !batch || !reach || kv_dtype > 1 ||
        (head_dim != 32 && head_dim != 64 && head_dim != 128 && head_dim != 256)) return fail(ADAMAH_ERR_INVALID, "attention_shape: bad arguments");
    const AttnShape s = attn_shape(n_head, n_head_kv, head_dim, kv_dtype ? 2u : 4u, batch, reach);
    out[0] = s.hpc; out[1] = s.pairs; out[2] = s.cluster; out[3] = s.cluster ? s.slots : 8u;
    out[4] = s.cluster ? (uint32_t)s.smem_cluster : 0u; out[5] = (uint32_t)s.smem;
    return ADAMAH_OK;
}

// Debug/verification read of an activation buffer of the last step:
// what = 0 hidden after the last layer [E] (steps that ran the LM head), 2 qkv, 4 attn_out, 5 proj [E], 6 act [FF].
extern "C" int adam_b200_decoder_read_buffer(uint32_t id, uint32_t what, uint32_t seq, float* out, uint32_t n) {
    Decoder* D = get_dec(id);
    if (!D) return ADAMAH_ERR_NOT_FOUND;
    const adam_b200_decoder_desc& d = D->d;
    const uint32_t q_dim = d.n_head * d.head_dim, k_dim = d.n_head_kv * d.head_dim;
    const float* bufs[7] = {D->hbuf[D->h_final], nullptr, D->qkv, nullptr, D->attn_out, D->proj, D->act};
    const uint32_t lds[7] = {d.n_embd, d.n_embd, q_dim + 2 * k_dim, q_dim, q_dim, d.n_embd, d.n_ff};
    if (what > 6 || !bufs[what] || !out || seq >= d.max_batch || n > lds[what]) return fail(ADAMAH_ERR_INVALID, "decoder_read_buffer: bad arguments");
    DCU(cudaMemcpyAsync(out, bufs[what] + (size_t)seq * lds[what], (size_t)n * 4, cudaMemcpyDeviceToHost, g.stream));
    DCU(cudaStreamSynchronize(g.stream));
    return ADAMAH_OK;
}
