// Attention of a prefill chunk: causal soft-max attention of many query rows over the paged cache
// (map_qk_norm_rope_x.comp, map_row_copy.comp, map_matmul_t.comp + map_attn_softmax_value.comp for every prompt position;
// adam/models/engine.py:3838-3847 walks the prompt one position at a time).
//
// The decode attention (k_attention in decoder.cu) gives every row its own pass over the cache on the fp32 pipe; for a
// prompt that is rows x context cache reads.  Here 32, 64 or 128 query rows (positions x the query heads of one kv head)
// share each tile of the cache, and both products run on mma.sync tensor instructions with the operands kept at the
// precision of the fp32 path: the cache's fp16 values are exact operands, and a query row or a row of probabilities goes
// in as two fp16 terms (22 bits); an fp32 cache takes three tf32 products (x_hi y_hi + x_hi y_lo + x_lo y_hi) instead.
// mma.sync rather than tcgen05: the rows of a chunk are a few dozen tiles per layer, about a tenth of the chunk's
// arithmetic, and the score tile needs a tanh and an exponential per element between the two products, which keeps it in
// registers here.  A tile's P.V goes into fresh accumulators and is added to the running output in fp32 with the
// rescaling that the online soft-max needs anyway, so the tensor core's round-to-zero sums stay a few instructions long.
// Bound by the latency of one CTA's chain (load a tile, scores, soft-max, P.V), so the rows are spread over as many SMs and
// warps as there are: with four warps per 64 rows and one cache tile in flight a tile of 64 positions took 8 us, four times its
// mma.sync time, and a 13-row prompt 32 us per layer (one CTA, unrolled code that the launch finds cold); now 10.8 us.  1B
// shape, whole prefill: 32 prompts x 512 129 -> 106 ms, 1500 tokens 15.9 -> 12.3 ms (fp16 cache), 23.9 -> 17.3 ms (fp32).
#include "attn_prefill.cuh"

namespace ab {

constexpr float AP_NEG = -1.0e30f;

// ---- QK-norm + RoPE + append: one warp per (row, head); the arithmetic of k_attention's row prologue ----------------
template <typename T, int HD>
__global__ void __launch_bounds__(256) k_qkv_prep(const AttnPrefillArgs a) {
    pdl_launch_dependents();
    // What the host wrote ahead of the pass (positions, pages) and the tables are read before the wait for the kernel in front:
    // that chain of dependent loads, here and in the attention kernels, was 1.5 us per layer (12 prompt rows, 1B: 1.43 -> 1.40 ms).
    const uint32_t lane = threadIdx.x & 31, w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, per_row = a.n_head + 2 * a.geo.n_kv;
    const bool live = w < a.n_rows * per_row;
    const uint32_t r = live ? w / per_row : 0u, h = w % per_row;
    const bool is_q = h < a.n_head, is_v = h >= a.n_head + a.geo.n_kv;
    const int32_t p = a.row_pos[r];
    float* src = a.qkv + (size_t)r * a.qkv_ld + (size_t)h * HD;
    const uint32_t page_no = (uint32_t)p / a.geo.page;
    const int32_t page_id = page_no < a.geo.max_pages ? a.block_table[(size_t)a.row_seq[r] * a.geo.max_pages + page_no] : -1;
    constexpr uint32_t half = HD / 2;
    constexpr int NP = (HD / 2 + 31) / 32;
    const uint32_t pp = (uint32_t)p < a.n_pos ? (uint32_t)p : a.n_pos - 1;
    const float *ct = a.cos_t + (size_t)pp * half, *sn_t = a.sin_t + (size_t)pp * half, *wt = is_q ? a.q_norm : a.k_norm;
    float c[NP], sn[NP], w0[NP], w1[NP];
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        const uint32_t i = min(lane + 32 * j, half - 1);
        c[j] = ct[i]; sn[j] = sn_t[i];
        w0[j] = wt ? wt[i] : 1.f; w1[j] = wt ? wt[i + half] : 1.f;
    }
    pdl_wait();
    if (!live) return;
    T* dst = nullptr;
    if (!is_q) {
        if (page_id < 0 || (uint32_t)p >= a.n_pos) { if (lane == 0) atomicOr(a.err, DEVERR_OOB_MAP); return; }
        dst = reinterpret_cast<T*>(a.kv_pool) + kv_index(a.geo, (uint32_t)page_id, a.layer, is_v ? 1u : 0u, (h - a.n_head) % a.geo.n_kv, (uint32_t)p % a.geo.page);
    }
    if (is_v) {
        for (uint32_t i = lane; i < HD; i += 32) st_kv(dst + i, src[i]);
        return;
    }
    float x0[NP], x1[NP], ss = 0.f;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        const uint32_t i = lane + 32 * j;
        x0[j] = i < half ? src[i] : 0.f;
        x1[j] = i < half ? src[i + half] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < NP; ++j) ss = fmaf(x0[j], x0[j], ss);
#pragma unroll
    for (int j = 0; j < NP; ++j) ss = fmaf(x1[j], x1[j], ss);
    float rms = 1.f;
    if (wt) { ss = warp_sum(ss); rms = sqrtf(ss / (float)HD + a.eps); }
    const float rcp = __frcp_rn(rms);
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        const uint32_t i = lane + 32 * j;
        if (i < half) {
            float a0 = x0[j], a1 = x1[j];
            if (wt) { a0 = div_by(a0, rms, rcp) * w0[j]; a1 = div_by(a1, rms, rcp) * w1[j]; }
            const float y0 = __fsub_rn(__fmul_rn(a0, c[j]), __fmul_rn(a1, sn[j])), y1 = __fadd_rn(__fmul_rn(a0, sn[j]), __fmul_rn(a1, c[j]));
            if (is_q) { src[i] = y0; src[i + half] = y1; }
            else { st_kv(dst + i, y0); st_kv(dst + i + half, y1); }
        }
    }
}

// ---- small helpers -------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t ap_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ap_cp16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void ap_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ap_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_h(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_t(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void tf32_split(float x, uint32_t& hi, uint32_t& lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(x - __uint_as_float(hi)));
}
__device__ __forceinline__ void half_split(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h); lo = *reinterpret_cast<const uint32_t*>(&l);
}

// What a query row of a tile is: row r -> position r / group, head r % group of the kv head's group.
struct ApRow { int pos; bool ok; size_t q, o; };
__device__ __forceinline__ ApRow ap_row(const AttnPrefillArgs& a, const AttnTile& t, uint32_t kvh, uint32_t group, uint32_t r, uint32_t HD) {
    const uint32_t tok = r / group, head = kvh * group + r % group;
    ApRow x;
    x.ok = tok < (uint32_t)t.n_tok && r < (uint32_t)t.n_tok * group;
    const uint32_t tk = x.ok ? tok : 0u;
    x.pos = t.pos + (int)tk;
    x.q = (size_t)(t.row + tk) * a.qkv_ld + (size_t)head * HD;
    x.o = (size_t)(t.row + tk) * a.n_head * HD + (size_t)head * HD;
    return x;
}

// tanh(x) for soft-capped scores: where the whole warp is below 1/4 (scores below a quarter of the cap, nearly always) its
// power series (the first term left out is 9e-9 of the value), else 1 - 2 / (1 + e^2x).
__device__ __forceinline__ float ap_tanh_small(float x) {
    const float y = x * x;
    return fmaf(x * y, fmaf(y, fmaf(y, fmaf(y, 62.f / 2835.f, -17.f / 315.f), 2.f / 15.f), -1.f / 3.f), x);
}
__device__ __forceinline__ float ap_tanh(float x) {
    const float d = 1.f + expf(fminf(2.f * x, 80.f));
    return fabsf(x) < 0.25f ? ap_tanh_small(x) : 1.f - div_by(2.f, d, rcp_newton(d));
}

// Online soft-max of one tile of scores (NT tiles of 8 positions from kv0): c becomes the probabilities, alpha the factor
// of the rows' earlier sums.  Row h of this thread is rows g + 8 h of the warp.
template <int NT>
__device__ __forceinline__ void ap_softmax(float (&c)[NT][4], const AttnPrefillArgs& a, const float (&scl)[2], const int (&pos)[2], int kv0, bool edge,
                                           float (&m)[2], float (&l)[2], float (&alpha)[2]) {
    const int lane = threadIdx.x & 31, q = lane & 3;
    const float rcap = a.cap > 0.f ? __frcp_rn(a.cap) : 0.f;
    float mx[2] = {AP_NEG, AP_NEG};
    if (a.cap > 0.f) {
        float big = 0.f;
        const float sx[2] = {scl[0] * rcap, scl[1] * rcap};
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) { c[j][e] *= sx[e >> 1]; big = fmaxf(big, fabsf(c[j][e])); }
        if (__all_sync(0xffffffffu, big < 0.25f)) {
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) c[j][e] = ap_tanh_small(c[j][e]) * a.cap;
        } else {
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) c[j][e] = ap_tanh(c[j][e]) * a.cap;
        }
    } else {
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) c[j][e] *= scl[e >> 1];
    }
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int h = e >> 1, kp = kv0 + 8 * j + 2 * q + (e & 1);
            float s = c[j][e];
            if (edge && (kp > pos[h] || (a.window > 0 && kp + (int)a.window <= pos[h]))) s = AP_NEG;
            c[j][e] = s;
            mx[h] = fmaxf(mx[h], s);
        }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
        const float mn = fmaxf(m[h], mx[h]);
        alpha[h] = expf(m[h] - mn);
        m[h] = mn;
        l[h] *= alpha[h];
    }
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float p = c[j][e] > 0.5f * AP_NEG ? expf(c[j][e] - m[e >> 1]) : 0.f;
            c[j][e] = p;
            l[e >> 1] += p;
        }
}

// The KH warps of a row group hold soft-max sums over different positions of the same rows: added up through shared memory
// (`ex`: KH / 2 slots per row group of m, l and the output, lane by lane), the result in the warps kh = 0.
template <int HD, int RG, int KH>
__device__ __forceinline__ void ap_merge(float4* ex, int rg, int kh, int lane, float (&o)[HD / 8][4], float (&m)[2], float (&l)[2]) {
#pragma unroll 1
    for (int step = KH / 2; step > 0; step >>= 1) {
        float4* at = ex + (size_t)((kh & (step - 1)) * RG + rg) * (HD / 8 + 1) * 32 + lane;
        __syncthreads();
        if (kh >= step && kh < 2 * step) {
            at[0] = make_float4(m[0], m[1], l[0], l[1]);
#pragma unroll
            for (int j = 0; j < HD / 8; ++j) at[(j + 1) * 32] = make_float4(o[j][0], o[j][1], o[j][2], o[j][3]);
        }
        __syncthreads();
        if (kh < step) {
            const float4 y = at[0];
            const float ym[2] = {y.x, y.y}, yl[2] = {y.z, y.w};
            float s0[2], s1[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float mn = fmaxf(m[h], ym[h]);
                s0[h] = expf(m[h] - mn); s1[h] = expf(ym[h] - mn);
                m[h] = mn;
                l[h] = l[h] * s0[h] + yl[h] * s1[h];
            }
#pragma unroll
            for (int j = 0; j < HD / 8; ++j) {
                const float4 v = at[(j + 1) * 32];
                o[j][0] = o[j][0] * s0[0] + v.x * s1[0]; o[j][1] = o[j][1] * s0[0] + v.y * s1[0];
                o[j][2] = o[j][2] * s0[1] + v.z * s1[1]; o[j][3] = o[j][3] * s0[1] + v.w * s1[1];
            }
        }
    }
}
template <int HD>
__device__ __forceinline__ void ap_store(const AttnPrefillArgs& a, const AttnTile& t, uint32_t kvh, uint32_t group, int r0, int lane, const float (&o)[HD / 8][4],
                                         const float (&l_part)[2], float unit) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float l = l_part[h];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        const ApRow r = ap_row(a, t, kvh, group, r0 + (lane >> 2) + 8 * h, HD);
        if (!r.ok) continue;
        const float d = l * unit, rd = __frcp_rn(d);
#pragma unroll
        for (int j = 0; j < HD / 8; ++j)
            *reinterpret_cast<float2*>(a.out + r.o + 8 * j + 2 * (lane & 3)) = make_float2(div_by(o[j][2 * h], d, rd), div_by(o[j][2 * h + 1], d, rd));
    }
}

// Where a tile's rows lie in the cache: looked up once per row and an iteration ahead (a look-up per 16-byte copy, with its
// dependent load of the page table, made a tile take 12 us).
template <int BN>
__device__ __forceinline__ void ap_locate(const AttnPrefillArgs& a, const int32_t* bt, uint32_t kvh, int kv0, int kv_hi, size_t (&rows)[2][BN]) {
    if (threadIdx.x < BN) {
        const int p = min(kv0 + (int)threadIdx.x, kv_hi - 1);
        const uint32_t pn = (uint32_t)p / a.geo.page;
        const int32_t page = pn < a.geo.max_pages ? max(bt[pn], 0) : 0;
        rows[(kv0 / BN) & 1][threadIdx.x] = kv_index(a.geo, (uint32_t)page, a.layer, 0, kvh, (uint32_t)p % a.geo.page);
    }
}

// The kernels below: RG groups of 16 query rows, KH warps to a group, each with its share of every tile's positions.  Two
// tiles of K and V in shared memory.  The loop's first two turns only request tiles (one copy of the code: a launch runs
// through most of it once or twice, and each instruction's first fetch counts).

// ---- fp16 cache: m16n8k16, two terms on the query / probability side; tiles of 64 positions -------------------------
template <int HD, int RG, int KH>
__global__ void __launch_bounds__(RG * KH * 32, 1) k_attn_prefill_h(const AttnPrefillArgs a) {
    constexpr int ROWS = RG * 16, BN = 64, PB = BN / KH, NCH = HD / 8, NTH = RG * KH * 32;
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ size_t s_row[2][BN];
    __shared__ float s_inv[ROWS];
    __half* sQh = reinterpret_cast<__half*>(sm);
    __half* sQl = sQh + ROWS * HD;
    const uint32_t qh_s = ap_smem(sQh), ql_s = ap_smem(sQl), kv_s = ql_s + ROWS * HD * 2;
    constexpr uint32_t TILE = BN * HD * 2;                                              // stage s: K at kv_s + 2 s TILE, V behind it
    const int tid = threadIdx.x, warp = tid >> 5, rg = warp % RG, kh = warp / RG, lane = tid & 31, g = lane >> 2;
    pdl_launch_dependents();
    const AttnTile t = a.tiles[blockIdx.x];
    const uint32_t kvh = blockIdx.y, group = a.n_head / a.geo.n_kv;
    const __half* pool = reinterpret_cast<const __half*>(a.kv_pool);
    const int32_t* bt = a.block_table + (size_t)t.seq * a.geo.max_pages;
    auto sw = [](int r, int ch) { return NCH >= 8 ? ch ^ (r & 7) : ch ^ ((r >> 1) & (NCH - 1)); };
    const int kv_hi = t.pos + t.n_tok;                                                  // positions [.., kv_hi)
    const int kv_lo = a.window > 0 && t.pos + 1 > (int)a.window ? (t.pos + 1 - (int)a.window) / BN * BN : 0;
    const size_t v_off = (size_t)a.geo.n_kv * a.geo.page * HD;                          // a value row lies this far behind its key row
    const int pos[2] = {ap_row(a, t, kvh, group, rg * 16 + g, HD).pos, ap_row(a, t, kvh, group, rg * 16 + g + 8, HD).pos};
    // the warp's range of positions, to leave out tiles that it does not attend to
    const int tok_lo = (rg * 16) / (int)group, tok_hi = min((rg * 16 + 15) / (int)group, t.n_tok - 1);
    const bool live = tok_lo < t.n_tok;
    const int p_lo = t.pos + tok_lo, p_hi = t.pos + tok_hi;
    float o[HD / 8][4], m[2] = {AP_NEG, AP_NEG}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < HD / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[j][e] = 0.f;

    ap_locate<BN>(a, bt, kvh, kv_lo, kv_hi, s_row);     // the plan and the pages come from the host: no need to wait for them
    pdl_wait();
#pragma unroll 1
    for (int kv0 = kv_lo - 2 * BN; kv0 < kv_hi; kv0 += BN) {
        if (kv0 >= kv_lo) ap_wait<1>();
        __syncthreads();
        if (kv0 + 3 * BN < kv_hi) ap_locate<BN>(a, bt, kvh, kv0 + 3 * BN, kv_hi, s_row);
        const uint32_t k_s = kv_s + (uint32_t)((kv0 / BN) & 1) * 2u * TILE, v_s = k_s + TILE;
        const int part = kv0 + kh * PB;
        const bool work = kv0 >= kv_lo && live && part <= p_hi && !(a.window > 0 && part + PB - 1 + (int)a.window <= p_lo);
        if (kv0 == kv_lo - BN) {
            // the query rows: power-of-two scale per row, two fp16 terms; the row group's warps share them out
            constexpr int EPL = HD / 32, RB = KH == 4 ? 4 : 2;                          // values per lane, rows at a time
#pragma unroll 1
            for (int r0 = kh * (16 / KH); r0 < (kh + 1) * (16 / KH); r0 += RB) {
                float x[RB][EPL];
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    const ApRow row = ap_row(a, t, kvh, group, rg * 16 + r0 + r, HD);
#pragma unroll
                    for (int e = 0; e < EPL; ++e) x[r][e] = row.ok ? a.qkv[row.q + lane * EPL + e] : 0.f;
                }
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    float mxv = 0.f;
#pragma unroll
                    for (int e = 0; e < EPL; ++e) mxv = fmaxf(mxv, fabsf(x[r][e]));
                    mxv = warp_max(mxv);
                    int ex = 0;                                                         // largest element into [2^7, 2^8)
                    if (mxv > 0.f && mxv < 3.0e38f) ex = max(-100, min(100, 134 - (int)((__float_as_uint(mxv) >> 23) & 0xFFu)));
                    const float s = __uint_as_float((uint32_t)(127 + ex) << 23);
                    const int rr = rg * 16 + r0 + r;
                    if (lane == 0) s_inv[rr] = __uint_as_float((uint32_t)(127 - ex) << 23);
#pragma unroll
                    for (int e = 0; e < EPL; ++e) {
                        const int d = lane * EPL + e;
                        const float v = x[r][e] * s;
                        const __half h = __float2half_rn(v);
                        const int at = rr * HD + sw(rr, d >> 3) * 8 + (d & 7);
                        sQh[at] = h;
                        sQl[at] = __float2half_rn(v - __half2float(h));
                    }
                }
            }
        }
        if (work) {
            const bool edge = part + PB - 1 > p_lo || (a.window > 0 && part + (int)a.window <= p_hi);
            float c[PB / 8][4], alpha[2] = {1.f, 1.f};
            const float scl[2] = {s_inv[rg * 16 + g] * a.scale, s_inv[rg * 16 + g + 8] * a.scale};
#pragma unroll
            for (int j = 0; j < PB / 8; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) c[j][e] = 0.f;
#pragma unroll KH
            for (int k = 0; k < HD / 16; ++k) {
                uint32_t qh[4], ql[4];
                const int qr = rg * 16 + (lane & 15), qc = 2 * k + (lane >> 4);
                const uint32_t qo = (uint32_t)(qr * HD + sw(qr, qc) * 8) * 2u;
                ldsm4(qh_s + qo, qh);
                ldsm4(ql_s + qo, ql);
#pragma unroll
                for (int n = 0; n < PB / 16; ++n) {
                    uint32_t b[4];
                    const int kr = kh * PB + n * 16 + (lane >> 4) * 8 + (lane & 7), kc = 2 * k + ((lane >> 3) & 1);
                    ldsm4(k_s + (uint32_t)(kr * HD + sw(kr, kc) * 8) * 2u, b);
                    mma_h(c[2 * n], ql, b[0], b[1]); mma_h(c[2 * n + 1], ql, b[2], b[3]);
                    mma_h(c[2 * n], qh, b[0], b[1]); mma_h(c[2 * n + 1], qh, b[2], b[3]);
                }
            }
            uint32_t ph[PB / 16][4], pl[PB / 16][4];
            ap_softmax<PB / 8>(c, a, scl, pos, part, edge, m, l, alpha);
#pragma unroll
            for (int s = 0; s < PB / 16; ++s)
#pragma unroll
                for (int f = 0; f < 4; ++f) {           // times 256: the low terms stay clear of the fp16 subnormals
                    const float* p = &c[2 * s + (f >> 1)][2 * (f & 1)];
                    half_split(p[0] * 256.f, p[1] * 256.f, ph[s][f], pl[s][f]);
                }
            constexpr int DC = HD == 256 ? 32 : HD >= 64 ? 64 : HD;     // dims per round: what the registers beside `o` allow
#pragma unroll
            for (int d0 = 0; d0 < HD; d0 += DC) {
                float acc[DC / 8][4];
#pragma unroll
                for (int j = 0; j < DC / 8; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
                for (int s = 0; s < PB / 16; ++s)
#pragma unroll
                    for (int n = 0; n < DC / 16; ++n) {
                        uint32_t b[4];
                        const int vr = kh * PB + s * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), vc = d0 / 8 + 2 * n + (lane >> 4);
                        ldsm4t(v_s + (uint32_t)(vr * HD + sw(vr, vc) * 8) * 2u, b);
                        mma_h(acc[2 * n], pl[s], b[0], b[1]); mma_h(acc[2 * n + 1], pl[s], b[2], b[3]);
                        mma_h(acc[2 * n], ph[s], b[0], b[1]); mma_h(acc[2 * n + 1], ph[s], b[2], b[3]);
                    }
#pragma unroll
                for (int j = 0; j < DC / 8; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[d0 / 8 + j][e] = fmaf(o[d0 / 8 + j][e], alpha[e >> 1], acc[j][e]);
            }
        }
        __syncthreads();
        if (kv0 + 2 * BN < kv_hi) {
            const size_t* rows = s_row[(kv0 / BN) & 1];
#pragma unroll 4
            for (int i = tid; i < BN * NCH; i += NTH) {
                const int r = i / NCH, ch = i % NCH;
                const __half* src = pool + rows[r] + ch * 8;
                const uint32_t dst = (uint32_t)(r * HD + sw(r, ch) * 8) * 2u;
                ap_cp16(k_s + dst, src);
                ap_cp16(v_s + dst, src + v_off);
            }
        }
        ap_commit();
    }
    ap_wait<0>();
    ap_merge<HD, RG, KH>(reinterpret_cast<float4*>(sm), rg, kh, lane, o, m, l);
    if (kh == 0) ap_store<HD>(a, t, kvh, group, rg * 16, lane, o, l, 256.f);
}

// ---- fp32 cache: m16n8k8 tf32, three products per pair; tiles of 32 positions ---------------------------------------
// Operands stay fp32 in shared memory (rows padded by 4 floats: the fragment reads below are free of bank conflicts) and
// are split into two tf32 terms as they are read.
template <int HD, int RG, int KH>
__global__ void __launch_bounds__(RG * KH * 32, 1) k_attn_prefill_f(const AttnPrefillArgs a) {
    constexpr int ROWS = RG * 16, BN = 32, PB = BN / KH, LD = HD + 4, NTH = RG * KH * 32;
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ size_t s_row[2][BN];
    float *sQ = reinterpret_cast<float*>(sm), *sKV = sQ + ROWS * LD;                    // stage s: K at sKV + 2 s BN LD, V behind it
    const int tid = threadIdx.x, warp = tid >> 5, rg = warp % RG, kh = warp / RG, lane = tid & 31, g = lane >> 2, q = lane & 3;
    pdl_launch_dependents();
    const AttnTile t = a.tiles[blockIdx.x];
    const uint32_t kvh = blockIdx.y, group = a.n_head / a.geo.n_kv;
    const float* pool = reinterpret_cast<const float*>(a.kv_pool);
    const int32_t* bt = a.block_table + (size_t)t.seq * a.geo.max_pages;
    const int kv_hi = t.pos + t.n_tok;
    const int kv_lo = a.window > 0 && t.pos + 1 > (int)a.window ? (t.pos + 1 - (int)a.window) / BN * BN : 0;
    const size_t v_off = (size_t)a.geo.n_kv * a.geo.page * HD;
    const float scl[2] = {a.scale, a.scale};
    const int pos[2] = {ap_row(a, t, kvh, group, rg * 16 + g, HD).pos, ap_row(a, t, kvh, group, rg * 16 + g + 8, HD).pos};
    const int tok_lo = (rg * 16) / (int)group, tok_hi = min((rg * 16 + 15) / (int)group, t.n_tok - 1);
    const bool live = tok_lo < t.n_tok;
    const int p_lo = t.pos + tok_lo, p_hi = t.pos + tok_hi;
    float o[HD / 8][4], m[2] = {AP_NEG, AP_NEG}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < HD / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[j][e] = 0.f;

    ap_locate<BN>(a, bt, kvh, kv_lo, kv_hi, s_row);     // the plan and the pages come from the host: no need to wait for them
    pdl_wait();
#pragma unroll 1
    for (int kv0 = kv_lo - 2 * BN; kv0 < kv_hi; kv0 += BN) {
        if (kv0 >= kv_lo) ap_wait<1>();
        __syncthreads();
        if (kv0 + 3 * BN < kv_hi) ap_locate<BN>(a, bt, kvh, kv0 + 3 * BN, kv_hi, s_row);
        float *sK = sKV + (size_t)((kv0 / BN) & 1) * 2 * BN * LD, *sV = sK + BN * LD;
        const int part = kv0 + kh * PB;
        const bool work = kv0 >= kv_lo && live && part <= p_hi && !(a.window > 0 && part + PB - 1 + (int)a.window <= p_lo);
        if (kv0 == kv_lo - BN)
#pragma unroll 2
            for (int r = kh * (16 / KH); r < (kh + 1) * (16 / KH); ++r) {
                const ApRow row = ap_row(a, t, kvh, group, rg * 16 + r, HD);
#pragma unroll
                for (int d = lane; d < HD; d += 32) sQ[(rg * 16 + r) * LD + d] = row.ok ? a.qkv[row.q + d] : 0.f;
            }
        if (work) {
            const bool edge = part + PB - 1 > p_lo || (a.window > 0 && part + (int)a.window <= p_hi);
            float c[PB / 8][4], alpha[2] = {1.f, 1.f};
#pragma unroll
            for (int j = 0; j < PB / 8; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) c[j][e] = 0.f;
#pragma unroll KH
            for (int k = 0; k < HD; k += 8) {
                const float* qp = sQ + (rg * 16 + g) * LD + k + q;
                uint32_t ah[4], al[4];
                tf32_split(qp[0], ah[0], al[0]); tf32_split(qp[8 * LD], ah[1], al[1]);
                tf32_split(qp[4], ah[2], al[2]); tf32_split(qp[8 * LD + 4], ah[3], al[3]);
#pragma unroll
                for (int n = 0; n < PB / 8; ++n) {
                    const float* kp = sK + (kh * PB + n * 8 + g) * LD + k + q;
                    uint32_t b0h, b0l, b1h, b1l;
                    tf32_split(kp[0], b0h, b0l); tf32_split(kp[4], b1h, b1l);
                    mma_t(c[n], al, b0h, b1h); mma_t(c[n], ah, b0l, b1l); mma_t(c[n], ah, b0h, b1h);
                }
            }
            ap_softmax<PB / 8>(c, a, scl, pos, part, edge, m, l, alpha);
            // the order of the positions inside a step of 8 is free: slots t and t + 4 are positions 2 t and 2 t + 1, which is
            // how the scores lie in the registers
            uint32_t ph[PB / 8][4], pl[PB / 8][4];
#pragma unroll
            for (int s = 0; s < PB / 8; ++s) {
                tf32_split(c[s][0], ph[s][0], pl[s][0]); tf32_split(c[s][2], ph[s][1], pl[s][1]);
                tf32_split(c[s][1], ph[s][2], pl[s][2]); tf32_split(c[s][3], ph[s][3], pl[s][3]);
            }
            constexpr int DC = HD >= 64 ? 64 : HD;
#pragma unroll
            for (int d0 = 0; d0 < HD; d0 += DC) {
                float acc[DC / 8][4];
#pragma unroll
                for (int j = 0; j < DC / 8; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
                for (int s = 0; s < PB / 8; ++s)
#pragma unroll
                    for (int n = 0; n < DC / 8; ++n) {
                        const float* vp = sV + (kh * PB + s * 8 + 2 * q) * LD + d0 + n * 8 + g;
                        uint32_t b0h, b0l, b1h, b1l;
                        tf32_split(vp[0], b0h, b0l); tf32_split(vp[LD], b1h, b1l);
                        mma_t(acc[n], pl[s], b0h, b1h); mma_t(acc[n], ph[s], b0l, b1l); mma_t(acc[n], ph[s], b0h, b1h);
                    }
#pragma unroll
                for (int j = 0; j < DC / 8; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[d0 / 8 + j][e] = fmaf(o[d0 / 8 + j][e], alpha[e >> 1], acc[j][e]);
            }
        }
        __syncthreads();
        if (kv0 + 2 * BN < kv_hi) {
            const size_t* rows = s_row[(kv0 / BN) & 1];
            const uint32_t k_s = ap_smem(sK), v_s = ap_smem(sV);
#pragma unroll 4
            for (int i = tid; i < BN * (HD / 4); i += NTH) {
                const int r = i / (HD / 4), ch = i % (HD / 4);
                const float* src = pool + rows[r] + ch * 4;
                const uint32_t dst = (uint32_t)(r * LD + ch * 4) * 4u;
                ap_cp16(k_s + dst, src);
                ap_cp16(v_s + dst, src + v_off);
            }
        }
        ap_commit();
    }
    ap_wait<0>();
    ap_merge<HD, RG, KH>(reinterpret_cast<float4*>(sm), rg, kh, lane, o, m, l);
    if (kh == 0) ap_store<HD>(a, t, kvh, group, rg * 16, lane, o, l, 1.f);
}

// ---- host ----------------------------------------------------------------------------------------------------------
template <typename T>
static int prep_t(const AttnPrefillArgs& a, cudaStream_t stream, bool pdl) {
    const uint32_t warps = a.n_rows * (a.n_head + 2 * a.geo.n_kv);
    const dim3 grid((warps + 7) / 8);
    switch (a.head_dim) {
    case 32: launch_k(k_qkv_prep<T, 32>, grid, dim3(256), 0, stream, pdl, a); break;
    case 64: launch_k(k_qkv_prep<T, 64>, grid, dim3(256), 0, stream, pdl, a); break;
    case 128: launch_k(k_qkv_prep<T, 128>, grid, dim3(256), 0, stream, pdl, a); break;
    default: launch_k(k_qkv_prep<T, 256>, grid, dim3(256), 0, stream, pdl, a); break;
    }
    count_launch();
    return check_launch("qkv_prep");
}
int launch_qkv_prep(const AttnPrefillArgs& a, bool kv_half, cudaStream_t stream, bool pdl) {
    return kv_half ? prep_t<__half>(a, stream, pdl) : prep_t<float>(a, stream, pdl);
}

template <int HD, int RG, int KH>
static int attn_t(const AttnPrefillArgs& a, bool kv_half, cudaStream_t stream, bool pdl) {
    constexpr size_t rows = RG * 16, smem_h = (2 * rows + 4 * 64) * HD * 2, smem_f = (rows + 4 * 32) * (HD + 4) * 4;
    constexpr size_t merge = (size_t)(KH / 2) * RG * (HD / 8 + 1) * 32 * 16;
    static_assert(merge <= smem_h && merge <= smem_f && smem_h <= 225 * 1024 && smem_f <= 225 * 1024, "shared memory");
    void (*k)(const AttnPrefillArgs) = kv_half ? k_attn_prefill_h<HD, RG, KH> : k_attn_prefill_f<HD, RG, KH>;
    const size_t smem = kv_half ? smem_h : smem_f;
    static bool set[2] = {false, false};
    if (!set[kv_half]) {
        if (cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return fail(ADAMAH_ERR_BACKEND, "attn_prefill: cannot raise the shared-memory limit");
        set[kv_half] = true;
    }
    launch_k(k, dim3(a.n_tiles, a.geo.n_kv), dim3(RG * KH * 32), smem, stream, pdl, a);
    count_launch();
    return check_launch("attn_prefill");
}
template <int HD>
static int attn_r(const AttnPrefillArgs& a, bool kv_half, uint32_t rows, cudaStream_t stream, bool pdl) {
    if constexpr (HD <= 128)
        if (rows == 128) return attn_t<HD, 8, 1>(a, kv_half, stream, pdl);
    return rows == 64 ? attn_t<HD, 4, 2>(a, kv_half, stream, pdl) : attn_t<HD, 2, 4>(a, kv_half, stream, pdl);
}
int launch_attn_prefill(const AttnPrefillArgs& a, bool kv_half, uint32_t tile_rows, cudaStream_t stream, bool pdl) {
    switch (a.head_dim) {
    case 32: return attn_r<32>(a, kv_half, tile_rows, stream, pdl);
    case 64: return attn_r<64>(a, kv_half, tile_rows, stream, pdl);
    case 128: return attn_r<128>(a, kv_half, tile_rows, stream, pdl);
    default: return attn_r<256>(a, kv_half, tile_rows, stream, pdl);
    }
}

}  // namespace ab
