// Dequant-fused GEMM  y[b][n] = sum_k W[n][k] x[b][k]  for a few activation rows b (decode batches, short prompts) over
// the row-tiled Q4_0 / Q4_K copies (tile.cu), on mma.sync.  Same operator as gemm_tc.cu (the reference's Q4 mat-vec shader
// adamah-MAIN/adamah/shaders/src/f32/map_matvec_t_xq4.comp and map_fused_gateup_t_xq4.comp run once per row by adamah.c:8606-8691).
//
// Why not tcgen05 here.  Its weight operand is w = d (q - 8), rebuilt as two fp16 terms: 7.6 thread instructions per weight
// whatever the rows, which is all of the time of a call with few.  An accumulator that restarts with every block of 32 weights
// lets the operand be the code q itself and the block scale meet the block's sums instead of its weights.  In tensor memory that
// accumulator would have to be read back for every block; the registers of mma.sync.m16n8k16 are where the sums are wanted.
//
// Arithmetic.  A row of activations is scaled by a power of two and split into two fp16 terms x_hi + x_lo (22 bits of every
// element; k_quant_rows); two columns of B hold a row's terms.  A block is two instructions (K = 16 each) that add up
// sum((q - 8) x) from zero, and acc += d * sum in fp32, the two terms apart until the end.  Q4_K: w = d sc (q - 8) +
// (8 d sc - dmin m); the second part multiplies the block's sum of activations, kept in fp32.  The tensor core rounds towards
// zero, but only within a block (two additions): relative error of a product 6e-8 to 1.7e-7, with activations of mean 1 too,
// where gemm_tc.cu has 2e-7 to 3.4e-7 and the GEMV 1.8e-7 to 7e-7.  (A nibble masked out of its word is a subnormal half, q 2^-24
// or q 2^-20, and needs no conversion; but the tensor core aligns its products by their nominal exponents: 4e-7 to 1e-6.)
//
// One CTA per SM: 16 warps at most that multiply (12 where their sums need the registers) and one that fetches.  A unit is GW row
// groups of 16 rows (for a gate / up product the same 16 rows of both matrices); warp (r, s) owns unit
// r of the CTA's U and slice s of KS of every stage's K.  A stage is KS * C tile pairs (64 values of K each) of all units and the
// same K of the activation image, by bulk copies onto one mbarrier.  Work is dealt out as whole items (U units over all of
// K) or, where those leave SMs idle, as stages of all items in a row; an item that several CTAs share is added up by the one
// that ends last, in the order of K, so results do not depend on timing.
// Every wait is bounded: when one runs out the kernel records DEVERR_WAIT, stops waiting and returns.
#include "gemm_tc.cuh"
#include "gemv_mma.cuh"

#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <unordered_map>

namespace ab {

constexpr int GM_SMEM = 220 * 1024;
constexpr int GM_MAX_STAGES = 8;
__host__ __device__ constexpr int gm_warps(int ntl, int gw) { return gw == 2 && ntl > 1 ? 12 : 16; }        // warps that multiply, at most

struct GmArgs {
    const uint8_t *t0, *t1;                             // row-tiled weights; t1: up rows of a pair
    const uint8_t* img; const float* inv; uint32_t* err;
    float* y; int ldy;
    int N, n_rg, pairs, B;                              // rows, row groups and tile pairs along K of one matrix
    int pair, swiglu;
    int U, KS, C, NS, spi, items, shared;               // see above; spi = stages per item
    float* part; unsigned int* tickets;                 // shared items: per CTA the sums of its first and last one; arrivals, by the CTA in which an item begins
    unsigned long long* best; unsigned int* ticket;     // arg-max: one key per activation row (0 between launches), CTAs that are done
    int* out_tok; float *out_val, *out_tok_f32, softcap;
};

// D (+)= A (16 x 16, fp16) * B (16 x 8, fp16), fp32 sums
__device__ __forceinline__ void hmma_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void hmma_add(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t h2_add(uint32_t v, float c) {
    const __half2 r = __hadd2(*reinterpret_cast<__half2*>(&v), __float2half2_rn(c));
    return *reinterpret_cast<const uint32_t*>(&r);
}
// The eight codes of a word, less 8, as pairs of halves: low nibbles of bytes (0, 2) and (1, 3) to p[0], p[2], the high ones to
// p[4], p[6].  A nibble lands in the mantissa of 1024 (bits 0..3) or of 64 (bits 4..7).  The constants come in registers that the
// compiler cannot look into: one lop3 takes only one literal.
struct GmMasks { uint32_t lo, hi, k1024, k64; };
__device__ __forceinline__ GmMasks gm_masks() {
    GmMasks m;
    asm volatile("mov.u32 %0, 0x000F000F;\n\tmov.u32 %1, 0x00F000F0;\n\tmov.u32 %2, 0x64006400;\n\tmov.u32 %3, 0x54005400;" : "=r"(m.lo), "=r"(m.hi), "=r"(m.k1024), "=r"(m.k64));
    return m;
}
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ void codes_h2(const GmMasks& m, uint32_t w, uint32_t* p) {
    const uint32_t v = w >> 8;
    p[0] = h2_add(and_or(w, m.lo, m.k1024), -1032.f);
    p[2] = h2_add(and_or(v, m.lo, m.k1024), -1032.f);
    p[4] = h2_add(and_or(w, m.hi, m.k64), -72.f);
    p[6] = h2_add(and_or(v, m.hi, m.k64), -72.f);
}
__device__ __forceinline__ uint4 lds4(uint32_t at) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at));
    return v;
}
__device__ __forceinline__ uint2 lds2(uint32_t at) { uint2 v; asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(at)); return v; }
__device__ __forceinline__ float lds1(uint32_t at) { float v; asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at)); return v; }
// Packed fp32 pairs (one instruction for two).
__device__ __forceinline__ float2 add_2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 ra, rb;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tadd.rn.f32x2 ra, ra, rb;\n\tmov.b64 {%0, %1}, ra;\n\t}" : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 mul_2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 ra, rb;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmul.rn.f32x2 ra, ra, rb;\n\tmov.b64 {%0, %1}, ra;\n\t}" : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
// Bytes i and j of a word as floats: into the mantissa of 2^23.
__device__ __forceinline__ float2 bytes_2(uint32_t w, uint32_t i, uint32_t j) {
    return add_2(make_float2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | i)), __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | j))), make_float2(-8388608.f, -8388608.f));
}

template <int WT, int NTL, int GW, bool HEAD>           // NTL: groups of four activation rows; GW: row groups per warp
__global__ void __launch_bounds__((gm_warps(NTL, GW) + 1) * 32, 1) k_gemm_mma(const GmArgs a) {
    constexpr int BP = 4 * NTL, TILE = MmaGeo<false, WT>::TILE, BLK = gm_block_bytes(WT, BP), NV = NTL * 2 * GW;      // NV: sums per lane
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ __align__(8) uint64_t full[GM_MAX_STAGES], empty[GM_MAX_STAGES];
    __shared__ bool s_last;
    __shared__ float s_inv[BP];
    [[maybe_unused]] __shared__ unsigned long long s_best[HEAD ? BP : 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int U = a.U, KS = a.KS, C = a.C, NS = a.NS, n_mul = U * KS, step = KS * C, spi = a.spi;
    const bool pair = GW == 2 && !HEAD && a.pair != 0;
    const uint32_t w_bytes = (uint32_t)(U * GW * step * TILE), st_bytes = w_bytes + (uint32_t)(step * 2 * BLK);
    float* red = reinterpret_cast<float*>(sm + (size_t)NS * st_bytes);                  // [n_mul][NV][32] (KS > 1)
    const long long all = (long long)a.items * spi;
    const int cta = (int)blockIdx.x, n_cta = (int)gridDim.x;
    auto q_begin = [&](int c) { return (int)(c * all / n_cta); };
    const int q0 = a.shared ? q_begin(cta) : 0, q1 = a.shared ? q_begin(cta + 1) : (a.items - cta + n_cta - 1) / n_cta * spi;
    auto item_of = [&](int i) { return a.shared ? i : cta + i * n_cta; };
    if (tid == 0) {
        for (int i = 0; i < NS; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], (uint32_t)n_mul); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if constexpr (HEAD) { if (tid < BP) s_best[tid] = 0; }
    __syncthreads();
    bool dead = false;
    auto wait_on = [&](uint64_t* bar, uint32_t parity) {
        if (!dead && !mbar_wait(bar, parity)) { dead = true; atomicOr(a.err, DEVERR_WAIT); }
    };
    pdl_launch_dependents();

    if (warp == n_mul) {
        // ---- fetch: a lane per row group, lane 0 the activations too; the first stages' weights ahead of the wait ----
        const uint8_t* base = pair && (lane & 1) ? a.t1 : a.t0;
        auto weights = [&](int q, int slot) {
            const int i = q / spi, p0 = (q - i * spi) * step, n = min(step, a.pairs - p0);
            if (lane == 0) mbar_expect_tx(&full[slot], (uint32_t)(n * (U * GW * TILE + 2 * BLK)));
            __syncwarp();
            if (lane < U * GW) {
                const int at = pair ? item_of(i) * U + (lane >> 1) : item_of(i) * U * GW + lane;
                bulk_g2s(sm + (size_t)slot * st_bytes + lane * step * TILE, base + ((size_t)min(at, a.n_rg - 1) * a.pairs + p0) * TILE, (uint32_t)(n * TILE), &full[slot]);
            }
        };
        auto rows = [&](int q, int slot) {
            const int p0 = (q % spi) * step, n = min(step, a.pairs - p0);
            if (lane == 0) bulk_g2s(sm + (size_t)slot * st_bytes + w_bytes, a.img + (size_t)p0 * 2 * BLK, (uint32_t)(n * 2 * BLK), &full[slot]);
        };
        const int pre = min(NS, q1 - q0);
        for (int n = 0; n < pre; ++n) weights(q0 + n, n);
        pdl_wait();
        for (int n = 0; n < pre; ++n) rows(q0 + n, n);
        int slot = 0; uint32_t par = 0;
        for (int q = q0 + pre; q < q1; ++q) {
            wait_on(&empty[slot], par);
            weights(q, slot);
            rows(q, slot);
            if (++slot == NS) { slot = 0; par ^= 1u; }
        }
        // no copy may be in flight when the CTA ends, whatever became of the waits
        const int total = q1 - q0;
        for (int n = total - pre; n < total; ++n) mbar_wait(&full[n % NS], (uint32_t)(n / NS) & 1u);
    } else if (warp < n_mul) {
        const int g = lane >> 2, t = lane & 3, r_own = warp / KS, s_own = warp - r_own * KS;
        auto sync_mul = [&]() { asm volatile("bar.sync 1, %0;" :: "r"(n_mul * 32) : "memory"); };
        auto sync_unit = [&]() { asm volatile("bar.sync %0, %1;" :: "r"(2 + r_own), "r"(KS * 32) : "memory"); };      // KS > 1: at most 8 units
        float acc[GW][NTL][4];                          // rows g and g + 8: the sums with x_hi and x_lo
#pragma unroll
        for (int w = 0; w < GW; ++w)
#pragma unroll
            for (int i = 0; i < NTL; ++i) acc[w][i][0] = acc[w][i][1] = acc[w][i][2] = acc[w][i][3] = 0.f;
        [[maybe_unused]] float best_v[HEAD ? NTL : 1];
        [[maybe_unused]] int best_r[HEAD ? NTL : 1];
        if constexpr (HEAD) {
#pragma unroll
            for (int i = 0; i < NTL; ++i) { best_v[i] = 0.f; best_r[i] = -1; }
        }
        pdl_wait();
        for (int b = tid; b < a.B; b += n_mul * 32) s_inv[b] = a.inv[b];
        sync_mul();
        // The sum of row `row` of a unit's matrix (i: which of the lane's activation rows) goes out; a pair gives gate and up.
        auto store = [&](int i, int row, float v, float up) {
            const int b = 4 * i + t;
            if (b >= a.B || row >= a.N) return;
            v *= s_inv[b];
            if (pair) v = gated(v, a.swiglu ? silu_arg(v) : gelu_arg(v)) * (up * s_inv[b]);
            if constexpr (HEAD) {                       // NaN counts as -FLT_MAX, ties go to the lower row: a lane's rows ascend
                const float f = v == v ? v : -3.402823466e+38f;
                if (f > best_v[i] || best_r[i] < 0) { best_v[i] = f; best_r[i] = row; }
                if (a.y) a.y[(size_t)b * a.ldy + row] = a.softcap > 0.f ? tanhf(v / a.softcap) * a.softcap : v;
            } else a.y[(size_t)b * a.ldy + row] = v;
        };
        const uint32_t sm_s = smem_u32(sm);
        const GmMasks masks = gm_masks();
        int slot = 0; uint32_t par = 0;
        for (int q = q0; q < q1;) {
            const int i0 = q / spi, j0 = q - i0 * spi, j1 = min(spi, j0 + q1 - q), item = item_of(i0);
            q += j1 - j0;
            for (int j = j0; j < j1; ++j) {
                wait_on(&full[slot], par);
                uint32_t wb = sm_s + (uint32_t)slot * st_bytes + (uint32_t)((r_own * GW * step + s_own * C) * TILE);
                uint32_t xb = sm_s + (uint32_t)slot * st_bytes + w_bytes + (uint32_t)(s_own * C * 2 * BLK) + lane * 16;
                const int n = min(C, a.pairs - j * step - s_own * C);
                uint4 qn[GW]; uint2 sn[GW], hn[GW];     // the next tile pair's codes and scales
                auto fetch = [&](uint32_t at) {
#pragma unroll
                    for (int w = 0; w < GW; ++w) {
                        const uint32_t tile = at + (uint32_t)(w * step * TILE);
                        qn[w] = lds4(tile + lane * 16);
                        sn[w] = lds2(tile + 512 + g * 8);
                        if constexpr (WT == WT_Q4_K) hn[w] = lds2(tile + 576 + g * 8);
                    }
                };
                if (n > 0) fetch(wb);
#pragma unroll 1
                for (int k = 0; k < n; ++k, xb += 2 * BLK) {
                    uint4 qv[GW]; uint2 sc[GW];
                    [[maybe_unused]] float2 dm[GW][2];
#pragma unroll
                    for (int w = 0; w < GW; ++w) {
                        qv[w] = qn[w]; sc[w] = sn[w];
                        if constexpr (WT == WT_Q4_K) {
                            dm[w][0] = __half22float2(*reinterpret_cast<const __half2*>(&hn[w].x));
                            dm[w][1] = __half22float2(*reinterpret_cast<const __half2*>(&hn[w].y));
                        }
                    }
                    if (k + 1 < n) wb += TILE;
                    fetch(wb);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        uint32_t p[GW][8];              // A fragments of the low nibbles (rows g and g + 8 in turn), then of the high ones
                        float d[GW][2];
                        [[maybe_unused]] float o[GW][2];
#pragma unroll
                        for (int w = 0; w < GW; ++w) {
                            const uint32_t wg = u ? qv[w].z : qv[w].x, wh = u ? qv[w].w : qv[w].y, s2 = u ? sc[w].y : sc[w].x;
                            codes_h2(masks, wg, &p[w][0]);
                            codes_h2(masks, wh, &p[w][1]);
                            if constexpr (WT == WT_Q4_0) {
                                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&s2));
                                d[w][0] = f.x; d[w][1] = f.y;
                            } else {
                                const float2 es = mul_2(make_float2(dm[w][0].x, dm[w][1].x), bytes_2(s2, 0, 2)), em = mul_2(make_float2(dm[w][0].y, dm[w][1].y), bytes_2(s2, 1, 3));
                                d[w][0] = es.x; d[w][1] = es.y;
                                o[w][0] = fmaf(8.f, es.x, -em.x); o[w][1] = fmaf(8.f, es.y, -em.y);
                            }
                        }
#pragma unroll
                        for (int i = 0; i < NTL; ++i) {
                            const uint4 b = lds4(xb + u * BLK + i * 512);
                            [[maybe_unused]] float sx;
                            if constexpr (WT == WT_Q4_K) sx = lds1(xb - lane * 16 + t * 4 + u * BLK + 128 * BP + 16 * i);
#pragma unroll
                            for (int w = 0; w < GW; ++w) {
                                float s[4], (&ac)[4] = acc[w][i];
                                hmma_zero(s, p[w][0], p[w][1], p[w][2], p[w][3], b.x, b.y);
                                hmma_add(s, p[w][4], p[w][5], p[w][6], p[w][7], b.z, b.w);
                                ac[0] = fmaf(d[w][0], s[0], ac[0]); ac[1] = fmaf(d[w][0], s[1], ac[1]);
                                ac[2] = fmaf(d[w][1], s[2], ac[2]); ac[3] = fmaf(d[w][1], s[3], ac[3]);
                                if constexpr (WT == WT_Q4_K) {
                                    ac[0] = fmaf(o[w][0], sx, ac[0]);
                                    ac[2] = fmaf(o[w][1], sx, ac[2]);
                                }
                            }
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(&empty[slot])) : "memory");
                if (++slot == NS) { slot = 0; par ^= 1u; }
            }
            // ---- the item's sums (or this CTA's part of them) ----
            const int unit = item * U + r_own;          // of the call
            auto row_of = [&](int w, int h) { return (pair ? unit * 16 : (unit * GW + w) * 16) + 8 * h + g; };
            const bool part = j1 - j0 < spi;
            if (KS == 1 && !part) {
#pragma unroll
                for (int w = 0; w < GW; ++w)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (pair && w == 1) continue;
#pragma unroll
                        for (int i = 0; i < NTL; ++i)
                            store(i, row_of(w, h), acc[w][i][2 * h] + acc[w][i][2 * h + 1], acc[GW - 1][i][2 * h] + acc[GW - 1][i][2 * h + 1]);
                    }
            }
            float* mine = red + (size_t)warp * NV * 32 + lane;
#pragma unroll
            for (int w = 0; w < GW; ++w)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < NTL; ++i) {     // sum (w, h, i) of a lane
                        if (KS > 1 || part) mine[((w * 2 + h) * NTL + i) * 32] = acc[w][i][2 * h] + acc[w][i][2 * h + 1];
                        acc[w][i][2 * h] = acc[w][i][2 * h + 1] = 0.f;
                    }
            if (KS == 1 && !part) continue;
            if (KS > 1) sync_unit(); else __syncwarp();
            auto sum_of = [&](int v) {                  // over the slices of K
                const float* f = red + (size_t)(r_own * KS) * NV * 32 + v * 32 + lane;
                float r = f[0];
                for (int s = 1; s < KS; ++s) r += f[(size_t)s * NV * 32];
                return r;
            };
            int c_lo = 0, c_hi = 0;
            auto slot_of = [&](int c) { return a.part + (size_t)(2 * c + (c == c_lo ? 1 : 0)) * GEMM_SLOT + (size_t)r_own * NV * 32 + lane; };     // it begins here, or before
            if (part) {
                // an item that several CTAs share: leave the partial sums; the CTA that arrives last adds all of them
                auto cta_of = [&](int qq) {
                    int c = (int)((long long)qq * n_cta / all);
                    while (q_begin(c) > qq) --c;
                    while (q_begin(c + 1) <= qq) ++c;
                    return c;
                };
                c_lo = cta_of(item * spi); c_hi = cta_of(item * spi + spi - 1);
                float* out = slot_of(cta);
                for (int v = s_own; v < NV; v += KS) out[v * 32] = sum_of(v);
                __threadfence();
                sync_mul();
                if (tid == 0) {
                    const unsigned int seen = atomicAdd(a.tickets + c_lo, 1u);
                    s_last = seen == (unsigned int)(c_hi - c_lo);
                    if (s_last) a.tickets[c_lo] = 0u;
                }
                sync_mul();
                const bool last = s_last;
                sync_mul();
                if (!last) continue;
                __threadfence();
            }
            auto total_of = [&](int v) {
                if (!part) return sum_of(v);
                float r = 0.f;
                for (int c = c_lo; c <= c_hi; ++c) r += __ldcg(slot_of(c) + v * 32);
                return r;
            };
#pragma unroll
            for (int i = 0; i < NTL; ++i)
                for (int wh = s_own; wh < (pair ? 2 : 2 * GW); wh += KS) {
                    const float v = total_of(wh * NTL + i), up = pair ? total_of((2 + wh) * NTL + i) : 0.f;
                    store(i, row_of(wh >> 1, wh & 1), v, up);
                }
            if (KS > 1) sync_unit();                    // the exchange is free again
        }
        if constexpr (HEAD) {                           // the lanes' winners to the CTA's; the last CTA to end decodes the GPU's and clears the keys
#pragma unroll
            for (int i = 0; i < NTL; ++i) {
                unsigned long long key = 0;
                if (best_r[i] >= 0) {
                    const uint32_t bits = __float_as_uint(best_v[i] + 0.f), ord = bits ^ ((uint32_t)((int)bits >> 31) | 0x80000000u);
                    key = ((unsigned long long)ord << 32) | (0xffffffffu - (uint32_t)best_r[i]);
                }
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) { const unsigned long long k = __shfl_xor_sync(0xffffffffu, key, o); if (k > key) key = k; }
                if (g == 0 && key) atomicMax(&s_best[4 * i + t], key);
            }
            sync_mul();
            for (int b = tid; b < a.B; b += n_mul * 32) if (s_best[b]) atomicMax(a.best + b, s_best[b]);
            __threadfence();
            sync_mul();
            if (tid == 0) s_last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
            sync_mul();
            if (s_last) {
                __threadfence();
                for (int b = tid; b < a.B; b += n_mul * 32) {
                    const unsigned long long key = __ldcg(a.best + b);
                    const uint32_t ord = (uint32_t)(key >> 32);
                    const int tok = (int)(0xffffffffu - (uint32_t)key);
                    if (a.out_tok) a.out_tok[b] = tok;
                    if (a.out_tok_f32) a.out_tok_f32[b] = (float)tok;
                    if (a.out_val) a.out_val[b] = __uint_as_float(ord & 0x80000000u ? ord ^ 0x80000000u : ~ord);
                    a.best[b] = 0;
                }
                if (tid == 0) *a.ticket = 0u;
            }
        }
    }
}

// ---- host ----------------------------------------------------------------------------------------------------------
typedef void (*GmKernel)(const GmArgs);
template <int WT, int GW, bool HEAD> static GmKernel gm_kernel(int ntl) {
    return ntl == 1 ? k_gemm_mma<WT, 1, GW, HEAD> : ntl == 2 ? k_gemm_mma<WT, 2, GW, HEAD> : ntl == 3 ? k_gemm_mma<WT, 3, GW, HEAD> : k_gemm_mma<WT, 4, GW, HEAD>;
}
int gemm_mma_pad(int B) { return (B + 3) / 4 * 4; }

bool gemm_mma_supports(int wtype, const GemvArgs& a) {
    return (wtype == WT_Q4_0 || wtype == WT_Q4_K) && a.B <= GM_MAX_ROWS && a.N % 16 == 0 && a.K % (wtype == WT_Q4_0 ? 64 : 256) == 0;
}

struct GmCall { bool q40, pair, head; int N, K, B; };
struct GmShape { int gw, U, KS, C, NS, grid; bool shared; };
static int gm_groups(const GmCall& p) { return (p.B + 3) / 4; }
static int gm_wt(const GmCall& p) { return p.q40 ? WT_Q4_0 : WT_Q4_K; }
static size_t gm_stage_bytes(const GmCall& p, const GmShape& f) {
    return (size_t)f.KS * f.C * ((size_t)f.U * f.gw * mma_tile_bytes(gm_wt(p)) + 2 * gm_block_bytes(gm_wt(p), 4 * gm_groups(p)));
}
static size_t gm_red_bytes(const GmCall& p, const GmShape& f) { return f.KS > 1 || f.shared ? (size_t)f.U * f.KS * gm_groups(p) * 2 * f.gw * 128 : 0; }
static int gm_steps(const GmCall& p, const GmShape& f) { return (p.K / 64 + f.KS * f.C - 1) / (f.KS * f.C); }      // stages per item
static int gm_items(const GmCall& p, const GmShape& f) {
    const int n_rg = p.N / 16, units = p.pair ? n_rg : (n_rg + f.gw - 1) / f.gw;
    return (units + f.U - 1) / f.U;
}
static int gm_item_floats(const GmCall& p, const GmShape& f) { return f.U * gm_groups(p) * 2 * f.gw * 32; }         // sums of one item
// Number of stages that fit (f.NS); false where that is too few, or where a shared item's sums do not fit the workspace.  One stage
// is enough for a CTA that has one item; with more it would fetch nothing while it multiplies: 21504 x 5376 Q4_K on 4 rows 33.2 us
// instead of 24.2, 131072 x 2560 Q4_0 on 4 rows 61.2 instead of 47.7, 65536 x 1536 Q4_0 on 16 rows 41.3 instead of 29.2.
static bool gm_fits(const GmCall& p, GmShape& f, int sm_count) {
    if (f.shared && gm_item_floats(p, f) > GEMM_SLOT) return false;
    const size_t room = GM_SMEM - gm_red_bytes(p, f), st = gm_stage_bytes(p, f);
    f.NS = room < st ? 0 : (int)(room / st);
    if (f.NS > GM_MAX_STAGES) f.NS = GM_MAX_STAGES;
    return f.NS >= 2 || (f.NS == 1 && gm_steps(p, f) == 1 && !f.shared && gm_items(p, f) <= sm_count);
}
// Shape: the cheapest under an estimate in SM cycles, fitted to sweeps of shapes on 262144 x 1152, 21504 x 5376, 1536 x 1152, 6912 x 1152
// and 1152 x 6912 (2, 8 and 16 rows) and on ten products with long K (8, 12 and 16 rows, 2520 shapes in all): a warp's tile pair
// takes 137 cycles of latency and a share of the SM's pipes that grows with the warps and the rows, no less than its bytes from HBM
// and those of the activation image from L2 (86 a cycle); a stage some 140 cycles, 60 for each of its bulk copies and 60 more where
// the next one alone is in flight; an item its exchange, the slices of K one after the other; sharing items the workspace (about 8 us).
// The shapes chosen so are 1.5 % slower than the best measured ones, 5.6 % without the image and with a cheaper exchange and
// workspace: 2560 x 10240 Q4_K on 12 rows 22.0 us and 19.4, 24576 x 1024
// Q4_0 on 16 rows 13.2 and 10.6, 131072 x 2560 Q4_0 on 8 rows 71.2 and 56.6; 6912 x 1152 Q4_0 on 8 rows 5.49 and 5.69.
static GmShape gm_search(const GmCall& p, int sm_count) {
    const int ntl = gm_groups(p), pairs = p.K / 64;
    GmShape s = {};
    double best = 1e300;
    const double share = (p.q40 ? 15.0 : 21.0) + (p.q40 ? 10.0 : 11.0) * ntl, bytes = mma_tile_bytes(gm_wt(p)) / 23.0, img = 2 * gm_block_bytes(gm_wt(p), 4 * ntl) / 86.0;
    for (int gw = p.pair ? 2 : 1; gw <= (p.head ? 1 : 2); ++gw)
        for (int U = 1; U <= gm_warps(ntl, gw) && U * gw <= 32; ++U)
            for (int ks = 1; U * ks <= gm_warps(ntl, gw) && ks <= pairs && (U <= 8 || ks == 1); ++ks)
                for (int c = 1; c <= 8 && (c == 1 || ks * (c - 1) < pairs); ++c)
                    for (int sh = 0; sh < 2; ++sh) {
                        GmShape f = {gw, U, ks, c, 0, 0, sh != 0};
                        if (!gm_fits(p, f, sm_count)) continue;
                        const int step = ks * c, spi = gm_steps(p, f), items = gm_items(p, f), rest = pairs - (spi - 1) * step;
                        const double nw = U * ks, lone = (137.0 + 30.0 * (gw - 1)) + nw * gw * share, mem = nw * gw * bytes + ks * img;
                        const double per_pair = lone > mem ? lone : mem, fixed = 140.0 + 60.0 * U * gw + (f.NS == 2 ? 60.0 : 0.0);
                        const double finish = 400.0 + (ks > 1 ? 1000.0 + 14.0 * ks * ntl * gw : 0.0);
                        const double item = (spi - 1) * (c * per_pair + fixed) + (rest < c ? rest : c) * per_pair + fixed;
                        const int whole = items < sm_count ? items : sm_count;
                        double cost;
                        if (sh) {
                            const long long all = (long long)items * spi;
                            if (all <= sm_count || items % sm_count == 0) continue;
                            const double per = (double)((all + sm_count - 1) / sm_count);
                            cost = per * (c * per_pair + fixed) + (1.0 + per / spi) * finish + 15000.0 + spi / per * 300.0;
                            f.grid = sm_count;
                        } else { cost = (double)((items + whole - 1) / whole) * (item + finish); f.grid = whole; }
                        if (cost < best * 0.999) { best = cost; s = f; }
                    }
    return s;
}

// ADAM_B200_GM_SHAPE="row groups per warp,units,k_slices,tile pairs,shared" (a tuning aid, read once) in place of the estimate
// wherever a call can be launched so.
static GmShape gm_forced(const GmCall& p, int sm_count, GmShape s) {
    struct Force { bool set; int v[5]; };
    static const Force force = [] {
        Force f = {};
        const char* e = getenv("ADAM_B200_GM_SHAPE");
        f.set = e && sscanf(e, "%d,%d,%d,%d,%d", &f.v[0], &f.v[1], &f.v[2], &f.v[3], &f.v[4]) == 5;
        return f;
    }();
    if (!force.set) return s;
    GmShape f = {p.pair ? 2 : p.head ? 1 : force.v[0], force.v[1], force.v[2], force.v[3], 0, 0, force.v[4] != 0};
    const int warps = gm_warps(gm_groups(p), f.gw);
    if ((f.gw != 1 && f.gw != 2) || f.U < 1 || f.U > warps || f.U * f.gw > 32 || f.KS < 1 || f.KS > warps / f.U || f.KS > p.K / 64 || f.C < 1 || f.C > 8 || (f.U > 8 && f.KS > 1))
        return s;
    const int items = gm_items(p, f);
    if ((long long)items * gm_steps(p, f) <= sm_count) f.shared = false;
    if (!gm_fits(p, f, sm_count)) return s;
    f.grid = f.shared || items > sm_count ? sm_count : items;
    return f;
}
// The search takes 4 to 16 us, as long as a small product: a shape is kept for the next call of the same problem.
static GmShape gm_shape(const GmCall& p, int sm_count) {
    static std::mutex lock;
    static std::unordered_map<uint64_t, GmShape> known;
    const uint64_t key = (uint64_t)(uint32_t)(p.N / 16) | (uint64_t)(p.K / 64) << 28 | (uint64_t)gm_groups(p) << 40 | (uint64_t)(p.q40 ? 1 : 0) << 44 |
                         (uint64_t)(p.pair ? 1 : p.head ? 2 : 0) << 45 | (uint64_t)sm_count << 48;
    std::lock_guard<std::mutex> work(lock);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    const GmShape s = gm_forced(p, sm_count, gm_search(p, sm_count));
    if (known.size() >= 4096) known.clear();
    known[key] = s;
    if (getenv("ADAM_B200_DEBUG"))
        fprintf(stderr, "[gemm_mma] N %d K %d rows %d pair %d: %d,%d,%d,%d,%d, %d stages, grid %d\n", p.N, p.K, 4 * gm_groups(p), (int)p.pair, s.gw, s.U, s.KS, s.C, (int)s.shared, s.NS, s.grid);
    return s;
}

int gemm_mma_ctas(int wtype, const GemvArgs& a) {
    const GmCall p = {wtype == WT_Q4_0, a.epi == EPI_GEGLU || a.epi == EPI_SWIGLU, a.epi == EPI_ARGMAX, a.N, a.K, a.B};
    return gm_shape(p, g.sm_count).grid;
}

int launch_gemm_mma(int wtype, const uint8_t* t0, const uint8_t* t1, const GemvArgs& a, const GemmWork& w, cudaStream_t stream) {
    const bool pair = a.epi == EPI_GEGLU || a.epi == EPI_SWIGLU, head = a.epi == EPI_ARGMAX, q40 = wtype == WT_Q4_0;
    const GmCall p = {q40, pair, head, a.N, a.K, a.B};
    const int ntl = gm_groups(p), pairs = a.K / 64, n_rg = a.N / 16;
    const GmShape s = gm_shape(p, g.sm_count);
    if (!s.U) return fail(ADAMAH_ERR_INVALID, "gemm_mma: shape not supported");
    GmArgs m = {};
    m.t0 = t0; m.t1 = t1; m.img = w.img; m.inv = w.inv; m.err = g.dev_err; m.y = a.y; m.ldy = a.ldy;
    m.N = a.N; m.n_rg = n_rg; m.pairs = pairs; m.B = a.B; m.pair = pair; m.swiglu = a.epi == EPI_SWIGLU;
    m.U = s.U; m.KS = s.KS; m.C = s.C; m.NS = s.NS; m.spi = gm_steps(p, s); m.items = gm_items(p, s); m.shared = s.shared;
    m.part = w.part; m.tickets = w.tickets;
    if (head) { m.best = w.best; m.ticket = w.ticket; m.out_tok = a.out_tok; m.out_val = a.out_val; m.out_tok_f32 = a.out_tok_f32; m.softcap = a.softcap; }
    const GmKernel k = head ? (q40 ? gm_kernel<WT_Q4_0, 1, true>(ntl) : gm_kernel<WT_Q4_K, 1, true>(ntl))
                     : s.gw == 2 ? (q40 ? gm_kernel<WT_Q4_0, 2, false>(ntl) : gm_kernel<WT_Q4_K, 2, false>(ntl))
                                 : (q40 ? gm_kernel<WT_Q4_0, 1, false>(ntl) : gm_kernel<WT_Q4_K, 1, false>(ntl));
    static bool attr[2][3][5];
    bool& known = attr[q40 ? 0 : 1][head ? 2 : s.gw - 1][ntl];
    if (!known) {
        if (cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, GM_SMEM) != cudaSuccess)
            return fail(ADAMAH_ERR_BACKEND, "gemm_mma: cannot raise the shared-memory limit");
        known = true;
    }
    const cudaError_t e = launch_k(k, dim3((unsigned)s.grid), dim3((unsigned)(s.U * s.KS + 1) * 32), s.NS * gm_stage_bytes(p, s) + gm_red_bytes(p, s), stream, true, m);
    if (e != cudaSuccess) return fail(ADAMAH_ERR_BACKEND, "gemm_mma: launch failed: %s", cudaGetErrorString(e));
    count_launch();
    ++g_gemm_counts[GC_FEW];
    if (s.shared) ++g_gemm_counts[GC_FEW_SHARED];
    return ADAMAH_OK;
}

}  // namespace ab

// The launch shape that a product would get on a GPU of `sm_count` SMs, without a GPU: out[0..9] = row groups per warp, units, K slices,
// tile pairs per stage and slice, stages, CTAs, items shared (0 / 1), floats of an item's sums, of the room for them in the workspace,
// bytes of shared memory.
extern "C" int adam_b200_few_rows_shape(uint32_t ggml_type, uint32_t n, uint32_t k, uint32_t rows, uint32_t kind, uint32_t sm_count, uint32_t* out) {
    using namespace ab;
    const int wt = ggml_type == 2 ? WT_Q4_0 : WT_Q4_K;
    GemvArgs a = {};
    a.N = (int)n; a.K = (int)k; a.B = (int)rows;
    if ((ggml_type != 2 && ggml_type != 12) || kind > 2 || !out || !rows || rows > GM_MAX_ROWS || !n || !k || n > (1u << 30) || k > 32768 || !sm_count || sm_count > 1024 ||
        !gemm_mma_supports(wt, a))
        return ADAMAH_ERR_INVALID;
    const GmCall p = {wt == WT_Q4_0, kind == 1, kind == 2, a.N, a.K, a.B};
    const GmShape s = gm_shape(p, (int)sm_count);
    const uint32_t v[10] = {(uint32_t)s.gw, (uint32_t)s.U, (uint32_t)s.KS, (uint32_t)s.C, (uint32_t)s.NS, (uint32_t)s.grid, s.shared ? 1u : 0u,
                            (uint32_t)gm_item_floats(p, s), (uint32_t)GEMM_SLOT, (uint32_t)(s.NS * gm_stage_bytes(p, s) + gm_red_bytes(p, s))};
    for (int i = 0; i < 10; ++i) out[i] = v[i];
    return ADAMAH_OK;
}
