// Dequant GEMV for two to four activation rows and a matrix that the shared memory of all SMs holds at once: k_gemv_row
// (gemv_row.cuh) for the step of a few sequences.
//
// A decode step of a few sequences over matrices of a few megabytes is the same chain of latencies as that of one, so the same
// things are kept short: one launch per product with the norm chain inside it, weights requested ahead of the wait, every
// K slice of a row staged by one warp with a scale of its own, 1 / rms of the stream as a factor of the result.  Differences:
//   * One CTA per SM, of RG row groups (as many as give every SM one): its warps are RG x KS, each with PPW tile pairs.  A row's
//     slice is staged once per CTA: warp (rg, ks) stages slice ks of the rows rg, rg + RG, ...
//   * Weights wait in shared memory (bulk copies), registers hold the activations being staged.
//   * Two rows share an MMA (columns 0-3 and 4-7), and a tile is unpacked once for all rows.
//   * Activations keep four signed bytes, 31 bits relative to the slice's largest value: the fourth column of a row costs nothing,
//     and a product's relative error is 6e-8 to 9e-8 whatever the activations' tails (k_gemv_mma 2.9e-7 to 2.2e-6).
#pragma once
#include "gemv_row.cuh"

namespace ab {

// KS slices x RG row groups = the CTA's warps; NR: rows at most (2, 4); JW: rows a warp stages at most.
template <bool PAIR, int WT, bool CHAIN, int PPW, int NR, int JW, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_gemv_rows(const GemvArgs a, const uint8_t* __restrict__ t0, const uint8_t* __restrict__ t1, int KS, float inv_k) {
    pdl_launch_dependents();
    constexpr int NM = PAIR ? 2 : 1, NV = PPW / 2, UNITS = 2 * PPW, TILE = MmaGeo<PAIR, WT>::TILE, NP = NR / 2;
    constexpr int LD = 36;                                                  // floats per row of the slices' sums: rows on different banks
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) float s_part[2][NR][ROW_MAX_WARPS];            // the slices' sums of squares: branch, stream
    __shared__ float s_inv[NR][ROW_MAX_WARPS];                              // what undoes the slices' scales
    __shared__ __align__(8) uint64_t s_bar[ROW_MAX_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int rg_l = warp / KS, ks = warp - rg_l * KS, RG = n_warps / KS;
    const int n_rg = a.N >> 4, pairs = a.K >> 6, B = a.B;
    const int rg = min((int)blockIdx.x * RG + rg_l, n_rg - 1);              // past the end: the last group again, not stored
    const int p0 = ks * PPW, np = min(PPW, pairs - p0);
    // [slice][unit][row][4 columns of 32 bytes], column c (hi, mid, lo, lowest) of unit u at c ^ (u & 3); each warp's tile pairs;
    // [row group][row][matrix * 16 + row of it][LD] sums; Q4_K: [slice][unit][row][2] activation sums
    unsigned char* xb = smem_raw + ks * (UNITS * NR * 128);
    unsigned char* wb = smem_raw + KS * (UNITS * NR * 128) + warp * (NM * PPW * TILE);
    float* red = reinterpret_cast<float*>(smem_raw + KS * (UNITS * NR * 128) + n_warps * (NM * PPW * TILE));
    float* s_sx = red + RG * (NR * NM * 16 * LD);

    // ---- ahead of the dependency wait ----
    if (lane == 0) {
        mbar_init(&s_bar[warp], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&s_bar[warp], (uint32_t)(np * TILE * NM));
        const size_t off = ((size_t)rg * pairs + p0) * TILE;
        bulk_g2s(wb, t0 + off, (uint32_t)(np * TILE), &s_bar[warp]);
        if (PAIR) bulk_g2s(wb + PPW * TILE, t1 + off, (uint32_t)(np * TILE), &s_bar[warp]);
    }
    __syncwarp();                                                           // every lane waits on the barrier, a warp without rows with nothing in between
    const int f0 = p0 * 16 + lane, nf = np * 16 - lane;                     // this lane's first float4; how far the slice goes from there
    float4 vp[NV], vw[NV];
    if (CHAIN) {
        const float4 o4 = make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
        for (int j = 0; j < NV; ++j) vp[j] = vw[j] = o4;
        if (a.w_post) {
#pragma unroll
            for (int j = 0; j < NV; ++j) if (32 * j < nf) vp[j] = reinterpret_cast<const float4*>(a.w_post)[f0 + 32 * j];
        }
        if (a.w_pre) {
#pragma unroll
            for (int j = 0; j < NV; ++j) if (32 * j < nf) vw[j] = reinterpret_cast<const float4*>(a.w_pre)[f0 + 32 * j];
        }
    }
    for (int i = threadIdx.x; i < RG * NR * NM * 16 * 4; i += blockDim.x) {  // zeros behind the last slice's sums (read four at a time)
        const int k = (KS & ~3) + (i & 3);
        if (k >= KS) red[(i >> 2) * LD + k] = 0.f;
    }
    for (int i = threadIdx.x; i < 2 * NR * 4; i += blockDim.x) {
        const int k = (KS & ~3) + (i & 3);
        if (k >= KS && k < ROW_MAX_WARPS) s_part[0][0][(i >> 2) * ROW_MAX_WARPS + k] = 0.f;
    }
    const int ng = (KS + 3) >> 2;
    auto total = [&](const float* p) {
        float4 s = reinterpret_cast<const float4*>(p)[0];
#pragma unroll
        for (int i = 1; i < ROW_MAX_WARPS / 4; ++i) {
            if (i < ng) { const float4 v = reinterpret_cast<const float4*>(p)[i]; s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; }
        }
        return (s.x + s.y) + (s.z + s.w);
    };
    pdl_wait();

    // ---- this warp's rows of its slice ----
    float4 x[JW][NV];
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < JW; ++q) {
        const int r = rg_l + q * RG;
#pragma unroll
        for (int j = 0; j < NV; ++j)
            x[q][j] = (r < B && 32 * j < nf) ? reinterpret_cast<const float4*>((CHAIN ? a.h_in : a.x) + (size_t)r * a.ldx)[f0 + 32 * j] : z4;
    }
    if (CHAIN) {
        if (a.add_src) {
            float4 va[JW][NV];
#pragma unroll
            for (int q = 0; q < JW; ++q) {
                const int r = rg_l + q * RG;
#pragma unroll
                for (int j = 0; j < NV; ++j)
                    va[q][j] = (r < B && 32 * j < nf) ? reinterpret_cast<const float4*>(a.add_src + (size_t)r * a.ldx)[f0 + 32 * j] : z4;
            }
            if (a.w_post) {
#pragma unroll
                for (int q = 0; q < JW; ++q) {
                    const int r = rg_l + q * RG;
                    if (r < B) {
                        float s = 0.f;
#pragma unroll
                        for (int j = 0; j < NV; ++j) s += fmaf(va[q][j].x, va[q][j].x, va[q][j].y * va[q][j].y) + fmaf(va[q][j].z, va[q][j].z, va[q][j].w * va[q][j].w);
                        s = warp_sum(s);
                        if (lane == 0) s_part[0][r][ks] = s;
                    }
                }
                __syncthreads();
            }
#pragma unroll
            for (int q = 0; q < JW; ++q) {
                const int r = rg_l + q * RG;
                if (r < B) {
                    const float ra = a.w_post ? rsqrt_newton(fmaf(total(s_part[0][r]), inv_k, a.eps)) : 1.f;
#pragma unroll
                    for (int j = 0; j < NV; ++j) {
                        x[q][j].x = fmaf(va[q][j].x * ra, vp[j].x, x[q][j].x); x[q][j].y = fmaf(va[q][j].y * ra, vp[j].y, x[q][j].y);
                        x[q][j].z = fmaf(va[q][j].z * ra, vp[j].z, x[q][j].z); x[q][j].w = fmaf(va[q][j].w * ra, vp[j].w, x[q][j].w);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < JW; ++q) {
        const int r = rg_l + q * RG;
        if (r < B) {
            if (CHAIN) {
                if (a.h_out && blockIdx.x == 0) {
                    float4* ho = reinterpret_cast<float4*>(a.h_out + (size_t)r * a.ldx) + f0;
#pragma unroll
                    for (int j = 0; j < NV; ++j) if (32 * j < nf) ho[32 * j] = x[q][j];
                }
                if (a.w_pre) {
                    float s = 0.f;
#pragma unroll
                    for (int j = 0; j < NV; ++j) {
                        s += fmaf(x[q][j].x, x[q][j].x, x[q][j].y * x[q][j].y) + fmaf(x[q][j].z, x[q][j].z, x[q][j].w * x[q][j].w);
                        x[q][j].x *= vw[j].x; x[q][j].y *= vw[j].y; x[q][j].z *= vw[j].z; x[q][j].w *= vw[j].w;
                    }
                    s = warp_sum(s);
                    if (lane == 0) s_part[1][r][ks] = s;
                }
            }
            float scale, inv;
            slice_scale<30>(largest(x[q]), scale, inv);
            if (lane == 0) s_inv[r][ks] = inv;
            unsigned char* xs = xb + (lane >> 3) * (NR * 128) + r * 128 + (lane & 3) * 8 + (lane & 4);
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const float v[4] = {x[q][j].x * scale, x[q][j].y * scale, x[q][j].z * scale, x[q][j].w * scale};
                uint32_t d[4];
                split4_x4(v, d);
                unsigned char* p = xs + j * (4 * NR * 128);
                *reinterpret_cast<uint32_t*>(p + ((0 ^ (lane >> 3)) * 32)) = d[0];
                *reinterpret_cast<uint32_t*>(p + ((1 ^ (lane >> 3)) * 32)) = d[1];
                *reinterpret_cast<uint32_t*>(p + ((2 ^ (lane >> 3)) * 32)) = d[2];
                *reinterpret_cast<uint32_t*>(p + ((3 ^ (lane >> 3)) * 32)) = d[3];
                if (WT == WT_Q4_K) {
                    int s0 = __dp4a((int)d[0], 0x01010101, 0) * 256 + __dp4a((int)d[1], 0x01010101, 0), s1 = __dp4a((int)d[2], 0x01010101, 0) * 256 + __dp4a((int)d[3], 0x01010101, 0);
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1) { s0 += __shfl_xor_sync(0xffffffffu, s0, o); s1 += __shfl_xor_sync(0xffffffffu, s1, o); }
                    if ((lane & 7) == 0)
                        *reinterpret_cast<float2*>(s_sx + ((ks * UNITS + (lane >> 3) + 4 * j) * NR + r) * 2) = make_float2(-16.f * (float)s0, -16.f * (float)s1);
                }
            }
        }
    }
    const bool landed = __all_sync(0xffffffffu, mbar_wait(&s_bar[warp], 0u));
    if (!landed && lane == 0) atomicOr(a.err, DEVERR_WAIT);                 // the result is wrong and said to be; see the end
    __syncthreads();

    // ---- products: rows 2 i and 2 i + 1 share the MMAs i of a block ----
    float acc[NM][NP][2];
#pragma unroll
    for (int m = 0; m < NM; ++m)
#pragma unroll
        for (int i = 0; i < NP; ++i) acc[m][i][0] = acc[m][i][1] = 0.f;
    const unsigned char* xl = xb + (g >> 2) * 128 + t * 8;
#pragma unroll
    for (int i = 0; i < PPW; ++i) {
        uint4 q[NM]; uint2 sc[NM], hd[NM];
        const bool in = i < np;                                             // no pair: scale 0, whatever its bytes and activations
#pragma unroll
        for (int m = 0; m < NM; ++m) {
            const unsigned char* tile = wb + (m * PPW + i) * TILE;
            q[m] = reinterpret_cast<const uint4*>(tile)[lane];
            const uint2 s = reinterpret_cast<const uint2*>(tile + 512)[g];
            sc[m] = in ? s : make_uint2(0u, 0u);
            if (WT == WT_Q4_K) { const uint2 h = reinterpret_cast<const uint2*>(tile + 576)[g]; hd[m] = in ? h : make_uint2(0u, 0u); }
        }
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
            const int u = 2 * i + blk;
            uint2 bx[NP];
#pragma unroll
            for (int n = 0; n < NP; ++n) bx[n] = *reinterpret_cast<const uint2*>(xl + u * (NR * 128) + n * 256 + (((g & 3) ^ (u & 3)) * 32));
#pragma unroll
            for (int m = 0; m < NM; ++m) {
                const uint32_t w0 = blk ? q[m].z : q[m].x, w1 = blk ? q[m].w : q[m].y, s2 = blk ? sc[m].y : sc[m].x;
                const uint32_t M = 0xF0F0F0F0u, X = WT == WT_Q4_0 ? 0x80808080u : 0u;
                const uint32_t a0 = ((w0 << 4) & M) ^ X, a1 = ((w1 << 4) & M) ^ X, a2 = (w0 & M) ^ X, a3 = (w1 & M) ^ X;
                float e0, e1, o0 = 0.f, o1 = 0.f;
                if constexpr (WT == WT_Q4_0) {
                    const float2 d = __half22float2(*reinterpret_cast<const __half2*>(&s2));
                    e0 = d.x; e1 = d.y;
                } else {
                    const float2 dm0 = __half22float2(*reinterpret_cast<const __half2*>(&hd[m].x)), dm1 = __half22float2(*reinterpret_cast<const __half2*>(&hd[m].y));
                    e0 = dm0.x * (float)(s2 & 0xFFu); o0 = dm0.y * (float)((s2 >> 8) & 0xFFu);
                    e1 = dm1.x * (float)((s2 >> 16) & 0xFFu); o1 = dm1.y * (float)(s2 >> 24);
                }
#pragma unroll
                for (int n = 0; n < NP; ++n) {
                    if (2 * n < B) {
                        int dd[4];
                        if constexpr (WT == WT_Q4_0) imma16832_s(dd, a0, a1, a2, a3, bx[n].x, bx[n].y);
                        else {
                            imma16832(dd, a0, a1, a2, a3, bx[n].x, bx[n].y);
                            const float sx = s_sx[((ks * UNITS + u) * NR + 2 * n + (t >> 1)) * 2 + (t & 1)];
                            acc[m][n][0] = fmaf(o0, sx, acc[m][n][0]); acc[m][n][1] = fmaf(o1, sx, acc[m][n][1]);
                        }
                        acc[m][n][0] = fmaf(e0, (float)(dd[0] * 256 + dd[1]), acc[m][n][0]);
                        acc[m][n][1] = fmaf(e1, (float)(dd[2] * 256 + dd[3]), acc[m][n][1]);
                    }
                }
            }
        }
    }
    // Even lanes hold 16 (256 hi + mid), odd ones 16 (256 lo + lowest): times 65536 / 16 and 1 / 16, both exact.  Lane t / 2: row.
    const float cm = (t & 1) ? 1.0f / 16.0f : 4096.0f;
#pragma unroll
    for (int n = 0; n < NP; ++n) {
        const int r = 2 * n + (t >> 1);
        if (2 * n < B) {
            const float f = cm * s_inv[r][ks];                              // (a row that is not there has no scale, and nobody reads its sums)
#pragma unroll
            for (int m = 0; m < NM; ++m) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float v = acc[m][n][h] * f;
                    v += __shfl_xor_sync(0xffffffffu, v, 1);
                    if (!(t & 1)) red[((rg_l * NR + r) * (NM * 16) + m * 16 + g + 8 * h) * LD + ks] = v;
                }
            }
        }
    }
    __syncthreads();
    // ---- the slices' sums: a warp per (row group, activation row), lane = row of the group (and matrix) ----
    for (int c = warp; c < RG * B; c += n_warps) {
        const int gl = c / B, r = c - gl * B, grp = (int)blockIdx.x * RG + gl;
        float v = total(red + ((gl * NR + r) * (NM * 16) + (PAIR ? lane : lane & 15)) * LD);
        if (CHAIN && a.w_pre) v *= rsqrt_newton(fmaf(total(s_part[1][r]), inv_k, a.eps));
        const float up = PAIR ? __shfl_down_sync(0xffffffffu, v, 16) : 0.f;
        if (lane < 16 && grp < n_rg) {
            const float o = !PAIR ? v : (a.epi == EPI_GEGLU ? gelu_tanh(v) : silu_clip(v)) * up;
            a.y[(size_t)r * a.ldy + grp * 16 + lane] = o;
        }
    }
    if (!landed) mbar_wait(&s_bar[warp], 0u);                               // a bounded chance to land before the shared memory is given up
}

// ADAMAH_ERR_INVALID where gemv_rows_takes() says no.
bool gemv_rows_takes(int wtype, const GemvArgs& a);
int launch_gemv_rows(int wtype, const uint8_t* t0, const uint8_t* t1, GemvArgs a, cudaStream_t stream);

}  // namespace ab
