// Dequant GEMV for one activation row and a matrix that has to be streamed: k_gemv_mma's ring of bulk copies with the staging
// of k_gemv_row (gemv_row.cuh).
//
// The warps of a CTA are the K slices of one 16-row group at a time; every warp stages only the activations of its slice, with
// a scale of its own (31 bits, four signed bytes), and its weights stream through its own ring.  k_gemv_mma stages the whole
// vector in every CTA behind three CTA-wide reductions, and while that runs a ring takes no more than it holds (25 MB over all
// SMs): at the 27B shape 16 of a layer's 72 us.  Here it takes 2.3 us per product (QKV 8.3 -> 7.3 us behind its wait, o-proj 6.3
// -> 3.7, down 20.4 -> 14.5).  Matrices of many row groups per CTA stay with k_gemv_mma (gemv_ring.cu).
#pragma once
#include "gemv_row.cuh"

namespace ab {

constexpr int RING_WARPS = 16;

// NV: float4 of activations per lane at most; NST: ring stages per warp.  grid: CTAs (each takes every gridDim.x-th row group).
template <bool PAIR, int WT, bool CHAIN, int NV, int NST>
__global__ void __launch_bounds__(RING_WARPS * 32, 1) k_gemv_ring(const GemvArgs a_in, const uint8_t* __restrict__ t0, const uint8_t* __restrict__ t1, float inv_k) {
    const GemvArgs& a = a_in;
    GM_STAMP2(0);
    constexpr int NM = PAIR ? 2 : 1, CH = MmaGeo<PAIR, WT>::CH, STAGE_BYTES = MmaGeo<PAIR, WT>::STAGE_BYTES, TILE = MmaGeo<PAIR, WT>::TILE;
    constexpr int KS = RING_WARPS, NG = KS / 4, LD = KS + 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];               // [unit][4 columns of 32 bytes]; Q4_K: [unit][2] sums; rings
    __shared__ __align__(16) float s_red[2][NM * 16][LD];
    __shared__ __align__(16) float s_part[2][KS];                           // the slices' sums of squares: branch, stream
    __shared__ __align__(8) uint64_t s_bar[KS][NST];
    const int lane = threadIdx.x & 31, ks = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int pairs = a.K >> 6, n_rg = a.N >> 4;
    const int p0 = ks * pairs / KS, np = (ks + 1) * pairs / KS - p0;
    const int my_sets = (n_rg - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    unsigned char* xb = smem_raw + (size_t)p0 * 256;
    float* s_sx = reinterpret_cast<float*>(smem_raw + (size_t)pairs * 256) + p0 * 4;
    unsigned char* ring = smem_raw + (size_t)pairs * (WT == WT_Q4_K ? 272 : 256) + (size_t)ks * NST * STAGE_BYTES;
    const int nch = (np + CH - 1) / CH, n_chunks = my_sets * nch;           // chunks per row group, of this warp in all

    // ---- ahead of the dependency wait: the ring's first stages, norm weights ----
    if (lane == 0) {
#pragma unroll
        for (int st = 0; st < NST; ++st) mbar_init(&s_bar[ks][st], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    int i_c = 0, i_j = 0, i_st = 0;
    size_t i_off = ((size_t)blockIdx.x * pairs + p0) * TILE;                // the row group's slice
    auto issue_next = [&]() {                                               // lane 0 only
        const int n = min(CH, np - i_j * CH);
        const size_t off = i_off + (size_t)(i_j * CH) * TILE;
        unsigned char* dst = ring + (size_t)i_st * STAGE_BYTES;
        mbar_expect_tx(&s_bar[ks][i_st], (uint32_t)(n * TILE * NM));
        bulk_g2s(dst, t0 + off, (uint32_t)(n * TILE), &s_bar[ks][i_st]);
        if (PAIR) bulk_g2s(dst + CH * TILE, t1 + off, (uint32_t)(n * TILE), &s_bar[ks][i_st]);
        ++i_c;
        if (++i_st == NST) i_st = 0;
        if (++i_j == nch) { i_j = 0; i_off += (size_t)gridDim.x * pairs * TILE; }
    };
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < NST; ++c) if (i_c < n_chunks) issue_next();
    }
    const int f0 = p0 * 16 + lane, nf = np * 16 - lane;                     // this lane's first float4; how far the slice goes from there
    float4 vp[CHAIN ? NV : 1], vw[CHAIN ? NV : 1];
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
    GM_STAMP2(1);
    pdl_launch_dependents();
    pdl_wait();
    GM_STAMP2(2);

    // ---- this warp's activations ----
    float4 x[NV];
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4* hp = reinterpret_cast<const float4*>(CHAIN ? a.h_in : a.x) + f0;
#pragma unroll
    for (int j = 0; j < NV; ++j) x[j] = 32 * j < nf ? hp[32 * j] : z4;
    if (CHAIN) {
        if (a.add_src) {
            const float4* ap = reinterpret_cast<const float4*>(a.add_src) + f0;
            float4 va[NV];
#pragma unroll
            for (int j = 0; j < NV; ++j) va[j] = 32 * j < nf ? ap[32 * j] : z4;
            float ra = 1.f;
            if (a.w_post) {
                float s = 0.f;
#pragma unroll
                for (int j = 0; j < NV; ++j) s += fmaf(va[j].x, va[j].x, va[j].y * va[j].y) + fmaf(va[j].z, va[j].z, va[j].w * va[j].w);
                s = warp_sum(s);
                if (lane == 0) s_part[0][ks] = s;
                __syncthreads();
                ra = rsqrt_newton(fmaf(row_total<NG>(s_part[0]), inv_k, a.eps));
            }
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                x[j].x = fmaf(va[j].x * ra, vp[j].x, x[j].x); x[j].y = fmaf(va[j].y * ra, vp[j].y, x[j].y);
                x[j].z = fmaf(va[j].z * ra, vp[j].z, x[j].z); x[j].w = fmaf(va[j].w * ra, vp[j].w, x[j].w);
            }
        }
        GM_STAMP2(5);
        if (a.h_out && blockIdx.x == 0) {
            float4* ho = reinterpret_cast<float4*>(a.h_out) + f0;
#pragma unroll
            for (int j = 0; j < NV; ++j) if (32 * j < nf) ho[32 * j] = x[j];
        }
        if (a.w_pre) {
            float s = 0.f;
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                s += fmaf(x[j].x, x[j].x, x[j].y * x[j].y) + fmaf(x[j].z, x[j].z, x[j].w * x[j].w);
                x[j].x *= vw[j].x; x[j].y *= vw[j].y; x[j].z *= vw[j].z; x[j].w *= vw[j].w;
            }
            s = warp_sum(s);
            if (lane == 0) s_part[1][ks] = s;
        }
    }
    float scale, inv;
    slice_scale<30>(largest(x), scale, inv);
    GM_STAMP2(6);
    unsigned char* xs = xb + (lane >> 3) * 128 + (lane & 3) * 8 + (lane & 4);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        if (32 * j < np * 16) {                                             // whole warps: a half-full float4 row stores zeros that nobody reads ...
            uint32_t d[4];
            const float v[4] = {x[j].x * scale, x[j].y * scale, x[j].z * scale, x[j].w * scale};
            split4_x4(v, d);
            if (32 * j < nf) {                                              // ... but not behind the slice, where the next warp's is
                unsigned char* p = xs + j * 512;
#pragma unroll
                for (int c = 0; c < 4; ++c) *reinterpret_cast<uint32_t*>(p + ((c ^ (lane >> 3)) * 32)) = d[c];
            }
            if (WT == WT_Q4_K) {
                int s0 = __dp4a((int)d[0], 0x01010101, 0) * 256 + __dp4a((int)d[1], 0x01010101, 0), s1 = __dp4a((int)d[2], 0x01010101, 0) * 256 + __dp4a((int)d[3], 0x01010101, 0);
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) { s0 += __shfl_xor_sync(0xffffffffu, s0, o); s1 += __shfl_xor_sync(0xffffffffu, s1, o); }
                if ((lane & 7) == 0 && 32 * j < nf) *reinterpret_cast<float2*>(s_sx + ((lane >> 3) + 4 * j) * 2) = make_float2(-16.f * (float)s0, -16.f * (float)s1);
            }
        }
    }
    __syncwarp();
    GM_STAMP2(3);

    // ---- the stream ----
    float acc[NM][2];
#pragma unroll
    for (int m = 0; m < NM; ++m) acc[m][0] = acc[m][1] = 0.f;
    const unsigned char* xl = xb + t * 8;
    const int c0 = (g & 3) * 32;
    const float* sxl = s_sx + (t & 1);
    // pair `idx` of the slice, tile pair k of the stage
    auto do_pair = [&](const unsigned char* buf, int k, int idx) {
        const unsigned char* xu = xl + idx * 256;
        const int sw = (idx & 1) * 64;                                      // column c of unit u stands at c ^ (u & 3)
        const uint2 b0 = *reinterpret_cast<const uint2*>(xu + (c0 ^ sw)), b1 = *reinterpret_cast<const uint2*>(xu + 128 + (c0 ^ sw ^ 32));
#pragma unroll
        for (int m = 0; m < NM; ++m) {
            const unsigned char* tile = buf + (m * CH + k) * TILE;
            const uint4 q = reinterpret_cast<const uint4*>(tile)[lane];
            const uint2 sc = reinterpret_cast<const uint2*>(tile + 512)[g];
#pragma unroll
            for (int blk = 0; blk < 2; ++blk) {
                const uint32_t w0 = blk ? q.z : q.x, w1 = blk ? q.w : q.y, s2 = blk ? sc.y : sc.x, M = 0xF0F0F0F0u;
                const uint2 b = blk ? b1 : b0;
                int dd[4];
                if constexpr (WT == WT_Q4_0) {
                    const uint32_t X = 0x80808080u;
                    imma16832_s(dd, ((w0 << 4) & M) ^ X, ((w1 << 4) & M) ^ X, (w0 & M) ^ X, (w1 & M) ^ X, b.x, b.y);
                    const float2 d = __half22float2(*reinterpret_cast<const __half2*>(&s2));
                    acc[m][0] = fmaf(d.x, (float)(dd[0] * 256 + dd[1]), acc[m][0]);
                    acc[m][1] = fmaf(d.y, (float)(dd[2] * 256 + dd[3]), acc[m][1]);
                } else {
                    imma16832(dd, (w0 << 4) & M, (w1 << 4) & M, w0 & M, w1 & M, b.x, b.y);
                    const uint2 hd = reinterpret_cast<const uint2*>(tile + 576)[g];
                    const float2 dm0 = __half22float2(*reinterpret_cast<const __half2*>(&hd.x)), dm1 = __half22float2(*reinterpret_cast<const __half2*>(&hd.y));
                    const float es0 = dm0.x * (float)(s2 & 0xFFu), em0 = dm0.y * (float)((s2 >> 8) & 0xFFu);
                    const float es1 = dm1.x * (float)((s2 >> 16) & 0xFFu), em1 = dm1.y * (float)(s2 >> 24);
                    const float sx = sxl[(2 * idx + blk) * 2];
                    acc[m][0] = fmaf(es0, (float)(dd[0] * 256 + dd[1]), fmaf(em0, sx, acc[m][0]));
                    acc[m][1] = fmaf(es1, (float)(dd[2] * 256 + dd[3]), fmaf(em1, sx, acc[m][1]));
                }
            }
        }
    };
    // Even lanes hold 16 (256 hi + mid), odd ones 16 (256 lo + lowest): times 65536 / 16 and 1 / 16, both exact.
    const float cm = ((t & 1) ? 1.0f / 16.0f : 4096.0f) * inv;
    float r_pre = 1.f;
    bool timed_out = false;
    int st = 0;
    uint32_t ph = 0;
    for (int s = 0; s < my_sets; ++s) {
        for (int j = 0; j < nch; ++j) {
            if (!timed_out && !__all_sync(0xffffffffu, mbar_wait(&s_bar[ks][st], ph))) {
                // A copy never came: say so and stop touching the ring, but keep meeting the CTA's barriers.
                timed_out = true;
                if (lane == 0) atomicOr(a.err, DEVERR_WAIT);
            }
            if (!timed_out) {
                const unsigned char* buf = ring + (size_t)st * STAGE_BYTES;
                const int n = np - j * CH;
                if (n >= CH) {
#pragma unroll
                    for (int k = 0; k < CH; ++k) do_pair(buf, k, j * CH + k);
                } else {
#pragma unroll 1
                    for (int k = 0; k < n; ++k) do_pair(buf, k, j * CH + k);
                }
                __syncwarp();                               // every lane is done with this stage
                if (lane == 0 && i_c < n_chunks) issue_next();
            }
            if (++st == NST) { st = 0; ph ^= 1u; }
        }
#pragma unroll
        for (int m = 0; m < NM; ++m) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float v = acc[m][h] * cm;
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                if (t == 0) s_red[s & 1][m * 16 + g + 8 * h][ks] = v;
                acc[m][h] = 0.f;
            }
        }
        // Two sets of sums: whoever reads set s does so before its own arrival for set s + 1, behind which set s + 2 is written.
        __syncthreads();
        if (CHAIN && s == 0 && a.w_pre) r_pre = rsqrt_newton(fmaf(row_total<NG>(s_part[1]), inv_k, a.eps));
        if (ks == s % KS) {                                 // the warps take turns
            const float v = row_total<NG>(s_red[s & 1][PAIR ? lane : lane & 15]) * r_pre;
            const float up = PAIR ? __shfl_down_sync(0xffffffffu, v, 16) : 0.f;
            if (lane < 16)
                a.y[((int)blockIdx.x + s * (int)gridDim.x) * 16 + lane] = !PAIR ? v : (a.epi == EPI_GEGLU ? gelu_tanh(v) : silu_clip(v)) * up;
        }
    }
    GM_STAMP2(4);
    if (timed_out) {
        // give the copies still in flight a bounded chance to land before the shared memory is given up
        for (int s2 = 0; s2 < NST; ++s2) { mbar_wait(&s_bar[ks][s2], 0u); mbar_wait(&s_bar[ks][s2], 1u); }
    }
}

// ADAMAH_ERR_INVALID where gemv_ring_takes() says no.
bool gemv_ring_takes(int wtype, const GemvArgs& a);
int launch_gemv_ring(int wtype, const uint8_t* t0, const uint8_t* t1, GemvArgs a, cudaStream_t stream);

}  // namespace ab
