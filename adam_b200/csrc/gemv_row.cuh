// Dequant GEMV for one activation row and a matrix that fits the registers of all SMs at once.
//
// One token of one sequence is a chain of products of a few megabytes each, and what such a product takes is not its
// bytes but the chain of latencies from "the previous kernel is done" to "the last row is stored": the activations' trip
// through L2, the reductions of the norm chain, the split into bytes, a few MMAs, the sum over K slices.  This kernel
// keeps that chain as short as it gets; k_gemv_mma (gemv_mma.cuh), whose warps share one staged copy of the activations
// behind three CTA-wide reductions, is for matrices that have to be streamed.
//   * A CTA is one group of 16 rows, its warps are the K slices: PPW tile pairs (64 weights each) per warp.  All CTAs are
//     resident together, so a warp holds its whole share of the matrix in registers, requested ahead of the dependency
//     wait: no ring, no stage barriers, no loop.
//   * A warp stages only the 64 * PPW activations that it multiplies, with a power-of-two scale of its own: no CTA-wide
//     maximum, no CTA barrier between staging and product.  (Its integers are relative to the slice's largest value, so
//     they are never coarser than those of one scale for the vector.)
//   * Of the input chain only the branch's RMS is needed ahead of the product.  1 / rms of the stream is a factor of the
//     whole result and its sum of squares meets the K slices' sums at the one barrier that adds them.
//   * Q4_0 codes enter the MMA as signed bytes 16 (q - 8): a nibble in a byte's upper half, its top bit flipped, IS that
//     byte, so nothing is subtracted per block.  (Q4_K: unsigned 16 q, its offsets take the block's activation sums.)
// Measured on a B200 at the 1B shape (Q4_0), from the end of the dependency wait to the last store, k_gemv_mma -> here: QKV
// 1536 x 1152 3.3 -> 1.6 us, o-proj 1152 x 1024 2.3 -> 0.9, gate / up 2 x 6912 x 1152 4.1 -> 2.1, down 1152 x 6912 4.5 -> 1.7.
// Relative error of a product 2.8e-7 to 3.3e-7 (N(0, 1) activations; before the same), 5.5e-7 to 8.1e-7 where they have heavy
// tails (before 8.1e-7 to 2.0e-6).  Tried and not kept: weights in shared memory by bulk copy (+0.3 us per product, an SM takes
// four CTAs of the gate / up product and another two), three row groups per CTA behind one staging (all 27 warps of an SM in
// step: products 0.75 -> 1.25 us), the code run once on nothing ahead of the wait (the same times: it is in the instruction cache).
// The arithmetic otherwise is that of k_gemv_mma: |x s| <= 2^22, three signed bytes per activation, mma.m16n8k32 in
// integers, block scale and sums in fp32.
#pragma once
#include "gemv_mma.cuh"

namespace ab {

constexpr int ROW_MAX_WARPS = 32;

__device__ __forceinline__ uint4 ld_weight(const uint8_t* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ld_weight2(const uint8_t* p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

// Four scaled activations (integers of at most 31 bits after rounding) as four words of signed bytes, the highest digits first:
// the digits of split_x4, of which the top one needs no flip.
__device__ __forceinline__ void split4_x4(const float (&f)[4], uint32_t (&d)[4]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = ((uint32_t)__float2int_rn(f[i]) + 0x00808080u) ^ 0x00808080u;
    const uint32_t l01 = __byte_perm(w[0], w[1], 0x5140), l23 = __byte_perm(w[2], w[3], 0x5140);      // bytes 0, 0, 1, 1
    const uint32_t h01 = __byte_perm(w[0], w[1], 0x7362), h23 = __byte_perm(w[2], w[3], 0x7362);      // bytes 2, 2, 3, 3
    d[0] = __byte_perm(h01, h23, 0x7632); d[1] = __byte_perm(h01, h23, 0x5410);
    d[2] = __byte_perm(l01, l23, 0x7632); d[3] = __byte_perm(l01, l23, 0x5410);
}

// The sum of NG groups of four floats at a 16-byte aligned place.
template <int NG>
__device__ __forceinline__ float row_total(const float* p) {
    float4 t = reinterpret_cast<const float4*>(p)[0];
#pragma unroll
    for (int i = 1; i < NG; ++i) {
        const float4 v = reinterpret_cast<const float4*>(p)[i];
        t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
    }
    return (t.x + t.y) + (t.z + t.w);
}

// The largest absolute value of a lane's activations, NaN if one of them is.
template <int NV>
__device__ __forceinline__ float largest(const float4 (&x)[NV]) {
    float am = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) am = max_nan(am, max_nan(max_nan(fabsf(x[j].x), fabsf(x[j].y)), max_nan(fabsf(x[j].z), fabsf(x[j].w))));
    return am;
}
// The power of two that brings a slice's largest value m * 2^e, 1/2 <= m < 1, to m * 2^BITS (less for values below 2^(BITS - 126)) and
// what undoes it.  |x|'s bits are in the values' order, infinity and NaN last: a slice that has one has no finite result,
// whatever its integers are.
template <int BITS>
__device__ __forceinline__ void slice_scale(float am, float& scale, float& inv) {
    const uint32_t eb = max(__reduce_max_sync(0xffffffffu, __float_as_uint(am)) >> 23, (uint32_t)BITS);
    scale = __uint_as_float((253u + BITS - eb) << 23);
    inv = __uint_as_float(eb == 255u ? 0x7FFFFFFFu : (eb - (BITS - 1)) << 23);
}

#ifdef ADAM_B200_STEP_TRACE
// CTAs 0 to 6 stamp their own rows, row 7 has the latest stamp of any CTA.
#define GR_STAMP(slot) do { if (threadIdx.x == 0 && blockIdx.y == 0 && a.trace) { \
        if (blockIdx.x < 7) STEP_STAMP(a.trace, blockIdx.x * 8 + (slot)); \
        atomicMax(reinterpret_cast<unsigned long long*>(a.trace) + 56 + (slot), (unsigned long long)step_trace_now()); } } while (0)
#else
#define GR_STAMP(slot) do { } while (0)
#endif

#ifdef ADAM_B200_STEP_TRACE
#define GM_STAMP2(slot) do { if (threadIdx.x == 0 && blockIdx.x < 8) STEP_STAMP(a_in.trace, blockIdx.x * 8 + (slot)); } while (0)
#else
#define GM_STAMP2(slot) do { } while (0)
#endif

// grid (row groups, activation rows), 32 * slices threads; PPW: tile pairs per warp; THREADS, CTAS: the launch bounds.
//
// An SM has up to 27 such warps that all wait for the same event and then run through this code together: what it takes is
// their instructions.  So no instruction here is about what the launch already knows: slices are PPW pairs (the last may be
// shorter: it loads its last pair again, with scales of zero), sums are over a fixed number of slices (zeros behind the last),
// addresses are made ahead of the wait, a value becomes an integer by an addition (1.5 * 2^23: the integer is in the low bits).
template <bool PAIR, int WT, bool CHAIN, int PPW, int THREADS, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS) k_gemv_row(const GemvArgs a, const uint8_t* __restrict__ t0, const uint8_t* __restrict__ t1, float inv_k) {
    GR_STAMP(0);
    pdl_launch_dependents();
    constexpr int NM = PAIR ? 2 : 1, NV = PPW / 2, UNITS = 2 * PPW, TILE = MmaGeo<PAIR, WT>::TILE;
    constexpr int NG = (THREADS / 32 + 3) / 4, LD = NG % 2 ? NG * 4 : NG * 4 + 4;          // groups of four slices; floats per row of their sums: rows on different banks
    static_assert(PPW % 2 == 0, "a warp's 32 lanes load two tile pairs' activations at a time");
    extern __shared__ __align__(16) unsigned char smem_raw[];               // per warp: UNITS * 128 bytes
    __shared__ __align__(16) float s_red[NM * 16][LD];
    __shared__ __align__(16) float s_part[2][NG * 4];                       // the slices' sums of squares: branch, stream
    __shared__ float s_sx[WT == WT_Q4_K ? ROW_MAX_WARPS * UNITS * 2 : 1];   // Q4_K: activation sums of the units, in the lanes' units
    const int lane = threadIdx.x & 31, ks = threadIdx.x >> 5, KS = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int rg = blockIdx.x, b = blockIdx.y;
    const int pairs = a.K >> 6;
    const int p0 = ks * PPW, np = min(PPW, pairs - p0);

    // ---- ahead of the dependency wait: weights, norm weights, what stays constant in shared memory ----
    uint4 q[NM][PPW];
    uint2 sc[NM][PPW], hd[NM][PPW];
    {
        const size_t off = ((size_t)rg * pairs + p0) * TILE;
#pragma unroll
        for (int i = 0; i < PPW; ++i) {
            const int at = (i < np ? i : np - 1) * TILE;
#pragma unroll
            for (int m = 0; m < NM; ++m) {
                const uint8_t* tile = (m ? t1 : t0) + off + at;
                q[m][i] = ld_weight(tile + lane * 16);
                sc[m][i] = ld_weight2(tile + 512 + g * 8);
                if (WT == WT_Q4_K) hd[m][i] = ld_weight2(tile + 576 + g * 8);
            }
        }
    }
    if (lane == 0) {
        const uint32_t wi = (uint32_t)(rg * KS + ks);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const uint32_t at = wi * a.pf_part[r];
            if (at < a.pf_bytes[r])
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(a.pf[r] + at), "r"(min(a.pf_part[r], a.pf_bytes[r] - at)) : "memory");
        }
    }
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
    // Unit u of the slice is 128 bytes, column c (hi, mid, lo, zero) of it at c ^ (u & 3).  Stores: lane's unit is lane / 8 (+ 4 per
    // further float4), its place (lane & 3) * 8 + (lane & 4).  Loads: lane (g, t) reads column g & 3 of every unit.
    unsigned char* xb = smem_raw + ks * (UNITS * 128);
    unsigned char* xs = xb + (lane >> 3) * 128 + (lane & 3) * 8 + (lane & 4);
    unsigned char *x_hi = xs + ((0 ^ (lane >> 3)) * 32), *x_mid = xs + ((1 ^ (lane >> 3)) * 32), *x_lo = xs + ((2 ^ (lane >> 3)) * 32);
    const unsigned char* xl = xb + (g & 3) * 32 + t * 8;
    const int step = ((g & 1) ? -32 : 32), step2 = ((g & 2) ? -64 : 64);    // to column c ^ 1, c ^ 2
#pragma unroll
    for (int j = 0; j < NV; ++j) *reinterpret_cast<uint32_t*>(xs + j * 512 + ((3 ^ (lane >> 3)) * 32)) = 0u;
    if (ks == 0) {
        for (int k = KS; k < NG * 4; ++k) {
            if (lane < NM * 16) s_red[lane][k] = 0.f;
            if (lane < 2) s_part[lane][k] = 0.f;
        }
    }
    const float4* hp = reinterpret_cast<const float4*>((CHAIN ? a.h_in : a.x) + (size_t)b * a.ldx) + f0;
    const float4* ap = reinterpret_cast<const float4*>(a.add_src + (size_t)b * a.ldx) + f0;
    GR_STAMP(1);
    pdl_wait();
    GR_STAMP(2);

    // ---- this warp's activations ----
    float4 x[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) { x[j] = make_float4(0.f, 0.f, 0.f, 0.f); if (32 * j < nf) x[j] = hp[32 * j]; }
    if (CHAIN) {
        if (a.add_src) {
            float4 va[NV];
#pragma unroll
            for (int j = 0; j < NV; ++j) { va[j] = make_float4(0.f, 0.f, 0.f, 0.f); if (32 * j < nf) va[j] = ap[32 * j]; }
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
        GR_STAMP(5);
        if (a.h_out && rg == 0) {
            float4* ho = reinterpret_cast<float4*>(a.h_out + (size_t)b * a.ldx) + f0;
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
    slice_scale<22>(largest(x), scale, inv);
    GR_STAMP(6);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const float v[4] = {x[j].x, x[j].y, x[j].z, x[j].w};
        uint32_t w[4];
        // x * scale + 1.5 * 2^23 has the integer in its low 23 bits; its three signed bytes as in split_x4
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = (__float_as_uint(fmaf(v[i], scale, 12582912.f)) + (0x00808080u - 0x4B400000u)) ^ 0x00808080u;
        const uint32_t wl = __byte_perm(__byte_perm(w[0], w[1], 0x0040), __byte_perm(w[2], w[3], 0x0040), 0x5410);
        const uint32_t wm = __byte_perm(__byte_perm(w[0], w[1], 0x0051), __byte_perm(w[2], w[3], 0x0051), 0x5410);
        const uint32_t wh = __byte_perm(__byte_perm(w[0], w[1], 0x0062), __byte_perm(w[2], w[3], 0x0062), 0x5410);
        *reinterpret_cast<uint32_t*>(x_hi + j * 512) = wh;
        *reinterpret_cast<uint32_t*>(x_mid + j * 512) = wm;
        *reinterpret_cast<uint32_t*>(x_lo + j * 512) = wl;
        if (WT == WT_Q4_K) {
            int sh = __dp4a((int)wh, 0x01010101, 0), sm = __dp4a((int)wm, 0x01010101, 0), sl = __dp4a((int)wl, 0x01010101, 0);
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                sh += __shfl_xor_sync(0xffffffffu, sh, o);
                sm += __shfl_xor_sync(0xffffffffu, sm, o);
                sl += __shfl_xor_sync(0xffffffffu, sl, o);
            }
            if ((lane & 7) == 0)
                *reinterpret_cast<float2*>(s_sx + (ks * UNITS + (lane >> 3) + 4 * j) * 2) = make_float2(-16.f * (float)(sh * 256 + sm), -16.f * (float)(sl * 256));
        }
    }
    __syncwarp();
    GR_STAMP(3);

    // ---- products ----
    float acc[NM][2];
#pragma unroll
    for (int m = 0; m < NM; ++m) acc[m][0] = acc[m][1] = 0.f;
#pragma unroll
    for (int i = 0; i < PPW; ++i) {
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
            const int u = 2 * i + blk;
            const uint2 bx = *reinterpret_cast<const uint2*>(xl + u * 128 + ((u & 1) ? step : 0) + ((u & 2) ? step2 : 0));   // lanes g >= 4 fill columns that nobody reads
#pragma unroll
            for (int m = 0; m < NM; ++m) {
                const uint32_t w0 = blk ? q[m][i].z : q[m][i].x, w1 = blk ? q[m][i].w : q[m][i].y;
                const uint32_t s2 = i < np ? (blk ? sc[m][i].y : sc[m][i].x) : 0u;
                int dd[4];
                if constexpr (WT == WT_Q4_0) {
                    const uint32_t M = 0xF0F0F0F0u, X = 0x80808080u;
                    imma16832_s(dd, ((w0 << 4) & M) ^ X, ((w1 << 4) & M) ^ X, (w0 & M) ^ X, (w1 & M) ^ X, bx.x, bx.y);
                    const float2 d = __half22float2(*reinterpret_cast<const __half2*>(&s2));
                    acc[m][0] = fmaf(d.x, (float)(dd[0] * 256 + dd[1]), acc[m][0]);
                    acc[m][1] = fmaf(d.y, (float)(dd[2] * 256 + dd[3]), acc[m][1]);
                } else {
                    const uint32_t M = 0xF0F0F0F0u;
                    imma16832(dd, (w0 << 4) & M, (w1 << 4) & M, w0 & M, w1 & M, bx.x, bx.y);
                    const float2 dm0 = __half22float2(*reinterpret_cast<const __half2*>(&hd[m][i].x)), dm1 = __half22float2(*reinterpret_cast<const __half2*>(&hd[m][i].y));
                    const float es0 = dm0.x * (float)(s2 & 0xFFu), em0 = dm0.y * (float)((s2 >> 8) & 0xFFu);
                    const float es1 = dm1.x * (float)((s2 >> 16) & 0xFFu), em1 = dm1.y * (float)(s2 >> 24);
                    const float sx = s_sx[(ks * UNITS + u) * 2 + (t & 1)];
                    acc[m][0] = fmaf(es0, (float)(dd[0] * 256 + dd[1]), fmaf(em0, sx, acc[m][0]));
                    acc[m][1] = fmaf(es1, (float)(dd[2] * 256 + dd[3]), fmaf(em1, sx, acc[m][1]));
                }
            }
        }
    }
    // Even lanes hold 16 (256 hi + mid), odd ones 16 * 256 lo: times 65536 / 256 / 16 and 1 / 256 / 16, both exact.
    const float cm = ((t & 1) ? 1.0f / 4096.0f : 16.0f) * inv;
#pragma unroll
    for (int m = 0; m < NM; ++m) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float v = acc[m][h] * cm;
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            if (t == 0) s_red[m * 16 + g + 8 * h][ks] = v;
        }
    }
    __syncthreads();
    // ---- the slices' sums: lane = row (and matrix) ----
    if (ks == 0) {
        float v = row_total<NG>(s_red[PAIR ? lane : lane & 15]);
        if (CHAIN && a.w_pre) v *= rsqrt_newton(fmaf(row_total<NG>(s_part[1]), inv_k, a.eps));
        const float up = PAIR ? __shfl_down_sync(0xffffffffu, v, 16) : 0.f;
        if (lane < 16) {
            const float r = !PAIR ? v : (a.epi == EPI_GEGLU ? gelu_tanh(v) : silu_clip(v)) * up;
            a.y[(size_t)b * a.ldy + rg * 16 + lane] = r;
        }
    }
    GR_STAMP(4);
}

// ADAMAH_ERR_INVALID where gemv_row_takes() says no.
bool gemv_row_takes(int wtype, const GemvArgs& a);
int launch_gemv_row(int wtype, const uint8_t* t0, const uint8_t* t1, GemvArgs a, cudaStream_t stream);

}  // namespace ab
