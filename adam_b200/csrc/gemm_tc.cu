// Dequant-fused GEMM  y[b][n] = sum_k W[n][k] x[b][k]  for many activation rows b (prompt rows, decode batches) on the
// 5th-generation tensor cores: tcgen05.mma with the weight operand and the accumulator in tensor memory (TMEM).  Same
// operator as the GEMV kernels (the reference's Q4 mat-vec shader adamah-MAIN/adamah/shaders/src/f32/map_matvec_t_xq4.comp
// and map_fused_gateup_t_xq4.comp run once per row by adamah.c:8606-8691).
//
// Arithmetic.  A row of activations is scaled by a power of two (largest element near 2^15) and split into two fp16
// terms, x = x_hi + x_lo (22 bits of every element).  A weight is rebuilt exactly as two fp16 terms, w = w_hi + w_lo:
//   Q4_0  w = d (q - 8): w_hi = RN16(d (q - 8)), w_lo = fma(d, q - 8, -w_hi), exact because d (q - 8) has 14 bits
//   Q4_K  w = d sc (q - 8) + (8 d sc - dmin m): the first product has 20 bits and splits the same way; the second is the
//         same for 32 neighbouring weights, so it becomes one more "weight" per 32 that multiplies the sum of their 32
//         activations (a few extra steps of K, 1/32 of the work).  The codes are centred because d sc q is never negative:
//         taken apart as d sc q and dmin m, activations with a mean make two sums of many times the result, and what
//         the tensor core rounds off is relative to them (256 x 5376, 9 rows of N(1, 1): 3.7e-5 of the result; the test asks for 5e-6).
//   Q8_0  w = d q: 19 bits, as Q4_0
// and w_hi x_hi + w_lo x_hi + w_hi x_lo is accumulated over K in fp32 (w_lo x_lo lies below 2^-22 of the product).
// Limit, what fp16 holds: 8 d (Q4_0), 128 d (Q8_0), 8 d sc and 32 |8 d sc - dmin m| (Q4_K) below 65504.  Uploads look for
// blocks beyond it, and tensors of a map that got one stay on the GEMV kernels.
//
// Two kernels:
//   k_quant_rows  one CTA per activation row: the optional input chain (residual add + RMS norms, as the GEMV prologue),
//                 the row's scale, and its two fp16 planes written in the B operand's shared-memory order (K-major,
//                 128-byte swizzle), so that the GEMM fetches operand tiles with plain bulk copies.
//   k_gemm_tc     see there.
// Every wait is bounded: when one runs out the kernel records DEVERR_WAIT, stops waiting, and still frees its tensor memory.
#include "gemm_tc.cuh"
#include "gemv_mma.cuh"
#include "gemv_rows.cuh"

#include <atomic>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <vector>

namespace ab {

// ---- workspace: the operand image of the activations and the rows' inverse scales -----------------------------
constexpr int TC_GROUP = 64;                            // rows of one image group
constexpr int TC_STEP_IMG = TC_GROUP * 128;             // one plane of one group and step (64 values of K): 8 KB
constexpr size_t TC_IMG_MAX = 256u << 20;               // largest image kept; longer calls run in row chunks
constexpr int TC_MAX_K = 32768;

struct TcWork { uint8_t* img; size_t img_cap; float* inv; int inv_cap; unsigned long long* best; float* part; unsigned int* tickets; std::vector<void*> retired; };   // best: arg-max keys [inv_cap], then a ticket
static TcWork g_tc = {};
static std::mutex g_tc_lock;            // the two kernels of a call are enqueued together: the image is one for all
static uint64_t g_tc_calls = 0;
uint64_t g_gemm_counts[GC_COUNTS] = {};
static std::atomic<int> g_tc_policy{-1};  // 0 never, 1 where it is expected to be faster, 2 whenever the shape allows; -1 = take it from ADAM_B200_TC

static int tc_main_steps(int K) { return (K + 63) / 64; }
static int tc_min_steps(int wtype, int K) { return wtype == WT_Q4_K ? (K / 32 + 63) / 64 : 0; }
static size_t tc_group_bytes(int wtype, int K) { return (size_t)(tc_main_steps(K) + tc_min_steps(wtype, K)) * 2 * TC_STEP_IMG; }
static int tc_pad_rows(int rows) { return (rows + 127) / 128 * 128; }

// Room for `rows` activation rows of length K (either block type); false when out of memory.  Recorded graphs hold the
// buffers' addresses, so a buffer that is outgrown stays until the release; sizes at least double, which bounds the sum.
bool gemm_tc_prepare(int rows, int K) {
    if (rows < 1 || K < 1 || K > TC_MAX_K) return false;
    std::lock_guard<std::mutex> work(g_tc_lock);
    const int pad = tc_pad_rows(rows);
    size_t need = (size_t)(pad / TC_GROUP) * tc_group_bytes(WT_Q4_K, K);
    if (need > TC_IMG_MAX) need = TC_IMG_MAX;
    auto grow = [&](void** p, size_t bytes) {
        void* q = nullptr;
        if (cudaMalloc(&q, bytes) != cudaSuccess) { cudaGetLastError(); return false; }
        cudaMemsetAsync(q, 0, bytes, g.stream);
        if (*p) g_tc.retired.push_back(*p);
        *p = q;
        return true;
    };
    if (!g_tc.part) {                                   // two slots of sums and two tickets per CTA
        if (!grow((void**)&g_tc.tickets, (size_t)g.sm_count * 8) || !grow((void**)&g_tc.part, (size_t)g.sm_count * 2 * GEMM_SLOT * 4)) return false;
    }
    if (need > g_tc.img_cap) {
        size_t cap = need > 2 * g_tc.img_cap ? need : 2 * g_tc.img_cap;
        if (cap > TC_IMG_MAX) cap = TC_IMG_MAX;
        if (!grow((void**)&g_tc.img, cap)) return false;
        g_tc.img_cap = cap;
    }
    if (pad > g_tc.inv_cap) {
        const int cap = pad > 2 * g_tc.inv_cap ? pad : 2 * g_tc.inv_cap;
        if (!grow((void**)&g_tc.best, (size_t)cap * 8 + 8)) return false;
        if (!grow((void**)&g_tc.inv, (size_t)cap * 4)) return false;
        g_tc.inv_cap = cap;
    }
    return true;
}

void gemm_tc_release() {
    cudaFree(g_tc.img); cudaFree(g_tc.inv); cudaFree(g_tc.best); cudaFree(g_tc.part); cudaFree(g_tc.tickets);
    for (void* p : g_tc.retired) cudaFree(p);
    g_tc = TcWork{};
}
static int tc_rows_fit(int wtype, int K) {              // rows of one pass: whole 128-row tiles
    const long long fit = (long long)(g_tc.img_cap / (2 * tc_group_bytes(wtype, K))) * 128;
    return (int)(fit < g_tc.inv_cap ? fit : g_tc.inv_cap / 128 * 128);
}

// ---- activations: chain, scale, two fp16 planes in B-operand order -------------------------------------------
// Bound by the latency of its chain (one row per CTA: load, up to two reductions of one barrier each, store), not by its 12
// bytes per value; the row stays in registers (MAXV float4 per thread), all loads are issued before the first use, the norm
// weights ahead of the dependency wait.
// Four consecutive values of K are stored in the order 0, 2, 1, 3: the order in which a word of nibbles is taken apart
// two at a time (see k_gemm_tc); K order is free as long as both operands agree.
__device__ __forceinline__ uint32_t swz_off(int r, int kb) { return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((((kb >> 4) ^ r) & 7) << 4) + (kb & 15)); }

__device__ __forceinline__ void split_half(float v, __half& hi, __half& lo) {
    hi = __float2half_rn(v);
    lo = __float2half_rn(v - __half2float(hi));
}

// FEW: the image of gemm_mma.cu instead: per 32 values of K the rows' 2 x 32 halves in the order of its B fragments, for
// Q4_K (n_min > 0) followed by a float per row, the sum of the 32 values; n_steps is then the number of rows it has room for.
template <int MAXV, bool CHAIN, bool FEW>
__global__ void __launch_bounds__(512) k_quant_rows(const GemvArgs a, uint8_t* __restrict__ img, float* __restrict__ inv_out, int n_min, int n_steps) {
    __shared__ __align__(16) float red[3][16];          // the warps' sums: branch, stream; their maxima
    const int r = blockIdx.x, tid = threadIdx.x, K = a.K, n4 = K >> 2, nt = blockDim.x;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f), o4 = make_float4(1.f, 1.f, 1.f, 1.f);
    const bool post = CHAIN && a.add_src && a.w_post, pre = CHAIN && a.w_pre;
    float4 v[MAXV], vp[CHAIN ? MAXV : 1], vw[CHAIN ? MAXV : 1];
    pdl_launch_dependents();
    // ahead of the wait: the norm weights (a step's matrices have pushed them out of L2), zeros behind the last warp's sum
    if constexpr (CHAIN) {
#pragma unroll
        for (int j = 0; j < MAXV; ++j) {
            const int i = tid + j * nt;
            vp[j] = (i < n4 && post) ? reinterpret_cast<const float4*>(a.w_post)[i] : o4;
            vw[j] = (i < n4 && pre) ? reinterpret_cast<const float4*>(a.w_pre)[i] : o4;
        }
    }
    if (tid < 16) {
#pragma unroll
        for (int k = 0; k < 3; ++k) if (tid >= nt >> 5) red[k][tid] = 0.f;
    }
    const float inv_k = 1.0f / (float)K;
    pdl_wait();
    const size_t row = (size_t)r * a.ldx;
    if constexpr (CHAIN) {
        const float* ap = a.add_src ? a.add_src + row : nullptr;
        float4 va[MAXV];
#pragma unroll
        for (int j = 0; j < MAXV; ++j) {
            const int i = tid + j * nt;
            const bool in = i < n4;
            v[j] = in ? reinterpret_cast<const float4*>(a.h_in + row)[i] : z4;
            va[j] = (in && ap) ? reinterpret_cast<const float4*>(ap)[i] : z4;
        }
        float ra = 1.f;
        if (post) {
            float ss = 0.f;
#pragma unroll
            for (int j = 0; j < MAXV; ++j) ss += fmaf(va[j].x, va[j].x, va[j].y * va[j].y) + fmaf(va[j].z, va[j].z, va[j].w * va[j].w);
            ss = warp_sum(ss);
            if ((tid & 31) == 0) red[0][tid >> 5] = ss;
            __syncthreads();
            ra = rsqrt_newton(fmaf(row_total<4>(red[0]), inv_k, a.eps));
        }
        if (ap) {
#pragma unroll
            for (int j = 0; j < MAXV; ++j) {
                v[j].x = fmaf(va[j].x * ra, vp[j].x, v[j].x); v[j].y = fmaf(va[j].y * ra, vp[j].y, v[j].y);
                v[j].z = fmaf(va[j].z * ra, vp[j].z, v[j].z); v[j].w = fmaf(va[j].w * ra, vp[j].w, v[j].w);
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < MAXV; ++j) {
            const int i = tid + j * nt;
            v[j] = i < n4 ? reinterpret_cast<const float4*>(a.x + row)[i] : z4;
        }
    }
    // the stream's sum of squares and the largest value (ahead of the division by the RMS) in one round
    float ss = 0.f, am = 0.f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
        if constexpr (CHAIN) {
            const int i = tid + j * nt;
            if (i < n4 && a.h_out) reinterpret_cast<float4*>(a.h_out + row)[i] = v[j];
            ss += fmaf(v[j].x, v[j].x, v[j].y * v[j].y) + fmaf(v[j].z, v[j].z, v[j].w * v[j].w);
            v[j].x *= vw[j].x; v[j].y *= vw[j].y; v[j].z *= vw[j].z; v[j].w *= vw[j].w;
        }
        am = fmaxf(am, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
    }
    am = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(am)));          // not negative: the bits are in the values' order
    if (pre) ss = warp_sum(ss);
    if ((tid & 31) == 0) { red[1][tid >> 5] = ss; red[2][tid >> 5] = am; }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 m = reinterpret_cast<const float4*>(red[2])[k];
        am = fmaxf(am, fmaxf(fmaxf(m.x, m.y), fmaxf(m.z, m.w)));
    }
    float rp = 1.f;                                     // 1 / RMS of the stream, a factor of every value
    if (pre) { rp = rsqrt_newton(fmaf(row_total<4>(red[1]), inv_k, a.eps)); am = am * rp * 1.000001f; }
    float s, inv;
    pow2_scale(am, s, inv);                             // largest element in (2^21, 2^22] ...
    s *= 0.0078125f; inv *= 128.f;                      // ... in (2^14, 2^15]
    if (pre) {
#pragma unroll
        for (int j = 0; j < MAXV; ++j) { v[j].x *= rp; v[j].y *= rp; v[j].z *= rp; v[j].w *= rp; }
    }
    if (tid == 0) inv_out[r] = inv;
    if constexpr (FEW) {
        const int blk = gm_block_bytes(n_min ? WT_Q4_K : WT_Q4_0, n_steps);
#pragma unroll
        for (int j = 0; j < MAXV; ++j) {
            const int i = tid + j * nt;                 // values 4 i .. 4 i + 3: piece i & 3 of the low or high half of block i >> 3
            const float4 f = make_float4(v[j].x * s, v[j].y * s, v[j].z * s, v[j].w * s);
            uint8_t* d = img + (size_t)(i >> 3) * blk;
            if (i < n4) {
                __half h[4], l[4];
                split_half(f.x, h[0], l[0]); split_half(f.z, h[1], l[1]); split_half(f.y, h[2], l[2]); split_half(f.w, h[3], l[3]);
                uint2* q = reinterpret_cast<uint2*>(d) + (r * 8 + (i & 3)) * 2 + ((i >> 2) & 1);
                q[0] = *reinterpret_cast<const uint2*>(h);
                q[8] = *reinterpret_cast<const uint2*>(l);
            }
            if (n_min) {
                float t = (f.x + f.y) + (f.z + f.w);
                t += __shfl_xor_sync(0xffffffffu, t, 1);
                t += __shfl_xor_sync(0xffffffffu, t, 2);
                t += __shfl_xor_sync(0xffffffffu, t, 4);
                if (i < n4 && (i & 7) == 0) reinterpret_cast<float*>(d + 128 * n_steps)[r] = t;
            }
        }
        return;
    }
    const int r64 = r & 63;
    uint8_t* base = img + (size_t)(r >> 6) * n_steps * (2 * TC_STEP_IMG);
    auto put4 = [&](int k0, float4 f) {                 // values k0 .. k0+3, already scaled
        __half h[4], l[4];
        split_half(f.x, h[0], l[0]); split_half(f.z, h[1], l[1]); split_half(f.y, h[2], l[2]); split_half(f.w, h[3], l[3]);
        uint8_t* d = base + (size_t)(n_min + (k0 >> 6)) * (2 * TC_STEP_IMG) + swz_off(r64, (k0 & 63) * 2);
        *reinterpret_cast<uint2*>(d) = *reinterpret_cast<const uint2*>(h);
        *reinterpret_cast<uint2*>(d + TC_STEP_IMG) = *reinterpret_cast<const uint2*>(l);
    };
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
        const int i = tid + j * nt;
        const float4 f = make_float4(v[j].x * s, v[j].y * s, v[j].z * s, v[j].w * s);
        if (i < n4) put4(4 * i, f);
        if (n_min) {                                    // sums over 32 neighbouring values (eight lanes), over 32: what Q4_K's block offset multiplies
            float t = (f.x + f.y) + (f.z + f.w);
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            t += __shfl_xor_sync(0xffffffffu, t, 2);
            t += __shfl_xor_sync(0xffffffffu, t, 4);
            if (i < n4 && (i & 7) == 0) {
                const int sub = i >> 3;
                __half h, l;
                split_half(t * 0.03125f, h, l);
                uint8_t* d = base + (size_t)(sub >> 6) * (2 * TC_STEP_IMG) + swz_off(r64, (sub & 63) * 2);
                *reinterpret_cast<__half*>(d) = h;
                *reinterpret_cast<__half*>(d + TC_STEP_IMG) = l;
            }
        }
    }
    // what the last steps hold beyond the row's end multiplies as zero
    for (int i = n4 + tid; i < (n_steps - n_min) * 16; i += nt) put4(4 * i, z4);
    for (int sub = (K >> 5) + tid; sub < n_min * 64; sub += nt) {
        uint8_t* d = base + (size_t)(sub >> 6) * (2 * TC_STEP_IMG) + swz_off(r64, (sub & 63) * 2);
        *reinterpret_cast<__half*>(d) = __half(0.f);
        *reinterpret_cast<__half*>(d + TC_STEP_IMG) = __half(0.f);
    }
}

// ---- tcgen05 primitives --------------------------------------------------------------------------------------
// Shared-memory matrix descriptor, K-major with the 128-byte swizzle (layout 2 at bit 61): start address and the
// distance between 8-row groups (1024 bytes), in 16-byte units, plus the descriptor version of this architecture (bit 46).
// The 16 values of K of one instruction are 32 bytes of a row: the next instruction's descriptor starts 32 bytes further.
#define TC_DESC_HI ((uint32_t)(1024u >> 4) | (1u << 14) | (2u << 29))
// Instruction descriptor of kind::f16: D = f32 (1 at bit 4), A = B = f16 (0 at bits 7 and 10), both operands K-major,
// N / 8 at bit 17, M / 16 at bit 24.
template <int N> constexpr uint32_t TC_IDESC = (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void tc_alloc(uint32_t* slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// D[tmem] (+)= A[tmem] * B[smem]; one instruction covers 16 values of K.
__device__ __forceinline__ void tc_mma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 :: "r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// The mbarrier gets one arrival when all tensor-core operations issued so far by this thread are done.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(bar)) : "memory");
}
// 16 and 8 consecutive 32-bit columns of this thread's TMEM lane, to and from registers.
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&r)[16]) {       // valid after tc_ld_wait()
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]),
                   "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16_l1(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }
__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ float ld_cluster(uint32_t saddr, uint32_t rank) {
    uint32_t a; float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

// ---- nibbles -> two fp16 terms ----------------------------------------------------------------------------------
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
// The low or high nibbles of a word's four bytes, two at a time, as halves: bytes (0, 2) and (1, 3) as 1024 + q (low) or
// 1024 + 16 q (high), by masking them into the mantissa of 1024.0.
template <bool HIGH> __device__ __forceinline__ void nib_pairs(uint32_t w, uint32_t (&p)[2]) {
    constexpr uint32_t M = HIGH ? 0x00F000F0u : 0x000F000Fu;
    p[0] = (w & M) | 0x64006400u;
    p[1] = ((w >> 8) & M) | 0x64006400u;
}
// The high nibbles as 64 + q, in the mantissa of 64.0.
__device__ __forceinline__ void nib_pairs_64(uint32_t w, uint32_t (&p)[2]) {
    p[0] = (w & 0x00F000F0u) | 0x54005400u;
    p[1] = ((w >> 8) & 0x00F000F0u) | 0x54005400u;
}
// v * d as w_hi + w_lo (v two exact small integers)
__device__ __forceinline__ void split_h2(__half2 v, __half2 d, uint32_t& whi, uint32_t& wlo) {
    const __half2 h = __hmul2_rn(v, d);                    // rounded once, not contracted
    whi = as_u32(h);
    wlo = as_u32(__hfma2(v, d, __hneg2(h)));
}
// Scales and minima of group g (64 weights = sub-blocks 2g, 2g+1) of a Q4_K header: sub-block 2g in bits 0..7, 2g+1 in 8..15.
__device__ __forceinline__ void q4k_codes(const uint4& h, int g, uint32_t& sp, uint32_t& mp) {
    const int sh = (g & 1) * 16;
    const uint32_t s16 = (h.y >> sh) & 0xFFFFu, m16 = (h.z >> sh) & 0xFFFFu, t16 = (h.w >> sh) & 0xFFFFu;
    if (g < 2) { sp = s16 & 0x3F3Fu; mp = m16 & 0x3F3Fu; }
    else { sp = (t16 & 0x0F0Fu) | ((s16 >> 2) & 0x3030u); mp = ((t16 >> 4) & 0x0F0Fu) | ((m16 >> 2) & 0x3030u); }
}

// ---- the GEMM ---------------------------------------------------------------------------------------------------
// One CTA per SM.  A CTA's tile is 128 weight rows (or 64 gate rows in TMEM lanes 0..63 and the same 64 up rows in lanes
// 64..127) by NT activation rows: D is 2 NT columns of TMEM (NT = 256: NT), the rest a ring of weight tiles (128 rows x 64
// values of K as w_hi | w_lo, 64 columns each).  K is walked in stages of SP steps of 64 values, NS stages in flight; a stage has one
// barrier for everything that fills it (its activation tiles, and the warps that rebuild its weight tiles) and one that
// the tensor core's commit releases.
//   warp roles   Warpgroup 0: warp 0 issues the tensor-core instructions, warp 1 fetches activation tiles.  Warpgroup 1 reads
//                results back.  The others rebuild weights, a weight tile each in turn.  setmaxnreg moves registers from
//                warpgroup 0 to the reader, which holds NT sums per thread.
//   weights      A lane owns a row.  Its codes come by cp.async into the warp's own ring in shared memory (R tiles ahead,
//                across the end of a tile, two lanes per row so that a sector is fetched whole), are taken apart in fp16
//                pairs (4.25 instructions per two weights) and go to TMEM with tcgen05.st: no shared-memory operand image,
//                no swizzle, and the shared memory's 128 bytes per cycle are left to the activation operand.
//   activations  x_hi | x_lo tiles of 64 values of K by bulk copies from the image.
//   products     per 16 values of K two tcgen05.mma (M 128): w_hi x [x_hi | x_lo] with N = 2 NT into D1 | D2, and
//                w_lo x x_hi with N = NT into D2; 6 cycles per step and activation row, the tensor core's rate.
//                What the loop costs besides is the issuing warp's own latency, about 100 cycles per barrier and 20 per
//                instruction, because the queue in front of the tensor core is short: with two barriers and two commits per
//                step the bare loop took 671 cycles at NT = 64 and 520 at NT = 16, with one of each per two steps 448 and
//                246 (NT = 128: 878 and 772, the rate of the instructions).  One elected lane issues, but the whole warp
//                walks the loop: inside a one-lane branch it took half as long again.
//   rounding     The tensor core rounds its running sum towards zero, an error that grows with the number of instructions
//                added up.  So the cross terms, 2^-11 of the result, have D2 to themselves, and every two (NT = 128: three)
//                steps D1 is added to registers and restarted.  Relative error of a 1152 x 6912 product by the steps
//                between: all of K 6.1e-6, eight 5.8e-7, four 3.4e-7, three 2.8e-7, two 2.1e-7; the GEMV, which adds
//                integers up within a block, has 2.9e-7 to 4.7e-7, and two or three steps stay below it for every size.
//                Up to NT = 64 a stage has a pair D1 | D2 of its own and the reader's arrivals count among those that
//                fill the stage, so the issuing warp waits for nothing more.  At NT = 128 there is room for one pair:
//                the stage that restarts D1 issues its products for D2 first, two thirds of its time, while D1 is
//                read.  32 prompts x 512 at the 1B shape: 141 ms with eight steps, 157 with two and no second pair, 148 so.
//   NT = 256     halves the rebuilding per product, which is energy (long prompts run at the power limit).  One accumulator of 256
//                columns and no D2: a stage of two steps issues the cross terms of both, then both main terms, and is read
//                out, so the additions at full magnitude are the eight of two steps.  Activations come plane by plane, each slot
//                given back as soon as its last product is done; a step's weights and planes share one barrier, because a wait of
//                the issuing warp costs 86 cycles even if satisfied and only some four instructions queue ahead of the tensor
//                core (a barrier per plane: 640 us instead of 598).  A round trip over the accumulator costs 289 cycles and the
//                reading of 128 columns 280 more, twice per 3072 cycles of products; two warpgroups read.  Bound by these
//                trips and the waits (tensor pipe 63 % active at 21504 x 5376 Q4_K on 1024 rows), not by rebuilding (leaving it out: -7 %).
//   work split   Three ways, by an estimate of their times (launch_rows).  Whole tiles, dealt in turn.  Or all stages
//                of all tiles in a row, dealt out evenly: a tile that several CTAs share is added up by the one that ends
//                last (atomic ticket, partial sums in a workspace), in the order of K; 168 tiles on 148 SMs take 1.14 tiles'
//                time, not 2, but the adding up costs 2 to 5 us.  Or, where the tiles alone leave SMs idle, clusters of S
//                CTAs that take a part of K each, leave their sums in their own shared memory and add each other's columns
//                through distributed shared memory, again in the order of K: results do not depend on timing.
//   code size    Every launch finds the instruction cache cold, and fetching code costs about 12 cycles per instruction executed
//                for the first time: with every loop unrolled and an instance per kind of result, 6000 to 15000 of a layer's
//                15000 to 25000 cycles.  So stored and gate/up products share an instance (the flag is uniform), and
//                loops whose registers allow it are rolled.
// The request for shared memory is at least 120 KB, so that an SM never holds two of these CTAs: one that waits for
// tensor memory held by a cluster that waits for it would never end.
constexpr int TC_SMEM_MIN = 120 * 1024;
struct TcGemm {
    WeightRef w0, w1;
    float* y; int ldy;
    const uint8_t* img; const float* inv; uint32_t* err;
    int N, units, B;                                    // units = K / 32
    int pair, swiglu;                                   // gate / up tiles, and which activation
    int n_min, n_main, tiles_n, items;                  // items = tiles_n (weight tiles) * tiles of NT rows
    int S, shared;                                      // K splits; whether CTAs share tiles
    float* part; unsigned int* tickets;                 // shared tiles: per CTA the sums of its first and last one; arrivals, by the CTA in which a tile begins
    unsigned long long* best; unsigned int* ticket;     // arg-max: one key per activation row (0 between launches), CTAs that are done
    int* out_tok; float *out_val, *out_tok_f32, softcap;
};
template <int WT, int NT> struct TcGeo {
    static constexpr int NH = NT == 256 ? 2 : 1, NC = NT / NH;               // reading warpgroups, columns that each reads
    static constexpr int SP = NT == 128 ? 1 : 2, NS = NT == 128 ? 4 : 2;     // steps per stage, stages
    static constexpr int BANKS = NT >= 128 ? 1 : NS, PERIOD = NT == 128 ? 3 : 1;        // sets of accumulators; stages between two read-outs
    static constexpr int DCOLS = NT == 256 ? NT : BANKS * 2 * NT;            // columns of accumulators
    static constexpr int GROUPS = NT == 256 ? 2 : NT == 128 ? 3 : 4, THREADS = (1 + NH + GROUPS) * 128;     // warpgroups that rebuild weights, a step each in turn
    static constexpr int REG_LOW = NT == 256 ? 32 : 40, REG_READ = NT == 256 ? 152 : NT == 128 ? 200 : 120, REG_MAKE = NT == 256 ? 72 : 80;    // sum = what the CTA is launched with
    static constexpr int R = WT == WT_Q8_0 && NT >= 128 ? 3 : 4;                  // weight ring: tiles ahead per warp
    static constexpr int QB = WT == WT_Q8_0 ? 64 : 32;                       // bytes of a row's codes per step
    static constexpr int SLOT = 32 * QB + (WT == WT_Q4_K ? 512 : 128);       // 32 rows: codes, then block scales / superblock headers
    static constexpr int BSTEP = NT * 256, PLANE = NT * 128;                 // both planes of one step, one plane
    static constexpr int RING = (NT == 256 ? 2 : NS * SP) * BSTEP, XCH = RING + GROUPS * 4 * R * SLOT;     // offsets: weight rings, columns of results on their way out
    static constexpr int XCOLS = NC < 32 ? NC : 32;                          // so many columns at a time
    static constexpr int SMEM_USED = XCH + NH * XCOLS * 512 + 1024;
    static constexpr int SMEM = SMEM_USED > TC_SMEM_MIN ? SMEM_USED : TC_SMEM_MIN;
    static_assert(SMEM <= 226 * 1024 && DCOLS + 64 * NS * SP <= 512 && GROUPS % SP == 0 && GROUPS <= NS * SP, "shared or tensor memory");
    static_assert(REG_LOW + NH * REG_READ + GROUPS * REG_MAKE <= 65536 / THREADS / 8 * 8 * (1 + NH + GROUPS), "registers");
};
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(p));
    return p != 0;
}
template <int N> __device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(N)); }
template <int N> __device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(N)); }
template <int N, int HAVE> __device__ __forceinline__ void reg_set() { if constexpr (N > HAVE) reg_inc<N>(); else if constexpr (N < HAVE) reg_dec<N>(); }
template <int WT, int NT, bool HEAD>
__global__ void __launch_bounds__(TcGeo<WT, NT>::THREADS, 1) k_gemm_tc(const TcGemm a) {
    using G = TcGeo<WT, NT>;
    const bool pair = !HEAD && WT != WT_Q8_0 && a.pair != 0;
    constexpr int SP = G::SP, NS = G::NS, NH = G::NH, NC = G::NC;
    extern __shared__ __align__(1024) uint8_t sm_raw[];
    uint8_t* sm = sm_raw + ((1024u - (smem_u32(sm_raw) & 1023u)) & 1023u);     // the swizzle works on address bits
    uint8_t* smB = sm;
    __shared__ __align__(8) uint64_t full[NT == 256 ? 2 * NS : NS], empty[NS], d_full, d_empty, p_empty[4];
    __shared__ uint32_t s_tmem;
    __shared__ bool s_last[NH];
    __shared__ float s_inv[NT];
    [[maybe_unused]] __shared__ unsigned long long s_best[HEAD ? NT : 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wg = warp >> 2;
    const int S = a.S, split = S > 1 ? (int)(blockIdx.x % (uint32_t)S) : 0;     // a cluster's CTAs are neighbours along x
    // this split's share of the steps: first those of the block offsets, then those of the products
    const int mn0 = split * a.n_min / S, mn1 = (split + 1) * a.n_min / S;
    const int ma0 = split * a.n_main / S, ma1 = (split + 1) * a.n_main / S;
    const int nmn = mn1 - mn0, nst = nmn + ma1 - ma0, n_steps = a.n_min + a.n_main;
    const int spi = (nst + SP - 1) / SP;                                        // stages per item; the last may hold one step only
    // This CTA's stages [q0, q1), counted through its items; the i-th of them is item_of(i).  Whole tiles are dealt in turn, so
    // that CTAs side by side read the same activation tile at about the same time.
    const long long all = (long long)a.items * spi;
    auto q_begin = [&](int cta) { return (int)(cta * all / gridDim.x); };       // shared tiles: stages of all items in a row
    const int cta = (int)blockIdx.x, n_cta = (int)gridDim.x;
    const int q0 = a.shared ? q_begin(cta) : 0, q1 = a.shared ? q_begin(cta + 1) : S > 1 ? spi : (a.items - cta + n_cta - 1) / n_cta * spi;
    auto item_of = [&](int i) { return a.shared ? i : S > 1 ? cta / S : cta + i * n_cta; };
    auto m_of = [&](int item) { return item / a.tiles_n * NT; };                // first activation row and weight tile of an item
    auto n_of = [&](int item) { return item % a.tiles_n; };
    if (tid == 0) {
        for (int i = 0; i < NS; ++i) { if (NT != 256) mbar_init(&full[i], 4 * SP + 1 + (G::BANKS > 1 ? 4 : 0)); mbar_init(&empty[i], 1); }
        mbar_init(&d_full, 1); mbar_init(&d_empty, 4 * NH);
        if constexpr (NT == 256) for (int i = 0; i < 4; ++i) { mbar_init(&full[i], 4 + 2); mbar_init(&p_empty[i], 1); }      // a step: four warps of weights, two planes
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) tc_alloc(&s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    constexpr uint32_t A_COL = G::DCOLS;       // first column of the weight ring
    bool dead = false;
    auto wait_on = [&](uint64_t* bar, uint32_t parity) {
        if (!dead && !mbar_wait(bar, parity)) { dead = true; atomicOr(a.err, DEVERR_WAIT); }
    };
    const int row = (warp & 3) * 32 + lane;             // this lane's TMEM lane
    const uint32_t tlane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    auto act = [&](float gate, float up) { return gated(gate, a.swiglu ? silu_arg(gate) : gelu_arg(gate)) * up; };     // no branch
    // The end of a split item: the cluster's sums lie in the exchange; every CTA finishes the columns c = split, split + S, ...
    auto finish_split = [&]() {
        cl_arrive();
        cl_wait();
        const uint32_t ex_s = smem_u32(smB);
        auto total_of = [&](int c, int r) {             // all loads in flight, then one order of addition
            float p[8], v = 0.f;
#pragma unroll
            for (int q = 0; q < 8; ++q) p[q] = q < S ? ld_cluster(ex_s + (uint32_t)(c * 128 + r) * 4u, (uint32_t)q) : 0.f;
#pragma unroll
            for (int q = 0; q < 8; ++q) v += p[q];
            return v;
        };
        const int item = item_of(0), tn = n_of(item), m0 = m_of(item), n_col = min(NT, a.B - m0);
        const int r = pair ? row & 63 : row, n_out = pair ? tn * 64 + r : tn * 128 + r;
        float* yp = a.y + (size_t)m0 * a.ldy + n_out;
        const int lanes = pair ? 2 : 1;                 // a pair's 64 rows: each half of the lanes takes its own columns
#pragma unroll 1
        for (int c = split + S * ((wg - 1) * lanes + (pair ? row >> 6 : 0)); c < n_col; c += (G::GROUPS + 1) * lanes * S) {
            const float sc = a.inv[m0 + c];
            float v = total_of(c, r) * sc;
            if (pair) v = act(v, total_of(c, 64 + r) * sc);
            if (n_out < a.N) yp[(size_t)c * a.ldy] = v;
        }
        cl_arrive();
        cl_wait();
    };
    pdl_launch_dependents();

    if (wg == 0) {
        reg_dec<G::REG_LOW>();
        pdl_wait();                                     // the image comes from the kernel before this one; no bounded wait below spans that kernel
        const bool lead = elect_one();
        if (warp == 1) {
            // ---- activation tiles ----
            if constexpr (NT == 256) {
                // planes of 256 rows in the order in which they are multiplied and room for them becomes free (see the products)
                const size_t group_bytes = (size_t)n_steps * (2 * TC_STEP_IMG);
                uint32_t x[4] = {0, 1, 2, 3}, par = 0xFu;               // slots of a stage's planes lo 0, hi 0, hi 1, lo 1; parities of their waits
                for (int q = q0; q < q1; ++q) {
                    const int i = q / spi, st0 = (q - i * spi) * SP, m0 = m_of(item_of(i));
                    uint64_t* fs = full + ((q - q0) & 1) * 2;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int st = st0 + (k >> 1), lo = k == 0 || k == 3 ? 1 : 0;
                        const uint32_t s = x[k];
                        if (st >= nst) {                // no second step: its barrier gets what it counts all the same
                            if (lead) mbar_arrive(fs + 1);
                            __syncwarp();
                            continue;
                        }
                        wait_on(&p_empty[s], par >> s & 1u);
                        par ^= 1u << s;
                        if (lead) {
                            mbar_expect_tx(fs + (k >> 1), G::PLANE);
                            const size_t at = (size_t)(st < nmn ? mn0 + st : a.n_min + ma0 + st - nmn) * (2 * TC_STEP_IMG) + lo * TC_STEP_IMG;
#pragma unroll
                            for (int g4 = 0; g4 < 4; ++g4) {            // groups without rows take the first's: their sums are dropped
                                const int group = m0 / TC_GROUP + (m0 + g4 * TC_GROUP < a.B ? g4 : 0);
                                bulk_g2s(smB + s * G::PLANE + g4 * TC_STEP_IMG, a.img + group * group_bytes + at, TC_STEP_IMG, fs + (k >> 1));
                            }
                        }
                        __syncwarp();
                    }
                    const uint32_t x1 = x[1];
                    x[1] = x[3]; x[3] = x[2]; x[2] = x1;
                }
                // no copy may be in flight when the CTA ends, whatever became of the waits above: the last two stages
                for (int n = max(0, q1 - q0 - 2); n < q1 - q0; ++n)
                    for (int t = 0; t < 2; ++t) mbar_wait(&full[(n & 1) * 2 + t], (uint32_t)(n >> 1) & 1u);
            } else {
                uint32_t s = 0, par = 1, n = 0;
                const size_t group_bytes = (size_t)n_steps * (2 * TC_STEP_IMG);
                for (int q = q0; q < q1;) {
                    const int i = q / spi, j0 = q - i * spi, j1 = min(spi, j0 + q1 - q);
                    q += j1 - j0;
                    const uint8_t* group = a.img + (size_t)(item_of(i) / a.tiles_n) * (NT == 128 ? 2 : 1) * group_bytes;
                    for (int j = j0; j < j1; ++j, ++n) {
                        if (n >= (uint32_t)NS) wait_on(&empty[s], par);
                        const int st0 = j * SP, n_sub = SP == 1 ? 1 : min(SP, nst - st0);
                        if (lead) {
                            mbar_expect_tx(&full[s], (uint32_t)(n_sub * G::BSTEP));
                            for (int t = 0; t < n_sub; ++t) {
                                const int st = st0 + t;
                                const uint8_t* src = group + (size_t)(st < nmn ? mn0 + st : a.n_min + ma0 + st - nmn) * (2 * TC_STEP_IMG);
                                uint8_t* dst = smB + (s * SP + t) * G::BSTEP;
                                if constexpr (NT == TC_GROUP) bulk_g2s(dst, src, G::BSTEP, &full[s]);
                                else {                      // both planes of the first NT rows, or of two groups
                                    constexpr int ROWS = NT < TC_GROUP ? NT : TC_GROUP;
                                    bulk_g2s(dst, src, ROWS * 128, &full[s]);
                                    bulk_g2s(dst + NT * 128, src + TC_STEP_IMG, ROWS * 128, &full[s]);
                                    if constexpr (NT > TC_GROUP) {
                                        bulk_g2s(dst + TC_STEP_IMG, src + group_bytes, TC_STEP_IMG, &full[s]);
                                        bulk_g2s(dst + NT * 128 + TC_STEP_IMG, src + group_bytes + TC_STEP_IMG, TC_STEP_IMG, &full[s]);
                                    }
                                }
                            }
                        }
                        __syncwarp();
                        if (++s == (uint32_t)NS) { s = 0; par ^= 1u; }
                    }
                }
                // no copy may be in flight when the CTA ends, whatever became of the waits above
                for (uint32_t i = n > (uint32_t)NS ? n - NS : 0; i < n; ++i) mbar_wait(&full[i % NS], (i / NS) & 1u);
            }
        } else if (warp == 0) {
            // ---- products ----
            const uint32_t b_lo = (smem_u32(smB) & 0x3FFFFu) >> 4;
            auto desc = [&](uint32_t lo) { return ((uint64_t)TC_DESC_HI << 32) | lo; };
            if constexpr (NT == 256) {
                // A stage: the cross terms of its (up to) two steps, then their main terms, one accumulator of 256 columns.
                // A plane x_lo is done with after a third of the stage, x_hi after five sixths: lo 0, lo 1, hi 0, hi 1 in
                // this order leave their slots to the next stage's lo 0, hi 0, hi 1, lo 1.
                uint32_t s = 0, par = 0, x[4] = {0, 1, 2, 3};
                for (int q = q0; q < q1; ++q) {
                    const int n_sub = min(SP, nst - (q % spi) * SP);
#pragma unroll
                    for (int t = 0; t < SP; ++t) {
                        wait_on(&full[s * 2 + t], par);
                        if (t == n_sub) break;
                        if (t == 0 && q > q0) wait_on(&d_empty, (uint32_t)(q - q0 - 1) & 1u);
                        const uint32_t xl = t ? x[3] : x[0], xh = t ? x[2] : x[1], ac = tmem + A_COL + (s * SP + t) * 64u;
                        tc_fence_after();
                        if (lead) {
                            const uint32_t bl = b_lo + xl * (uint32_t)(G::PLANE / 16), bh = b_lo + xh * (uint32_t)(G::PLANE / 16);
#pragma unroll
                            for (uint32_t k = 0; k < 4; ++k) tc_mma_ts(tmem, ac + k * 8u, desc(bl + k * 2u), TC_IDESC<NT>, t || k ? 1u : 0u);
                            tc_commit(&p_empty[xl]);
#pragma unroll
                            for (uint32_t k = 0; k < 4; ++k) tc_mma_ts(tmem, ac + 32u + k * 8u, desc(bh + k * 2u), TC_IDESC<NT>, 1u);
                        }
                        __syncwarp();
                    }
                    if (lead) {
#pragma unroll
                        for (int t = 0; t < SP; ++t) {
                            if (t == n_sub) break;
                            const uint32_t xh = t ? x[2] : x[1], ac = tmem + A_COL + (s * SP + t) * 64u, bh = b_lo + xh * (uint32_t)(G::PLANE / 16);
#pragma unroll
                            for (uint32_t k = 0; k < 4; ++k) tc_mma_ts(tmem, ac + k * 8u, desc(bh + k * 2u), TC_IDESC<NT>, 1u);
                            tc_commit(&p_empty[xh]);
                        }
                        tc_commit(&d_full);
                        tc_commit(&empty[s]);
                    }
                    __syncwarp();
                    if (++s == (uint32_t)NS) { s = 0; par ^= 1u; }
                    const uint32_t x1 = x[1];
                    x[1] = x[3]; x[3] = x[2]; x[2] = x1;
                }
            } else {
                uint32_t s = 0, par = 0, periods = 0;
                for (int q = q0; q < q1;) {
                    const int j0 = q % spi, j1 = min(spi, j0 + q1 - q);
                    q += j1 - j0;
                    for (int j = j0; j < j1; ++j) {
                        if constexpr (G::BANKS > 1) {       // a stage has accumulators of its own
                            wait_on(&full[s], par);
                            tc_fence_after();
                            if (lead) {
                                const uint32_t d1 = tmem + s * 2 * NT, d2 = d1 + NT;
#pragma unroll
                                for (int t = 0; t < SP; ++t) {
                                    if (t == 1 && 2 * j + 1 >= nst) break;
                                    const uint32_t slot = s * SP + t, ac = tmem + A_COL + slot * 64u, bh = b_lo + slot * (uint32_t)(G::BSTEP / 16);
#pragma unroll
                                    for (uint32_t q = 0; q < 4; ++q) {
                                        tc_mma_ts(d1, ac + q * 8u, desc(bh + q * 2u), TC_IDESC<2 * NT>, t + q > 0 ? 1u : 0u);
                                        tc_mma_ts(d2, ac + 32u + q * 8u, desc(bh + q * 2u), TC_IDESC<NT>, 1u);
                                    }
                                }
                                tc_commit(&empty[s]);       // for the reading warpgroup too
                            }
                        } else {
                            const bool fresh = (j - j0) % G::PERIOD == 0;   // D1 starts again; D2 only with an item
                            if (j == j0 && periods) wait_on(&d_empty, (periods - 1u) & 1u);
                            wait_on(&full[s], par);
                            tc_fence_after();
                            const uint32_t d1 = tmem, d2 = tmem + NT, ac = tmem + A_COL + s * 64u, bh = b_lo + s * (uint32_t)(G::BSTEP / 16);
                            if (fresh && j > j0) {          // the products for D2 while D1 is read
                                if (lead) {
#pragma unroll
                                    for (uint32_t q = 0; q < 4; ++q) {
                                        tc_mma_ts(d2, ac + q * 8u, desc(bh + NT * 8 + q * 2u), TC_IDESC<NT>, 1u);
                                        tc_mma_ts(d2, ac + 32u + q * 8u, desc(bh + q * 2u), TC_IDESC<NT>, 1u);
                                    }
                                }
                                __syncwarp();
                                wait_on(&d_empty, (periods - 1u) & 1u);
                                tc_fence_after();
                                if (lead) {
#pragma unroll
                                    for (uint32_t q = 0; q < 4; ++q) tc_mma_ts(d1, ac + q * 8u, desc(bh + q * 2u), TC_IDESC<NT>, q > 0 ? 1u : 0u);
                                }
                            } else if (lead) {
#pragma unroll
                                for (uint32_t q = 0; q < 4; ++q) {
                                    tc_mma_ts(d1, ac + q * 8u, desc(bh + q * 2u), TC_IDESC<2 * NT>, (q > 0 || j > j0) ? 1u : 0u);
                                    tc_mma_ts(d2, ac + 32u + q * 8u, desc(bh + q * 2u), TC_IDESC<NT>, 1u);
                                }
                            }
                            periods += fresh ? 1u : 0u;
                            if (lead) {
                                tc_commit(&empty[s]);
                                if ((j - j0) % G::PERIOD == G::PERIOD - 1 || j == j1 - 1) tc_commit(&d_full);
                            }
                        }
                        __syncwarp();
                        if (++s == (uint32_t)NS) { s = 0; par ^= 1u; }
                    }
                }
            }
        }
        __syncwarp();
        if (S > 1) { cl_arrive(); cl_wait(); cl_arrive(); cl_wait(); }
    } else if (wg <= NH) {
        // ---- results: the accumulators into registers; an item's end: scale back, activation, store ----
        reg_inc<G::REG_READ>();
        pdl_wait();
        // Which half it reads, and its thread.  rd and the barrier's number are constants where one warpgroup reads: in registers they
        // cost spills at NT = 64 (a text of 65 tokens at the 1B shape is scored in 3960 us instead of 3900).  rt comes from wg: from
        // rd it costs spills in the Q4_K instance of NT = 128 (a 27B prompt of 100 tokens and 24 steps 24.08 ms instead of 23.98).
        const int rd = NH == 1 ? 0 : wg - 1, rt = tid - wg * 128;
        auto sync_rd = [&]() { asm volatile("bar.sync %0, 128;" :: "r"(rd + 1) : "memory"); };
        float* xch = reinterpret_cast<float*>(sm + G::XCH) + rd * (G::XCOLS * 128);
        uint32_t nth = 0;                               // accumulation period
        if constexpr (G::BANKS > 1) { if (lane < NS) mbar_arrive(&full[lane]); }        // all accumulators are free
        if constexpr (HEAD) {
            if (rt < NT) s_best[rt] = 0;
            sync_rd();
        }
        [[maybe_unused]] auto flush_best = [&](int m0) {
            sync_rd();
            if (rt < min(NT, a.B - m0)) {
                if (s_best[rt]) atomicMax(a.best + m0 + rt, s_best[rt]);
                s_best[rt] = 0;
            }
            sync_rd();
        };
        for (int q = q0; q < q1;) {
            const int i0 = q / spi, j0 = q - i0 * spi, j1 = min(spi, j0 + q1 - q), item = item_of(i0), tn = n_of(item), m0 = m_of(item) + rd * NC;
            const int np = (j1 - j0 + G::PERIOD - 1) / G::PERIOD;                       // accumulation periods
            q += j1 - j0;
            float acc[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) acc[c] = 0.f;
#pragma unroll 1
            for (int p = 0; p < np; ++p, ++nth) {
                const uint32_t bank = nth % G::BANKS;
                if constexpr (G::BANKS > 1) wait_on(&empty[bank], (nth / G::BANKS) & 1u);
                else wait_on(&d_full, nth & 1u);
                tc_fence_after();
                auto take = [&](uint32_t col) {         // the tensor core may wait for this: few round trips
                    constexpr int CH = NT == 256 || NC < 32 ? 16 : 32;
#pragma unroll
                    for (int ch = 0; ch < NC; ch += CH) {
                        float v[CH / 16][16];
#pragma unroll
                        for (int h = 0; h < CH / 16; ++h) tc_ld16(col + ch + 16 * h, v[h]);
                        tc_ld_wait();
                        if (NT == 256 && ch == NC - CH) {       // all of it is in registers
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&d_empty);
                        }
#pragma unroll
                        for (int c = 0; c < CH; c += 2) fma2(acc[ch + c], acc[ch + c + 1], v[c / 16][c % 16], v[c / 16][c % 16 + 1], 1.f, 1.f);
                    }
                };
                if constexpr (NT == 256) take(tlane + rd * NC);
                else {
#pragma unroll 1
                    for (int h = 0; h < (G::BANKS > 1 || p == np - 1 ? 2 : 1); ++h) take(tlane + bank * 2 * NT + h * NT);
                }
                if constexpr (NT != 256) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(G::BANKS > 1 ? &full[bank] : &d_empty);
                }
            }
            if (S > 1) {                                // one item per cluster, and the activation ring is drained: it becomes the exchange
                float* ex = reinterpret_cast<float*>(smB);
#pragma unroll
                for (int c = 0; c < NC; ++c) ex[c * 128 + row] = acc[c];
                break;
            }
            if (j1 - j0 < spi) {
                // a tile that several CTAs share: leave the partial sums; the CTA that arrives last adds all of them
                auto cta_of = [&](int qq) {
                    int c = (int)((long long)qq * n_cta / all);
                    while (q_begin(c) > qq) --c;
                    while (q_begin(c + 1) <= qq) ++c;
                    return c;
                };
                const int c_lo = cta_of(item * spi), c_hi = cta_of(item * spi + spi - 1);
                auto slot_of = [&](int c) { return a.part + (size_t)((2 * c + (c == c_lo ? 1 : 0)) * NH + rd) * (NC * 128) + row; };   // it begins here, or before
                float* out = slot_of(cta);
#pragma unroll
                for (int c = 0; c < NC; ++c) out[c * 128] = acc[c];
                __threadfence();
                sync_rd();
                if (rt == 0) {
                    unsigned int* ticket = a.tickets + c_lo * NH + rd;
                    const unsigned int seen = atomicAdd(ticket, 1u);
                    s_last[rd] = seen == (unsigned int)(c_hi - c_lo);
                    if (s_last[rd]) *ticket = 0u;
                }
                sync_rd();
                const bool last = s_last[rd];
                sync_rd();
                if (!last) continue;
                __threadfence();
                constexpr int CH = NT == 256 || NC < 32 ? 16 : 32;     // columns whose loads are in flight together
#pragma unroll
                for (int ch = 0; ch < NC; ch += CH) {
                    const float* in = slot_of(c_lo) + ch * 128;
#pragma unroll
                    for (int c = 0; c < CH; ++c) acc[ch + c] = __ldcg(in + c * 128);
                }
#pragma unroll 1
                for (int other = c_lo + 1; other <= c_hi; ++other) {
                    const float* in = slot_of(other);
#pragma unroll
                    for (int ch = 0; ch < NC; ch += CH) {
                        float t[CH];
#pragma unroll
                        for (int c = 0; c < CH; ++c) t[c] = __ldcg(in + (ch + c) * 128);
#pragma unroll
                        for (int c = 0; c < CH; ++c) acc[ch + c] += t[c];
                    }
                }
            }
            // Out through shared memory, XC columns at a time, by rolled loops.
            constexpr int XC = G::XCOLS;
            const int n_col = min(NC, a.B - m0);
            const int r = pair ? row & 63 : row, n = pair ? tn * 64 + r : tn * 128 + r;
            float* yp = a.y + (size_t)m0 * a.ldy + n;
            if (rt < n_col) s_inv[rd * NC + rt] = a.inv[m0 + rt];
            sync_rd();
#pragma unroll 1
            for (int h0 = 0; h0 < n_col; h0 += XC) {
                const int m = min(XC, n_col - h0);
#pragma unroll
                for (int c = 0; c < XC; ++c) xch[c * 128 + row] = acc[c];
                if (pair) {                             // gate (lanes 0..63) and up rows meet; all lanes share the outputs
                    sync_rd();
#pragma unroll 4
                    for (int c = row >> 6; c < m; c += 2) {
                        const float sc = s_inv[rd * NC + h0 + c], v = act(xch[c * 128 + r] * sc, xch[c * 128 + 64 + r] * sc);
                        if (n < a.N) yp[(size_t)(h0 + c) * a.ldy] = v;
                    }
                    sync_rd();
                } else if constexpr (HEAD) {
                    // best of the warp's rows per column: NaN counts as -FLT_MAX, ties go to the lower row
                    unsigned long long mine = 0;        // lane c: column h0 + c
#pragma unroll 2
                    for (int c = 0; c < m; ++c) {
                        const float v = xch[c * 128 + row] * s_inv[rd * NC + h0 + c], f = (v == v ? v : -3.402823466e+38f) + 0.f;
                        const uint32_t bits = __float_as_uint(f), ord = n < a.N ? bits ^ ((uint32_t)((int)bits >> 31) | 0x80000000u) : 0u;
                        const uint32_t top = __reduce_max_sync(0xffffffffu, ord);
                        const uint32_t at = __reduce_min_sync(0xffffffffu, ord == top ? (uint32_t)n : 0xffffffffu);
                        if (lane == c) mine = ((unsigned long long)top << 32) | (0xffffffffu - at);
                        if (a.y && n < a.N) yp[(size_t)(h0 + c) * a.ldy] = a.softcap > 0.f ? tanhf(v / a.softcap) * a.softcap : v;
                    }
                    if (lane < m) atomicMax(&s_best[h0 + lane], mine);
                } else if (n < a.N) {
#pragma unroll 4
                    for (int c = 0; c < m; ++c) yp[(size_t)(h0 + c) * a.ldy] = xch[c * 128 + row] * s_inv[rd * NC + h0 + c];
                }
#pragma unroll
                for (int c = 0; c < NC - XC; ++c) acc[c] = acc[c + XC];
            }
            if constexpr (HEAD) { if (a.B > NT) flush_best(m0); }       // the columns change with the next item
            sync_rd();              // s_inv is free again
        }
        if (S > 1) finish_split();
        if constexpr (HEAD) {                           // the last CTA to end decodes the winners and clears the keys
            flush_best(0);
            __threadfence();
            sync_rd();
            if (rt == 0) s_last[0] = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
            sync_rd();
            if (s_last[0]) {
                __threadfence();
                for (int b = rt; b < a.B; b += 128) {
                    const unsigned long long key = __ldcg(a.best + b);
                    const uint32_t ord = (uint32_t)(key >> 32);
                    const int tok = (int)(0xffffffffu - (uint32_t)key);
                    if (a.out_tok) a.out_tok[b] = tok;
                    if (a.out_tok_f32) a.out_tok_f32[b] = (float)tok;
                    if (a.out_val) a.out_val[b] = __uint_as_float(ord & 0x80000000u ? ord ^ 0x80000000u : ~ord);
                    a.best[b] = 0;
                }
                if (rt == 0) *a.ticket = 0u;
            }
        }
    } else {
        // ---- weights ----
        reg_set<G::REG_MAKE, 65536 / G::THREADS / 8 * 8>();
        const int grp = wg - 1 - NH, quarter = warp & 3;
        // This group fills step `sub` of every GROUPS / SP-th stage of the CTA's range.  It waits for a ring slot to be emptied
        // without having followed every phase of it, which is sound because the slots empty in order: it has seen a later
        // one than the slot's last but one use empty (GROUPS <= NS * SP).
        const int sub = grp % SP;
        uint8_t* ring = sm + G::RING + (warp - 4 * (1 + NH)) * G::R * G::SLOT;
        const uint32_t ring_s = smem_u32(ring);
        const WeightRef w = (pair && quarter >= 2) ? a.w1 : a.w0;                      // lanes 64..127 of a pair: up rows
        const bool scales_async = WT == WT_Q4_K || ((a.units & 1) == 0 && ((uintptr_t)w.d & 3) == 0);
        auto row_of = [&](int tn, int r) { return min(pair ? tn * 64 + (r & 63) : tn * 128 + r, a.N - 1); };
        const int rpu = WT == WT_Q4_0 ? a.units : WT == WT_Q8_0 ? 2 * a.units : (a.units >> 3) * 9;     // uint4 per weight row
        struct Cursor { int q, i, j; };                 // stage: of the range, item of the range and stage of the item
        constexpr int HOP = G::GROUPS / SP;
        auto next = [&](Cursor& c) { c.q += HOP; c.j += HOP; while (c.j >= spi) { c.j -= spi; ++c.i; } };

        // fetch cursor, R tiles ahead of the production cursor
        const int q_first = q0 + grp / SP;
        Cursor f = {q_first, q_first / spi, q_first % spi};
        int f_k = -1; uint32_t f_n = 0;                 // item that the row pointers belong to; ring slot
        constexpr int LPR = G::QB / 16, FI = LPR;       // lanes per row and copies per lane of a step's codes
        const uint4 *f_q[FI], *f_h = nullptr; const __half* f_d = nullptr;
        auto fetch = [&]() {
            if (f.q < q1) {
                if (f_k != f.i) {
                    f_k = f.i;
                    const int tn = n_of(item_of(f.i));
#pragma unroll
                    for (int h = 0; h < FI; ++h) f_q[h] = w.q + (size_t)row_of(tn, quarter * 32 + (32 / FI) * h + lane / LPR) * rpu;
                    if constexpr (WT != WT_Q4_K) f_d = w.d + (size_t)row_of(tn, row) * a.units;
                    else f_h = w.q + (size_t)row_of(tn, row) * rpu;
                }
                const int st = f.j * SP + sub, ks = ma0 + st - nmn;
                if (st >= nmn && st < nst) {
                    const uint32_t dst = ring_s + f_n * G::SLOT;
                    const int piece = lane % LPR;
                    const int off = WT == WT_Q4_K ? (ks >> 2) * 9 + 1 + (ks & 3) * 2 + piece : min(LPR * ks + piece, rpu - 1);
#pragma unroll
                    for (int h = 0; h < FI; ++h) {      // 16-byte pieces are stored rotated: the reads below are free of bank conflicts
                        const int rl = (32 / FI) * h + lane / LPR;
                        cp_async16(dst + rl * G::QB + ((LPR == 2 ? piece ^ ((rl >> 2) & 1) : piece ^ ((rl >> 1) & 3)) << 4), f_q[h] + off);
                    }
                    if constexpr (WT != WT_Q4_K) { if (scales_async) cp_async4(dst + 32 * G::QB + lane * 4, f_d + 2 * ks); }
                    else cp_async16_l1(dst + 32 * G::QB + lane * 16, f_h + (ks >> 2) * 9);
                }
                next(f);
            }
            if (++f_n == (uint32_t)G::R) f_n = 0;
            cp_commit();
        };
        uint32_t at = 0;                                // weight ring slot
        bool waited = false;
        Cursor c = {q_first, q_first / spi, q_first % spi};
        // One copy of the loop body serves the start too: R - 1 fetches before the first tile is taken.
#pragma unroll 1
        for (int turn = 0; c.q < q1; ++turn) {
            fetch();
            if (turn < G::R - 1) continue;
            const int st = c.j * SP + sub, ks = ma0 + st - nmn;
            const uint32_t nth = (uint32_t)(c.q - q0), stage = nth % NS, acol = tlane + A_COL + (stage * SP + sub) * 64u;
            cp_wait<G::R - 1>();
            __syncwarp();
            const uint8_t* slot = ring + at * G::SLOT;
            const uint8_t* codes = slot + lane * G::QB;
            auto piece_at = [&](int p) { return *reinterpret_cast<const uint4*>(codes + ((LPR == 2 ? p ^ ((lane >> 2) & 1) : p ^ ((lane >> 1) & 3)) << 4)); };
            if (!waited) { pdl_wait(); waited = true; } // no bounded wait below spans an earlier kernel
            if (nth >= (uint32_t)NS) {                  // the tensor core is done with what the slot held
                wait_on(&empty[stage], (nth / NS - 1u) & 1u);
                tc_fence_after();
            }
            if (WT == WT_Q4_K ? st >= nmn && st < nst : st < nst) {
                uint32_t d01 = 0, sp = 0;               // two block scales; or a superblock's, and two sub-blocks' factors
                if constexpr (WT != WT_Q4_K) {
                    if (scales_async) d01 = *reinterpret_cast<const uint32_t*>(slot + 32 * G::QB + lane * 4);
                    else {                              // odd number of blocks per row: their scales are not pairs of aligned halves
                        const unsigned short* dp = reinterpret_cast<const unsigned short*>(w.d) + (size_t)row_of(n_of(item_of(c.i)), row) * a.units + 2 * ks;
                        d01 = (uint32_t)dp[0] | (2 * ks + 1 < a.units ? (uint32_t)dp[1] << 16 : 0u);
                    }
                } else {
                    const uint4 hdr = *reinterpret_cast<const uint4*>(slot + 32 * G::QB + lane * 16);
                    uint32_t mp;
                    q4k_codes(hdr, ks & 3, sp, mp);
                    d01 = (hdr.x & 0xFFFFu) * 0x10001u;
                }
#pragma unroll (NT == 128 || (NT < 128 && WT == WT_Q4_K) ? 2 : 1)
                for (int b = 0; b < 2; ++b) {           // 32 values of K: columns 16 b .. of w_hi and of w_lo
                    const uint32_t col = acol + b * 16u;
                    uint32_t whi[8], wlo[8], v[2];
                    if constexpr (WT == WT_Q8_0) {      // bytes + 128 into the mantissa of 1024, two at a time
                        const __half2 d = as_h2((d01 >> (16 * b) & 0xFFFFu) * 0x10001u);
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
                            const uint4 p4 = piece_at(2 * b + y);
                            const uint32_t qw[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                            for (int x = 0; x < 4; ++x) {
                                const uint32_t u = qw[x] ^ 0x80808080u;
                                v[0] = (u & 0x00FF00FFu) | 0x64006400u; v[1] = ((u >> 8) & 0x00FF00FFu) | 0x64006400u;
#pragma unroll
                                for (int p = 0; p < 2; ++p) split_h2(__hadd2(as_h2(v[p]), __float2half2_rn(-1152.f)), d, whi[2 * x + p], wlo[2 * x + p]);
                            }
                            tc_st8(col + y * 8u, whi);
                            tc_st8(col + 32u + y * 8u, wlo);
                        }
                    } else if constexpr (WT == WT_Q4_0) {       // block b: values 0..15 in the low nibbles, 16..31 in the high ones
                        const __half2 d = as_h2((d01 >> (16 * b) & 0xFFFFu) * 0x10001u);
                        const uint4 p4 = piece_at(b);
                        const uint32_t qw[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                        for (int x = 0; x < 4; ++x) {
                            nib_pairs<false>(qw[x], v);
#pragma unroll
                            for (int p = 0; p < 2; ++p) split_h2(__hadd2(as_h2(v[p]), __float2half2_rn(-1032.f)), d, whi[2 * x + p], wlo[2 * x + p]);
                        }
                        tc_st8(col, whi);
                        tc_st8(col + 32u, wlo);
#pragma unroll
                        for (int x = 0; x < 4; ++x) {
                            nib_pairs<true>(qw[x], v);
#pragma unroll
                            for (int p = 0; p < 2; ++p) split_h2(__hfma2(as_h2(v[p]), __float2half2_rn(0.0625f), __float2half2_rn(-72.f)), d, whi[2 * x + p], wlo[2 * x + p]);
                        }
                        tc_st8(col + 8u, whi);
                        tc_st8(col + 40u, wlo);
                    } else {                            // low nibbles = sub-block 2g, high nibbles = sub-block 2g + 1
                        const uint32_t code = sp >> (8 * b) & 0xFFu;
                        const __half2 sc = __hsub2(as_h2((code * 0x10001u) | 0x64006400u), __float2half2_rn(1024.f)), off = __hmul2(sc, __float2half2_rn(-72.f));
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
                            const uint4 p4 = piece_at(y);
                            const int up = 4 - 4 * b;
                            const uint32_t qw[4] = {p4.x << up, p4.y << up, p4.z << up, p4.w << up};
#pragma unroll
                            for (int x = 0; x < 4; ++x) {
                                nib_pairs_64(qw[x], v);
#pragma unroll
                                for (int p = 0; p < 2; ++p)       // sc * (q - 8), an integer of at most 504, exactly
                                    split_h2(__hfma2(as_h2(v[p]), sc, off), as_h2(d01), whi[2 * x + p], wlo[2 * x + p]);
                            }
                            tc_st8(col + y * 8u, whi);
                            tc_st8(col + 32u + y * 8u, wlo);
                        }
                    }
                }
            } else if (WT == WT_Q4_K && st < nmn) {
                // a step of block offsets: 32 (8 d sc - dmin m) of 64 sub-blocks (the image holds the sums over 32 activations / 32)
                const int sb0 = (mn0 + st) * 8, n_sb = a.units >> 3;
                const uint4* src = w.q + (size_t)row_of(n_of(item_of(c.i)), row) * rpu;
#pragma unroll 1
                for (int b = 0; b < 4; ++b) {
                    uint32_t whi[8], wlo[8];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int sb = sb0 + 2 * b + e;
                        const uint4 h = __ldg(src + (size_t)min(sb, n_sb - 1) * 9);
                        const bool in = sb < n_sb;
                        const float dm = in ? -32.f * __half2float(__ushort_as_half((unsigned short)(h.x >> 16))) : 0.f;
                        const float d8 = in ? 256.f * __half2float(__ushort_as_half((unsigned short)(h.x & 0xFFFFu))) : 0.f;
#pragma unroll
                        for (int gq = 0; gq < 4; ++gq) {
                            uint32_t sp, mp;
                            q4k_codes(h, gq, sp, mp);
                            const float v0 = fmaf(d8, (float)(sp & 0xFFu), dm * (float)(mp & 0xFFu)), v1 = fmaf(d8, (float)(sp >> 8), dm * (float)(mp >> 8));
                            const __half2 h2 = __floats2half2_rn(v0, v1);
                            const float2 f2 = __half22float2(h2);
                            whi[4 * e + gq] = as_u32(h2);
                            wlo[4 * e + gq] = as_u32(__floats2half2_rn(v0 - f2.x, v1 - f2.y));
                        }
                    }
                    tc_st8(acol + b * 8u, whi);
                    tc_st8(acol + 32u + b * 8u, wlo);
                }
            }
            tc_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[NT == 256 ? stage * 2 + sub : stage]);
            if (++at == (uint32_t)G::R) at = 0;
            next(c);
        }
        cp_wait<0>();
        if (S > 1) finish_split();
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tc_dealloc(tmem, 512);
}

// ---- host ----------------------------------------------------------------------------------------------------------
// Fewest rows from which the GEMM is faster than the GEMV kernels, measured in decode steps and single calls.  The GEMV
// passes over the weights once per 1, 2 or 4 rows.  Where the passes run side by side on idle SMs (matrices below some 10 MB)
// that costs little (1B shape: 8 rows 1.11 against 1.10 ms per step, a chunk of 8 prompt rows 1.39 against 1.45 ms; 10 rows:
// 1.22 against 1.15; 12: 1.35 against 1.16); where they fill the GPU it costs their number (27B shape with every matrix on
// one path, 4 rows: 1.62 against 2.02 ms, 6: 2.5 against 2.04, 12: 3.9 against 2.08).  An LM head of a narrow model is bound by
// rebuilding weights here (262144 x 1152: 75 us whatever the rows, the GEMV 43 us at 4 and 71 at 8).
// Without a row-tiled copy a GEMV takes one launch per four rows (7 us each).  Q8_0 / Q5_0 have no tensor-core GEMV; their
// product in fp32 is 1.2e-7 from the exact one, closer than the 2.1e-7 of this kernel, so a product that is asked for by itself
// stays there, and the Q8_0 heads of a model come here, whose logits carry 2e-6 from the layers.
static int tc_rows_from(int wtype, const GemvArgs& a, bool pair, bool tiled) {
    if (wtype == WT_Q8_0) return a.epi == EPI_ARGMAX ? 4 : 1 << 30;
    if (!tiled) return 5;
    const double bytes = (double)a.N * a.K * 0.5625 * (pair ? 2 : 1);
    if (a.epi == EPI_ARGMAX && a.K < 4096) return 9;
    return bytes > 10.0e6 ? 6 : 9;
}

static int tc_clusters_at_once(int s);
// Does the call take the mma.sync kernel (gemm_mma.cu)?  Matrices above 10 MB from 3 rows to 16, smaller ones and the heads of
// narrow models from 5 to 8.  us a call, row kernel included, with it and without (GEMV up to 5 rows, above that k_gemm_tc), by rows:
//   21504 x 5376 Q4_K   2: 26.7, 24.2   4: 24.1, 32.2   8: 29.4, 47.3   16: 42.1, 47.6   32: 75, 54.5
//   5376 x 21504 Q4_K   2: 30.3, 36.5   4: 30.1, 59.8   8: 34.2, 54.2   16: 47.9, 55.0   32: 77, 61.9
//   1152 x 6912 Q4_0    4: 6.1, 8.2     8: 7.7, 9.8     12: 9.3, 9.9    16: 10.7, 10.0
//   6912 x 1152 Q4_0    4: 4.7, 7.5     8: 5.7, 8.2     16: 7.3, 8.7
//   262144 x 1152 Q4_0  4: 48.5, 40.9   8: 65.6, 91.2   12: 86, 91.7    16: 108, 92.0
// and ms a decode step: 1B shape 4 rows 0.887 and 0.894, 5 to 8 rows 1.04 and 1.12 to 1.15, 10 rows 1.226 and 1.220, 16 rows 1.365
// and 1.242; 27B shape (8 layers) 2 rows 1.16 and 1.05, 3 rows 1.18 and 1.52, 8 rows 1.42 and 2.08, 16 rows 2.16 and 2.25.
// From 9 rows on only where it has CTAs for the SMs: a long K over few row groups leaves them idle, and k_gemm_tc's clusters do
// not.  CTAs here and there, us with it and without: 2560 x 10240 Q4_K 80, 120: 12 rows 19.4, 17.8, 16 rows 20.7, 18.0; on 16 rows
// 3072 x 12288 Q4_0 96, 120: 21.1, 19.8, 1536 x 14336 Q4_0 96, 96: 17.2, 15.5, but 4096 x 14336 Q4_0 128, 128: 23.6, 24.3; on 12 rows
// 3072 x 12288 Q4_0 17.1, 19.4, 1536 x 14336 Q4_0 14.8, 15.4.
static bool takes_mma(int wtype, const GemvArgs& a, const uint8_t* t0, const uint8_t* t1, int policy) {
    const bool pair = a.epi == EPI_GEGLU || a.epi == EPI_SWIGLU;
    if (!t0 || (pair && !t1) || policy != 1 || !gemm_mma_supports(wtype, a)) return false;
    const bool large = (double)a.N * a.K * 0.5625 * (pair ? 2 : 1) > 10.0e6 && !(a.epi == EPI_ARGMAX && a.K < 4096);
    if (large ? a.B < 3 : a.B < 5 || a.B > 8) return false;
    if (a.B > 8 && large) {
        const int ctas = gemm_mma_ctas(wtype, a), tiles = pair ? (a.N + 63) / 64 : (a.N + 127) / 128;
        if (a.B > 12 && 3 * ctas <= 2 * g.sm_count) return false;
        std::lock_guard<std::mutex> work(g_tc_lock);
        int there = tiles < g.sm_count ? tiles : g.sm_count;
        for (int s = 2; s <= 8 && a.epi != EPI_ARGMAX; ++s) if (tiles <= tc_clusters_at_once(s)) there = tiles * s;
        if (10 * ctas < 7 * there) return false;
    }
    return (size_t)(a.K / 32) * gm_block_bytes(wtype, gemm_mma_pad(a.B)) <= g_tc.img_cap && gemm_mma_pad(a.B) <= g_tc.inv_cap;
}

GemmRoute gemm_route(int wtype, const GemvArgs& a, const uint8_t* t0, const uint8_t* t1, bool wide) {
    const bool pair = a.epi == EPI_GEGLU || a.epi == EPI_SWIGLU;
    int policy = g_tc_policy;
    if (policy < 0) {
        const int first = getenv("ADAM_B200_TC") ? atoi(getenv("ADAM_B200_TC")) : 1;
        if (g_tc_policy.compare_exchange_strong(policy, first)) policy = first;
    }
    if (wtype != WT_Q4_0 && wtype != WT_Q4_K && (wtype != WT_Q8_0 || pair)) return GEMM_NONE;
    if (a.B < TC_MIN_ROWS || a.K <= 0 || a.K > TC_MAX_K || a.N < 16 || (!a.y && a.epi != EPI_ARGMAX) || (wtype == WT_Q4_K ? (a.K % 256) : (a.K % 32))) return GEMM_NONE;
    if (a.epi == EPI_ARGMAX && a.B > tc_rows_fit(wtype, a.K)) return GEMM_NONE;
    if ((a.ldx & 3) || (!a.h_in && (!a.x || ((uintptr_t)a.x & 15)))) return GEMM_NONE;
    if (policy == 1 && t0 && (t1 || !pair) && gemv_rows_takes(wtype, a)) return GEMM_NONE;
    if (takes_mma(wtype, a, t0, t1, policy)) return GEMM_FEW;
    if (wide) return GEMM_NONE;
    if (policy == 0 || (policy == 1 && a.B < tc_rows_from(wtype, a, pair, t0 && (t1 || !pair)))) return GEMM_NONE;
    return tc_rows_fit(wtype, a.K) >= 128 ? GEMM_TC : GEMM_NONE;
}

typedef void (*TcKernel)(const TcGemm);
struct TcPick { TcKernel k; int smem, threads; bool attr; };
template <int WT, int NT, bool HEAD> static TcPick& tc_pick() {
    static TcPick p = {k_gemm_tc<WT, NT, HEAD>, TcGeo<WT, NT>::SMEM, TcGeo<WT, NT>::THREADS, false};
    return p;
}
template <int WT, bool HEAD> static TcPick& tc_pick(int nt) {
    if constexpr (!HEAD && WT != WT_Q8_0) { if (nt == 256) return tc_pick<WT, 256, HEAD>(); }
    return nt == 16 ? tc_pick<WT, 16, HEAD>() : nt == 32 ? tc_pick<WT, 32, HEAD>() : nt == 64 ? tc_pick<WT, 64, HEAD>() : tc_pick<WT, 128, HEAD>();
}
template <int WT> static TcPick& tc_pick(int nt, bool head) { return head ? tc_pick<WT, true>(nt) : tc_pick<WT, false>(nt); }

// Clusters of `s` CTAs that run at the same time, one CTA per SM (clusters stay inside a GPC).
static int tc_clusters_at_once(int s) {
    static int known[9] = {};
    if (!known[s]) {
        TcPick& p = tc_pick<WT_Q4_0, 16, false>();
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)s); cfg.blockDim = dim3((unsigned)p.threads); cfg.dynamicSmemBytes = (size_t)p.smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)s; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.attrs = at; cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute((const void*)p.k, cudaFuncAttributeMaxDynamicSharedMemorySize, p.smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, (const void*)p.k, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
        known[s] = n > 0 ? n : -1;
    }
    return known[s];
}

// One CTA per row; the fewest float4 per thread that 512 threads allow.
template <bool FEW> static void launch_quant_rows(const GemvArgs& a, int n_min, int n_steps, cudaStream_t stream) {
    const int cand[5] = {1, 2, 4, 8, 16}, n4 = a.K / 4;
    int mv = 16;
    for (int c : cand) if ((n4 + c - 1) / c <= 512) { mv = c; break; }
    const int threads = ((n4 + mv - 1) / mv + 31) / 32 * 32;
    auto go = [&](auto kern) { launch_k(kern, dim3(a.B), dim3(threads), 0, stream, true, a, g_tc.img, g_tc.inv, n_min, n_steps); };
    const bool chain = a.h_in != nullptr;
    switch (mv) {
    case 1: if (chain) go(k_quant_rows<1, true, FEW>); else go(k_quant_rows<1, false, FEW>); break;
    case 2: if (chain) go(k_quant_rows<2, true, FEW>); else go(k_quant_rows<2, false, FEW>); break;
    case 4: if (chain) go(k_quant_rows<4, true, FEW>); else go(k_quant_rows<4, false, FEW>); break;
    case 8: if (chain) go(k_quant_rows<8, true, FEW>); else go(k_quant_rows<8, false, FEW>); break;
    default: if (chain) go(k_quant_rows<16, true, FEW>); else go(k_quant_rows<16, false, FEW>); break;
    }
    count_launch();
}

static int launch_rows(int wtype, const GemvArgs& a, cudaStream_t stream) {
    const bool pair = a.epi == EPI_GEGLU || a.epi == EPI_SWIGLU;
    const int n_min = tc_min_steps(wtype, a.K), n_main = tc_main_steps(a.K);
    launch_quant_rows<false>(a, n_min, n_min + n_main, stream);
    // Work split: the cheapest under an estimate in SM cycles.  A step costs the larger of its tensor-core time and what
    // the rebuilding of a weight tile allows.  Dealt out evenly, a CTA costs its stages and, where tiles are shared, the
    // adding up of P partial results of nt columns; as clusters of S, waves of CTAs and one exchange.  One set of figures for
    // all block types, although rebuilding a Q4_K weight takes longer than a Q4_0 one: they only rank the splits of one call.
    const bool head = a.epi == EPI_ARGMAX;
    const int tiles_n = pair ? (a.N + 63) / 64 : (a.N + 127) / 128;
    int nt = 0, S = 1, grid = 1;
    bool shared = false;
    double best = 1e300;
    auto offer_tiles = [&](int n, double step) {
        const int sp = n == 128 ? 1 : 2, spi1 = (n_min + n_main + sp - 1) / sp;
        const long long items = (long long)tiles_n * ((a.B + n - 1) / n), all = items * spi1;
        auto offer = [&](double cost, int s, int ctas, bool sh) { if (cost < best * 0.999) { best = cost; nt = n; S = s; grid = ctas; shared = sh; } };
        const int whole = (int)(items < g.sm_count ? items : g.sm_count);
        offer((double)((items + whole - 1) / whole) * spi1 * sp * step, 1, whole, false);
        if (all >= g.sm_count) {
            const double per = (double)((all + g.sm_count - 1) / g.sm_count), sharers = 2.0 + spi1 / per;
            offer(per * sp * step + 3000.0 + n * (20.0 + 40.0 * sharers), 1, g.sm_count, true);
        }
        for (int s = 2; s <= (head || n == 256 ? 1 : 8) && s <= n_main; ++s) {
            const int at_once = tc_clusters_at_once(s);
            if (at_once < 1 || (n == 128 && items > at_once)) continue;
            const int steps = (n_main + s - 1) / s + (n_min + s - 1) / s;
            offer((double)((items + at_once - 1) / at_once) * ((steps + sp - 1) / sp * sp * step + 2000.0), s, (int)items * s, false);
        }
    };
    // Clusters of 128-row tiles only where all of them run at once.  A second wave starts CTAs anew (barriers, tensor memory, an empty
    // pipeline), which the estimate does not see: us with and without it, 6912 pairs x 1152 on 320 rows 74.6 and 59.2, 1152 x 1024 on
    // 1280 rows 39.1 and 20.1, 1536 x 1152 on 2048 rows 54.2 and 34.0, 1152 x 6912 on 1280 rows 98.9 and 68.6, 4096 x 2560 on 300
    // rows 45.7 and 31.5.  Over 242 measured products (14 shapes, 65 to 2048 rows) the split chosen so takes 1.1 % longer than
    // the best of all, 5.0 % with second waves.
    // Tiles of 256 rows take 1.9 times a tile of 128 (13824 x 1152 on 2048 rows 166 against 175 us, 21504 x 5376 on 1024 rows 598
    // against 631), so they win where their number suits the SMs as well as that of the smaller ones does: 5376 x 4096 Q4_K on 768 rows,
    // 126 tiles, 97 against 100 us, but 1152 x 6912 on 2048 rows, 72 tiles, 120 against 92.
    if (a.B <= 64) offer_tiles(a.B <= 16 ? 16 : a.B <= 32 ? 32 : 64, a.B > 32 ? 620.0 : 500.0);
    else {
        offer_tiles(128, 1250.0);
        if (a.B > 128 && !head && wtype != WT_Q8_0) offer_tiles(256, 2380.0);
    }
    const int tiles_m = (a.B + nt - 1) / nt;
    TcGemm t = {};
    t.w0 = a.w0; t.w1 = a.w1; t.y = a.y; t.ldy = a.ldy; t.img = g_tc.img; t.inv = g_tc.inv; t.err = g.dev_err;
    t.N = a.N; t.units = a.K / 32; t.B = a.B; t.swiglu = a.epi == EPI_SWIGLU;
    t.n_min = n_min; t.n_main = n_main; t.S = S;
    t.tiles_n = tiles_n;
    t.items = tiles_n * tiles_m;
    t.part = g_tc.part; t.tickets = g_tc.tickets; t.shared = shared ? 1 : 0;
    t.pair = pair;
    if (head) {
        t.best = g_tc.best; t.ticket = (unsigned int*)(g_tc.best + g_tc.inv_cap);
        t.out_tok = a.out_tok; t.out_val = a.out_val; t.out_tok_f32 = a.out_tok_f32; t.softcap = a.softcap;
    }
    TcPick& p = wtype == WT_Q4_0 ? tc_pick<WT_Q4_0>(nt, head) : wtype == WT_Q4_K ? tc_pick<WT_Q4_K>(nt, head) : tc_pick<WT_Q8_0>(nt, head);
    if (!p.attr) {
        if (cudaFuncSetAttribute((const void*)p.k, cudaFuncAttributeMaxDynamicSharedMemorySize, p.smem) != cudaSuccess)
            return fail(ADAMAH_ERR_BACKEND, "gemm_tc: cannot raise the shared-memory limit");
        p.attr = true;
    }
    cudaError_t e;
    if (S == 1) e = launch_k(p.k, dim3((unsigned)grid), dim3(p.threads), (size_t)p.smem, stream, true, t);
    else e = launch_k_cluster(p.k, dim3((unsigned)grid), dim3(p.threads), (size_t)p.smem, stream, true, (unsigned)S, false, t);
    if (e != cudaSuccess) return fail(ADAMAH_ERR_BACKEND, "gemm_tc: launch failed: %s", cudaGetErrorString(e));
    count_launch();
    ++g_gemm_counts[nt == 16 ? GC_TILE_16 : nt == 32 ? GC_TILE_32 : nt == 64 ? GC_TILE_64 : nt == 128 ? GC_TILE_128 : GC_TILE_256];
    if (shared) ++g_gemm_counts[GC_SHARED];
    if (S > 1) ++g_gemm_counts[t.items > tc_clusters_at_once(S) ? GC_CLUSTER_WAVES : GC_CLUSTERS];
    return ADAMAH_OK;
}

// Rows that exceed the workspace run in chunks of whole 128-row tiles.
int launch_gemm(GemmRoute route, int wtype, const uint8_t* t0, const uint8_t* t1, const GemvArgs& a, cudaStream_t stream) {
    std::lock_guard<std::mutex> work(g_tc_lock);
    if (route == GEMM_FEW) {
        launch_quant_rows<true>(a, tc_min_steps(wtype, a.K), gemm_mma_pad(a.B), stream);
        const int rc = launch_gemm_mma(wtype, t0, t1, a, GemmWork{g_tc.img, g_tc.inv, g_tc.part, g_tc.tickets, g_tc.best, (unsigned int*)(g_tc.best + g_tc.inv_cap)}, stream);
        if (rc) return rc;
        ++g_tc_calls;
        return check_launch("gemm_mma");
    }
    const int fit = tc_rows_fit(wtype, a.K);
    for (int b0 = 0; b0 < a.B; b0 += fit) {
        GemvArgs c = a;
        c.B = a.B - b0 < fit ? a.B - b0 : fit;
        if (a.x) c.x = a.x + (size_t)b0 * a.ldx;
        if (a.h_in) c.h_in = a.h_in + (size_t)b0 * a.ldx;
        if (a.add_src) c.add_src = a.add_src + (size_t)b0 * a.ldx;
        if (a.h_out) c.h_out = a.h_out + (size_t)b0 * a.ldx;
        if (a.y) c.y = a.y + (size_t)b0 * a.ldy;
        const int rc = launch_rows(wtype, c, stream);
        if (rc) return rc;
    }
    ++g_tc_calls;
    return check_launch("gemm_tc");
}

}  // namespace ab

// Number of GEMMs enqueued on the tcgen05 path since the library was loaded (tests use it to
// see which kernel a call took).
extern "C" uint64_t adam_b200_tc_gemm_count(void) { return ab::g_tc_calls; }
// The same by kernel and split: the first n values of the enumeration in gemm_tc.cuh.
extern "C" int adam_b200_gemm_counts(uint64_t* out, uint32_t n) {
    if (!out) return ADAMAH_ERR_INVALID;
    std::lock_guard<std::mutex> work(ab::g_tc_lock);
    for (uint32_t i = 0; i < n; ++i) out[i] = i < ab::GC_COUNTS ? ab::g_gemm_counts[i] : 0;
    return ADAMAH_OK;
}
// 0 = never use the tcgen05 GEMM, 1 = where it is expected to be faster (default), 2 = whenever the shape allows.
extern "C" int adam_b200_tc_gemm_policy(int policy) {
    if (policy < 0 || policy > 2) return ADAMAH_ERR_INVALID;
    ab::g_tc_policy = policy;
    return ADAMAH_OK;
}
