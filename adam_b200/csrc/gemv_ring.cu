// Host-side launch logic of the streaming one-row GEMV (kernel in gemv_ring.cuh).
#include "gemv_ring.cuh"

namespace ab {

typedef void (*RingKernel)(const GemvArgs, const uint8_t*, const uint8_t*, float);
// Row groups per CTA at most: beyond, the staging that this kernel saves is less than its barrier per row group costs.  us by k_gemv_mma
// and here, cold, Q4_0 / Q4_K: 12000 x 5376 (5.1 per CTA) 14.3 and 11.4 / 16.8 and 14.8; 16000 x 5376 (6.8) 15.1 and 13.5 / 17.7
// and 17.3; 21504 x 5376 (9.1) 18.5 and 16.8 / 21.8 and 22.9; 32768 x 5376 (13.8) 22.7 and 23.0 / 27.9 and 31.0.  One line for both
// types, where Q4_K turns; Q4_0 turns between 9 and 14.
constexpr int RING_SETS = 7;
constexpr int RING_SMEM_LIMIT = 220 * 1024;

// Ring stages: three, two beside the staged form of a very long row (86 KB at K = 21504) where three do not fit.
template <int WT>
static RingKernel pick(bool pair, bool chain, int nv, int nst) {
    if (nst == 2) return pair || chain || nv > 12 ? nullptr : k_gemv_ring<false, WT, false, 12, 2>;
    if (pair) return chain && nv <= 4 ? k_gemv_ring<true, WT, true, 4, 3> : nullptr;
    if (chain) return nv <= 4 ? k_gemv_ring<false, WT, true, 4, 3> : nullptr;
    return nv <= 4 ? k_gemv_ring<false, WT, false, 4, 3> : nv <= 12 ? k_gemv_ring<false, WT, false, 12, 3> : nullptr;
}

struct RingShape { RingKernel k; size_t smem; };
// Rows of at least two tile pairs per slice (a set of sums costs a barrier), at most twelve float4 per lane (four where the norm chain
// holds four vectors: such rows come up to K = 6144, what gemv_mma_supports takes), beside which the rings fit.
static bool ring_shape(int wt, const GemvArgs& a, RingShape* out) {
    if (a.N <= 0 || a.K <= 0 || a.B != 1 || a.N % 16 || a.K % 64 || a.epi == EPI_ARGMAX) return false;
    if (wt != WT_Q4_0 && (wt != WT_Q4_K || a.K % 256)) return false;
    const void* x = a.h_in ? (const void*)a.h_in : (const void*)a.x;
    if ((uintptr_t)x & 15) return false;
    const int pairs = a.K >> 6, np = (pairs + RING_WARPS - 1) / RING_WARPS, nv = (np + 1) / 2;
    if (pairs < 2 * RING_WARPS || a.N / 16 > RING_SETS * g.sm_count) return false;
    const bool pair = a.epi == EPI_GEGLU || a.epi == EPI_SWIGLU, chain = a.h_in != nullptr;
    RingShape s;
    int nst = 3;
    const auto bytes = [&](int n) { return (size_t)pairs * (wt == WT_Q4_K ? 272 : 256) + (size_t)RING_WARPS * mma_ring_bytes_per_warp(wt, n); };
    if (bytes(nst) > (size_t)RING_SMEM_LIMIT) nst = 2;
    s.smem = bytes(nst);
    s.k = wt == WT_Q4_0 ? pick<WT_Q4_0>(pair, chain, nv, nst) : pick<WT_Q4_K>(pair, chain, nv, nst);
    if (!s.k || s.smem > (size_t)RING_SMEM_LIMIT) return false;
    static thread_local RingKernel known[12]; static thread_local int n_known = 0;
    bool is_known = false;
    for (int i = 0; i < n_known; ++i) is_known |= known[i] == s.k;
    if (!is_known) {
        if (!carveout_max((const void*)s.k, RING_SMEM_LIMIT)) return false;
        if (n_known < 12) known[n_known++] = s.k;
    }
    *out = s;
    return true;
}

bool gemv_ring_takes(int wt, const GemvArgs& a) {
    RingShape s;
    return ring_shape(wt, a, &s);
}

int launch_gemv_ring(int wt, const uint8_t* t0, const uint8_t* t1, GemvArgs a, cudaStream_t stream) {
    RingShape s;
    if (!ring_shape(wt, a, &s)) return fail(ADAMAH_ERR_INVALID, "gemv_ring: shape not supported");
    a.err = g.dev_err;
    const int n_rg = a.N / 16;
    if (launch_k(s.k, dim3(n_rg < g.sm_count ? n_rg : g.sm_count), dim3(RING_WARPS * 32), s.smem, stream, g.pdl, a, t0, t1, 1.0f / (float)a.K) != cudaSuccess)
        return fail(ADAMAH_ERR_BACKEND, "gemv_ring: launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    count_ran(RAN_GEMV_RING);
    return ADAMAH_OK;
}

}  // namespace ab
