// Host-side launch logic of the GEMV for two to four rows (kernel in gemv_rows.cuh).
#include "gemv_rows.cuh"

namespace ab {

typedef void (*RowsKernel)(const GemvArgs, const uint8_t*, const uint8_t*, int, float);
struct RowsShape { RowsKernel k; int ks, rgs; size_t smem; };
// 1B shape, ms per step with k_gemv_mma and with this kernel: 2 rows 0.730 and 0.502, 3 0.838 and 0.643, 4 0.901 and 0.694.  Instances
// for eight rows took 0.960 at 5 rows, 0.974 at 6 and 1.051 at 8, the few-row GEMM takes 0.927, 0.934 and 0.960: it keeps those calls.
constexpr int ROWS_MAX = 4;
constexpr int ROWS_SMEM_LIMIT = 220 * 1024;

template <int WT, int NR>
static RowsKernel pick(bool pair, bool chain, int ppw, bool one_group) {
    if (ppw == 4) return k_gemv_rows<false, WT, false, 4, NR, NR, 1024>;
    if (one_group) return pair ? k_gemv_rows<true, WT, true, 2, NR, NR, 512> : chain ? k_gemv_rows<false, WT, true, 2, NR, NR, 512> : k_gemv_rows<false, WT, false, 2, NR, NR, 512>;
    return pair ? k_gemv_rows<true, WT, true, 2, NR, NR / 2, 1024> : chain ? k_gemv_rows<false, WT, true, 2, NR, NR / 2, 1024> : k_gemv_rows<false, WT, false, 2, NR, NR / 2, 1024>;
}

// Two tile pairs per warp (a lane stages one float4 of a row's slice), four for plain rows longer than 16 such slices; row groups
// per CTA: as many as give every SM one.
template <int WT>
static RowsShape rows_shape(const GemvArgs& a) {
    const bool pair = a.epi == EPI_GEGLU || a.epi == EPI_SWIGLU, chain = a.h_in != nullptr;
    const int pairs = a.K >> 6, n_rg = a.N >> 4, nr = a.B <= 2 ? 2 : 4;
    RowsShape s = {};
    s.rgs = (n_rg + g.sm_count - 1) / g.sm_count;
    int ppw = 2;
    s.ks = (pairs + 1) / 2;
    if (s.rgs == 1 && s.ks > 16) {
        if (chain) return RowsShape{};
        ppw = 4;
        s.ks = (pairs + 3) / 4;
    }
    if (s.ks * s.rgs > ROW_MAX_WARPS || (pair && !chain)) return RowsShape{};
    s.k = nr == 2 ? pick<WT, 2>(pair, chain, ppw, s.rgs == 1) : pick<WT, 4>(pair, chain, ppw, s.rgs == 1);
    const size_t nm = pair ? 2 : 1, warps = (size_t)s.ks * s.rgs;
    s.smem = (size_t)s.ks * 2 * ppw * nr * 128 + warps * nm * ppw * mma_tile_bytes(WT) + (size_t)s.rgs * nr * nm * 16 * 36 * 4 +
             (WT == WT_Q4_K ? (size_t)s.ks * 2 * ppw * nr * 8 : 0);
    if (s.smem > (size_t)ROWS_SMEM_LIMIT) return RowsShape{};
    return s;
}

static bool rows_shape_for(int wt, const GemvArgs& a, RowsShape* out) {
    if (a.N <= 0 || a.K <= 0 || a.B < 2 || a.B > ROWS_MAX || a.N % 16 || a.K % 64 || a.epi == EPI_ARGMAX) return false;
    if (wt != WT_Q4_0 && (wt != WT_Q4_K || a.K % 256)) return false;
    const void* x = a.h_in ? (const void*)a.h_in : (const void*)a.x;
    if (((uintptr_t)x & 15) || (a.ldx & 3)) return false;
    const RowsShape s = wt == WT_Q4_0 ? rows_shape<WT_Q4_0>(a) : rows_shape<WT_Q4_K>(a);
    if (!s.k) return false;
    static thread_local RowsKernel known[64]; static thread_local int n_known = 0;
    bool is_known = false;
    for (int i = 0; i < n_known; ++i) is_known |= known[i] == s.k;
    if (!is_known) {
        if (!carveout_max((const void*)s.k, ROWS_SMEM_LIMIT)) return false;
        if (n_known < 64) known[n_known++] = s.k;
    }
    *out = s;
    return true;
}

bool gemv_rows_takes(int wt, const GemvArgs& a) {
    RowsShape s;
    return rows_shape_for(wt, a, &s);
}

int launch_gemv_rows(int wt, const uint8_t* t0, const uint8_t* t1, GemvArgs a, cudaStream_t stream) {
    RowsShape s;
    if (!rows_shape_for(wt, a, &s)) return fail(ADAMAH_ERR_INVALID, "gemv_rows: shape not supported");
    a.err = g.dev_err;
    if (launch_k(s.k, dim3((a.N / 16 + s.rgs - 1) / s.rgs), dim3(s.ks * s.rgs * 32), s.smem, stream, g.pdl, a, t0, t1, s.ks, 1.0f / (float)a.K) != cudaSuccess)
        return fail(ADAMAH_ERR_BACKEND, "gemv_rows: launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    count_ran(RAN_GEMV_ROWS);
    return ADAMAH_OK;
}

}  // namespace ab
