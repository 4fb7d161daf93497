// Host-side launch logic of the one-row GEMV (kernel in gemv_row.cuh).
#include "gemv_row.cuh"

#include <atomic>

namespace ab {

typedef void (*RowKernel)(const GemvArgs, const uint8_t*, const uint8_t*, float);
struct RowShape { RowKernel k; int id, ks; size_t smem; };        // id: which of a type's instances
constexpr int ROW_IDS = 9;

// Two tile pairs per warp: its 32 lanes hold one float4 of activations each, the shortest chain there is (K <= 4096); four for
// longer rows.  Up to nine slices (K <= 1152) a thread keeps to 56 registers: three such CTAs, what a matrix of 400 row groups
// needs of every SM, then leave room in each quarter of the register file for the kernels ahead of them, and all start in time.
constexpr int ROW_THREADS = 288, ROW_CTAS = 4;
template <int WT>
static RowShape row_shape(const GemvArgs& a) {
    const bool pair = a.epi == EPI_GEGLU || a.epi == EPI_SWIGLU, chain = a.h_in != nullptr;
    const int pairs = a.K >> 6;
    RowShape s = {};
    int ppw = 2;
    s.ks = (pairs + 1) / 2;
    s.id = (pair ? 1 : 0) + (chain ? 2 : 0);
    if (s.ks * 32 <= ROW_THREADS) {
        s.k = pair ? (chain ? k_gemv_row<true, WT, true, 2, ROW_THREADS, ROW_CTAS> : k_gemv_row<true, WT, false, 2, ROW_THREADS, ROW_CTAS>)
                   : (chain ? k_gemv_row<false, WT, true, 2, ROW_THREADS, ROW_CTAS> : k_gemv_row<false, WT, false, 2, ROW_THREADS, ROW_CTAS>);
    } else if (s.ks <= ROW_MAX_WARPS) {
        s.id += 4;
        s.k = pair ? (chain ? k_gemv_row<true, WT, true, 2, 1024, 1> : k_gemv_row<true, WT, false, 2, 1024, 1>)
                   : (chain ? k_gemv_row<false, WT, true, 2, 1024, 1> : k_gemv_row<false, WT, false, 2, 1024, 1>);
    } else {
        ppw = 4;
        s.id = 8;
        s.ks = (pairs + 3) / 4;
        if (pair || chain || s.ks > ROW_MAX_WARPS) return RowShape{};
        s.k = k_gemv_row<false, WT, false, 4, 1024, 1>;
    }
    s.smem = (size_t)s.ks * ppw * 256;
    return s;
}

static bool row_shape_for(int wt, const GemvArgs& a, RowShape* out) {
    if (a.N <= 0 || a.K <= 0 || a.B != 1 || a.N % 16 || a.K % 64 || a.epi == EPI_ARGMAX) return false;
    if (wt != WT_Q4_0 && (wt != WT_Q4_K || a.K % 256)) return false;
    const void* x = a.h_in ? (const void*)a.h_in : (const void*)a.x;
    if (((uintptr_t)x & 15) || (a.ldx & 3)) return false;
    const RowShape s = wt == WT_Q4_0 ? row_shape<WT_Q4_0>(a) : row_shape<WT_Q4_K>(a);
    if (!s.k) return false;
    // Every CTA resident at once: a second wave would request its weights only when the first is done, which is what the rings
    // of k_gemv_mma are for.  (Asked for once per instance and number of slices.)
    static std::atomic<int> known[2][ROW_IDS][ROW_MAX_WARPS + 1];           // CTAs per SM plus one, 0 = not asked yet
    std::atomic<int>& kn = known[wt == WT_Q4_0 ? 0 : 1][s.id][s.ks];
    int per_sm = kn - 1;
    if (per_sm < 0) {
        if (!carveout_max((const void*)s.k, 0) ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, s.k, s.ks * 32, s.smem) != cudaSuccess) { cudaGetLastError(); return false; }
        kn = per_sm + 1;
    }
    if ((long long)(a.N / 16) > (long long)per_sm * g.sm_count) return false;
    // and at most 48 warps per SM: more of them take the instructions of as many stagings (9472 x 1152, 36 warps per SM, 5.2 us by
    // k_gemv_mma and 3.4 here; 20000 x 1024, 68 warps, 7.4 and 7.7)
    if ((long long)(a.N / 16) * s.ks > 48ll * g.sm_count) return false;
    *out = s;
    return true;
}

bool gemv_row_takes(int wt, const GemvArgs& a) {
    RowShape s;
    return row_shape_for(wt, a, &s);
}

int launch_gemv_row(int wt, const uint8_t* t0, const uint8_t* t1, GemvArgs a, cudaStream_t stream) {
    RowShape s;
    if (!row_shape_for(wt, a, &s)) return fail(ADAMAH_ERR_INVALID, "gemv_row: shape not supported");
    const uint32_t n_w = (uint32_t)(a.N / 16 * s.ks);
    for (int r = 0; r < 3; ++r) {
        if (!a.pf[r]) a.pf_bytes[r] = 0;
        a.pf_part[r] = (a.pf_bytes[r] / n_w + 127u) & ~127u;
    }
    if (launch_k(s.k, dim3(a.N / 16, a.B), dim3(s.ks * 32), s.smem, stream, g.pdl, a, t0, t1, 1.0f / (float)a.K) != cudaSuccess)
        return fail(ADAMAH_ERR_BACKEND, "gemv_row: launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    count_ran(RAN_GEMV_ROW);
    return ADAMAH_OK;
}

}  // namespace ab
