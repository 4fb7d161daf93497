// Dequant-fused GEMM for many activation rows on the 5th-generation tensor cores (tcgen05, TMEM).
// Interface of gemm_tc.cu; see there for the design.
#pragma once
#include "common.cuh"
#include "gemv.cuh"

namespace ab {

constexpr int TC_MIN_ROWS = 2;         // fewer rows than this never leave the GEMV kernels
// Floats of one item's partial sums in the workspace; a CTA has two such slots, for its first and its last item.
constexpr int GEMM_SLOT = 128 * 256;

// Which GEMM a problem runs on, none for the GEMV kernels.  `t0`, `t1`: row-tiled copies of the weights, where there are any;
// `wide`: the weights' map says that fp16 may not hold them.  Asked once per call: the answer goes with it, for the policy may
// change in between.
enum GemmRoute { GEMM_NONE, GEMM_FEW, GEMM_TC };
GemmRoute gemm_route(int wtype, const GemvArgs& a, const uint8_t* t0, const uint8_t* t1, bool wide);
// Makes room for calls with up to `rows` activation rows of length K (outside any stream capture; longer calls run in
// chunks).  The workspace only grows; false when out of memory.
bool gemm_tc_prepare(int rows, int K);
void gemm_tc_release();
// Enqueues the row-quantisation kernel and the GEMM.  Returns ADAMAH_OK or an error code.
int launch_gemm(GemmRoute route, int wtype, const uint8_t* t0, const uint8_t* t1, const GemvArgs& a, cudaStream_t stream);

// Which kernels calls have taken, counted under the lock that orders them: the few-row kernel (also: with items shared between CTAs),
// k_gemm_tc by rows of a tile (16 .. 256), with tiles shared, as clusters, and as more clusters than run at once.
enum { GC_FEW, GC_FEW_SHARED, GC_TILE_16, GC_TILE_32, GC_TILE_64, GC_TILE_128, GC_TILE_256, GC_SHARED, GC_CLUSTERS, GC_CLUSTER_WAVES, GC_COUNTS };
extern uint64_t g_gemm_counts[GC_COUNTS];

// ---- gemm_mma.cu: the second kernel of a call with few rows ----
constexpr int GM_MAX_ROWS = 16;
// Bytes of the activation image per 32 values of K, with room for `rows` rows (a multiple of four).
__host__ __device__ constexpr int gm_block_bytes(int wtype, int rows) { return rows * (wtype == WT_Q4_K ? 132 : 128); }
struct GemmWork { const uint8_t* img; const float* inv; float* part; unsigned int* tickets; unsigned long long* best; unsigned int* ticket; };
bool gemm_mma_supports(int wtype, const GemvArgs& a);
int gemm_mma_pad(int rows);            // rows the image has room for
int gemm_mma_ctas(int wtype, const GemvArgs& a);        // CTAs that a supported call is launched with
int launch_gemm_mma(int wtype, const uint8_t* t0, const uint8_t* t1, const GemvArgs& a, const GemmWork& w, cudaStream_t stream);

}  // namespace ab
