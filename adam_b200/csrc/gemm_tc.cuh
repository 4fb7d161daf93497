// Dequant-fused GEMM for many activation rows on the 5th-generation tensor cores (tcgen05, TMEM).
// Interface of gemm_tc.cu; see there for the design.
#pragma once
#include "common.cuh"
#include "gemv.cuh"

namespace ab {

constexpr int TC_MIN_ROWS = 2;         // fewer rows than this never leave the GEMV kernels

// Does this problem run on the tcgen05 path?  `tiled`: the GEMV kernels would have row-tiled copies of the weights; `wide`:
// the weights' map says that fp16 may not hold them.
bool gemm_tc_supports(int wtype, const GemvArgs& a, bool tiled, bool wide);
// Makes room for calls with up to `rows` activation rows of length K (outside any stream capture; longer calls run in
// chunks).  The workspace only grows; false when out of memory.
bool gemm_tc_prepare(int rows, int K);
void gemm_tc_release();
// Enqueues the row-quantisation kernel and the GEMM.  Returns ADAMAH_OK or an error code.
int launch_gemm_tc(int wtype, const GemvArgs& a, cudaStream_t stream);

}  // namespace ab
