// Entry of the paired-SM GEMM (gemm_pair.cu) for the dispatch in gemm.cu.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace mx {

struct GemmPairParams {
  __nv_bfloat16* out;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  int* status;
  int M, N, K, ldo, ldr;
  int glu_offset, epilogue;
  float glu_alpha, glu_limit;
  const float* ssq_in;          // deferred RMSNorm, as in GemmParams
  float* ssq_out;
  float ssq_eps, ssq_inv_dim;
  int w_fresh;
  int tiles_m, tiles_n, raster; // filled by the launch
};

bool gemm_pair_wanted(const GemmPairParams& p, bool glu, int sms);
int gemm_pair_launch(const CUtensorMap& map_x, const CUtensorMap& map_w, GemmPairParams p, bool glu, int sms, cudaStream_t stream);

}  // namespace mx
