// Entry of the two-head prefill attention (attention_tc2.cu) for the dispatch in attention_tc.cu.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace mx {

struct PrefillTc2Params {
  const int* block_tables;
  const int* cu_q;
  const int* context_lens;
  const float* sinks;
  __nv_bfloat16* out;           // [tokens, Hq * D]
  int* status;
  int num_seqs, Hq, Hkv, max_blocks, window, tiles_per_seq;
  float scale_log2;
};

// Hq / Hkv even, D 64 or 128, scale_log2 > 0; grid = num_seqs * Hq / 2 * tiles_per_seq.
int prefill_tc2_launch(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, const PrefillTc2Params& p, int D,
                       int grid, cudaStream_t stream);

}  // namespace mx
