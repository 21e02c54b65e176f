// Chunked gated delta rule (delta_chunk.cu) as linear_attention.cu calls it.
#pragma once
#include <cuda_runtime.h>

namespace b200 {

struct DeltaChunkArgs {
  const void *q, *k, *v;               // bf16 [T, Hk, 128], [T, Hk, 128], [T, Hv, DV], token strides below
  long qk_stride, v_stride;
  const float *g, *beta;               // [T, Hv]
  float* state;                        // [slots, Hv, 128, DV]
  const int *cu, *slots, *has_init;
  void* out;                           // bf16
  long out_stride;
  int Hk, Hv, DV;
  float scale;
  int l2norm;
  long num_slots;
  int min_len;                         // sequences with fewer tokens are left alone
  int* status;
};

bool launch_delta_chunk(const DeltaChunkArgs& p, int B, int DK, cudaStream_t stream, int* rc);

}  // namespace b200
