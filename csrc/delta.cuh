// Arguments of the gated delta rule's kernels (delta.cu, delta_chunk.cu).
#pragma once
#include "common.cuh"

#define LLMSS_DELTA_PREPARED 13312      // bytes that a chunk of 32 tokens and a head take between the two launches over chunks

struct DeltaArgs {
  const float* q; int64_t ldq;
  const float* k; int64_t ldk;
  const float* v; int64_t ldv;
  const float* log_decay; int64_t ldg;   // [T, H]
  const float* beta; int64_t ldb;        // [T, H]
  float* out;                            // [T, H * dv]
  float* state;                          // [slots, H, dv, dk]
  const int* cu_q; const int* seq_lens; const int* slots;
  int H, rep, dk, dv, dvt;
  float unit_eps, q_scale;
  int unit, beta_sigmoid;
  int vec16;       // q / k / v rows, the key size and the value slices allow 16-byte copies
  uint8_t* prepared;                     // [T / 32 + sequences][H] x LLMSS_DELTA_PREPARED, on a 16-byte line
  int least, below;      // sequences of least .. below - 1 tokens are this launch's
};

int delta_chunk_launch(const DeltaArgs& a, int B, int max_q, cudaStream_t stream);
