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
  // Over chunks: [T / 32 + sequences][H] x LLMSS_DELTA_PREPARED, on a 16-byte line (else null).  A sequence of `least` tokens and more goes over chunks until
  // a chunk that its products cannot take; the record of its first chunk then says how many tokens are done, per 128 value columns, and
  // the token-by-token launch takes the others.
  uint8_t* prepared;
  int least, chunks;     // (chunks: the most that are prepared of one sequence)
};

constexpr int kDeltaChunk = 32, kDeltaCols = 128, kDeltaDone = 29;       // tokens of a chunk, value columns of a block over chunks, blocks that a record has room for

int delta_chunk_launch(DeltaArgs a, int B, int max_q, cudaStream_t stream);
// where in a record the tokens done lie: behind the tiles and the numbers per token
constexpr int kDeltaDoneAt = LLMSS_DELTA_PREPARED - 4 * kDeltaDone;
