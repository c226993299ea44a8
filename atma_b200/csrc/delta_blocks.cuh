// The gated delta rule in fp32 arithmetic for any type and head size (delta_blocks.cu), as its callers see it.
#pragma once

#include "common.cuh"

namespace atma {

struct DeltaBlocks {
  const void *q, *k, *v;           // [rows][Hq][dk], [rows][G][dk], [rows][G or H][dv] (dtype)
  void* o;                         // [rows][H][dv] (dtype)
  const float *q_inv, *k_inv;      // [rows][Hq], [rows][G]: factors of the rows; nullptr = see `normalize`
  int normalize;                   // without factors: 1 = rows are divided by their length (at least 1e-12), 0 = used as they are
  float q_scale;                   // times q, besides
  const float *log_decay, *beta;   // [rows][H]
  const int32_t* cu_rows;          // [n_seqs + 1], or nullptr = every sequence has `len` rows
  const int32_t* start_pos;        // [n_seqs]: 0 = starts from a zero state, < 0 = its outputs are zero; nullptr = starts from state_in
  const int64_t* slots;            // [n_seqs] planes of the state arrays (< 0 = its outputs are zero), or nullptr = sequence i's is i
  const float* state_in;           // [planes][H][dk][dv], or nullptr = zero
  float* state_out;                // may be state_in, or nullptr
  int64_t state_ss;                // elements between planes
  int n_seqs, len;
  int64_t total_rows;
  int H, Hq, G, Hv, dk, dv, dtype;
};

bool delta_blocks_supported(int64_t total_rows, int n_seqs, int H, int dk);
int64_t delta_blocks_scratch_bytes(int64_t total_rows, int n_seqs, int H, int dk, int dv);
int delta_blocks_scan(const DeltaBlocks& a, void* scratch, cudaStream_t st);

}  // namespace atma
