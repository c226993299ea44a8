// Shared between the gated-delta scan kernels (16-bit inputs, d_k = d_v = 128, chunk = 64): the
// per-chunk factor record that the chunk-local kernel writes and the recurrence kernels read, and
// the descriptors of packed ("varlen") batches and of recurrence-to-factor maps.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cstdint>

namespace atma {
namespace scan {

constexpr int kC = 64, kD = 128;
// One record per (sequence, head, chunk): three 16-bit row-major [64 p][64 s] tiles
//   Tw = -T diag(beta g k_inv) | Tu = T diag(beta) | Rq = tril((g_p / g_s) q^_p.k^_s)          T = (I + A)^-1
// and, in a second array, one float per row for each of g q_inv scale and (g_C / g) k_inv, then g_C.  Behind it, in
// fp16, whether the chunk has a row of a length outside of [1, 64] (kScalFar): k_inv is then split in all of its rows, a power of two per row,
// which the recurrence multiplies the K rows with, and a factor from 1/2 to 1, which takes its place here.  The power is there as
// two fp16 ones (kScalP), whose product can be beyond what fp16 holds.  The rows of q, k and v
// themselves are read again by the recurrence, which makes -W = Tw K and U0 = Tu V beside its chain: a record with
// W, U0, Qg and Kt in it is 72 KB of writes and reads for what takes 24, and rounds each of them to 16 bits.
constexpr int kTile64 = kC * kC * 2, kRecTw = 0, kRecTu = kTile64, kRecRq = 2 * kTile64, kRecBytes = 3 * kTile64;
constexpr int kScalQ = 0, kScalK = kC, kScalG = 2 * kC, kScalFar = 2 * kC + 1, kScalP = 3 * kC, kScal = 256;                    // floats
// Scratch per chunk and head: record, scalars, and the rows of q, k, v that scan_factors keeps for scan_recur (whose
// callers hand it nothing but the scratch), and the whole scans where results take the inputs' place.
constexpr int kScratchPerChunk = kRecBytes + kScal * 4 + 3 * kC * kD * 2;

template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (kBf16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  } else {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  }
}
template <bool kBf16>
__device__ __forceinline__ float2 unpack2(uint32_t v) {
  if constexpr (kBf16) return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
  else return __half22float2(*reinterpret_cast<__half2*>(&v));
}
// byte offset of the 16-byte chunk `chunk` (0..7) of row `row` inside a 128-byte-swizzled box
__device__ __forceinline__ uint32_t box_off(int row, int chunk) {
  return (uint32_t)(row * 128 + ((chunk ^ (row & 7)) << 4));
}

// Packed batches: sequences of different lengths back to back in one token axis.  Chunks never
// straddle sequences: sequence i owns chunk records cu_chunks[i] .. cu_chunks[i+1]-1.
struct VarLen {
  const int32_t* cu_seqlens;   // device [n_seqs + 1] token offsets; nullptr = dense (B, T) batch
  const int32_t* cu_chunks;    // device [n_seqs + 1] chunk offsets (built by varlen_chunk_offsets_kernel)
  int n_seqs;
  const int64_t* slots;        // device [n_seqs] rows of state_table, or nullptr (dense state arrays)
  const int32_t* has_initial;  // device [n_seqs] or nullptr (= every sequence starts from its table row)
  float* state_table;          // [rows][H][dk][dv] fp32, or nullptr
  int64_t slot_stride;         // elements between table rows
  // state snapshots for prefix reuse: after every snap_chunks chunks that lie wholly inside the
  // sequence, the fp32 state goes to snapshots[snap_offsets[seq] + j] ([...][H][dk][dv]); nullptr = none
  float* snapshots;
  const int32_t* snap_offsets; // device [n_seqs]
  int snap_chunks;
};

constexpr int kMaxRec = 64;   // recurrences per launch
struct RecMap {                 // recurrence i walks the chunk records of batch entry rec[i];
  int rec[kMaxRec];             // zero_u0[i] != 0 replaces U0 by zero (the "v = 0" recurrence that
  int zero_u0[kMaxRec];         // yields a segment's state-transfer matrix)
  int c_begin[kMaxRec];         // chunk range [c_begin, c_end) of the records that recurrence i walks
  int c_end[kMaxRec];           // (c_end = 0 means "all NC chunks")
  int o_row[kMaxRec];           // batch row of the output tensor that recurrence i writes (negative: no output)
  int state_row[kMaxRec];       // plane of initial_state / final_state that recurrence i reads / writes
};

// The rows that the factors were made from: q (tokens, H, 128), k, v (tokens, Hkv, 128), contiguous 16-bit.
struct Rows {
  const void *q, *k, *v;
  int is_bf16, H, Hkv;
  int64_t tokens;
};

}  // namespace scan

// Recurrence over the chunk records on the 5th-generation tensor cores (gated_delta_scan_sm100.cu).
// Dense form: n_rec recurrences over the records of a scratch built for B sequences of T tokens;
// packed form (var.cu_seqlens != nullptr): one recurrence per sequence.  o may be null (state only).
int gated_delta_recur_sm100(const scan::Rows& rows, const uint8_t* recs, const float* scal, int64_t n_records, const float* initial_state,
                            void* o, float* final_state, int Tlen, int NC, int n_rec, const scan::RecMap& map,
                            const scan::VarLen& var, cudaStream_t st);
int scan_sm100_status_fetch_and_clear(int* out);

// Chunk-local factors on the 5th-generation tensor cores (gated_delta_local_sm100.cu): g, beta (tokens, H) fp32; records and
// scalars as laid out above.  Dense form: B sequences of Tlen tokens (NC chunks each); packed form: var.cu_seqlens / cu_chunks.
int gated_delta_local_sm100(const scan::Rows& rows, const float* g, const float* beta, uint8_t* recs, float* scal, int B, int Tlen,
                            int NC, int normalize_qk, float scale, const scan::VarLen& var, cudaStream_t st);
int scan_local_status_fetch_and_clear(int* out);

// (d, head, token) view of a (tokens, heads, 128) 16-bit tensor; boxes of 64 channels x 64 tokens of one head
int make_rows_map(CUtensorMap* out, const void* base, int is_bf16, int heads, int64_t tokens);

}  // namespace atma
