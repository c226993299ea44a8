// Gated-delta chunked scan: the C entries.  16-bit inputs with d_k = d_v = 128 run on the tensor cores in chunks of 64 tokens,
// everything else in fp32 arithmetic in blocks of eight (delta_blocks.cu).
#include "delta_blocks.cuh"

namespace atma {

constexpr int kScanC = 64;            // tokens per chunk of the tensor-core form

// tensor-core version for 16-bit inputs with d_k = d_v = 128 (gated_delta_scan_mma.cu)
bool gated_delta_scan_mma_supported(int dtype, int dk, int dv);
int64_t gated_delta_scan_mma_scratch_bytes(int B, int T, int H);
int gated_delta_scan_mma(const void* q, const void* k, const void* v, int dtype, const float* g, const float* beta,
                         const float* initial_state, void* o, float* final_state, void* scratch, int B, int T, int H,
                         int Hkv, int normalize_qk, float scale, int segments, cudaStream_t st);

int gated_delta_scan_mma_factors(const void* q, const void* k, const void* v, int dtype, const float* g,
                                 const float* beta, void* scratch, int B, int T, int H, int Hkv, int normalize_qk,
                                 float scale, bool keep_rows, cudaStream_t st);
int gated_delta_scan_mma_recur(const void* q, const void* k, const void* v, int Hkv, void* scratch, int dtype, int B, int T, int H,
                               int n_rec, const int* rec_of, const int* zero_u0, const float* initial_state, void* o, float* final_state,
                               cudaStream_t st);
int64_t gated_delta_scan_mma_varlen_scratch_bytes(int64_t total_tokens, int n_seqs, int H);
int gated_delta_scan_mma_varlen(const void* q, const void* k, const void* v, int dtype, const float* g, const float* beta,
                                const int32_t* cu_seqlens, int n_seqs, int64_t total_tokens, const float* initial_state,
                                float* final_state, float* state_table, int64_t slot_stride, const int64_t* slots,
                                const int32_t* has_initial, void* o, void* scratch, int H, int Hkv, int normalize_qk,
                                float scale, float* snapshots, const int32_t* snap_offsets, int snap_chunks,
                                cudaStream_t st);

}  // namespace atma

using namespace atma;

static int scan_factors_impl(const void* q, const void* k, const void* v, int dtype, const float* g, const float* beta, void* scratch, int B,
                             int T, int H, int Hkv, int dk, int dv, int normalize_qk, float scale, bool keep_rows, void* stream) {
  ATMA_REQUIRE(gated_delta_scan_mma_supported(dtype, dk, dv),
               "gated_delta_scan_factors: needs 16-bit inputs with dk = dv = 128 (got dtype %d, dk %d, dv %d)", dtype, dk, dv);
  ATMA_REQUIRE(B > 0 && T > 0 && H > 0 && Hkv > 0 && H % Hkv == 0, "gated_delta_scan_factors: bad shape");
  ATMA_REQUIRE(scratch != nullptr && (uintptr_t)scratch % 256 == 0 && (uintptr_t)q % 16 == 0 && (uintptr_t)k % 16 == 0 &&
                   (uintptr_t)v % 16 == 0, "gated_delta_scan_factors: scratch must be 256-byte and inputs 16-byte aligned");
  return gated_delta_scan_mma_factors(q, k, v, dtype, g, beta, scratch, B, T, H, Hkv, normalize_qk, scale, keep_rows, (cudaStream_t)stream);
}

extern "C" int atma_gated_delta_scan_factors(const void* q, const void* k, const void* v, int dtype, const float* g,
                                             const float* beta, void* scratch, int B, int T, int H, int Hkv, int dk,
                                             int dv, int normalize_qk, float scale, void* stream) {
  return scan_factors_impl(q, k, v, dtype, g, beta, scratch, B, T, H, Hkv, dk, dv, normalize_qk, scale, true, stream);
}

extern "C" int atma_gated_delta_scan_factors_alone(const void* q, const void* k, const void* v, int dtype, const float* g,
                                                   const float* beta, void* scratch, int B, int T, int H, int Hkv, int dk,
                                                   int dv, int normalize_qk, float scale, void* stream) {
  return scan_factors_impl(q, k, v, dtype, g, beta, scratch, B, T, H, Hkv, dk, dv, normalize_qk, scale, false, stream);
}

extern "C" int atma_gated_delta_scan_recur(void* scratch, int dtype, int B, int T, int H, int dk, int dv, int n_rec,
                                           const int* rec_of, const int* zero_u0, const float* initial_state, void* o,
                                           float* final_state, void* stream) {
  ATMA_REQUIRE(gated_delta_scan_mma_supported(dtype, dk, dv), "gated_delta_scan_recur: needs 16-bit, dk = dv = 128");
  ATMA_REQUIRE(scratch != nullptr && B > 0 && T > 0 && H > 0, "gated_delta_scan_recur: bad arguments");
  return gated_delta_scan_mma_recur(nullptr, nullptr, nullptr, H, scratch, dtype, B, T, H, n_rec, rec_of, zero_u0, initial_state, o, final_state,
                                    (cudaStream_t)stream);
}

extern "C" int atma_gated_delta_scan_recur_rows(const void* q, const void* k, const void* v, int Hkv, void* scratch, int dtype, int B, int T,
                                                int H, int dk, int dv, int n_rec, const int* rec_of, const int* zero_u0,
                                                const float* initial_state, void* o, float* final_state, void* stream) {
  ATMA_REQUIRE(gated_delta_scan_mma_supported(dtype, dk, dv), "gated_delta_scan_recur_rows: needs 16-bit, dk = dv = 128");
  ATMA_REQUIRE(scratch != nullptr && B > 0 && T > 0 && H > 0 && Hkv > 0 && H % Hkv == 0, "gated_delta_scan_recur_rows: bad arguments");
  ATMA_REQUIRE(q != nullptr && k != nullptr && v != nullptr && (uintptr_t)q % 16 == 0 && (uintptr_t)k % 16 == 0 && (uintptr_t)v % 16 == 0,
               "gated_delta_scan_recur_rows: q, k and v must be 16-byte aligned");
  return gated_delta_scan_mma_recur(q, k, v, Hkv, scratch, dtype, B, T, H, n_rec, rec_of, zero_u0, initial_state, o, final_state,
                                    (cudaStream_t)stream);
}

extern "C" int64_t atma_gated_delta_scan_varlen_scratch_bytes(int64_t total_tokens, int n_seqs, int H, int dk, int dv) {
  if (!gated_delta_scan_mma_supported(ATMA_BF16, dk, dv) || total_tokens < 0 || n_seqs < 0) return 0;
  return gated_delta_scan_mma_varlen_scratch_bytes(total_tokens, n_seqs, H);
}

static int scan_varlen_impl(const void* q, const void* k, const void* v, int dtype, const float* g,
                                            const float* beta, const int32_t* cu_seqlens, int n_seqs,
                                            int64_t total_tokens, const float* initial_state, float* final_state,
                                            float* state_table, int64_t slot_stride, const int64_t* slots,
                                            const int32_t* has_initial, void* o, void* scratch, int H, int Hkv, int dk,
                                            int dv, int normalize_qk, float scale, float* snapshots,
                                            const int32_t* snap_offsets, int snap_every_tokens, void* stream) {
  ATMA_REQUIRE(gated_delta_scan_mma_supported(dtype, dk, dv),
               "gated_delta_scan_varlen: needs 16-bit inputs with dk = dv = 128 (got dtype %d, dk %d, dv %d)", dtype, dk, dv);
  ATMA_REQUIRE(n_seqs >= 0 && total_tokens >= 0 && H > 0 && Hkv > 0 && H % Hkv == 0, "gated_delta_scan_varlen: bad shape");
  ATMA_REQUIRE(total_tokens / kScanC + n_seqs < (1 << 30), "gated_delta_scan_varlen: too many chunks");
  ATMA_REQUIRE(n_seqs <= 65535, "gated_delta_scan_varlen: at most 65535 sequences per call (got %d)", n_seqs);
  ATMA_REQUIRE(snapshots == nullptr || (snap_offsets != nullptr && snap_every_tokens > 0 && snap_every_tokens % kScanC == 0),
               "gated_delta_scan_varlen: snapshots need offsets and a spacing that is a multiple of %d tokens", kScanC);
  if (n_seqs == 0) return ATMA_OK;
  ATMA_REQUIRE(cu_seqlens != nullptr, "gated_delta_scan_varlen: cu_seqlens is required");
  ATMA_REQUIRE(state_table == nullptr || slots != nullptr, "gated_delta_scan_varlen: a state table needs slots");
  ATMA_REQUIRE(state_table == nullptr || (initial_state == nullptr && final_state == nullptr),
               "gated_delta_scan_varlen: pass either a slot-indexed state table or dense state arrays, not both");
  ATMA_REQUIRE(scratch != nullptr && (uintptr_t)scratch % 256 == 0 && (uintptr_t)q % 16 == 0 && (uintptr_t)k % 16 == 0 &&
                   (uintptr_t)v % 16 == 0, "gated_delta_scan_varlen: scratch must be 256-byte and inputs 16-byte aligned");
  return gated_delta_scan_mma_varlen(q, k, v, dtype, g, beta, cu_seqlens, n_seqs, total_tokens, initial_state, final_state,
                                     state_table, slot_stride, slots, has_initial, o, scratch, H, Hkv, normalize_qk, scale,
                                     snapshots, snap_offsets, snapshots ? snap_every_tokens / kScanC : 0, (cudaStream_t)stream);
}

extern "C" int atma_gated_delta_scan_varlen(const void* q, const void* k, const void* v, int dtype, const float* g,
                                            const float* beta, const int32_t* cu_seqlens, int n_seqs,
                                            int64_t total_tokens, const float* initial_state, float* final_state,
                                            float* state_table, int64_t slot_stride, const int64_t* slots,
                                            const int32_t* has_initial, void* o, void* scratch, int H, int Hkv, int dk,
                                            int dv, int normalize_qk, float scale, void* stream) {
  return scan_varlen_impl(q, k, v, dtype, g, beta, cu_seqlens, n_seqs, total_tokens, initial_state, final_state, state_table,
                          slot_stride, slots, has_initial, o, scratch, H, Hkv, dk, dv, normalize_qk, scale, nullptr, nullptr, 0,
                          stream);
}

extern "C" int atma_gated_delta_scan_varlen_snapshots(const void* q, const void* k, const void* v, int dtype, const float* g,
                                                      const float* beta, const int32_t* cu_seqlens, int n_seqs,
                                                      int64_t total_tokens, float* state_table, int64_t slot_stride,
                                                      const int64_t* slots, const int32_t* has_initial, void* o,
                                                      void* scratch, int H, int Hkv, int dk, int dv, int normalize_qk,
                                                      float scale, float* snapshots, const int32_t* snap_offsets,
                                                      int snap_every_tokens, void* stream) {
  ATMA_REQUIRE(snapshots != nullptr, "gated_delta_scan_varlen_snapshots: the snapshot buffer is required");
  return scan_varlen_impl(q, k, v, dtype, g, beta, cu_seqlens, n_seqs, total_tokens, nullptr, nullptr, state_table, slot_stride,
                          slots, has_initial, o, scratch, H, Hkv, dk, dv, normalize_qk, scale, snapshots, snap_offsets,
                          snap_every_tokens, stream);
}

extern "C" int64_t atma_gated_delta_scan_scratch_bytes(int B, int T, int H, int dk, int dv) {
  const int64_t fp32_path = delta_blocks_scratch_bytes((int64_t)B * T, B, H, dk, dv);
  const int64_t mma_path = gated_delta_scan_mma_scratch_bytes(B, T, H);
  return fp32_path > mma_path ? fp32_path : mma_path;
}

extern "C" int atma_gated_delta_scan(const void* q, const void* k, const void* v, int dtype,
                                     const float* g, const float* beta, const float* initial_state,
                                     void* o, float* final_state, void* scratch, int B, int T, int H,
                                     int Hkv, int dk, int dv, int normalize_qk, float scale,
                                     void* stream) {
  return atma_gated_delta_scan_segmented(q, k, v, dtype, g, beta, initial_state, o, final_state, scratch, B, T, H, Hkv, dk, dv,
                                         normalize_qk, scale, 0, stream);
}

extern "C" int atma_gated_delta_scan_segmented(const void* q, const void* k, const void* v, int dtype,
                                               const float* g, const float* beta, const float* initial_state,
                                               void* o, float* final_state, void* scratch, int B, int T, int H,
                                               int Hkv, int dk, int dv, int normalize_qk, float scale,
                                               int segments, void* stream) {
  ATMA_REQUIRE(segments >= 0 && segments <= 16, "gated_delta_scan: segments=%d outside 0..16", segments);
  ATMA_REQUIRE(dtype_ok(dtype), "gated_delta_scan: unsupported dtype %d", dtype);
  ATMA_REQUIRE(dk >= 1 && dk <= 128 && dv >= 1 && dv <= 128, "gated_delta_scan: dk=%d dv=%d outside 1..128", dk, dv);
  ATMA_REQUIRE(B >= 0 && T >= 0 && H > 0, "gated_delta_scan: bad shape");
  ATMA_REQUIRE(Hkv > 0 && H % Hkv == 0, "gated_delta_scan: H=%d is not a multiple of Hkv=%d", H, Hkv);
  ATMA_REQUIRE(scratch != nullptr || B * T == 0, "gated_delta_scan: scratch is required");
  cudaStream_t st = (cudaStream_t)stream;
  if (B == 0) return ATMA_OK;
  if (T == 0) {                                     // nothing to scan: the state passes through
    if (final_state && initial_state)
      ATMA_CUDA_OK(cudaMemcpyAsync(final_state, initial_state, sizeof(float) * (size_t)B * H * dk * dv,
                                   cudaMemcpyDeviceToDevice, st));
    else if (final_state)
      ATMA_CUDA_OK(cudaMemsetAsync(final_state, 0, sizeof(float) * (size_t)B * H * dk * dv, st));
    return ATMA_OK;
  }
  if (gated_delta_scan_mma_supported(dtype, dk, dv) && ((uintptr_t)q % 16 == 0) && ((uintptr_t)k % 16 == 0) &&
      ((uintptr_t)v % 16 == 0) && ((uintptr_t)scratch % 256 == 0))
    return gated_delta_scan_mma(q, k, v, dtype, g, beta, initial_state, o, final_state, scratch, B, T, H, Hkv,
                                normalize_qk, scale, segments, st);
  ATMA_REQUIRE(delta_blocks_supported((int64_t)B * T, B, H, dk), "gated_delta_scan: grid limits");
  DeltaBlocks a{};
  a.q = q; a.k = k; a.v = v; a.o = o;
  a.normalize = normalize_qk; a.q_scale = scale;
  a.log_decay = g; a.beta = beta;
  a.state_in = initial_state; a.state_out = final_state; a.state_ss = (int64_t)H * dk * dv;
  a.n_seqs = B; a.len = T; a.total_rows = (int64_t)B * T;
  a.H = H; a.Hq = H; a.G = Hkv; a.Hv = Hkv; a.dk = dk; a.dv = dv; a.dtype = dtype;
  return delta_blocks_scan(a, scratch, st);
}
