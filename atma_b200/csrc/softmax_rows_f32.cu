// Causal softmax attention of fp32 prompts over a paged cache: on the tensor cores (attend_tf32.cuh) where there are rows enough,
// else in fp32 arithmetic, 64 rows x 64 keys per step.  One or two maps,
// windows, a sink, the differential combination and the output gate as in softmax_rows_kernel, which keeps the other types
// and sizes and short steps.
//
// There a lane owns one key and a warp two rows: two loads from shared memory for two FMAs.  Here a thread owns 4 x 4 scores
// and 4 rows x 4 VM channels (rows_f32.cuh), so that FMAs and shared memory are both busy; K and V take turns in one buffer,
// V under the statistics, and two CTAs share an SM, one loading while the other computes.  Later rows have more keys, so
// those of all heads come first.  Measured, 1500 rows, 8 heads, two maps of 64, 128 value channels: 1089 -> 534 us (679 with
// the heads one after another).
#include "attend_tf32.cuh"
#include "rows_f32.cuh"
#include "softmax_attention.cuh"

namespace atma {

namespace {

using namespace rows_f32;

// rows q0 .. q0 + 63 of a sequence's head
template <int M, int VM, int kOf>
__device__ __forceinline__ void softmax_block(const atma_softmax_args& a, int s, int h, int q0, float* sm) {
  const int kd = M * a.dim, ld = kd + kPad;
  float* sQ = sm;                              // [64][ld]
  float* sKV = sQ + kM * ld;                   // K [64][ld], then V [64][64 VM]
  float* sP = sKV + kN * max(ld, 64 * VM);     // [M][64][kLdP]
  const int tid = threadIdx.x & (kThreads - 1), lane = tid & 31, warp = tid >> 5, tx = lane & 15, ty = 2 * warp + (lane >> 4);
  const int r_begin = a.cu_rows[s], n_rows = a.cu_rows[s + 1] - r_begin, start = a.start_pos[s], g = h / (a.H / a.G);
  float* out = static_cast<float*>(a.out);
  if (start < 0) {                             // padded sequence
    for (int i = tid; i < min(kM, n_rows - q0) * a.vdim; i += kThreads)
      out[(int64_t)(r_begin + q0 + i / a.vdim) * a.out_rs + (int64_t)h * a.vdim + i % a.vdim] = 0.f;
    return;
  }
  const float* Q = static_cast<const float*>(a.q);
  const float* K = static_cast<const float*>(a.k_cache);
  const float* V = static_cast<const float*>(a.v_cache);
  for (int i = tid; i < kM * (kd / 4); i += kThreads) {
    const int r = i / (kd / 4), c = 4 * (i - r * (kd / 4));
    float4 x = {0.f, 0.f, 0.f, 0.f};
    if (q0 + r < n_rows) x = *reinterpret_cast<const float4*>(Q + ((int64_t)(r_begin + q0 + r) * a.H + h) * kd + c);
    *reinterpret_cast<float4*>(sQ + r * ld + c) = make_float4(x.x * a.scale, x.y * a.scale, x.z * a.scale, x.w * a.scale);
  }
  const int last_pos = start + min(q0 + kM, n_rows) - 1;      // the last row's own position
  const int n_keys = min(last_pos + 1, a.max_blocks * a.block_size);
  const KeyTiles tiles(start + q0, last_pos, a.max_blocks * a.block_size, a.window, a.keep_first, kN);
  const int32_t* bt = a.block_tables + s * a.bt_stride;
  const int first_pos = start + q0 + 8 * warp;                // of this warp's eight rows

  float m[4][M], l[4][M];
  uint64_t acc[M][4][2 * VM];
#pragma unroll
  for (int t = 0; t < M; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      m[i][t] = a.sink;                        // the sink is a key that was seen before the others
      l[i][t] = a.sink > -INFINITY ? 1.f : 0.f;
#pragma unroll
      for (int c = 0; c < 2 * VM; ++c) acc[t][i][c] = 0;
    }

  for (int kt = 0; kt < tiles.n; ++kt) {
    const int k0 = tiles[kt] * kN;
    auto fetch = [&](const float* cache, int width, int row_len, int dst_ld) {      // the tile's rows of one cache, zeros behind them
      const int per_row = row_len / 4;
      for (int i = tid; i < kN * per_row; i += kThreads) {
        const int j = i / per_row, c = 4 * (i - j * per_row), pos = k0 + j;
        const float* src = cache;
        const bool there = pos < n_keys && c < width;
        if (there) {
          const int blk = pos / a.block_size;
          const int phys = min(max(bt[blk], 0), a.num_blocks - 1);
          src = cache + (((int64_t)phys * a.block_size + (pos - blk * a.block_size)) * a.G + g) * width + c;
        }
        copy16(sKV + j * dst_ld + c, src, there);
      }
    };
    block_sync<kOf>();                           // the last tile's V is read
    fetch(K, kd, kd, ld);
    copies_done<kOf>();
    // columns that some of the warp's rows see (j0 to j1 - 1) and those that all of them do (f0 to f1 - 1)
    const int kept = a.keep_first - k0, opens = first_pos - a.window + 1 - k0;
    int j1 = min(min(kN, n_keys - k0), first_pos + 8 - k0);
    if (kept > 0 && opens >= kN) j1 = min(j1, kept);
    const int j0 = kept > 0 ? 0 : max(opens, 0) & ~3, f1 = min(j1, first_pos + 1 - k0), f0 = kept >= f1 ? 0 : (opens + 7 + 3) & ~3;
    auto sees = [&](int i, int j) { return key_visible(start + q0 + 4 * ty + i, k0 + j, a.window, a.keep_first); };
#pragma unroll
    for (int t = 0; t < M; ++t) {
      float sc[4][4];
      dots<M == 1>(sQ + t * a.dim, sKV + t * a.dim, ld, a.dim / 4, ty, tx, sc);
      if (t == M - 1) {
        block_sync<kOf>();                       // K is read
        fetch(V, a.vdim, 64 * VM, 64 * VM);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int pos = start + q0 + 4 * ty + i;
        float top = -INFINITY;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = k0 + tx + 16 * j;
          sc[i][j] = key < n_keys && key_visible(pos, key, a.window, a.keep_first) ? sc[i][j] : -INFINITY;
          top = fmaxf(top, sc[i][j]);
        }
        const float mn = fmaxf(m[i][t], row_max(top));
        const float al = mn == -INFINITY ? 1.f : expf(m[i][t] - mn);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float p = mn == -INFINITY ? 0.f : expf(sc[i][j] - mn);
          sP[(t * kM + 4 * ty + i) * kLdP + tx + 16 * j] = p;
          sum += p;
        }
        l[i][t] = l[i][t] * al + row_sum(sum);
        m[i][t] = mn;
        times<VM>(acc[t][i], al);
      }
    }
    copies_done<kOf>();
#pragma unroll
    for (int t = 0; t < M; ++t) weigh<VM>(sP + t * kM * kLdP, sKV, ty, tx, j0, j1, f0, f1, sees, acc[t]);
  }

  const bool vec = a.out_rs % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = q0 + 4 * ty + i;
    float o[4 * VM], ss = 0.f;
#pragma unroll
    for (int c = 0; c < 4 * VM; ++c) {
      o[c] = l[i][0] > 0.f ? at<VM>(acc[0][i], c) / l[i][0] : 0.f;
      if constexpr (M == 2) o[c] -= l[i][M - 1] > 0.f ? a.lambda * (at<VM>(acc[M - 1][i], c) / l[i][M - 1]) : 0.f;
      ss = fmaf(o[c], o[c], ss);               // channels behind vdim are zero
    }
    float f = 1.f;
    if constexpr (M == 2) f = a.out_scale / sqrtf(row_sum(ss) / (float)a.vdim + a.eps);
    if (row < n_rows) {
      float* op = out + (int64_t)(r_begin + row) * a.out_rs + (int64_t)h * a.vdim;
      const float* gp = a.gate == nullptr ? nullptr : static_cast<const float*>(a.gate) + (int64_t)(r_begin + row) * a.gate_rs + (int64_t)h * a.vdim;
#pragma unroll
      for (int c = 0; c < VM; ++c) {
        const int at0 = 64 * c + 4 * tx;
        if (at0 >= a.vdim) continue;
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = o[4 * c + e] * f * (gp != nullptr ? sigmoid_gate(gp[at0 + e]) : 1.f);
        if (vec) *reinterpret_cast<float4*>(op + at0) = make_float4(y[0], y[1], y[2], y[3]);
        else
#pragma unroll
          for (int e = 0; e < 4; ++e) op[at0 + e] = y[e];
      }
    }
  }
}

template <int M, int VM>
__global__ void __launch_bounds__(kThreads, 2)
softmax_rows_f32_kernel(const atma_softmax_args a, int marked) {
  extern __shared__ __align__(16) float sm[];
  const int s = blockIdx.y, h = blockIdx.x % a.H, q0 = ((int)(gridDim.x - blockIdx.x) - 1) / a.H * kM;
  if (q0 >= a.cu_rows[s + 1] - a.cu_rows[s]) return;
  // behind the tensor-core kernel: only the blocks that it has marked
  if (marked && __float_as_uint(static_cast<const float*>(a.out)[(int64_t)(a.cu_rows[s] + q0) * a.out_rs + (int64_t)h * a.vdim]) != attend_tf32::kRedo) return;
  softmax_block<M, VM, 1>(a, s, h, q0, sm);
}

// ---- the same on the tensor cores, 128 rows of a head per CTA: 128 channels of q and k in all, 128 of v ------------------
__device__ int g_softmax_tf32_status = 0;

// a block of the tensor-core kernel's CTA, `at` bytes into its shared memory (a pointer would not be known to be shared); a function of
// its own, so that it takes none of that kernel's registers
template <int M>
__device__ __noinline__ void softmax_half_block(const atma_softmax_args& a, int s, int h, int q0, int at) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  softmax_block<M, 2, 2>(a, s, h, q0, reinterpret_cast<float*>(smem_raw + at));
}

template <int M>
struct SoftmaxFront {
  struct Row {
    int pos, n_keys, window, keep;
    float sink;
    __device__ __forceinline__ float score(float s) const { return s; }
    __device__ __forceinline__ bool sees(int key) const { return (key < n_keys) & (key <= pos) & ((pos - key < window) | (key < keep)); }
    __device__ __forceinline__ bool sees_all(int first, int last) const { return (last < n_keys) & (last <= pos) & ((pos - first < window) | (last < keep)); }
    __device__ __forceinline__ float start(int) const { return sink; }      // the sink is a key that was seen before the others
    __device__ __forceinline__ float start_sum(int) const { return sink > -INFINITY ? 1.f : 0.f; }
  };
  const atma_softmax_args& a;
  int s, h, g, q0, r_begin, n_rows, first, n_keys;
  KeyTiles kt;

  __device__ __forceinline__ SoftmaxFront(const atma_softmax_args& args, int seq, int head, int row0, int begin, int rows, int start)
      : a(args), s(seq), h(head), g(head / (args.H / args.G)), q0(row0), r_begin(begin), n_rows(rows), first(start + row0),
        n_keys(min(start + min(row0 + attend_tf32::kM, rows), args.max_blocks * args.block_size)),
        kt(start + row0, start + min(row0 + attend_tf32::kM, rows) - 1, args.max_blocks * args.block_size, args.window, args.keep_first, kN) {}
  __device__ __forceinline__ int tiles() const { return kt.n; }
  __device__ __forceinline__ int key0(int j) const { return kt[j] * kN; }
  __device__ __forceinline__ float q_scale() const { return a.scale; }
  __device__ __forceinline__ bool has(int r) const { return q0 + r < n_rows; }
  __device__ __forceinline__ bool few(int r) const {
    const int last = min(first + r + 1, n_keys), opens = first + r + 1 - a.window;      // keys [opens, last) and those that are kept
    const int seen = opens > 0 ? max(last - opens, 0) + min(max(a.keep_first, 0), opens) : last;
    return has(r) && seen > 0 && seen < attend_tf32::few_keys(M);
  }
  __device__ __forceinline__ float* result(int r) const {
    return static_cast<float*>(a.out) + (int64_t)(r_begin + q0 + r) * a.out_rs + (int64_t)h * attend_tf32::kD;
  }
  __device__ __forceinline__ void mark(int block) const { if (has(64 * block)) *result(64 * block) = __uint_as_float(attend_tf32::kRedo); }
  // blocks of few keys in fp32 arithmetic, half of the CTA's threads each
  __device__ __forceinline__ void plain() const {
    constexpr int kBytes = 4 * (kM * (attend_tf32::kD + kPad) + kN * (attend_tf32::kD + kPad) + M * kM * kLdP);
    static_assert(M == 2 || 2 * kBytes <= attend_tf32::kSmemBytes, "two blocks fit");
    const int block = threadIdx.x >> 8;
    if (has(64 * block)) softmax_half_block<M>(a, s, h, q0 + 64 * block, block * kBytes);
  }
  __device__ __forceinline__ const float* any() const { return static_cast<const float*>(a.q); }
  __device__ __forceinline__ const float* q_row(int r) const {
    return q0 + r < n_rows ? static_cast<const float*>(a.q) + ((int64_t)(r_begin + q0 + r) * a.H + h) * attend_tf32::kD : nullptr;
  }
  __device__ __forceinline__ const float* cached(const void* cache, int pos) const {
    if (pos >= n_keys) return nullptr;
    const int blk = pos / a.block_size, phys = min(max(a.block_tables[s * a.bt_stride + blk], 0), a.num_blocks - 1);
    return static_cast<const float*>(cache) + (((int64_t)phys * a.block_size + (pos - blk * a.block_size)) * a.G + g) * attend_tf32::kD;
  }
  __device__ __forceinline__ const float* k_row(int key) const { return cached(a.k_cache, key); }
  __device__ __forceinline__ const float* v_row(int key) const { return cached(a.v_cache, key); }
  __device__ __forceinline__ Row row(int r) const { return Row{first + r, n_keys, a.window, a.keep_first, a.sink}; }
  __device__ __forceinline__ void finish(const Row&, int r, int half, const float (&)[M], const float (&l)[M], float, float (&O)[M][64],
                                         attend_tf32::Shared& sh) const {
    using namespace attend_tf32;
    const bool ok = q0 + r < n_rows;
#pragma unroll
    for (int t = 0; t < M; ++t) {
      sh.sum[half][t][r] = l[t];
      if (ok && !trusted(O[t], l[t])) sh.redo[r >> 6] = 1;
    }
    rows_sync();
    float L[M], ss = 0.f;
#pragma unroll
    for (int t = 0; t < M; ++t) L[t] = l[t] + sh.sum[half ^ 1][t][r];
#pragma unroll
    for (int c = 0; c < 64; ++c) {
      O[0][c] = L[0] > 0.f ? O[0][c] / L[0] : 0.f;
      if constexpr (M == 2) O[0][c] -= L[M - 1] > 0.f ? a.lambda * (O[M - 1][c] / L[M - 1]) : 0.f;
      ss = fmaf(O[0][c], O[0][c], ss);
    }
    sh.sum[half][2][r] = ss;
    rows_sync();
    if (!ok) return;
    float* op = result(r) + 64 * half;
    if (sh.redo[r >> 6]) {
      if (half == 0 && (r & 63) == 0) mark(r >> 6);
      return;
    }
    float f = 1.f;
    if constexpr (M == 2) f = a.out_scale / sqrtf((ss + sh.sum[half ^ 1][2][r]) / (float)kD + a.eps);
    const float* gp = a.gate == nullptr ? nullptr : static_cast<const float*>(a.gate) + (int64_t)(r_begin + q0 + r) * a.gate_rs + (int64_t)h * kD + 64 * half;
    const bool vec = (reinterpret_cast<uintptr_t>(op) & 15) == 0;
#pragma unroll
    for (int c = 0; c < 64; c += 4) {
      float y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = O[0][c + e] * f * (gp != nullptr ? sigmoid_gate(gp[c + e]) : 1.f);
      if (vec) *reinterpret_cast<float4*>(op + c) = make_float4(y[0], y[1], y[2], y[3]);
      else
#pragma unroll
        for (int e = 0; e < 4; ++e) op[c + e] = y[e];
    }
  }
};

template <int M>
__global__ void __launch_bounds__(attend_tf32::kThreads, 1)
softmax_tf32_kernel(const __grid_constant__ atma_softmax_args a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ attend_tf32::Shared sh;
  const int s = blockIdx.y, h = blockIdx.x % a.H;
  const int r_begin = a.cu_rows[s], n_rows = a.cu_rows[s + 1] - r_begin, start = a.start_pos[s];
  const int q0 = attend_tf32::first_row<M>(a.H);
  if (q0 >= n_rows) return;
  if (start < 0) {                             // padded sequence
    float* out = static_cast<float*>(a.out);
    for (int i = threadIdx.x; i < min(attend_tf32::kM, n_rows - q0) * attend_tf32::kD; i += attend_tf32::kThreads)
      out[(int64_t)(r_begin + q0 + i / attend_tf32::kD) * a.out_rs + (int64_t)h * attend_tf32::kD + i % attend_tf32::kD] = 0.f;
    return;
  }
  SoftmaxFront<M> front(a, s, h, q0, r_begin, n_rows, start);
  attend_tf32::attend<SoftmaxFront<M>, M>(front, smem, sh, &g_softmax_tf32_status);
}

// 128 channels in one map or two, 128 of v, and enough rows.  Two maps, 8 heads, the call's own launches counted: 1500 rows 547 us on
// the 64 x 64 kernel, 173 here; 400 rows 156 and 83; 256 rows 104 and 73.  One map: 363 and 130, 106 and 80, 72 and 77.  Results that take the place of q or the gate: the mark would be in
// the rows that are read again.  Short windows: with one map every block would be left to the 64 x 64 kernel (few_keys); with two that is
// faster while its CTAs have an SM each (a window of 8, 400 rows 59 us against 69, 1500 rows 76 against 73; of 64, 66 and 69, 86 and 71).
bool softmax_tf32_supported(const atma_softmax_args& a) {
  const int64_t ctas = (int64_t)(a.max_rows + kM - 1) / kM * a.H * a.n_seqs, seen = (int64_t)a.window + (a.keep_first > 0 ? a.keep_first : 0);
  if (seen < attend_tf32::few_keys(1) && (a.maps == 1 || ctas <= sm_count_of_current_device())) return false;
  return a.maps * a.dim == attend_tf32::kD && a.vdim == attend_tf32::kD && a.max_rows >= (a.maps == 1 ? 257 : 256) && a.out != a.q && a.out != a.gate;
}

template <int M>
int launch_tf32(const atma_softmax_args& a, cudaStream_t st) {
  ATMA_CUDA_OK(cudaFuncSetAttribute(softmax_tf32_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, attend_tf32::kSmemBytes));
  softmax_tf32_kernel<M><<<dim3((a.max_rows + attend_tf32::kM - 1) / attend_tf32::kM * a.H, a.n_seqs), attend_tf32::kThreads, attend_tf32::kSmemBytes, st>>>(a);
  return launch_status("softmax attention (fp32, tensor cores)");
}

int smem_bytes(const atma_softmax_args& a) {
  const int ld = a.maps * a.dim + kPad, vm = a.vdim <= 64 ? 64 : 128;
  return 4 * (kM * ld + kN * (ld > vm ? ld : vm) + a.maps * kM * kLdP);
}

template <int M, int VM>
int launch(const atma_softmax_args& a, cudaStream_t st) {
  const int smem = smem_bytes(a);
  const bool tf32 = softmax_tf32_supported(a);
  if (tf32) {
    const int rc = launch_tf32<M>(a, st);
    if (rc != ATMA_OK) return rc;
  }
  ATMA_CUDA_OK(cudaFuncSetAttribute(softmax_rows_f32_kernel<M, VM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  softmax_rows_f32_kernel<M, VM><<<dim3((a.max_rows + kM - 1) / kM * a.H, a.n_seqs), kThreads, smem, st>>>(a, tf32);
  return launch_status("softmax attention (fp32, 64 x 64)");
}

}  // namespace

// Rows in quadruples of channels, sizes that leave room for two CTAs, and more rows than two CTAs of the other kernel hold.  With
// two maps and one page of keys at most, the other kernel's four times as many CTAs are faster while this one's leave most SMs
// without any (8 heads, one prompt: 33 rows 23 us against 28, 128 rows 48 against 51; with 8000 keys in front 3470 against 2516).
bool softmax_rows_f32_supported(const atma_softmax_args& a) {
  const int64_t ctas = (int64_t)(a.max_rows + kM - 1) / kM * a.H * a.n_seqs;
  if (a.maps == 2 && a.max_rows <= 128 && (int64_t)a.max_blocks * a.block_size <= 256 && 8 * ctas <= sm_count_of_current_device()) return false;
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return a.dtype == ATMA_F32 && a.max_rows > 32 && a.dim % 4 == 0 && a.vdim % 4 == 0 && a.maps * a.dim <= 128 && a.vdim <= 128 && al(a.q) &&
         al(a.k_cache) && al(a.v_cache);
}

int softmax_tf32_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  ATMA_CUDA_OK(cudaMemcpyFromSymbol(&v, g_softmax_tf32_status, sizeof(int)));
  if (v != 0) ATMA_CUDA_OK(cudaMemcpyToSymbol(g_softmax_tf32_status, &zero, sizeof(int)));
  *out = v;
  return ATMA_OK;
}

int softmax_rows_f32(const atma_softmax_args& a, cudaStream_t st) {
  if (a.maps == 1) return a.vdim <= 64 ? launch<1, 1>(a, st) : launch<1, 2>(a, st);
  return a.vdim <= 64 ? launch<2, 1>(a, st) : launch<2, 2>(a, st);
}

}  // namespace atma
