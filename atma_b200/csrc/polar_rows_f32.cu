// Polar Attention prefill of fp32 tensors with a head size of 64 or 128: on the tensor cores (attend_tf32.cuh) where there are
// rows enough, else in fp32 arithmetic, 64 rows x 64 keys per step, with the same results as polar_prefill_simt_kernel, which
// keeps the other types and sizes.
//
// There a lane owns one key and a warp four rows, with a shuffle for every weight; here a thread owns 4 x 4 scores and
// 4 rows x DK / 16 channels (rows_f32.cuh).  K and V take turns in one buffer, V under the statistics, and two CTAs share an
// SM; later rows have more keys, so those of all heads come first.  Measured, 2048 rows, 8 heads of 128: 1049 -> 423 us (527
// with the heads one after another and the scores one channel at a time).
#include "attend_tf32.cuh"
#include "polar_prefill.cuh"
#include "rows_f32.cuh"

namespace atma {

namespace {

using namespace rows_f32;
constexpr float kNegBig = -1e38f;

template <int DK> constexpr int kBlockBytes = 4 * (kM * (DK + kPad) + kN * (DK + kPad) + kM * kLdP);

// rows q0 .. q0 + 63 of a head
template <int DK, int kOf>
__device__ __forceinline__ void polar_block(const atma_polar_prefill_args& a, int h, int b, int q0, float* sm, float (*s_n)[2]) {
  constexpr int VM = DK / 64, ld = DK + kPad;
  float* sQ = sm;                              // [64][ld]
  float* sKV = sQ + kM * ld;                   // K [64][ld], then V [64][DK]
  float* sP = sKV + kN * ld;                   // [64][kLdP]
  const int tid = threadIdx.x & (kThreads - 1), lane = tid & 31, warp = tid >> 5, tx = lane & 15, ty = 2 * warp + (lane >> 4);
  const int kvh = h / (a.H / a.Hkv), q_limit = a.Tq, k_limit = a.Tk;
  const float* Q = static_cast<const float*>(a.q) + b * a.q_sb + h * a.q_sh;
  const float* K = static_cast<const float*>(a.k) + b * a.k_sb + kvh * a.k_sh;
  const float* V = static_cast<const float*>(a.v) + b * a.v_sb + kvh * a.v_sh;
  for (int i = tid; i < kM * (DK / 4); i += kThreads) {
    const int r = i / (DK / 4), c = 4 * (i - r * (DK / 4));
    const bool there = q0 + r < q_limit;
    copy16(sQ + r * ld + c, there ? Q + (int64_t)(q0 + r) * a.q_st + c : Q, there);
  }

  float n[4], temp[4], m[4], L[4], Q2[4];
  uint64_t acc[4][2 * VM];
  float lo = 3.0e38f, hi = -1.0f;              // key counts of this warp's rows
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = q0 + 4 * ty + i;
    const bool ok = r < q_limit;
    n[i] = !ok ? 0.f : (a.n_keys ? a.n_keys[r] : a.n_base + (float)(r + 1));
    const float nc = fmaxf(a.window > 0 ? fminf(n[i], (float)a.window) : n[i], 1.0f);
    temp[i] = 1.0f + a.spg[h] * logf(nc);
    if (ok) { lo = fminf(lo, n[i]); hi = fmaxf(hi, n[i]); }
    m[i] = kNegBig; L[i] = 0.f; Q2[i] = 0.f;
#pragma unroll
    for (int c = 0; c < 2 * VM; ++c) acc[i][c] = 0;
    if (a.stats_in_m != nullptr && ok) {
      const int64_t row = ((int64_t)b * a.H + h) * a.Tq + r;
      m[i] = a.stats_in_m[row]; L[i] = a.stats_in_l[row]; Q2[i] = a.stats_in_q2[row];
#pragma unroll
      for (int c = 0; c < VM; ++c) {
        const float* p = a.stats_in_s + row * DK + 64 * c + 4 * tx;
        acc[i][2 * c] = pack2(p[0], p[1]);
        acc[i][2 * c + 1] = pack2(p[2], p[3]);
      }
    }
  }
  const float inv_sqrt_dk = rsqrtf((float)DK);
  lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, 16));
  hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, 16));
  if (lane == 0) { s_n[warp][0] = lo; s_n[warp][1] = hi; }
  block_sync<kOf>();
  float all_lo = lo, all_hi = hi;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) { all_lo = fminf(all_lo, s_n[w][0]); all_hi = fmaxf(all_hi, s_n[w][1]); }

  // ---- key tiles that some row sees ----
  const float koff = (float)a.key_offset;
  const int j_end = max((int)fminf((float)k_limit, ceilf(all_hi - koff)), 0);
  int j_begin = 0;
  if (a.window > 0) {
    const float first = all_lo - (float)a.window - koff;
    if (first > 0.f) j_begin = (int)fminf(first, (float)k_limit) / kN * kN;
  }
  for (int k0 = j_begin; k0 < j_end; k0 += kN) {
    auto fetch = [&](const float* src, int64_t stride, int dst_ld) {
      for (int i = tid; i < kN * (DK / 4); i += kThreads) {
        const int j = i / (DK / 4), c = 4 * (i - j * (DK / 4));
        const bool there = k0 + j < k_limit;
        copy16(sKV + j * dst_ld + c, there ? src + (int64_t)(k0 + j) * stride + c : src, there);
      }
    };
    block_sync<kOf>();                           // the last tile's V is read
    fetch(K, a.k_st, ld);
    copies_done<kOf>();
    float sc[4][4];
    dots<true>(sQ, sKV, ld, DK / 4, ty, tx, sc);
    block_sync<kOf>();
    fetch(V, a.v_st, DK);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float f = temp[i] * inv_sqrt_dk;
      float top = kNegBig;
      bool valid[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = k0 + tx + 16 * j;
        const float pos = (float)key + koff;
        valid[j] = key < k_limit && pos < n[i] && (a.window <= 0 || pos >= n[i] - (float)a.window);
        sc[i][j] = valid[j] ? sc[i][j] * f : kNegBig;
        top = fmaxf(top, sc[i][j]);
      }
      const float mn = fmaxf(m[i], row_max(top));
      const float al = expf(m[i] - mn);
      float sum = 0.f, sq = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = valid[j] ? expf(sc[i][j] - mn) : 0.f;
        sP[(4 * ty + i) * kLdP + tx + 16 * j] = p;
        sum += p;
        sq = fmaf(p, p, sq);
      }
      L[i] = L[i] * al + row_sum(sum);
      Q2[i] = Q2[i] * al * al + row_sum(sq);
      m[i] = mn;
      times<VM>(acc[i], al);
    }
    // keys that some of the warp's rows see (j0 to j1 - 1) and those that all of them do (f0 to f1 - 1)
    auto within = [&](float key) { return (int)fminf(fmaxf(key - koff - (float)k0, 0.f), (float)kN); };
    const int j1 = min(min(kN, k_limit - k0), within(ceilf(hi))), f1 = min(j1, within(ceilf(lo)));
    const int j0 = a.window > 0 ? within(lo - (float)a.window) & ~3 : 0, f0 = a.window > 0 ? (within(ceilf(hi) - (float)a.window) + 3) & ~3 : 0;
    auto sees = [&](int i, int j) {
      const float pos = (float)(k0 + j) + koff;
      return pos < n[i] && (a.window <= 0 || pos >= n[i] - (float)a.window);
    };
    copies_done<kOf>();
    weigh<VM>(sP, sKV, ty, tx, j0, j1, f0, f1, sees, acc);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");

  // ---- result ----
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = q0 + 4 * ty + i;
    const bool ok = r < q_limit;
    const int64_t row = ((int64_t)b * a.H + h) * a.Tq + r;
    if (!a.finalize) {
      if (ok) {
        if (tx == 0) { a.stats_out_m[row] = m[i]; a.stats_out_l[row] = L[i]; a.stats_out_q2[row] = Q2[i]; }
#pragma unroll
        for (int c = 0; c < 4 * VM; ++c) a.stats_out_s[row * DK + 64 * (c >> 2) + 4 * tx + (c & 3)] = at<VM>(acc[i], c);
      }
      continue;
    }
    const float nc = fmaxf(a.window > 0 ? fminf(n[i], (float)a.window) : n[i], 1.0f);
    const float a_n = temp[i] * (a.null_base[h] + a.sps[h] * sqrtf(logf(nc + 1.0f)));
    const float mn = fmaxf(m[i], a_n);
    const float al = expf(m[i] - mn);
    const float Lf = L[i] * al, Q2f = Q2[i] * al * al;
    const float p_n = expf(a_n - mn);
    const float Z = Lf + p_n;
    float sv[4 * VM], sq = 0.f;
#pragma unroll
    for (int c = 0; c < 4 * VM; ++c) {
      sv[c] = at<VM>(acc[i], c) * al + p_n * a.v_null[h * DK + 64 * (c >> 2) + 4 * tx + (c & 3)];
      sq = fmaf(sv[c], sv[c], sq);
    }
    const float inv = 1.0f / fmaxf(sqrtf(row_sum(sq)), a.eps);
    if (ok) {
      float* cp = static_cast<float*>(a.c) + b * a.c_sb + h * a.c_sh + (int64_t)r * a.c_st;
#pragma unroll
      for (int c = 0; c < 4 * VM; ++c) cp[64 * (c >> 2) + 4 * tx + (c & 3)] = sv[c] * inv;
      if (tx == 0) {
        const float n_eff = Lf * Lf / fmaxf(Q2f, 1e-30f);
        const float m_eff = n_eff * (Lf / fmaxf(Z, a.eps));
        static_cast<float*>(a.mag)[b * a.mag_sb + h * a.mag_sh + (int64_t)r * a.mag_st] = tanhf(a.beta[h] * log1pf(m_eff));
      }
    }
  }
}

template <int DK>
__global__ void __launch_bounds__(kThreads, 2)
polar_rows_f32_kernel(const atma_polar_prefill_args a, int marked) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float s_n[kThreads / 32][2];
  const int h = blockIdx.x % a.H, b = blockIdx.y, q0 = ((int)(gridDim.x - blockIdx.x) - 1) / a.H * kM;
  // behind the tensor-core kernel: only the blocks that it has marked
  if (marked && __float_as_uint(static_cast<const float*>(a.c)[b * a.c_sb + h * a.c_sh + (int64_t)q0 * a.c_st]) != attend_tf32::kRedo) return;
  polar_block<DK, 1>(a, h, b, q0, sm, s_n);
}

// ---- the same on the tensor cores, 128 rows of a head per CTA ----------------------------------------------------------
// a block of the tensor-core kernel's CTA, `at` bytes into its shared memory (a pointer would not be known to be shared); a function of
// its own, so that it takes none of that kernel's registers
__device__ __noinline__ void polar_half_block(const atma_polar_prefill_args& a, int h, int b, int q0, int at) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ float s_n[2][8][2];
  polar_block<attend_tf32::kD, 2>(a, h, b, q0, reinterpret_cast<float*>(smem_raw + at), s_n[threadIdx.x >> 8]);
}

__device__ int g_polar_tf32_status = 0;

struct PolarFront {
  struct Row {
    float n, f, temp, nc, koff;
    int k_limit, window;
    __device__ __forceinline__ float score(float s) const { return s * f; }
    __device__ __forceinline__ bool sees(int key) const {
      const float pos = (float)key + koff;
      return (key < k_limit) & (pos < n) & ((window <= 0) | (pos >= n - (float)window));
    }
    __device__ __forceinline__ bool sees_all(int first, int last) const { return sees(first) & sees(last); }      // keys that are seen follow one another
    __device__ __forceinline__ float start(int) const { return kNegBig; }
    __device__ __forceinline__ float start_sum(int) const { return 0.f; }
  };
  const atma_polar_prefill_args& a;
  int h, b, kvh, q0, j_begin, j_end;

  __device__ __forceinline__ float count(int r) const {
    return r >= a.Tq ? 0.f : (a.n_keys ? a.n_keys[r] : a.n_base + (float)(r + 1));
  }
  __device__ __forceinline__ PolarFront(const atma_polar_prefill_args& args, float (*s_n)[2]) : a(args) {
    h = blockIdx.x % a.H; b = blockIdx.y; kvh = h / (a.H / a.Hkv);
    q0 = attend_tf32::first_row<1>(a.H);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < 4) {
      const int r = q0 + 32 * warp + lane;
      float lo = r < a.Tq ? count(r) : 3.0e38f, hi = r < a.Tq ? lo : -1.0f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      }
      if (lane == 0) { s_n[warp][0] = lo; s_n[warp][1] = hi; }
    }
    __syncthreads();
    float lo = s_n[0][0], hi = s_n[0][1];
#pragma unroll
    for (int w = 1; w < 4; ++w) { lo = fminf(lo, s_n[w][0]); hi = fmaxf(hi, s_n[w][1]); }
    const float koff = (float)a.key_offset;
    j_end = max((int)fminf((float)a.Tk, ceilf(hi - koff)), 0);
    j_begin = 0;
    if (a.window > 0) {
      const float first = lo - (float)a.window - koff;
      if (first > 0.f) j_begin = (int)fminf(first, (float)a.Tk) / kN * kN;
    }
  }
  __device__ __forceinline__ int tiles() const { return max(j_end - j_begin + kN - 1, 0) / kN; }
  __device__ __forceinline__ int key0(int j) const { return j_begin + j * kN; }
  __device__ __forceinline__ float q_scale() const { return 1.f; }
  __device__ __forceinline__ bool has(int r) const { return q0 + r < a.Tq; }
  __device__ __forceinline__ bool few(int r) const {
    const float n = count(q0 + r), first = fmaxf(a.window > 0 ? n - (float)a.window : 0.f, (float)a.key_offset);
    const float seen = fminf(n, (float)a.key_offset + (float)a.Tk) - first;
    return has(r) && seen > 0.f && seen < (float)attend_tf32::few_keys(1);
  }
  __device__ __forceinline__ float* result(int r) const { return static_cast<float*>(a.c) + b * a.c_sb + h * a.c_sh + (int64_t)(q0 + r) * a.c_st; }
  __device__ __forceinline__ void mark(int block) const { if (has(64 * block)) *result(64 * block) = __uint_as_float(attend_tf32::kRedo); }
  // blocks of few keys in fp32 arithmetic, half of the CTA's threads each
  __device__ __forceinline__ void plain() const {
    static_assert(2 * kBlockBytes<attend_tf32::kD> <= attend_tf32::kSmemBytes, "two blocks fit");
    const int block = threadIdx.x >> 8;
    if (has(64 * block)) polar_half_block(a, h, b, q0 + 64 * block, block * kBlockBytes<attend_tf32::kD>);
  }
  __device__ __forceinline__ const float* any() const { return static_cast<const float*>(a.q); }
  __device__ __forceinline__ const float* q_row(int r) const {
    return q0 + r < a.Tq ? static_cast<const float*>(a.q) + b * a.q_sb + h * a.q_sh + (int64_t)(q0 + r) * a.q_st : nullptr;
  }
  __device__ __forceinline__ const float* k_row(int key) const {
    return key < a.Tk ? static_cast<const float*>(a.k) + b * a.k_sb + kvh * a.k_sh + (int64_t)key * a.k_st : nullptr;
  }
  __device__ __forceinline__ const float* v_row(int key) const {
    return key < a.Tk ? static_cast<const float*>(a.v) + b * a.v_sb + kvh * a.v_sh + (int64_t)key * a.v_st : nullptr;
  }
  __device__ __forceinline__ Row row(int r) const {
    Row w;
    w.n = count(q0 + r);
    w.nc = fmaxf(a.window > 0 ? fminf(w.n, (float)a.window) : w.n, 1.0f);
    w.temp = 1.0f + a.spg[h] * logf(w.nc);
    w.f = w.temp * rsqrtf((float)attend_tf32::kD);
    w.koff = (float)a.key_offset; w.k_limit = a.Tk; w.window = a.window;
    return w;
  }
  __device__ __forceinline__ void finish(const Row& w, int r, int half, const float (&m)[1], const float (&l)[1], float q2, float (&O)[1][64],
                                         attend_tf32::Shared& sh) const {
    using namespace attend_tf32;
    const bool ok = q0 + r < a.Tq;
    sh.sum[half][0][r] = l[0]; sh.sum[half][1][r] = q2;
    if (ok && !trusted(O[0], l[0])) sh.redo[r >> 6] = 1;
    rows_sync();
    const float a_n = w.temp * (a.null_base[h] + a.sps[h] * sqrtf(logf(w.nc + 1.0f)));
    const float mn = fmaxf(m[0], a_n), al = expf(m[0] - mn), p_n = expf(a_n - mn);
    const float Lf = (l[0] + sh.sum[half ^ 1][0][r]) * al, Q2f = (q2 + sh.sum[half ^ 1][1][r]) * al * al, Z = Lf + p_n;
    const float* vn = a.v_null + h * kD + 64 * half;
    float sq = 0.f;
#pragma unroll
    for (int c = 0; c < 64; ++c) {
      O[0][c] = fmaf(O[0][c], al, p_n * vn[c]);
      sq = fmaf(O[0][c], O[0][c], sq);
    }
    sh.sum[half][2][r] = sq;
    rows_sync();
    if (!ok) return;
    float* cp = result(r) + 64 * half;
    if (sh.redo[r >> 6]) {
      if (half == 0 && (r & 63) == 0) mark(r >> 6);
      return;
    }
    const float inv = 1.0f / fmaxf(sqrtf(sq + sh.sum[half ^ 1][2][r]), a.eps);
    if ((reinterpret_cast<uintptr_t>(cp) & 15) == 0) {
#pragma unroll
      for (int c = 0; c < 64; c += 4)
        *reinterpret_cast<float4*>(cp + c) = make_float4(O[0][c] * inv, O[0][c + 1] * inv, O[0][c + 2] * inv, O[0][c + 3] * inv);
    } else {
#pragma unroll
      for (int c = 0; c < 64; ++c) cp[c] = O[0][c] * inv;
    }
    if (half == 0) {
      const float n_eff = Lf * Lf / fmaxf(Q2f, 1e-30f), m_eff = n_eff * (Lf / fmaxf(Z, a.eps));
      static_cast<float*>(a.mag)[b * a.mag_sb + h * a.mag_sh + (int64_t)(q0 + r) * a.mag_st] = tanhf(a.beta[h] * log1pf(m_eff));
    }
  }
};

__global__ void __launch_bounds__(attend_tf32::kThreads, 1)
polar_tf32_kernel(const __grid_constant__ atma_polar_prefill_args a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ attend_tf32::Shared sh;
  __shared__ float s_n[4][2];
  PolarFront front(a, s_n);
  attend_tf32::attend<PolarFront, 1>(front, smem, sh, &g_polar_tf32_status);
}

// Head size 128, no statistics carried in or out (a marked block is done again from the inputs alone), and enough rows: 2048
// rows, 8 heads, the call's own launches counted, 432 us on the 64 x 64 kernel, 136 here; 512 rows 100 and 60; 300 rows 66 and 60; 256 rows 55 and
// 58 (with two CTAs a head one is for fp32 arithmetic).
// Results that take the place of q: the mark would be in the rows that are read again.  Windows of fewer than few_keys keys: every block
// would be left to the 64 x 64 kernel.
bool polar_tf32_supported(const atma_polar_prefill_args& a) {
  return a.dk == 128 && a.finalize && a.stats_in_m == nullptr && a.Tq > 256 && a.c != a.q && (a.window <= 0 || a.window >= attend_tf32::few_keys(1));
}

template <int DK>
int launch(const atma_polar_prefill_args& a, cudaStream_t st) {
  const bool tf32 = polar_tf32_supported(a);
  if (tf32) {
    ATMA_CUDA_OK(cudaFuncSetAttribute(polar_tf32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, attend_tf32::kSmemBytes));
    polar_tf32_kernel<<<dim3((a.Tq + attend_tf32::kM - 1) / attend_tf32::kM * a.H, a.B), attend_tf32::kThreads, attend_tf32::kSmemBytes, st>>>(a);
    const int rc = launch_status("polar_prefill (fp32, tensor cores)");
    if (rc != ATMA_OK) return rc;
  }
  constexpr int smem = kBlockBytes<DK>;
  ATMA_CUDA_OK(cudaFuncSetAttribute(polar_rows_f32_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  polar_rows_f32_kernel<DK><<<dim3((a.Tq + kM - 1) / kM * a.H, a.B), kThreads, smem, st>>>(a, tf32);
  return launch_status("polar_prefill (fp32, 64 x 64)");
}

}  // namespace

// Rows in quadruples of channels, and more rows than one CTA of the other kernel holds.  Packed batches stay with that: they
// are for 16-bit types.
bool polar_rows_f32_supported(const atma_polar_prefill_args& a) {
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  auto rows = [](int64_t sb, int64_t sh, int64_t st) { return sb % 4 == 0 && sh % 4 == 0 && st % 4 == 0; };
  return a.dtype == ATMA_F32 && (a.dk == 64 || a.dk == 128) && a.n_tiles == 0 && a.Tq > 32 && al(a.q) && al(a.k) && al(a.v) &&
         rows(a.q_sb, a.q_sh, a.q_st) && rows(a.k_sb, a.k_sh, a.k_st) && rows(a.v_sb, a.v_sh, a.v_st);
}

int polar_tf32_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  ATMA_CUDA_OK(cudaMemcpyFromSymbol(&v, g_polar_tf32_status, sizeof(int)));
  if (v != 0) ATMA_CUDA_OK(cudaMemcpyToSymbol(g_polar_tf32_status, &zero, sizeof(int)));
  *out = v;
  return ATMA_OK;
}

int polar_rows_f32(const atma_polar_prefill_args& a, cudaStream_t st) { return a.dk == 64 ? launch<64>(a, st) : launch<128>(a, st); }

}  // namespace atma
