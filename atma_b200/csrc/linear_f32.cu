// fp32 matrix product on the tensor cores: out[m][n] = sum_k x[m][k] w[n][k] + bias[n], at fp32 accuracy.
//
// fp32 arithmetic outside the tensor cores reaches 40-50 TFLOP/s here.  A row times a power of two that brings its largest
// value into [2^14, 2^15) is the sum of an fp16 term and 2^-11 times another, to 2^-22 of a value (2^-51 of the row's
// largest, where a value is that much smaller).  Three products of terms - lo hi, hi lo, hi hi, small ones first, the last
// scaling down what is there by 2^11 on its way - leave out 2^-22 of a product, with random signs.  The tensor core rounds
// its fp32 sums towards zero, so a sum stays there for 64 columns only; the columns' sums are added in registers, rounded to
// nearest.  Error against 64 bits, 2-norm, beside the library's fp32 product (1500 rows, random normal): K = 1024 1.1e-7
// against 4.1e-7, K = 5120 1.5e-7 against 9.0e-7.
//   split kernel: one CTA per row of x and of w, two fp16 planes each and the row's power of two.
//   product kernel: a CTA owns 128 rows x BN columns.  Warp 0 TMA (both planes of 64 columns of x and of w per stage),
//   warp 1 MMA, warps 2-9 add the sums of one stage out of one half of the accumulator columns while the next stage's
//   products go to the other half, scale them back and write whole 128-byte lines.
// Bound by L2 -> shared memory traffic (96 KB per 64 columns and CTA at BN = 256, 62 B per clock and SM if the tensor cores
// were to wait for nothing).  Narrower BN where wide tiles would leave SMs without one; see pick_bn.
// Infinities and NaN have no fp16 terms: a tile that meets one in its rows is computed in fp32 arithmetic instead.
// Measured with the split, out of HBM, beside the library's: 1500 x 8192 x 1024 120 us (497), 1500 x 1024 x 5120 93 us (353),
// 4096 x 8192 x 1024 261 us (1195).  Below 128 rows, 64 columns or K = 64 the split costs more than it gives (32 x 512 x
// 2048: 36 us against 26) and callers stay with the library.
// Every mbarrier wait is bounded; on expiry the CTA frees its TMEM, returns and leaves a status word for the host.
#include <climits>

#include "common.cuh"
#include "linear_f32.cuh"
#include "sm100.cuh"

namespace atma {

namespace {

using namespace sm100;

constexpr int kBM = 128, kBK = 64;
constexpr int kThreads = 320;
constexpr int kNotFinite = INT_MIN;
constexpr int kLoBits = 11;                 // the second plane is 2^11 times what the first leaves

__device__ int g_linear_status = 0;

__device__ __forceinline__ float pow2i(int n) { return __int_as_float((n + 127) << 23); }      // -126 <= n <= 127

// ---- rows into two fp16 planes ----------------------------------------------------------------------------------------
template <bool VEC>
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ x, int64_t x_rs, int M, const float* __restrict__ w, int N, int K, int Kp,
                  __half* __restrict__ xp, __half* __restrict__ wp, int* __restrict__ exps) {
  __shared__ uint32_t s_max[8];
  const int tid = threadIdx.x;
  const bool is_x = (int)blockIdx.x < M;
  const int64_t row = is_x ? blockIdx.x : blockIdx.x - M;
  const float* src = is_x ? x + row * x_rs : w + row * K;
  __half* hi = (is_x ? xp : wp) + row * Kp;
  __half* lo = hi + (int64_t)(is_x ? M : N) * Kp;
  auto load = [&](int i) {                  // four values from column 4 i
    float4 v = {0.f, 0.f, 0.f, 0.f};
    if (VEC) {
      if (4 * i < K) v = reinterpret_cast<const float4*>(src)[i];
    } else {
      if (4 * i < K) v.x = src[4 * i];
      if (4 * i + 1 < K) v.y = src[4 * i + 1];
      if (4 * i + 2 < K) v.z = src[4 * i + 2];
      if (4 * i + 3 < K) v.w = src[4 * i + 3];
    }
    return v;
  };
  constexpr int kKept = 4;                  // rows of up to 4096 stay in registers between the two passes
  float4 kept[kKept];
  uint32_t most = 0;
  auto largest = [&](const float4& v) {
    most = max(max(most, __float_as_uint(v.x) & 0x7fffffffu), max(__float_as_uint(v.y) & 0x7fffffffu,
               max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu)));
  };
#pragma unroll
  for (int j = 0; j < kKept; ++j) { kept[j] = load(tid + 256 * j); largest(kept[j]); }
  for (int i = tid + 256 * kKept; 4 * i < K; i += 256) largest(load(i));
  most = __reduce_max_sync(0xffffffffu, most);
  if ((tid & 31) == 0) s_max[tid >> 5] = most;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; ++j) most = max(most, s_max[j]);
  const bool finite = most < 0x7f800000u;
  const int s = min(14 + 127 - (int)(most >> 23), 126);
  if (tid == 0) exps[blockIdx.x] = finite ? s : kNotFinite;
  const float scale = finite ? pow2i(s) : 0.f;
  auto store = [&](int i, const float4& v) {
    const float e[4] = {v.x * scale, v.y * scale, v.z * scale, v.w * scale};
    alignas(8) __half h[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) { h[j] = __float2half_rn(e[j]); l[j] = __float2half_rn((e[j] - __half2float(h[j])) * (1 << kLoBits)); }
    reinterpret_cast<uint2*>(hi)[i] = *reinterpret_cast<const uint2*>(h);
    reinterpret_cast<uint2*>(lo)[i] = *reinterpret_cast<const uint2*>(l);
  };
#pragma unroll
  for (int j = 0; j < kKept; ++j)
    if (4 * (tid + 256 * j) < Kp) store(tid + 256 * j, kept[j]);
  for (int i = tid + 256 * kKept; 4 * i < Kp; i += 256) store(i, load(i));
}

// D[tmem] = A * B + 2^-kLoBits D
__device__ __forceinline__ void mma_ss_onto_lo(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, %4;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "n"(kLoBits)
      : "memory");
}

// ---- product ------------------------------------------------------------------------------------------------------------
template <int BN>
struct Tile {
  static constexpr int kStages = BN == 256 ? 2 : (BN == 128 ? 3 : 4);
  static constexpr int kPlaneA = kBM * kBK * 2, kPlaneB = BN * kBK * 2;
  static constexpr int kStageBytes = 2 * (kPlaneA + kPlaneB);
  static constexpr int kSmem = kStages * kStageBytes + 1024;
  static constexpr int kCols = 2 * BN;      // TMEM columns
};

struct Product {
  const float *x, *w, *bias;
  const int* exps;
  float* out;
  int64_t x_rs, out_rs;
  int M, N, K, Kp;
};

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
linear_f32_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, const Product p) {
  using L = Tile<BN>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[L::kStages], empty[L::kStages], acc_full[2], acc_empty[2];
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort_v;
  __shared__ int s_ex[kBM];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;

  int bad = 0;
  for (int i = tid; i < kBM; i += kThreads) {
    s_ex[i] = m0 + i < p.M ? p.exps[m0 + i] : 0;
    bad |= s_ex[i] == kNotFinite;
  }
  for (int i = tid; i < BN; i += kThreads) bad |= n0 + i < p.N && p.exps[p.M + n0 + i] == kNotFinite;
  if (__syncthreads_or(bad)) {
    for (int i = tid; i < kBM * BN; i += kThreads) {
      const int m = m0 + i / BN, n = n0 + i % BN;
      if (m >= p.M || n >= p.N) continue;
      const float *xr = p.x + m * p.x_rs, *wr = p.w + (int64_t)n * p.K;
      float acc = 0.f;
      for (int k = 0; k < p.K; ++k) acc = fmaf(xr[k], wr[k], acc);
      p.out[m * p.out_rs + n] = acc + (p.bias ? p.bias[n] : 0.f);
    }
    return;
  }

  if (warp == 0) tmem_alloc(&s_tmem, L::kCols);
  if (tid == 32) {
    for (int i = 0; i < L::kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 256); }
    s_abort_v = 0;
    fence_barrier_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const int NK = p.Kp / kBK;
  volatile int* abort = &s_abort_v;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (; it < NK; ++it) {
        const int st = it % L::kStages;
        if (it >= L::kStages && !mbar_wait(&empty[st], (it / L::kStages - 1) & 1, abort)) break;
        uint8_t* a = smem + st * L::kStageBytes;
        mbar_arrive_expect_tx(&full[st], L::kStageBytes);
        tma_load_4d(a, &tm_x, &full[st], it * kBK, m0, 0, 0);
        tma_load_4d(a + 2 * L::kPlaneA, &tm_w, &full[st], it * kBK, n0, 0, 0);
      }
      volatile int alone = 0;               // whatever the others do, the CTA does not end before its copies
      for (int i = max(0, it - L::kStages); i < it; ++i) mbar_wait(&full[i % L::kStages], (i / L::kStages) & 1, &alone);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(kBM, BN, 0, 0, 0);
      for (int it = 0; it < NK; ++it) {
        const int st = it % L::kStages, buf = it & 1;
        if (it >= 2 && !mbar_wait(&acc_empty[buf], (it / 2 - 1) & 1, abort)) break;
        if (!mbar_wait(&full[st], (it / L::kStages) & 1, abort)) break;
        tc_fence_after();
        const uint32_t a = smem_u32(smem + st * L::kStageBytes), b = a + 2 * L::kPlaneA, d = tmem + buf * BN;
#pragma unroll
        for (int t = 0; t < 3; ++t) {       // lo hi, hi lo, hi hi
          const uint32_t at = a + (t == 0 ? L::kPlaneA : 0), bt = b + (t == 1 ? L::kPlaneB : 0);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) {
            const uint64_t ad = make_sdesc_sw128(at + 32 * k, 16, 1024), bd = make_sdesc_sw128(bt + 32 * k, 16, 1024);
            if (t == 2 && k == 0) mma_ss_onto_lo(d, ad, bd, idesc);
            else mma_ss(d, ad, bd, idesc, t > 0 || k > 0);
          }
        }
        tc_commit(&empty[st]);
        tc_commit(&acc_full[buf]);
      }
    }
  } else {
    constexpr int kMine = BN / 2;           // columns of a thread's row
    const int quarter = warp & 3, side = (warp - 2) >> 2;
    const uint32_t at = tmem + (uint32_t(32 * quarter) << 16) + side * kMine;
    float acc[kMine];
#pragma unroll
    for (int i = 0; i < kMine; ++i) acc[i] = 0.f;
    bool ok = true;
    for (int it = 0; it < NK; ++it) {
      const int buf = it & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[buf], (it / 2) & 1, abort));
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < kMine; c += 32) {
        uint32_t r[32];
        tmem_ld32(at + buf * BN + c, r);
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[c + i] += __uint_as_float(r[i]);
      }
      tc_fence_before();
      mbar_arrive(&acc_empty[buf]);
    }
    if (ok) {                               // every product is done: the stages' memory is free
      float* s = reinterpret_cast<float*>(smem) + (warp - 2) * 32 * 33;
#pragma unroll
      for (int c = 0; c < kMine; c += 32) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 32; ++i) s[lane * 33 + i] = acc[c + i];
        __syncwarp();
        const int n = n0 + side * kMine + c + lane;
        const bool in = n < p.N;
        const int ew = in ? p.exps[p.M + n] : 0;
        const float bias = in && p.bias ? p.bias[n] : 0.f;
        for (int r = 0; r < 32; ++r) {
          const int m = 32 * quarter + r;
          if (m0 + m >= p.M) break;
          const int e = -(s_ex[m] + ew);
          const float v = s[r * 33 + lane] * pow2i(e / 2) * pow2i(e - e / 2);
          if (in) p.out[(m0 + m) * p.out_rs + n] = v + bias;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, L::kCols);
  if (tid == 0 && s_abort_v) atomicExch(&g_linear_status, 1);
}

int make_map(CUtensorMap* out, const __half* planes, int rows, int Kp, int box_rows) {
  const uint64_t dims[4] = {(uint64_t)Kp, (uint64_t)rows, 2, 1};
  const int64_t strides[3] = {Kp, (int64_t)rows * Kp, 2 * (int64_t)rows * Kp};
  const uint32_t box[4] = {kBK, (uint32_t)box_rows, 2, 1};
  return make_tmap_16bit_4d(out, planes, 0, dims, strides, box);
}

template <int BN>
int launch(const Product& p, const __half* xp, const __half* wp, cudaStream_t st) {
  CUtensorMap mx, mw;
  int rc = make_map(&mx, xp, p.M, p.Kp, kBM);
  if (rc == ATMA_OK) rc = make_map(&mw, wp, p.N, p.Kp, BN);
  if (rc != ATMA_OK) return rc;
  ATMA_CUDA_OK(cudaFuncSetAttribute(linear_f32_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<BN>::kSmem));
  linear_f32_kernel<BN><<<dim3((p.M + kBM - 1) / kBM, (p.N + BN - 1) / BN), kThreads, Tile<BN>::kSmem, st>>>(mx, mw, p);
  return launch_status("linear_f32 (tcgen05)");
}

// The widest tile moves the fewest bytes per product, but a whole wave of tiles costs the same however few there are: the
// choice is the one whose waves times bytes per stage are fewest.
int pick_bn(int M, int N) {
  int best = 0;
  int64_t least = INT64_MAX;
  for (int bn : {256, 128, 64}) {
    const int64_t tiles = (int64_t)((M + kBM - 1) / kBM) * ((N + bn - 1) / bn), sms = sm_count_of_current_device();
    const int64_t cost = (tiles + sms - 1) / sms * (kBM + bn);
    if (cost < least) { least = cost; best = bn; }
  }
  return best;
}

int padded(int K) { return (K + kBK - 1) / kBK * kBK; }
int64_t round256(int64_t n) { return (n + 255) & ~(int64_t)255; }

}  // namespace

int linear_f32_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  ATMA_CUDA_OK(cudaMemcpyFromSymbol(&v, g_linear_status, sizeof(int)));
  if (v != 0) ATMA_CUDA_OK(cudaMemcpyToSymbol(g_linear_status, &zero, sizeof(int)));
  *out = v;
  return ATMA_OK;
}

}  // namespace atma

using namespace atma;

extern "C" int64_t atma_linear_f32_scratch_bytes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  return round256((int64_t)M * padded(K) * 4) + round256((int64_t)N * padded(K) * 4) + round256(((int64_t)M + N) * 4) + 256;
}

extern "C" int atma_linear_f32(const float* x, int64_t x_rs, const float* w, const float* bias, float* out, int64_t out_rs, int M, int N,
                               int K, void* scratch, void* stream) {
  if (M <= 0 || N <= 0) return ATMA_OK;
  ATMA_REQUIRE(x != nullptr && w != nullptr && out != nullptr && scratch != nullptr, "linear_f32: null pointer");
  ATMA_REQUIRE(K > 0 && K <= (1 << 24) && (int64_t)M + N < (int64_t(1) << 30), "linear_f32: bad shape (%d, %d, %d)", M, N, K);
  const int bn = pick_bn(M, N), Kp = padded(K);
  ATMA_REQUIRE((N + bn - 1) / bn <= 65535, "linear_f32: too many columns (%d)", N);
  cudaStream_t st = (cudaStream_t)stream;
  uint8_t* at = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(scratch) + 255) & ~(uintptr_t)255);
  __half* xp = reinterpret_cast<__half*>(at);
  __half* wp = reinterpret_cast<__half*>(at + round256((int64_t)M * Kp * 4));
  int* exps = reinterpret_cast<int*>(at + round256((int64_t)M * Kp * 4) + round256((int64_t)N * Kp * 4));
  const bool vec = K % 4 == 0 && x_rs % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
  if (vec) split_rows_kernel<true><<<M + N, 256, 0, st>>>(x, x_rs, M, w, N, K, Kp, xp, wp, exps);
  else split_rows_kernel<false><<<M + N, 256, 0, st>>>(x, x_rs, M, w, N, K, Kp, xp, wp, exps);
  int rc = launch_status("linear_f32 (split)");
  if (rc != ATMA_OK) return rc;
  const Product p{x, w, bias, exps, out, x_rs, out_rs, M, N, K, Kp};
  if (bn == 256) return launch<256>(p, xp, wp, st);
  if (bn == 128) return launch<128>(p, xp, wp, st);
  return launch<64>(p, xp, wp, st);
}
