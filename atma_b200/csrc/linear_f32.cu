// fp32 matrix product on the tensor cores: out[m][n] = sum_k x[m][k] w[n][k] + bias[n], at fp32 accuracy.
//
// fp32 arithmetic outside the tensor cores reaches 40-50 TFLOP/s here.  A row times a power of two that brings its largest
// value into [2^14, 2^15) is the sum of an fp16 term and 2^-11 times another, to 2^-22 of a value that is not 2^28 times
// smaller than that.  Three products of terms - lo hi, hi lo, hi hi, small ones first, the last scaling down what is there by
// 2^11 on its way - leave out 2^-22 of a product, with random signs.  The tensor core rounds
// its fp32 sums towards zero, so a sum stays there for 64 columns only; the columns' sums are added in registers, rounded to
// nearest.  Error against 64 bits, 2-norm, beside the library's fp32 product (1500 rows, random normal): K = 1024 1.1e-7
// against 4.1e-7, K = 5120 1.5e-7 against 9.0e-7.
// What the smaller values of a row lose is summed when it is split.  A result that this could change by more than 2^-24 of
// itself - large values that meet zeros and small ones that do not - is summed again in fp32 from the inputs, a warp for
// four, and so are the results of a row with an infinity or a NaN, which has no fp16 terms.  Rows of random values, squared
// activations among them, have next to none, and the test costs nothing that shows; where every result needs it, 1500 x 8192 x
// 1024 takes 9.9 ms instead of 0.11 (7.7 while every tile had its CTA), with one such row of x 0.31.
//   split kernel: one CTA per row of x and of w, two fp16 planes each, the row's power of two and what it lost.
//   product kernel: a CTA per SM takes tiles of 128 rows x BN columns in turn (a very long K: a CTA per tile).  Warp 0 TMA (both planes of 64 columns of x and of
//   w per stage), warp 1 MMA, warps 2-9 add the sums of one stage out of one half of the accumulator columns while the next stage's
//   products go to the other half, scale them back and write them, under the first two stages of the next tile.
// Bound by the products (1536 clocks per 64 columns at BN = 256) and L2 -> shared memory traffic (96 KB for them, 1600 clocks) within
// a tile, 1780 measured; between tiles by the results' way out: 18000 clocks a tile, as long as ten stages, with a loop over rows
// and columns that loads, scales and stores one value, 6000 with four values at a time and the columns' figures fetched under the
// products.  Narrower BN where wide tiles would leave SMs without one; see pick_bn.
// Measured out of HBM, without the split (with it, beside the library's, 1500 x 8192 x 1024 103 us and 499): 1500 x 8192 x 1024
// 93 -> 83 us, 4096 x 8192 x 1024 227 -> 179, 2048 x 1024 x 4096 59 -> 51, 512 x 1024 x 1024 16.4 -> 13.3.  Where one side is short or
// few tiles walk a long K the library's is faster (32 x 512 x 2048: 26 us against 36) and callers stay with it.
// Every mbarrier wait is bounded; on expiry the CTA frees its TMEM, returns and leaves a status word for the host.
#include "common.cuh"
#include "linear_f32.cuh"
#include "sm100.cuh"

namespace atma {

namespace {

using namespace sm100;

constexpr int kBM = 128, kBK = 64;
constexpr int kOut = 16, kLd = kOut + 4;      // columns that leave at a time; floats between their rows: quarter warps meet no bank twice
constexpr int kThreads = 320;
constexpr int kLoBits = 11;                 // the second plane is 2^11 times what the first leaves
constexpr float kWhole = 1.0f / (1 << 13);  // scaled values from here on are in the two terms to 2^-22 of themselves
constexpr float kGone = 8.6736174e-19f;      // 2^-60: from there down nothing is left (and scaling may have made it zero already)
constexpr float kLossUnits = 4.6116860e18f; // 2^62: a row's loss, at most 2^-36 of each of 2^24 values, is counted in these

__device__ int g_linear_status = 0;

// From where on a sum whose row or column has that loss is trusted: it meets values below 2^15, and 2^-24 of the sum is accepted.
__device__ __forceinline__ float trusted_from(unsigned long long loss) { return (float)loss * (549755813888.0f / kLossUnits); }      // 2^39

__device__ __forceinline__ float pow2i(int n) { return __int_as_float((n + 127) << 23); }      // -126 <= n <= 127

// ---- rows into two fp16 planes ----------------------------------------------------------------------------------------
// Out of HBM and latency: a row of 1024 is one load, two barriers and one store per thread, so rows in flight count (9692 rows 20 us
// with 32 registers, 25 with 40; the bytes alone are 12).
// KEPT: groups of four values a thread has in registers between the two passes (1024 columns each); the others are read again.
template <bool VEC, int KEPT>
__global__ void __launch_bounds__(256, KEPT == 1 ? 8 : 6)
split_rows_kernel(const float* __restrict__ x, int64_t x_rs, int M, const float* __restrict__ w, int N, int K, int Kp,
                  __half* __restrict__ xp, __half* __restrict__ wp, int* __restrict__ exps, unsigned long long* __restrict__ losses) {
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
  float4 kept[KEPT];
  uint32_t most = 0;
  auto largest = [&](const float4& v) {
    most = max(max(most, __float_as_uint(v.x) & 0x7fffffffu), max(__float_as_uint(v.y) & 0x7fffffffu,
               max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu)));
  };
#pragma unroll
  for (int j = 0; j < KEPT; ++j) { kept[j] = load(tid + 256 * j); largest(kept[j]); }
  for (int i = tid + 256 * KEPT; 4 * i < K; i += 256) largest(load(i));
  most = __reduce_max_sync(0xffffffffu, most);
  if ((tid & 31) == 0) s_max[tid >> 5] = most;
  if (tid == 0) losses[blockIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; ++j) most = max(most, s_max[j]);
  if (most >= 0x7f800000u) {                // an infinity or a NaN: its results are summed in fp32
    for (int i = tid; 4 * i < Kp; i += 256) {
      reinterpret_cast<uint2*>(hi)[i] = uint2{0, 0};
      reinterpret_cast<uint2*>(lo)[i] = uint2{0, 0};
    }
    if (tid == 0) { exps[blockIdx.x] = 0; losses[blockIdx.x] = 1; }     // sums of zeros: none of them is trusted
    return;
  }
  const int s = min(14 + 127 - (int)(most >> 23), 126);
  if (tid == 0) exps[blockIdx.x] = s;
  const float scale = pow2i(s);
  const uint32_t small = 2 * __float_as_uint(kWhole / scale) - 1;     // twice the bits drop the sign, and a zero's less one are the largest
  auto store = [&](int i, const float4& v) {
    const float x[4] = {v.x, v.y, v.z, v.w};
    alignas(8) __half h[4], l[4];
    uint32_t least = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float e = x[j] * scale;
      h[j] = __float2half_rn(e);
      l[j] = __float2half_rn((e - __half2float(h[j])) * (1 << kLoBits));
      least = min(least, 2 * __float_as_uint(x[j]) - 1);
    }
    if (least < small) {                    // whole numbers: their sum has no order
      unsigned long long loss = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float e = x[j] * scale;
        if (fabsf(e) < kWhole && x[j] != 0.f)                  // what both terms leave: exact, as the differences are
          loss += (unsigned long long)ceilf(fmaxf(fabsf(e - __half2float(h[j]) - __half2float(l[j]) * (1.0f / (1 << kLoBits))),
                                                  fabsf(e) < kGone ? kGone : 0.f) * kLossUnits);
      }
      if (loss != 0) atomicAdd(losses + blockIdx.x, loss);
    }
    reinterpret_cast<uint2*>(hi)[i] = *reinterpret_cast<const uint2*>(h);
    reinterpret_cast<uint2*>(lo)[i] = *reinterpret_cast<const uint2*>(l);
  };
#pragma unroll
  for (int j = 0; j < KEPT; ++j)
    if (4 * (tid + 256 * j) < Kp) store(tid + 256 * j, kept[j]);
  for (int i = tid + 256 * KEPT; 4 * i < Kp; i += 256) store(i, load(i));
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
  static constexpr int kStaging = 8 * 32 * kLd * 4;                       // results on their way out, a warp's 32 rows x 16 columns
  static constexpr int kSmem = kStages * kStageBytes + kStaging + 1024;
  static constexpr int kCols = 2 * BN;      // TMEM columns
};

struct Product {
  const float *x, *w, *bias;
  const int* exps;                          // [M + N]
  const unsigned long long* losses;         // [M + N]
  float* out;
  int64_t x_rs, out_rs;
  int M, N, K, Kp;
};

// Results that the terms alone don't settle, in fp32 arithmetic: bit 4 i + j of a lane's `flags` is row m0 + lane / 4 + 8 i, column
// n0 + 4 (lane % 4) + j.  Four of a row at a time: their loads do not wait for one another, and x is read once for them (for each of
// them, 1500 x 8192 x 1024 with nothing but such results took 11.4 ms).
__device__ __noinline__ void sum_again(const Product& p, int m0, int n0, uint32_t flags) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    uint32_t mine = (flags >> (4 * i) & 15u) << (4 * (lane & 3));            // the row's 16 columns, from its four lanes
    mine |= __shfl_xor_sync(0xffffffffu, mine, 1);
    mine |= __shfl_xor_sync(0xffffffffu, mine, 2);
    uint32_t lanes = __ballot_sync(0xffffffffu, mine != 0) & 0x11111111u;
    while (lanes != 0) {
      const int from = __ffs(lanes) - 1, row = m0 + (from >> 2) + 8 * i;
      lanes &= lanes - 1;
      uint32_t cols = __shfl_sync(0xffffffffu, mine, from);
      const float* x = p.x + (int64_t)row * p.x_rs;
      while (cols != 0) {
        int c[4];
        float acc[4] = {};
        const float* w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          c[j] = j > 0 && cols == 0 ? c[0] : __ffs(cols) - 1;
          cols &= cols - 1;
          w[j] = p.w + (int64_t)(n0 + c[j]) * p.K;
        }
#pragma unroll 4
        for (int k = lane; k < p.K; k += 32) {
          const float a = x[k];
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[j] = fmaf(a, w[j][k], acc[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float sum = warp_sum(acc[j]);
          if (lane == j) p.out[(int64_t)row * p.out_rs + n0 + c[j]] = sum + (p.bias ? p.bias[n0 + c[j]] : 0.f);
        }
      }
    }
  }
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
linear_f32_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                  const __grid_constant__ Product p) {
  using L = Tile<BN>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[L::kStages], empty[L::kStages], acc_full[2], acc_empty[2];
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort_v;
  // A warp's own figures of its rows (the power of two) and columns (the same, from where on a sum is trusted, the bias).  Four warps
  // have the same columns, but no copy in common: a warp gives its accumulators away before it writes its results, so with K <= 128
  // the next tile's products can be through, and another warp two tiles ahead, while it still reads.
  __shared__ int s_ex[8][32];
  __shared__ __align__(16) int s_cex[8][BN / 2];
  __shared__ __align__(16) float s_cleast[8][BN / 2], s_cbias[8][BN / 2];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m_tiles = (p.M + kBM - 1) / kBM, tiles = m_tiles * ((p.N + BN - 1) / BN);

  if (warp == 0) tmem_alloc(&s_tmem, L::kCols);
  if (tid == 32) {
    for (int i = 0; i < L::kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
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
    if (elect_one()) {
      uint32_t n = 0;                       // stages so far, over all tiles
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int m0 = tile % m_tiles * kBM, n0 = tile / m_tiles * BN;
        for (int it = 0; it < NK; ++it, ++n) {
          const uint32_t st = n % L::kStages;
          if (n >= L::kStages && !(ok = mbar_wait(&empty[st], (n / L::kStages - 1) & 1, abort))) break;
          uint8_t* a = smem + st * L::kStageBytes;
          mbar_arrive_expect_tx(&full[st], L::kStageBytes);
          tma_load_4d(a, &tm_x, &full[st], it * kBK, m0, 0, 0);
          tma_load_4d(a + 2 * L::kPlaneA, &tm_w, &full[st], it * kBK, n0, 0, 0);
        }
      }
      volatile int alone = 0;               // whatever the others do, the CTA does not end before its copies
      for (uint32_t i = n > L::kStages ? n - L::kStages : 0; i < n; ++i) mbar_wait(&full[i % L::kStages], (i / L::kStages) & 1, &alone);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc(kBM, BN, 0, 0, 0);
      uint32_t n = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        for (int it = 0; it < NK; ++it, ++n) {
          const uint32_t st = n % L::kStages, buf = n & 1;
          ok = (n < 2 || mbar_wait(&acc_empty[buf], (n / 2 - 1) & 1, abort)) && mbar_wait(&full[st], (n / L::kStages) & 1, abort);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a = smem_u32(smem + st * L::kStageBytes), b = a + 2 * L::kPlaneA, d = tmem + buf * BN;
#pragma unroll
          for (int t = 0; t < 3; ++t) {     // lo hi, hi lo, hi hi
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
    }
  } else {
    constexpr int kMine = BN / 2;           // columns of a thread's row
    const int w = warp - 2, quarter = warp & 3, side = w >> 2;
    const uint32_t at = tmem + (uint32_t(32 * quarter) << 16) + side * kMine;
    float* s = reinterpret_cast<float*>(smem + L::kStages * L::kStageBytes) + w * 32 * kLd;
    const bool vec = p.out_rs % 4 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
    const int rr = lane >> 2, cc = 4 * (lane & 3);                   // what this lane stores: row rr + 8 i, four columns
    uint32_t n_st = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
      const int mw = tile % m_tiles * kBM + 32 * quarter, nw = tile / m_tiles * BN + side * kMine, rows = min(32, p.M - mw);
      const bool in_row = lane < rows;
      const int ex = in_row ? p.exps[mw + lane] : 0;
      const float row_least = in_row ? trusted_from(p.losses[mw + lane]) : 0.f, most_least = warp_max(row_least);
      int* cex = s_cex[w];
      float *cleast = s_cleast[w], *cbias = s_cbias[w];
      __syncwarp();                         // the last tile's figures have been read
      s_ex[w][lane] = ex;
      int most_e = -1000, least_e = 1000;
      // under the first products
#pragma unroll
      for (int i = lane; i < kMine; i += 32) {
        const bool in = nw + i < p.N;
        cex[i] = in ? p.exps[p.M + nw + i] : 0;
        cleast[i] = in ? trusted_from(p.losses[p.M + nw + i]) : -INFINITY;
        cbias[i] = in && p.bias ? p.bias[nw + i] : 0.f;
        most_e = max(most_e, cex[i]); least_e = min(least_e, cex[i]);
      }
      // whether every result's power of two is a normal number; else it comes as two factors
      const bool one_factor = __reduce_max_sync(0xffffffffu, most_e) + __reduce_max_sync(0xffffffffu, ex) <= 126 &&
                              __reduce_min_sync(0xffffffffu, least_e) + __reduce_min_sync(0xffffffffu, ex) >= -127;
      float acc[kMine];
#pragma unroll
      for (int i = 0; i < kMine; ++i) acc[i] = 0.f;
      for (int it = 0; it < NK; ++it, ++n_st) {
        const uint32_t buf = n_st & 1;
        ok = mbar_wait_warp(&acc_full[buf], (n_st / 2) & 1, abort);
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
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      }
      if (!ok || rows <= 0) continue;
      // 16 columns at a time through shared memory, so that rows leave in whole sectors.  The tensor cores have begun the next
      // tile, but wait after two stages of it, so the common case is kept short: whole tiles, powers of two that are normal numbers.
      const bool simple = one_factor && vec && rows == 32 && nw + kMine <= p.N;
      float* to = p.out + (int64_t)(mw + rr) * p.out_rs + nw + cc;
      const int64_t step = 8 * p.out_rs;
      uint32_t flags[kMine / 32];           // 16 results of this lane in each half
#pragma unroll
      for (int c = 0; c < kMine; c += kOut) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kOut; i += 4) *reinterpret_cast<float4*>(s + lane * kLd + i) = make_float4(acc[c + i], acc[c + i + 1], acc[c + i + 2], acc[c + i + 3]);
        const int4 ew = *reinterpret_cast<const int4*>(cex + c + cc);
        const float4 l4 = *reinterpret_cast<const float4*>(cleast + c + cc), bias = *reinterpret_cast<const float4*>(cbias + c + cc);
        const float least = fmaxf(fmaxf(l4.x, l4.y), fmaxf(l4.z, l4.w)) + most_least;
        __syncwarp();
        uint32_t again = 0;                 // four results that may have to be summed again, per row
        if (simple) {
          const int fx = (127 - ew.x) << 23, fy = (127 - ew.y) << 23, fz = (127 - ew.z) << 23, fw = (127 - ew.w) << 23;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 q = *reinterpret_cast<const float4*>(s + (rr + 8 * i) * kLd + cc);
            const int er = s_ex[w][rr + 8 * i] << 23;
            again |= fminf(fminf(fabsf(q.x), fabsf(q.y)), fminf(fabsf(q.z), fabsf(q.w))) < least ? 15u << (4 * i) : 0u;
            *reinterpret_cast<float4*>(to + i * step + c) =
                make_float4(fmaf(q.x, __int_as_float(fx - er), bias.x), fmaf(q.y, __int_as_float(fy - er), bias.y),
                            fmaf(q.z, __int_as_float(fz - er), bias.z), fmaf(q.w, __int_as_float(fw - er), bias.w));
          }
        } else {
          const int e4[4] = {ew.x, ew.y, ew.z, ew.w}, left = p.N - (nw + c + cc);
          const float b4[4] = {bias.x, bias.y, bias.z, bias.w};
#pragma unroll 1
          for (int i = 0; i < 4; ++i) {
            const int r = rr + 8 * i;
            if (r >= rows) break;
            const float4 q = *reinterpret_cast<const float4*>(s + r * kLd + cc);
            const float sum[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (j >= left) break;
              const int e = -(s_ex[w][r] + e4[j]);
              to[i * step + c + j] = fmaf(sum[j] * pow2i(e / 2), pow2i(e - e / 2), b4[j]);
              if (fabsf(sum[j]) < least) again |= (left >= 4 ? 15u : (1u << left) - 1) << (4 * i);      // all four, as above
            }
          }
        }
        if ((c / kOut) & 1) flags[c / 32] |= again << 16; else flags[c / 32] = again;
      }
#pragma unroll
      for (int c = 0; c < kMine; c += kOut) {
        const uint32_t f = flags[c / 32] >> (16 * ((c / kOut) & 1)) & 0xffffu;
        if (__any_sync(0xffffffffu, f != 0)) sum_again(p, mw, nw + c, f);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, L::kCols);
  if (tid == 0 && s_abort_v) atomicExch(&g_linear_status, 1);
}

// From here on a tile has a CTA to itself.  Tiles in turn have the next products wait while results are summed again, and a wait ends
// after 1.1 s: a tile of 128 x 256 with nothing else took 3.3 ms at K = 1024, 20 at 8192, 160 at 32704.  What tiles in turn save,
// some 12000 clocks each, is then less than 1.5 % of a tile's 512 stages.
constexpr int kAloneK = 1 << 15;

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
  const int64_t tiles = (int64_t)((p.M + kBM - 1) / kBM) * ((p.N + BN - 1) / BN);
  const int sms = sm_count_of_current_device();
  const bool in_turn = tiles > sms && p.Kp < kAloneK;
  linear_f32_kernel<BN><<<(unsigned)(in_turn ? sms : tiles), kThreads, Tile<BN>::kSmem, st>>>(mx, mw, p);
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
  return round256((int64_t)M * padded(K) * 4) + round256((int64_t)N * padded(K) * 4) + round256(((int64_t)M + N) * 4) + round256(((int64_t)M + N) * 8) + 256;
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
  auto* losses = reinterpret_cast<unsigned long long*>(reinterpret_cast<uint8_t*>(exps) + round256(((int64_t)M + N) * 4));
  const bool vec = K % 4 == 0 && x_rs % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
#define ATMA_SPLIT(VEC, KEPT) split_rows_kernel<VEC, KEPT><<<M + N, 256, 0, st>>>(x, x_rs, M, w, N, K, Kp, xp, wp, exps, losses)
  if (vec) { if (Kp <= 1024) ATMA_SPLIT(true, 1); else ATMA_SPLIT(true, 4); }
  else { if (Kp <= 1024) ATMA_SPLIT(false, 1); else ATMA_SPLIT(false, 4); }
#undef ATMA_SPLIT
  int rc = launch_status("linear_f32 (split)");
  if (rc != ATMA_OK) return rc;
  const Product p{x, w, bias, exps, losses, out, x_rs, out_rs, M, N, K, Kp};
  if (bn == 256) return launch<256>(p, xp, wp, st);
  if (bn == 128) return launch<128>(p, xp, wp, st);
  return launch<64>(p, xp, wp, st);
}
