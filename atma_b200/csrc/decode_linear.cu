// Weight-streaming linear layers for small decode batches (up to 16 rows): out = x W^T + b, optionally
// with the MLP's squared-ReLU gate applied to the two halves of the result before it is written
// (inference/models/atma.py:87-97: fc GEMM -> gate * relu(x)^2 -> proj GEMM; :631-673: in_proj / out_proj
// around the LFM2 conv).  At these batch sizes the products are bound by reading the weights once from
// HBM: every warp streams whole 16-row slabs of W with 16-byte loads (all loads of its K range in flight
// before the first use), keeps them in the register layout mma.sync wants without a shared-memory round
// trip, and multiplies by the x rows it reads from L1/L2.  A 16-byte piece of a weight row is eight
// consecutive k; the same eight k of an x row go to the matching B-operand registers, so the reduction
// index is permuted identically on both sides and no shuffle is needed.  K is split over the 16 warps of a
// CTA; their partial tiles meet in shared memory, where bias, rounding to the activation dtype (what the
// GEMM of the separate-op path would have written) and the gate are applied, one thread per result.
//
// Bound by latency: 2 to 17 MB of weights are 0.3 to 2.5 us of HBM time.  The kernel starts under the one in front (early.cuh)
// and asks for its weights then, a result's K splits are added by a thread of its own (one warp per unit used to do that
// alone, over a microsecond), and the compiler is told that one CTA per SM is meant: for two it keeps too few registers to
// have the loads of a K range in flight.  From the end of the kernel in front, 3 rows: 8192 x 1024 gated 5.8 -> 4.0 us,
// 1024 x 4096 4.7 -> 3.6, 1024 x 1024 3.4 -> 2.3; 8 rows: 1024 x 5120 5.2 -> 4.7.
#include <climits>

#include "common.cuh"
#include "early.cuh"
#include "gelu.cuh"
#include "mma_sync.cuh"

namespace atma {

namespace {

constexpr int kWarps = 16;                 // warps per CTA
constexpr int kAhead = 8;                  // lines of a row that are asked for under the kernel in front: 16 KB per warp, 38 MB in all
constexpr int kMaxRows = 16;               // batch rows (two n8 tiles)

struct LinArgs {
  const void* x; int64_t x_rs;             // [B][K]
  const void* w;                           // [N][K] row-major (torch Linear layout)
  const void* bias;                        // [N] or null
  void* out; int64_t out_rs;               // [B][N], or [B][N/2] where two halves are combined
  int B, N, K;
  int ks, kper;                            // K splits per unit (power of two <= 16), columns of one (a multiple of 32, the last
                                           // has what is left); units per CTA = 16 / ks
  int units;                               // 16-feature units (two halves: N/2/16, else N/16)
};

// One warp: its unit's rows [row0, row0+16) (and, gated, [row0 + N/2, ...)) over k in [k0, k1).
// kGated: 0 plain, 1 up * relu(gate)^2, 2 gelu_tanh(gate) * up, 3 relu(y)^2 of every feature (no second half)
template <typename T, int NT, int kGated>
__global__ void __launch_bounds__(kWarps * 32, 1)
decode_linear_kernel(const LinArgs a) {
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
  constexpr int kTiles = kGated == 1 || kGated == 2 ? 2 : 1;
  __shared__ float part[kWarps][kTiles][NT][4][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int upc = kWarps / a.ks;                              // units per CTA
  const int unit = blockIdx.x * upc + warp / a.ks;
  const int split = warp % a.ks;
  const int k0 = min(split * a.kper, a.K), kend = min(k0 + a.kper, a.K);
  const T* W = static_cast<const T*>(a.w);
  const T* X = static_cast<const T*>(a.x);
  if (unit < a.units) {                                       // the warp's first weights, a 128-byte line per lane
    constexpr int kLine = 128 / (int)sizeof(T);
    const int lines = min((kend - k0 + kLine - 1) / kLine, kAhead);
    for (int i = lane; i < 16 * kTiles * lines; i += 32) {
      const int r = i / lines, at = k0 + (i - r * lines) * kLine;
      prefetch_l2(W + ((int64_t)unit * 16 + (r & 15) + (r < 16 ? 0 : a.N / 2)) * a.K + at);
    }
  }
  early_start();
  // result e of the CTA: [unit][n][j][lane], feature (of the first half) and batch row of an accumulator register; the bias of
  // the thread's first one is requested with the weights
  auto place = [&](int e, int& feat, int& b) {
    const int u = blockIdx.x * upc + e / (NT * 128), j = e / 32 % 4, l = e % 32;
    feat = u < a.units ? u * 16 + (l >> 2) + (j >= 2 ? 8 : 0) : -1;
    b = 8 * (e / 128 % NT) + 2 * (l & 3) + (j & 1);
  };
  const T* bias = static_cast<const T*>(a.bias);
  float bias0[kTiles] = {};
  if (bias != nullptr && (int)threadIdx.x < upc * NT * 128) {
    int feat, b;
    place(threadIdx.x, feat, b);
    if (feat >= 0) {
#pragma unroll
      for (int i = 0; i < kTiles; ++i) bias0[i] = to_f32(bias[feat + i * (a.N / 2)]);
    }
  }
  float acc[kTiles][NT][4];
#pragma unroll
  for (int i = 0; i < kTiles; ++i)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][n][j] = 0.f;

  if (unit < a.units) {
    const int row0 = unit * 16;
    const T* wr[kTiles][2];
#pragma unroll
    for (int i = 0; i < kTiles; ++i) {
      const int64_t base = (int64_t)(row0 + (i ? a.N / 2 : 0));
      wr[i][0] = W + (base + g) * a.K + k0 + 8 * t;
      wr[i][1] = W + (base + g + 8) * a.K + k0 + 8 * t;
    }
    const T* xr[NT];
    bool xok[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      xok[n] = (8 * n + g) < a.B;
      xr[n] = X + (int64_t)(xok[n] ? 8 * n + g : 0) * a.x_rs + k0 + 8 * t;
    }
    constexpr int kUnroll = 4;                                // 32-k blocks requested together
    for (int kb = 0; kb < kend - k0; kb += 32 * kUnroll) {
      uint4 wv[kUnroll][kTiles][2], xv[kUnroll][NT];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const bool on = k0 + kb + 32 * u + 8 * t < kend;
#pragma unroll
        for (int i = 0; i < kTiles; ++i)
#pragma unroll
          for (int r = 0; r < 2; ++r)
            wv[u][i][r] = on ? __ldcs(reinterpret_cast<const uint4*>(wr[i][r] + kb + 32 * u)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int n = 0; n < NT; ++n)
          xv[u][n] = (on && xok[n]) ? *reinterpret_cast<const uint4*>(xr[n] + kb + 32 * u) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u)
#pragma unroll
        for (int i = 0; i < kTiles; ++i)
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            const uint32_t a0[4] = {wv[u][i][0].x, wv[u][i][1].x, wv[u][i][0].y, wv[u][i][1].y};
            const uint32_t a1[4] = {wv[u][i][0].z, wv[u][i][1].z, wv[u][i][0].w, wv[u][i][1].w};
            mma::mma16816<kBf16>(acc[i][n], a0, xv[u][n].x, xv[u][n].y);
            mma::mma16816<kBf16>(acc[i][n], a1, xv[u][n].z, xv[u][n].w);
          }
    }
  }
#pragma unroll
  for (int i = 0; i < kTiles; ++i)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int j = 0; j < 4; ++j) part[warp][i][n][j][lane] = acc[i][n][j];
  __syncthreads();
  // every thread adds the K splits of its results; bias, rounding and gate follow
  T* out = static_cast<T*>(a.out);
  for (int e = threadIdx.x; e < upc * NT * 128; e += kWarps * 32) {
    int feat, b;
    place(e, feat, b);
    if (feat < 0 || b >= a.B) continue;
    const int first = e / (NT * 128) * a.ks, n = e / 128 % NT, j = e / 32 % 4, l = e % 32;
    float y[kTiles];
#pragma unroll
    for (int i = 0; i < kTiles; ++i) {
      float s = 0.f;
#pragma unroll 4
      for (int k = 0; k < a.ks; ++k) s += part[first + k][i][n][j][l];
      if (bias != nullptr) s += e == (int)threadIdx.x ? bias0[i] : to_f32(bias[feat + i * (a.N / 2)]);
      y[i] = round_through<T>(s);                              // what the GEMM of the separate-op path writes
    }
    float v = y[0];
    if constexpr (kGated == 2) {
      v = gelu_tanh_16(y[0]) * y[1];
    } else if constexpr (kGated == 1) {
      const float p = fmaxf(y[0], 0.f);
      float sq = p * p;
      if constexpr (kBf16) sq = round_through<T>(sq);         // eager bf16 materialises relu(x)^2 before the multiply
      v = y[1] * sq;
    } else if constexpr (kGated == 3) {
      const float p = fmaxf(y[0], 0.f);
      v = p * p;
    }
    out[(int64_t)b * a.out_rs + feat] = from_f32<T>(v);
  }
}

}  // namespace
}  // namespace atma

using namespace atma;

static int decode_linear(const void* x, int64_t x_row_stride, const void* weight, const void* bias, void* out, int64_t out_row_stride,
                         int B, int N, int K, int gated, int dtype, void* stream) {
  ATMA_REQUIRE(dtype == ATMA_BF16 || dtype == ATMA_F16, "decode_linear: 16-bit activations and weights only (dtype %d)", dtype);
  ATMA_REQUIRE(B >= 0 && B <= kMaxRows, "decode_linear: %d rows; this entry serves decode batches of up to %d", B, kMaxRows);
  ATMA_REQUIRE(gated >= 0 && gated <= 3, "decode_linear: unknown form %d", gated);
  const bool halves = gated == 1 || gated == 2;
  ATMA_REQUIRE(N > 0 && N % (halves ? 32 : 16) == 0, "decode_linear: N=%d must be a multiple of %d", N, halves ? 32 : 16);
  ATMA_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(weight) & 15) == 0 && x_row_stride % 8 == 0,
               "decode_linear: x and weight must be 16-byte aligned with a row stride that is a multiple of 8 elements");
  if (B == 0) return ATMA_OK;
  LinArgs a{};
  a.x = x; a.x_rs = x_row_stride; a.w = weight; a.bias = bias; a.out = out; a.out_rs = out_row_stride;
  a.B = B; a.N = N; a.K = K;
  a.units = (halves ? N / 2 : N) / 16;
  // K splits per unit: a wave of CTAs costs its share of K and a latency of about 0.15 of a whole unit's (1024 columns), so
  // few units are split as far as one wave holds them and the LM head's 3144 in two: 393 CTAs, 20 us against 27 unsplit
  const int sms = sm_count_of_current_device();
  int ks = 1;
  for (int s = 1, best = INT_MAX; s <= kWarps; s <<= 1) {
    if (s > 1 && (K % 32 == 0 ? K % (32 * s) != 0 : K < 64 * s)) break;
    const int waves = ((a.units + kWarps / s - 1) / (kWarps / s) + sms - 1) / sms, cost = waves * (100 / s + 15);
    if (cost < best) { best = cost; ks = s; }
  }
  a.ks = ks;
  a.kper = (K + 32 * ks - 1) / (32 * ks) * 32;
  const int upc = kWarps / ks;
  const dim3 grid((a.units + upc - 1) / upc), block(kWarps * 32);
  cudaStream_t st = (cudaStream_t)stream;
#define ATMA_LIN(T, NT, G) launch_early(B, decode_linear_kernel<T, NT, G>, grid, block, 0, st, a)
#define ATMA_LIN_ANY(T, NT)                                                                  \
  do {                                                                                       \
    if (gated == 3) ATMA_LIN(T, NT, 3); else if (gated == 2) ATMA_LIN(T, NT, 2);            \
    else if (gated) ATMA_LIN(T, NT, 1); else ATMA_LIN(T, NT, 0);                             \
  } while (0)
  if (dtype == ATMA_BF16) {
    if (B <= 8) ATMA_LIN_ANY(__nv_bfloat16, 1); else ATMA_LIN_ANY(__nv_bfloat16, 2);
  } else {
    if (B <= 8) ATMA_LIN_ANY(__half, 1); else ATMA_LIN_ANY(__half, 2);
  }
#undef ATMA_LIN_ANY
#undef ATMA_LIN
  return launch_status("decode_linear");
}

extern "C" int atma_decode_linear(const void* x, int64_t x_row_stride, const void* weight, const void* bias, void* out,
                                  int64_t out_row_stride, int B, int N, int K, int gated, int dtype, void* stream) {
  ATMA_REQUIRE(K >= 32 && K % 32 == 0, "decode_linear: K=%d must be a multiple of 32", K);
  return decode_linear(x, x_row_stride, weight, bias, out, out_row_stride, B, N, K, gated, dtype, stream);
}

extern "C" int atma_decode_linear_k8(const void* x, int64_t x_row_stride, const void* weight, const void* bias, void* out,
                                     int64_t out_row_stride, int B, int N, int K, int gated, int dtype, void* stream) {
  ATMA_REQUIRE(K >= 32 && K % 8 == 0, "decode_linear_k8: K=%d must be a multiple of 8, 32 at least", K);
  return decode_linear(x, x_row_stride, weight, bias, out, out_row_stride, B, N, K, gated, dtype, stream);
}
