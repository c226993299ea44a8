// Pieces of the fp32 attention kernels that hold 64 query rows and 64 keys per step: 256 threads, thread (ty, tx) = 16 x 16
// owns rows 4 ty .. + 3 with keys tx + 16 j for the scores and channels 64 m + 4 tx .. + 3 for the weighted sum.  A row's 16
// threads are one half of a warp, so its statistics are four shuffles and its weights pass through shared memory without a
// barrier.  Per four channels of the scores a warp reads 12 lines of shared memory for 64 FMAs (in pairs, f32x2, where
// registers allow), per four keys of the sum 20 for 128 in pairs.
#pragma once

#include "common.cuh"
#include "f32x2.cuh"

namespace atma {
namespace rows_f32 {

constexpr int kM = 64, kN = 64, kThreads = 256;
constexpr int kLdP = kN + 4;
constexpr int kPad = 4;                     // floats behind a row of Q or K: rows 8 apart meet no bank twice

__device__ __forceinline__ void copy16(float* dst, const float* src, bool there) {      // zeros where there is nothing
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
               ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(there ? 16 : 0) : "memory");
}
// The 256 threads of a block of 64 rows: of a CTA, or (kOf 2) half of a CTA that has two blocks.
template <int kOf>
__device__ __forceinline__ void block_sync() {
  if constexpr (kOf == 1) __syncthreads();
  else asm volatile("bar.sync %0, 256;" ::"r"(1 + (int)(threadIdx.x >> 8)) : "memory");
}
template <int kOf>
__device__ __forceinline__ void copies_done() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  block_sync<kOf>();
}

// s[i][j] = row 4 ty + i times key tx + 16 j over n4 quadruples of channels.  PAIRS: even and odd channels in sums of their own,
// for kernels that have the registers.
template <bool PAIRS>
__device__ __forceinline__ void dots(const float* q, const float* k, int ld, int n4, int ty, int tx, float (&s)[4][4]) {
  const float *qr = q + 4 * ty * ld, *kr = k + tx * ld;
  if constexpr (PAIRS) {
    uint64_t t[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) t[i][j] = 0;
#pragma unroll 2
    for (int c = 0; c < n4; ++c) {
      ulonglong2 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(kr + 16 * j * ld + 4 * c);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(qr + i * ld + 4 * c);
#pragma unroll
        for (int j = 0; j < 4; ++j) t[i][j] = fma2(a.y, b[j].y, fma2(a.x, b[j].x, t[i][j]));
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack2(t[i][j]);
        s[i][j] = f.x + f.y;
      }
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 2
  for (int c = 0; c < n4; ++c) {
    float4 b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(kr + 16 * j * ld + 4 * c);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 a = *reinterpret_cast<const float4*>(qr + i * ld + 4 * c);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        s[i][j] = fmaf(a.w, b[j].w, fmaf(a.z, b[j].z, fmaf(a.y, b[j].y, fmaf(a.x, b[j].x, s[i][j]))));
    }
  }
}

// acc[i][.] += sum over keys j0 .. j1 - 1 of p[4 ty + i][j] v[j][.].  Every row of the warp sees the keys from f0 to f1 - 1 (f0 a
// multiple of 4 if there are four of them); for the others sees(i, j) tells, and a value that a row does not see stays out of
// its sums, be it infinite or no number at all.  Edges are short, so their keys go one by one.
template <int VM, typename Sees>
__device__ __forceinline__ void weigh(const float* p, const float* v, int ty, int tx, int j0, int j1, int f0, int f1, Sees sees,
                                      uint64_t (&acc)[4][2 * VM]) {
  const float* pr = p + 4 * ty * kLdP;
  auto add = [&](int i, float f, const ulonglong2 (&x)[VM]) {
    const uint64_t ff = pack2(f, f);
#pragma unroll
    for (int m = 0; m < VM; ++m) {
      acc[i][2 * m] = fma2(x[m].x, ff, acc[i][2 * m]);
      acc[i][2 * m + 1] = fma2(x[m].y, ff, acc[i][2 * m + 1]);
    }
  };
  auto edge = [&](int from, int to) {
#pragma unroll 1
    for (int j = from; j < to; ++j) {
      ulonglong2 x[VM];
#pragma unroll
      for (int m = 0; m < VM; ++m) x[m] = *reinterpret_cast<const ulonglong2*>(v + j * 64 * VM + 64 * m + 4 * tx);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (sees(i, j)) add(i, pr[i * kLdP + j], x);
    }
  };
  f0 = min(max(f0, j0), j1);
  f1 = f0 + max(min(f1, j1) - f0, 0) / 4 * 4;
  edge(j0, f0);
#pragma unroll 1
  for (int j = f0; j < f1; j += 4) {
    float4 w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(pr + i * kLdP + j);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      ulonglong2 x[VM];
#pragma unroll
      for (int m = 0; m < VM; ++m) x[m] = *reinterpret_cast<const ulonglong2*>(v + (j + e) * 64 * VM + 64 * m + 4 * tx);
#pragma unroll
      for (int i = 0; i < 4; ++i) add(i, e == 0 ? w[i].x : (e == 1 ? w[i].y : (e == 2 ? w[i].z : w[i].w)), x);
    }
  }
  edge(f1, j1);
}

// over the 16 threads of a row
__device__ __forceinline__ float row_max(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int VM>
__device__ __forceinline__ void times(uint64_t (&acc)[2 * VM], float f) {
  const uint64_t ff = pack2(f, f);
#pragma unroll
  for (int c = 0; c < 2 * VM; ++c) acc[c] = mul2(acc[c], ff);
}

// channel 64 m + 4 tx + e of a row's sums is at(acc, 4 m + e)
template <int VM>
__device__ __forceinline__ float at(const uint64_t (&acc)[2 * VM], int i) {
  const float2 f = unpack2(acc[i >> 1]);
  return i & 1 ? f.y : f.x;
}

}  // namespace rows_f32
}  // namespace atma
