// Attention of fp32 rows on the tensor cores at fp32 accuracy: 128 rows of one head x 64 keys per step, 128 channels of q and k
// (in one map, or two maps of 64), 128 of v.
//
// Every operand is the sum of two tf32 terms, x = hi + lo with hi rounded to nearest, which leaves 2^-22 of it; three products
// of terms - lo hi, hi lo, hi hi, small ones first - leave out 2^-22 of a product, with random signs.  The tensor core rounds its
// fp32 sums towards zero, which makes weights smaller together, so that next to a null key's weight they are off by more than
// fp32 arithmetic's.  So a sum stays there for 16 channels of a score (32 with two maps, where a score has 64) and for 64 keys of a
// result only; the others are made in registers.  What is
// elementwise (scores, maxima, exponentials, sums of weights) is fp32 arithmetic as in the other fp32 kernels.
// Errors of rows by the keys they see, 2-norm against 64 bits, products|64 x 64 kernels (2048 rows, 8 heads; 1e-7), and products with
// one sum for 64 channels:
//                         keys:  1       2-4     5-16    17-64   65-128  129-256 257-1024 -2048     1   2-4 -16 -64 -128 -256 -1024 -2048
//   Polar, null key             1.0|1.0 1.4|1.3 1.8|1.7 2.4|2.3 2.8|2.6 3.0|2.9 3.4|3.6  3.7|4.2    1.2 1.7 2.5 3.7 4.2  4.6  5.4  6.0
//   softmax, one map            0.4|0   1.2|1.0 1.6|1.6 2.4|2.2 2.8|2.7 2.9|3.4 3.1|5.2  3.2|7.4    0.4 1.4 2.1 3.2 3.7  3.9  4.2  4.3
//   softmax, two maps           0.8|0.7 1.3|1.3 1.6|1.8 1.9|2.5 2.1|3.3 2.2|4.1 2.4|5.9  2.6|8.5    0.8 1.6 1.8 2.2 2.5  2.6  2.9  3.0
// With one map, 64-row blocks with a row that sees fewer than 128 keys (few_keys) are for fp32 arithmetic: both blocks of a CTA, as a
// prompt's first two, are done so at once, half of the threads each, beside the other CTAs' longer walks; one alone is marked.
// A value that is infinite or no number, or results so small that their lo terms vanish, make a CTA mark 64-row blocks of its
// output (kRedo); the 64 x 64 kernels of rows_f32.cuh run behind it on marked blocks only, and decide what such values give.
//
//   warps 0-7    rows: thread = TMEM lane 32 (w % 4) + lane, half w / 4 of a step's keys and of the channels of v.  Scores out
//                of TMEM, weights back as two terms, the step's sums out of TMEM into registers
//   warps 8-11   keys: raw rows by cp.async a step ahead, then both terms of K [key][channel] and of V^T [channel][key] into
//                shared memory, K-major with 128-byte swizzle
//   warp 12      issues the products; owns the TMEM allocation (warps 13-15 fill the warpgroup)
// TMEM (512 columns): Q hi [0,128) lo [128,256) | two sums of scores [256,384), then the weights hi and lo in their place |
// the step's result [384,512), with one map the other two sums before.  With one map pairs of sums take the places in turn, the next
// pair's products under the reading of the one in front, for next to nothing; sum by sum it was 1500 clocks a step.
// A step of 64 keys takes 7800 clocks: three products at half the 16-bit rate, 1536 for the scores and 1536 for the result, with
// their waits 4000; 1400 for the weights; what is left are scores, sums and hand-overs.  TMEM is full, so the next scores wait
// for this step's result.
// Every mbarrier wait is bounded; on expiry the CTA frees its TMEM, returns and leaves a status word for the host.
#pragma once

#include "common.cuh"
#include "sm100.cuh"

namespace atma {
namespace attend_tf32 {

using namespace sm100;

constexpr int kM = 128, kN = 64, kD = 128, kThreads = 512;
constexpr int few_keys(int maps) { return maps == 1 ? kM : 0; }
constexpr uint32_t kRedo = 0x7fc0a11cu;              // a NaN that no arithmetic gives, in a block's first value
constexpr int kTerm = kN * kD * 4;                   // one term of K or V
constexpr int kOffK = 0, kOffV = 2 * kTerm, kOffRawK = 4 * kTerm, kOffRawV = 5 * kTerm, kSmemBytes = 6 * kTerm + 1024;
constexpr uint32_t kColQ = 0, kColS = 256, kColP = 256, kColO = 384;
constexpr int kRowRegs = 208, kKeyRegs = 56, kMmaRegs = 40;          // 256 x 208 + 128 x 56 + 128 x 40 = 512 x 128, as launched
static_assert(256 * kRowRegs + 128 * kKeyRegs + 128 * kMmaRegs <= kThreads * 128, "more registers than the block is launched with");

struct Shared {
  uint64_t q_ready, k_full, k_empty, v_full, v_empty, s_full[2], s_free[2], p_full, o_full, o_free;
  uint32_t tmem;
  int abort, redo[2];
  float max[2][kM], sum[2][3][kM];                   // what the two halves of a row tell each other
};

__device__ __forceinline__ void rows_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ void keys_sync() { asm volatile("bar.sync 2, 128;" ::: "memory"); }
__device__ __forceinline__ float hi_term(float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u); }
__device__ __forceinline__ void copy16(float* dst, const float* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void mma_ts_tf32(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__host__ __device__ constexpr uint32_t idesc_tf32(int N) { return (1u << 4) | (2u << 7) | (2u << 10) | (uint32_t(N >> 3) << 17) | (uint32_t(kM >> 4) << 24); }
__device__ __forceinline__ uint64_t desc(uint32_t addr) { return make_sdesc_sw128(addr, 16, 1024); }

// The CTA's first row.  Later rows have more keys, so they come first, but for the very first, which go row by row of keys (few_keys) and
// take as long as a dozen steps.
template <int M>
__device__ __forceinline__ int first_row(int heads) {
  const int tiles = gridDim.x / heads, at = blockIdx.x / heads;
  return (few_keys(M) > 0 ? (at == 0 ? 0 : tiles - at) : tiles - 1 - at) * kM;
}

// Front: what a kernel attends to.  Front(args, shared): the CTA's rows and keys, told by all threads together, ends with a barrier;
//   tiles(), key0(j)      steps and their first keys
//   has(r), few(r)        whether row r is there, and sees keys, but fewer than few_keys; plain() the CTA's rows in fp32 arithmetic
//   mark(block)           a block of 64 rows (0, 1), if it has any, to be done again
//   q_row(r), q_scale()   pointer to 128 channels of row r (0 .. 127) or null
//   k_row(key), v_row(key), or null
//   Row: row(r) with score(s), sees(key) and sees_all(first, last), without branches; start(t) and start_sum(t)
//   finish(row, r, half, m, l, q2, O, shared) = the row's half of the output; marks what has to be done again
template <typename Front, int M>
__device__ __forceinline__ void attend(Front& f, uint8_t* smem, Shared& sh, int* status) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool few = tid < kM && f.few(tid);
  const int few0 = __syncthreads_or(few && tid < kM / 2), few1 = __syncthreads_or(few && tid >= kM / 2);
  if constexpr (few_keys(M) > 0) {
    if (few0 && (few1 || !f.has(kM / 2))) {
      f.plain();
      return;
    }
  }
  if (tid == 0) {
    mbar_init(&sh.q_ready, 8); mbar_init(&sh.k_full, 4); mbar_init(&sh.k_empty, 1); mbar_init(&sh.v_full, 4); mbar_init(&sh.v_empty, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&sh.s_full[i], 1); mbar_init(&sh.s_free[i], 8); }
    mbar_init(&sh.p_full, 8); mbar_init(&sh.o_full, 1); mbar_init(&sh.o_free, 8);
    sh.abort = 0; sh.redo[0] = few0; sh.redo[1] = few1;
    fence_barrier_init();
  }
  if (warp == 12) tmem_alloc(&sh.tmem, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = sh.tmem;
  volatile int* abort_flag = &sh.abort;
  const int n_tiles = f.tiles();
  constexpr int kSum = M == 1 ? 16 : 32, kPairs = kD / M / (2 * kSum);           // channels that are summed in the tensor core; pairs of such sums

  if (warp < 8) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRowRegs));
    const int half = warp >> 2, r = 32 * (warp & 3) + lane;
    const uint32_t lane_base = tbase + (uint32_t(32 * (warp & 3)) << 16);
    const auto row = f.row(r);
    {                                                // this half's 64 channels of the row, both terms
      const float* q = f.q_row(r);
      const float scale = f.q_scale();
#pragma unroll 1
      for (int c = 0; c < 64; c += 16) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int e = 0; e < 16; e += 4) {
          const float4 x = q != nullptr ? *reinterpret_cast<const float4*>(q + 64 * half + c + e) : make_float4(0.f, 0.f, 0.f, 0.f);
          const float y[4] = {x.x * scale, x.y * scale, x.z * scale, x.w * scale};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            hi[e + i] = __float_as_uint(hi_term(y[i]));
            lo[e + i] = __float_as_uint(y[i] - __uint_as_float(hi[e + i]));
          }
        }
        tmem_st16(lane_base + kColQ + 64 * half + c, hi);
        tmem_st16(lane_base + kColQ + 128 + 64 * half + c, lo);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.q_ready);
    }
    float O[M][64], m[M], l[M], q2 = 0.f;
#pragma unroll
    for (int t = 0; t < M; ++t) {
      m[t] = row.start(t);
      l[t] = half == 0 ? row.start_sum(t) : 0.f;      // each half sums its own keys
#pragma unroll
      for (int c = 0; c < 64; ++c) O[t][c] = 0.f;
    }
    // after a wait that ran out every later one returns at once, and the warps keep walking the same barriers
    uint32_t it = 0;                                  // steps times maps
    for (int j = 0; j < n_tiles; ++j) {
      const int key0 = f.key0(j) + 32 * half;
#pragma unroll
      for (int t = 0; t < M; ++t, ++it) {
        float s[32] = {};
#pragma unroll 1
        for (int g = 0; g < kPairs; ++g) {
          mbar_wait_warp(&sh.s_full[g & 1], (kPairs > 2 ? g >> 1 : it) & 1u, abort_flag);
          tc_fence_after();
          const uint32_t at = lane_base + kColS + 128 * (g & 1) + 32 * half;
          if constexpr (M == 1) {
            uint32_t x[64];
            tmem_ld32_nowait(at, x);
            tmem_ld32_nowait(at + 64, x + 32);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 64; ++i) { reg_fence(x[i]); s[i & 31] += __uint_as_float(x[i]); }
          } else {
#pragma unroll
            for (int c = 0; c < 128; c += 64) {        // there are no registers for both
              uint32_t x[32];
              tmem_ld32(at + c, x);
#pragma unroll
              for (int i = 0; i < 32; ++i) s[i] += __uint_as_float(x[i]);
            }
          }
          if (g + 2 < kPairs) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.s_free[g & 1]);
          }
        }
        float top = -INFINITY;
#pragma unroll
        for (int i = 0; i < 32; ++i) s[i] = row.score(s[i]);
        if (!__all_sync(0xffffffffu, row.sees_all(key0, key0 + 31))) {
#pragma unroll
          for (int i = 0; i < 32; ++i) s[i] = row.sees(key0 + i) ? s[i] : -INFINITY;
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) top = fmaxf(top, s[i]);
        sh.max[half][r] = top;
        rows_sync();
        const float mn = fmaxf(m[t], fmaxf(top, sh.max[half ^ 1][r]));
        const float from = mn == -INFINITY ? 0.f : mn;
        const float al = expf(m[t] - from);           // 0 while nothing has been seen
        float sum = 0.f, sq = 0.f;
#pragma unroll
        for (int c = 0; c < 32; c += 16) {
          uint32_t hi[16], lo[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float p = expf(s[c + i] - from);
            sum += p;
            sq = fmaf(p, p, sq);
            hi[i] = __float_as_uint(hi_term(p));
            lo[i] = __float_as_uint(p - __uint_as_float(hi[i]));
          }
          tmem_st16(lane_base + kColP + 32 * half + c, hi);
          tmem_st16(lane_base + kColP + 64 + 32 * half + c, lo);
        }
        tmem_st_wait();
        tc_fence_before();
        rows_sync();                                  // the maxima are read, too
        if (lane == 0) mbar_arrive(&sh.p_full);
        l[t] = fmaf(l[t], al, sum);
        if (M == 1) q2 = fmaf(q2, al * al, sq);
        m[t] = mn;
        mbar_wait_warp(&sh.o_full, it & 1u, abort_flag);
        tc_fence_after();
        if constexpr (M == 1) {                       // the next step's second pair of sums waits for this place
          uint32_t o[64];
          tmem_ld32_nowait(lane_base + kColO + 64 * half, o);
          tmem_ld32_nowait(lane_base + kColO + 64 * half + 32, o + 32);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.o_free);
#pragma unroll
          for (int i = 0; i < 64; ++i) { reg_fence(o[i]); O[t][i] = fmaf(O[t][i], al, __uint_as_float(o[i])); }
        } else {
#pragma unroll
          for (int c = 0; c < 64; c += 16) {
            uint32_t o[16];
            tmem_ld16(lane_base + kColO + 64 * half + c, o);
#pragma unroll
            for (int i = 0; i < 16; ++i) O[t][c + i] = fmaf(O[t][c + i], al, __uint_as_float(o[i]));
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.o_free);
        }
      }
    }
    f.finish(row, r, half, m, l, q2, O, sh);
  } else if (warp < 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kKeyRegs));
    const int lw = warp - 8;
    float* raw_k = reinterpret_cast<float*>(smem + kOffRawK);
    float* raw_v = reinterpret_cast<float*>(smem + kOffRawV);
    auto fetch = [&](bool values, float* dst, int j) {
      if (j < n_tiles) {
        // a warp's rows are lw, lw + 4, ..., a lane's piece is its own; a lane finds one row for all of them
        const int at = f.key0(j) + lw + 4 * (lane & 15);
        const unsigned long long mine = reinterpret_cast<unsigned long long>(values ? f.v_row(at) : f.k_row(at));
#pragma unroll 4
        for (int i = 0; i < 16; ++i) {
          const float* src = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, mine, i));
          copy16(dst + (lw + 4 * i) * kD + 4 * lane, src != nullptr ? src + 4 * lane : f.any(), src != nullptr);
        }
      }
      copies_commit();
    };
    fetch(false, raw_k, 0);
    fetch(true, raw_v, 0);
    for (int j = 0; j < n_tiles; ++j) {
      copies_wait<1>();
      if (j > 0) mbar_wait_warp(&sh.k_empty, (uint32_t)(j - 1) & 1u, abort_flag);
#pragma unroll 4
      for (int i = 0; i < 16; ++i) {
        const int key = lw + 4 * i;
        const float4 x = *reinterpret_cast<const float4*>(raw_k + key * kD + 4 * lane);
        const float4 hi = make_float4(hi_term(x.x), hi_term(x.y), hi_term(x.z), hi_term(x.w));
        uint8_t* dst = smem + kOffK + (lane >> 3) * (kN * 128) + key * 128 + (((lane & 7) ^ (key & 7)) << 4);
        *reinterpret_cast<float4*>(dst) = hi;
        *reinterpret_cast<float4*>(dst + kTerm) = make_float4(x.x - hi.x, x.y - hi.y, x.z - hi.z, x.w - hi.w);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.k_full);
      fetch(false, raw_k, j + 1);
      copies_wait<1>();
      keys_sync();
      if (j > 0) mbar_wait_warp(&sh.v_empty, (uint32_t)(j - 1) & 1u, abort_flag);
      {
        const int d = 32 * lw + lane;
#pragma unroll 4
        for (int q = 0; q < 16; ++q) {                // four keys of a channel
          float x[4], hi[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) { x[e] = raw_v[(4 * q + e) * kD + d]; hi[e] = hi_term(x[e]); }
          uint8_t* dst = smem + kOffV + (q >> 3) * (kD * 128) + d * 128 + (((q & 7) ^ (d & 7)) << 4);
          *reinterpret_cast<float4*>(dst) = make_float4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<float4*>(dst + kTerm) = make_float4(x[0] - hi[0], x[1] - hi[1], x[2] - hi[2], x[3] - hi[3]);
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.v_full);
      keys_sync();                                    // the raw rows have been read
      fetch(true, raw_v, j + 1);
    }
    copies_wait<0>();
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kMmaRegs));
    if (warp == 12 && elect_one()) {
      const uint64_t k_desc = desc(smem_u32(smem + kOffK)), v_desc = desc(smem_u32(smem + kOffV));
      bool ok = n_tiles == 0 || mbar_wait(&sh.q_ready, 0, abort_flag);
      uint32_t it = 0;
      for (int j = 0; j < n_tiles && ok; ++j) {
        ok = mbar_wait(&sh.k_full, (uint32_t)j & 1u, abort_flag);
        for (int t = 0; t < M && ok; ++t, ++it) {
          tc_fence_after();
          for (int g = 0; g < kPairs && ok; ++g) {    // rolled: all descriptors at once would not fit this warp's registers
            // the second place is the result's: the one in front has been read
            if (g == 1 && it > 0) ok = mbar_wait(&sh.o_free, (it - 1) & 1u, abort_flag);
            if (g > 1) ok = mbar_wait(&sh.s_free[g & 1], it & 1u, abort_flag);
            if (!ok) break;
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
              // few instructions between products: 32 clocks each, and with descriptors made for every one the issue took twice that
              const int step = ((t * kPairs + g) * 2 + c) * (kSum / 8);
              const uint32_t d = tbase + kColS + 128 * (g & 1) + 64 * c, qa = tbase + kColQ + 8 * step;
              const uint64_t kd = k_desc + uint64_t(((step >> 2) * (kN * 128) + (step & 3) * 32) >> 4);
#pragma unroll
              for (int term = 0; term < 3; ++term)
#pragma unroll
                for (int k = 0; k < kSum / 8; ++k)
                  mma_ts_tf32(d, qa + (term == 0 ? 128 : 0) + 8 * k, kd + uint64_t(((term == 1 ? kTerm : 0) + 32 * k) >> 4), idesc_tf32(kN), (term > 0 || k > 0) ? 1u : 0u);
            }
            tc_commit(&sh.s_full[g & 1]);
          }
          if (!ok) break;
          if (t == M - 1) tc_commit(&sh.k_empty);
          ok = mbar_wait(&sh.p_full, it & 1u, abort_flag) && mbar_wait(&sh.v_full, (uint32_t)j & 1u, abort_flag) &&
               (kPairs > 1 || it == 0 || mbar_wait(&sh.o_free, (it - 1) & 1u, abort_flag));
          if (!ok) break;
          tc_fence_after();
#pragma unroll 1
          for (int term = 0; term < 3; ++term) {
            const uint32_t pa = tbase + kColP + (term == 0 ? 64 : 0);
            const uint64_t vd = v_desc + uint64_t((term == 1 ? kTerm : 0) >> 4);
#pragma unroll
            for (int k = 0; k < 8; ++k)
              mma_ts_tf32(tbase + kColO, pa + 8 * k, vd + uint64_t(((k >> 2) * (kD * 128) + (k & 3) * 32) >> 4), idesc_tf32(kD), (term > 0 || k > 0) ? 1u : 0u);
          }
          tc_commit(&sh.o_full);
          if (t == M - 1) tc_commit(&sh.v_empty);
        }
      }
    }
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && sh.abort) atomicExch(status, 1);
  if (warp == 12) tmem_dealloc(tbase, 512);
}

// Whether a row's half can be trusted: finite everywhere, and not so small that lo terms are lost (a row of zeros is).
__device__ __forceinline__ bool trusted(const float (&o)[64], float l) {
  float most = 0.f;
  bool finite = l < INFINITY;
#pragma unroll
  for (int c = 0; c < 64; ++c) {
    most = fmaxf(most, fabsf(o[c]));
    finite = finite && fabsf(o[c]) < INFINITY;
  }
  return finite && (most == 0.f || most > 1e-28f);
}

}  // namespace attend_tf32
}  // namespace atma
