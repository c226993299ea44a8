// Gated-delta scan, the chunk-local (state-independent) stage, on the 5th-generation tensor cores
// (sm_100a): K and Q tiles by TMA, the Gram matrices on tcgen05.mma with TMEM accumulators,
// the 64 x 64 unit-lower-triangular inverse per chunk in fp32 / tf32 by the worker warps.
//
// A persistent CTA walks over tiles of TWO 64-token chunks of one head (128 rows, rows 0-63 = the
// first chunk, 64-127 = the second; the two chunks only share the MMA shapes, every product that
// couples them is masked).  Per tile, with g the inclusive decay prefix inside a chunk, k^ and q^
// the L2-normalised rows:
//
//   MMA    Gkk = K K^T,  Gqk = Q K^T                               128 x 128 x 128 each (SS)
//   warps  A[p][s] = beta_p (g_p/g_s) k^_p.k^_s  (s < p)           fp32, shared memory
//          Rq[p][s] = (g_p/g_s) q^_p.k^_s        (s <= p)          -> record
//          T = (I + A)^-1: 16 x 16 diagonal blocks by substitution (fp32), then the blocks below
//          the diagonal level by level with mma.sync tf32 (G_il = -T_ii A_il; T_ij = sum_l G_il T_lj)
//          Tw[p][s] = -T[p][s] beta_s g_s k_inv_s,  Tu[p][s] = T[p][s] beta_s    -> record
//          (fp16: k_inv without a power of two, see gated_delta_scan.cuh)
//
// The row scalings of the right-hand sides are in the columns of T, so that the recurrence multiplies
// Tw and Tu with the K and V rows as they are.
// What bounds it is the serial chain of a tile's thread phases (Gram rows, substitution, four levels of
// blocks), so two CTAs share an SM: T takes the place of the K and Q tiles, which are dead once the Gram
// matrices are there (98 KB).  8 sequences of 16384 tokens, 8 heads: 330 us (0.75 GB
// moved); one CTA per SM that also made W and U0 and wrote 72 KB a chunk took 617 us.
//
//   warp 0      TMA producer        warp 1      MMA issuer; owns the TMEM allocation
//   warps 2-9   workers; warp w works on TMEM lanes / tile rows 32 (w % 4) .. +31 and on column
//               half (w - 2) / 4 of whatever it reads
// TMEM (256 columns): Gkk [0,128) Gqk [128,256).
// Every mbarrier wait is bounded; on expiry the CTA frees its TMEM, returns and leaves a status
// word for the host.
#include "common.cuh"
#include "sm100.cuh"
#include "gated_delta_scan.cuh"

namespace atma {

using namespace sm100;
using namespace scan;

namespace {

__device__ int g_local_status = 0;

constexpr int kThreads = 320;                     // TMA warp, MMA warp, eight worker warps
constexpr int kTile = 2 * kD * 128;               // a [128][128] 16-bit tile = two 64-column boxes of 16 KiB
constexpr int kLd = 68;                           // fp32 row stride of the A and T matrices
constexpr int kMat = 128 * kLd * 4;
// T over the K tile (and 2 KiB of Q); the Rq rows on their way to the record behind it
constexpr int kOffK = 0, kOffQ = kTile, kOffTf = 0, kOffRq = 40960, kOffAf = 2 * kTile, kSmemBytes = kOffAf + kMat + 1024;
static_assert(kMat <= kOffRq && kOffRq + 16384 <= kOffAf, "T and Rq lie over the K and Q tiles");

constexpr uint32_t kColKK = 0, kColQK = 128;

struct Barriers { uint64_t kq_full, g_done, tile_free; };

struct Meta { int64_t t0[2]; int rows[2]; int64_t rec[2]; int h, hk; };

struct Params {
  const float* g; const float* beta;
  uint8_t* recs; float* scal;
  int Tlen, H, Hkv, NC, B, normalize;
  float scale;
  int n_pairs; int64_t n_tiles;
  VarLen var;
};

// 1 / |k| of fp16 rows (2^-20 to 2^24, or there is no row) as a factor from 1/2 to 1 and the product of two powers of two
__device__ __forceinline__ float without_pow2(float x, __half2& pow2) {
  const uint32_t b = __float_as_uint(x);
  const int e = (int)(b >> 23) - 126;
  if (e < -24 || e > 26) { pow2 = __float2half2_rn(0.f); return 0.f; }
  pow2 = __floats2half2_rn(__int_as_float((127 + (e >> 1)) << 23), __int_as_float((127 + e - (e >> 1)) << 23));
  return __uint_as_float((b & 0x007fffffu) | 0x3f000000u);
}

__device__ __forceinline__ void worker_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// acc (16 x 16 as two 8-column tiles) += A (16 x 16, row-major, stride kLd) * B (16 x 16, row-major, stride kLd)
__device__ __forceinline__ void block_mma(float (&acc)[2][4], const float* A, const float* Bm, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) {
    uint32_t a[4];
    a[0] = __float_as_uint(A[g * kLd + 8 * ks + t]);
    a[1] = __float_as_uint(A[(g + 8) * kLd + 8 * ks + t]);
    a[2] = __float_as_uint(A[g * kLd + 8 * ks + t + 4]);
    a[3] = __float_as_uint(A[(g + 8) * kLd + 8 * ks + t + 4]);
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
      mma_tf32(acc[nt], a, __float_as_uint(Bm[(8 * ks + t) * kLd + 8 * nt + g]), __float_as_uint(Bm[(8 * ks + t + 4) * kLd + 8 * nt + g]));
  }
}
__device__ __forceinline__ void block_store(float* C, const float (&acc)[2][4], int lane, float sign) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    *reinterpret_cast<float2*>(C + g * kLd + 8 * nt + 2 * t) = make_float2(sign * acc[nt][0], sign * acc[nt][1]);
    *reinterpret_cast<float2*>(C + (g + 8) * kLd + 8 * nt + 2 * t) = make_float2(sign * acc[nt][2], sign * acc[nt][3]);
  }
}

__device__ __forceinline__ void tile_meta(const Params& p, int64_t tile, Meta& m) {
  m.h = (int)(tile % p.H);
  m.hk = m.h / (p.H / p.Hkv);
  const int64_t rest = tile / p.H;
  const int j = (int)(rest % p.n_pairs);
  const int b = (int)(rest / p.n_pairs);
#pragma unroll
  for (int ci = 0; ci < 2; ++ci) {
    const int c = 2 * j + ci;
    m.t0[ci] = 0; m.rows[ci] = 0; m.rec[ci] = -1;
    if (p.var.cu_seqlens != nullptr) {
      const int total = p.var.cu_chunks[p.var.n_seqs];
      if (c < total) {
        int lo = 0, hi = p.var.n_seqs;                // largest s with cu_chunks[s] <= c
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (p.var.cu_chunks[mid] <= c) lo = mid; else hi = mid;
        }
        m.t0[ci] = (int64_t)p.var.cu_seqlens[lo] + (int64_t)(c - p.var.cu_chunks[lo]) * kC;
        m.rows[ci] = (int)min((int64_t)kC, (int64_t)p.var.cu_seqlens[lo + 1] - m.t0[ci]);
        m.rec[ci] = (int64_t)m.h * p.NC + c;
      }
    } else if (c < p.NC) {
      m.t0[ci] = (int64_t)b * p.Tlen + (int64_t)c * kC;
      m.rows[ci] = min(kC, p.Tlen - c * kC);
      m.rec[ci] = ((int64_t)b * p.H + m.h) * p.NC + c;
    }
  }
}

template <bool kBf16>
__global__ void __launch_bounds__(kThreads, 2)
scan_local_sm100_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* Ks = smem + kOffK;
  uint8_t* Qs = smem + kOffQ;
  uint8_t* Rqs = smem + kOffRq;
  float* Af = reinterpret_cast<float*>(smem + kOffAf);
  float* Tf = reinterpret_cast<float*>(smem + kOffTf);
  __shared__ Barriers bar;
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  __shared__ float s_lg[128], s_bt[128], s_kinv[128], s_qinv[128], s_wsc[128], s_wsum[4];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(&bar.kq_full, 1); mbar_init(&bar.g_done, 1); mbar_init(&bar.tile_free, 8);
    s_abort = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(&s_tmem_base, 256);
  if (warp == 0 && lane == 0) { prefetch_tensormap(&tmap_q); prefetch_tensormap(&tmap_k); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = s_tmem_base;
  volatile int* abort_flag = &s_abort;

  if (warp == 0) {
    // =============================== TMA producer ================================================
    if (elect_one()) {
      uint32_t it = 0;
      for (int64_t tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x, ++it) {
        if (it > 0 && !mbar_wait(&bar.tile_free, (it - 1) & 1u, abort_flag)) break;
        Meta m;
        tile_meta(p, tile, m);
        mbar_arrive_expect_tx(&bar.kq_full, 2 * kTile);
#pragma unroll
        for (int ci = 0; ci < 2; ++ci)
#pragma unroll
          for (int cb = 0; cb < 2; ++cb) {
            tma_load_4d(Ks + cb * 16384 + ci * 8192, &tmap_k, &bar.kq_full, cb * 64, m.hk, (int)m.t0[ci], 0);
            tma_load_4d(Qs + cb * 16384 + ci * 8192, &tmap_q, &bar.kq_full, cb * 64, m.h, (int)m.t0[ci], 0);
          }
        // the tiles' place is taken until the end of this one; meanwhile the next inputs come into L2
        if (tile + gridDim.x < p.n_tiles) {
          Meta mn;
          tile_meta(p, tile + gridDim.x, mn);
#pragma unroll
          for (int ci = 0; ci < 2; ++ci)
#pragma unroll
            for (int cb = 0; cb < 2; ++cb) {
              tma_prefetch_l2_4d(&tmap_k, cb * 64, mn.hk, (int)mn.t0[ci], 0);
              tma_prefetch_l2_4d(&tmap_q, cb * 64, mn.h, (int)mn.t0[ci], 0);
            }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // =============================== MMA issuer =================================================
    if (elect_one()) {
      constexpr uint32_t idesc_kk = make_idesc(128, 128, kBf16 ? 1 : 0, 0, 0);     // both operands K-major
      const uint64_t hi_k = (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61) | (uint64_t(16 >> 4) << 16);
      const uint64_t kd = hi_k | uint64_t((smem_u32(Ks) >> 4) & 0x3FFFu), qd = hi_k | uint64_t((smem_u32(Qs) >> 4) & 0x3FFFu);
      uint32_t it = 0;
      for (int64_t tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x, ++it) {
        if (!mbar_wait(&bar.kq_full, it & 1u, abort_flag)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint64_t off = uint64_t(((kk >> 2) * 16384 + (kk & 3) * 32) >> 4);
          mma_ss(tbase + kColKK, kd + off, kd + off, idesc_kk, kk > 0);
        }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint64_t off = uint64_t(((kk >> 2) * 16384 + (kk & 3) * 32) >> 4);
          mma_ss(tbase + kColQK, qd + off, kd + off, idesc_kk, kk > 0);
        }
        tc_commit(&bar.g_done);
      }
    }
  } else {
    // =============================== workers ====================================================
    const int wtid = tid - 64;
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const int row = 32 * quad + lane;                  // tile row p (and TMEM lane)
    const int ci = row >> 6, pr = row & 63;            // chunk of the tile, row inside the chunk
    const uint32_t lane_base = tbase + (uint32_t(32 * quad) << 16);
    uint32_t it = 0;
    // the tile's coordinates, and g and beta of this thread's row (first column half only), are
    // fetched one tile ahead
    Meta m_next{};
    float g_pre = 0.f, b_pre = 0.f;
    auto prefetch_tile = [&](int64_t tile) {
      if (tile < p.n_tiles) {
        tile_meta(p, tile, m_next);
        if (half == 0) {
          const bool v = pr < (ci ? m_next.rows[1] : m_next.rows[0]);
          const int64_t gi = ((ci ? m_next.t0[1] : m_next.t0[0]) + pr) * p.H + m_next.h;
          g_pre = v ? p.g[gi] : 0.f;
          b_pre = v ? p.beta[gi] : 0.f;
        }
      }
    };
    prefetch_tile(blockIdx.x);
    for (int64_t tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x, ++it) {
      const Meta m = m_next;
      const bool valid = pr < (ci ? m.rows[1] : m.rows[0]);
      const int64_t rec = ci ? m.rec[1] : m.rec[0];

      // ---- decay prefix and beta: one row per thread of the first column half ---------------------
      float run = g_pre;
      if (half == 0) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const float up = __shfl_up_sync(0xffffffffu, run, o);
          if (lane >= o) run += up;
        }
      }
      worker_sync();                                     // every warp is done with the previous tile's arrays
      if (half == 0) {
        s_bt[row] = b_pre;
        if (lane == 31) s_wsum[quad] = run;
      }
      mbar_wait(&bar.kq_full, it & 1u, abort_flag);      // after a timeout every later wait returns at once; the warps keep
                                                         // walking the same barriers
      // ---- row norms: K by the first column half, Q by the second ------------------------------------
      {
        const uint8_t* src = half ? Qs : Ks;
        float sum[2] = {0.f, 0.f};
#pragma unroll
        for (int ch = 0; ch < 8; ++ch)
#pragma unroll
          for (int cb = 0; cb < 2; ++cb) {
            const uint4 u = *reinterpret_cast<const uint4*>(src + cb * 16384 + box_off(row, ch));
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 f = unpack2<kBf16>(w[e]);
              sum[cb] = fmaf(f.x, f.x, fmaf(f.y, f.y, sum[cb]));
            }
          }
        const float inv = p.normalize ? 1.0f / fmaxf(sqrtf(sum[0] + sum[1]), 1e-12f) : 1.0f;
        // rows behind the sequence's end are another's, or nothing: whatever they hold, their factors are zero
        if (half) s_qinv[row] = valid ? inv * p.scale : 0.f; else s_kinv[row] = valid ? inv : 0.f;
      }
      worker_sync();
      float k_left = s_kinv[row];                        // what Tw and the scalars have of k_inv, and what the K rows get
      __half2 k_pow2 = __float2half2_rn(1.f);
      bool far = false;
      if constexpr (!kBf16) {
        auto beyond = [](float x) { return x > 1.0078125f || (x > 0.f && x < 0.015625f); };
        far = __any_sync(0xffffffffu, p.normalize && (beyond(k_left) || beyond(s_kinv[row ^ 32])));       // of the chunk
        if (far) k_left = without_pow2(k_left, k_pow2);
      }
      if (half == 0) {
        if (quad & 1) run += s_wsum[quad - 1];           // second warp of the chunk
        s_lg[row] = run;
        s_wsc[row] = -s_bt[row] * __expf(run) * k_left;  // column scale of Tw
      }
      worker_sync();
      const float lg_p = s_lg[row], bt_p = s_bt[row], lg_C = s_lg[64 * ci + 63], kinv_p = s_kinv[row], qinv_p = s_qinv[row];
      if (half == 0 && rec >= 0) {
        float* sc = p.scal + rec * kScal;
        sc[kScalQ + pr] = valid ? __expf(lg_p) * qinv_p : 0.f;
        sc[kScalK + pr] = valid ? __expf(lg_C - lg_p) * k_left : 0.f;
        if (far) reinterpret_cast<__half2*>(sc)[kScalP + pr] = k_pow2;
        if (pr == kC - 1) { sc[kScalG] = __expf(run); sc[kScalFar] = far; }
      }

      // ---- A (fp32, shared memory) and Rq (record) from the Gram matrices -------------------------------
      mbar_wait(&bar.g_done, it & 1u, abort_flag);
      __syncwarp();
      tc_fence_after();
      {
        uint32_t rq[16];
        const int own = valid, sees = valid ? pr : 0;    // columns s < sees, and s = pr if the row is the sequence's
        // rows 0-31 of a chunk see no column of its second half: that warp only writes zeros
        if (half == 1 && (quad & 1) == 0) {
#pragma unroll
          for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(Af + row * kLd + 32 + j) = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int j = 0; j < 16; ++j) rq[j] = 0u;
        } else {
          uint32_t gk[32], gq[32];
          tmem_ld32_nowait(lane_base + kColKK + 64 * ci + 32 * half, gk);
          tmem_ld32_nowait(lane_base + kColQK + 64 * ci + 32 * half, gq);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            float a2[2], r2[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              reg_fence(gk[j + e]); reg_fence(gq[j + e]);
              const int s = 32 * half + j + e;
              const float dec = __expf(lg_p - s_lg[64 * ci + s]) * s_kinv[64 * ci + s];
              a2[e] = (s < sees) ? bt_p * dec * kinv_p * __uint_as_float(gk[j + e]) : 0.f;
              r2[e] = (s < sees + own) ? dec * qinv_p * __uint_as_float(gq[j + e]) : 0.f;
            }
            *reinterpret_cast<float2*>(Af + row * kLd + 32 * half + j) = make_float2(a2[0], a2[1]);
            rq[j >> 1] = pack2<kBf16>(r2[0], r2[1]);
          }
        }
        // the Q tile is dead: [128 rows][8 chunks of 16 bytes], chunk index xor (row & 7)
#pragma unroll
        for (int c4 = 0; c4 < 4; ++c4)
          *reinterpret_cast<uint4*>(Rqs + box_off(row, 4 * half + c4)) = make_uint4(rq[4 * c4], rq[4 * c4 + 1], rq[4 * c4 + 2], rq[4 * c4 + 3]);
      }
      tc_fence_before();
      worker_sync();
#pragma unroll
      for (int i = 0; i < 4; ++i) {                      // 16 KiB out, 512 contiguous bytes per warp instruction
        const int idx = wtid + 256 * i, r = idx >> 3, ch = idx & 7;
        const int64_t to = (r >> 6) ? m.rec[1] : m.rec[0];
        if (to >= 0)
          *reinterpret_cast<uint4*>(p.recs + to * (int64_t)kRecBytes + kRecRq + (r & 63) * 128 + ch * 16) =
              *reinterpret_cast<const uint4*>(Rqs + box_off(r, ch));
      }

      // ---- T = (I + A)^-1 per chunk: diagonal 16 x 16 blocks by substitution ----------------------------
      if (wtid < 128) {
        const int cc = wtid >> 6, blk = (wtid >> 4) & 3, j = wtid & 15;
        const float* Ab = Af + (64 * cc + 16 * blk) * kLd + 16 * blk;
        float* Tb = Tf + (64 * cc + 16 * blk) * kLd + 16 * blk;
        float x[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          float acc = (r == j) ? 1.f : 0.f;
#pragma unroll
          for (int s = 0; s < r; ++s) acc = fmaf(-Ab[r * kLd + s], x[s], acc);
          x[r] = acc;
          Tb[r * kLd + j] = acc;
        }
      }
      worker_sync();
      // G_il = -T_ii A_il for the six blocks below the diagonal of each chunk (in place over A_il)
      for (int blk = warp - 2; blk < 12; blk += 8) {
        const int cc = blk / 6, e = blk % 6;
        const int bi = (e == 0) ? 1 : (e < 3 ? 2 : 3), bl = (e == 0) ? 0 : (e < 3 ? e - 1 : e - 3);
        float acc[2][4] = {};
        float* Ail = Af + (64 * cc + 16 * bi) * kLd + 16 * bl;
        block_mma(acc, Tf + (64 * cc + 16 * bi) * kLd + 16 * bi, Ail, lane);
        __syncwarp();
        block_store(Ail, acc, lane, -1.f);
      }
      worker_sync();
      // T_ij = sum_{l=j}^{i-1} G_il T_lj, one level of blocks below the diagonal at a time
#pragma unroll 1
      for (int d = 1; d <= 3; ++d) {
        const int per = 4 - d;                          // blocks of this level per chunk
        for (int blk = warp - 2; blk < 2 * per; blk += 8) {
          const int cc = blk / per, bj = blk % per, bi = bj + d;
          float acc[2][4] = {};
          for (int l = bj; l < bi; ++l)
            block_mma(acc, Af + (64 * cc + 16 * bi) * kLd + 16 * l, Tf + (64 * cc + 16 * l) * kLd + 16 * bj, lane);
          block_store(Tf + (64 * cc + 16 * bi) * kLd + 16 * bj, acc, lane, 1.f);
        }
        worker_sync();
      }
      prefetch_tile(tile + gridDim.x);

      // ---- Tw and Tu -> record: eight threads per 128-byte row ------------------------------------------------
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int idx = wtid + 256 * i, r = idx >> 3, ch = idx & 7, rp = r & 63, c0 = 64 * (r >> 6) + 8 * ch;
        const int64_t to = (r >> 6) ? m.rec[1] : m.rec[0];
        uint32_t w4[4] = {}, u4[4] = {};
        if ((ch >> 1) <= (rp >> 4)) {                    // blocks above the diagonal are not there
          float t[8], wsc[8], bt[8];
#pragma unroll
          for (int e = 0; e < 8; e += 4) {
            *reinterpret_cast<float4*>(t + e) = *reinterpret_cast<const float4*>(Tf + r * kLd + 8 * ch + e);
            *reinterpret_cast<float4*>(wsc + e) = *reinterpret_cast<const float4*>(s_wsc + c0 + e);
            *reinterpret_cast<float4*>(bt + e) = *reinterpret_cast<const float4*>(s_bt + c0 + e);
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) t[e] = 8 * ch + e <= rp ? t[e] : 0.f;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            w4[e] = pack2<kBf16>(t[2 * e] * wsc[2 * e], t[2 * e + 1] * wsc[2 * e + 1]);
            u4[e] = pack2<kBf16>(t[2 * e] * bt[2 * e], t[2 * e + 1] * bt[2 * e + 1]);
          }
        }
        if (to >= 0) {
          uint8_t* dst = p.recs + to * (int64_t)kRecBytes + rp * 128 + ch * 16;
          *reinterpret_cast<uint4*>(dst + kRecTw) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
          *reinterpret_cast<uint4*>(dst + kRecTu) = make_uint4(u4[0], u4[1], u4[2], u4[3]);
        }
      }
      fence_proxy_async();                               // the next tile's TMA writes over T and Rq
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.tile_free);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0 && s_abort) atomicExch(&g_local_status, 1);
  if (warp == 1) tmem_dealloc(tbase, 256);
}

}  // namespace

int make_rows_map(CUtensorMap* out, const void* base, int is_bf16, int heads, int64_t tokens) {
  const uint64_t dims[4] = {128, (uint64_t)heads, (uint64_t)tokens, 1};
  const int64_t strides[3] = {128, (int64_t)heads * 128, (int64_t)heads * 128 * tokens};
  const uint32_t box[4] = {64, 1, 64, 1};
  return make_tmap_16bit_4d(out, base, is_bf16, dims, strides, box);
}

int gated_delta_local_sm100(const Rows& rows, const float* g, const float* beta, uint8_t* recs, float* scal, int B, int Tlen, int NC,
                            int normalize_qk, float scale, const VarLen& var, cudaStream_t st) {
  if (NC <= 0 || rows.tokens <= 0) return ATMA_OK;
  if (rows.tokens >= (int64_t(1) << 31)) return fail(ATMA_ERR_INVALID, "gated_delta_scan: %lld tokens exceed the tensor-map range", (long long)rows.tokens);
  CUtensorMap mq, mk;
  int rc = make_rows_map(&mq, rows.q, rows.is_bf16, rows.H, rows.tokens);
  if (rc == ATMA_OK) rc = make_rows_map(&mk, rows.k, rows.is_bf16, rows.Hkv, rows.tokens);
  if (rc != ATMA_OK) return rc;
  Params p{};
  p.g = g; p.beta = beta; p.recs = recs; p.scal = scal;
  p.Tlen = Tlen; p.H = rows.H; p.Hkv = rows.Hkv; p.NC = NC; p.B = B; p.normalize = normalize_qk; p.scale = scale;
  p.n_pairs = (NC + 1) / 2;
  p.n_tiles = (int64_t)(var.cu_seqlens != nullptr ? 1 : B) * p.n_pairs * p.H;
  p.var = var;
  const int sms = sm_count_of_current_device();
  const int grid = (int)(p.n_tiles < 2 * sms ? p.n_tiles : 2 * sms);
  auto kernel = rows.is_bf16 ? scan_local_sm100_kernel<true> : scan_local_sm100_kernel<false>;
  ATMA_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
  kernel<<<grid, kThreads, kSmemBytes, st>>>(mq, mk, p);
  return launch_status("gated_delta_scan (chunk-local, tcgen05)");
}

int scan_local_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  ATMA_CUDA_OK(cudaMemcpyFromSymbol(&v, g_local_status, sizeof(int)));
  if (v != 0) ATMA_CUDA_OK(cudaMemcpyToSymbol(g_local_status, &zero, sizeof(int)));
  *out = v;
  return ATMA_OK;
}

}  // namespace atma
