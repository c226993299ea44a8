// The gated delta rule over packed prompt rows on the 5th-generation tensor cores (sm_100a), 64 rows a chunk, at fp32
// accuracy: whatever stands between the 16-bit q, k, v and the fp32 state enters the 16-bit products as two terms
// (rounded value and remainder), and everything that is a scalar per row - unit-norm factors, decays, step sizes - is
// applied to fp32 accumulators instead of to 16-bit operands.
//
// With S the state before a chunk, a_s the inclusive decay prefix inside it, k^ = k k_inv, q^ = q q_inv:
//
//   R_s = v_s - a_s k_inv_s (S^T k_s)                                 residual against the old state
//   U   = M1 R,          M1 = (I + A)^-1 diag(beta),  A[p][s] = beta_p (a_p / a_s) k^_p.k^_s   (s < p)
//   O_p = a_p q_inv_p (S^T q_p) + (M2 R)_p,   M2 = Rq M1,  Rq[p][s] = (a_p / a_s) q^_p.k^_s    (s <= p)
//   S'  = a_C S + sum_s (a_C / a_s) k_inv_s k_s u_s^T
//
// factors (delta_factors_kernel): M1, M2 and the row scalars of every chunk and head, side by side.  A persistent CTA
//   takes two chunks of a head as one 128-row tile: Gram matrices K K^T and Q K^T by tcgen05.mma (exact products of the
//   16-bit rows), A and Rq in fp32, the inverse by 16 x 16 blocks - substitution on the diagonal, mma.sync tf32 with
//   split operands below it - and M2 the same way.  Two CTAs share an SM, so one's serial chain runs under the other's.
// recurrence (delta_recur_kernel): one CTA per (sequence, head, 128 value channels) holds S^T in fp32 registers and walks
//   the chunks.  v is on the 128 TMEM lanes of every accumulator; the A operands S^T, R^T, U^T sit in TMEM as two 16-bit
//   terms, the B operands are the K and Q rows exactly as TMA delivers them and M1, M2 as two terms.  Issue order per
//   chunk: P = S^T K^T | first half of S^T Q^T | U^T = R^T M1^T | second half of S^T Q^T | dS^T = U^T K | R^T M2^T, so that
//   the products the next step does not wait for run under the thread phases.  Few long sequences are cut into segments that
//   are walked side by side (plan_kernel, delta_compose_kernel).
//     warp 0 TMA producer (two stages), warp 1 MMA issuer, warps 2-17 state warps (TMEM lanes 32 (warp % 4) .. + 31, column
//     quarter (warp - 2) / 4); what a thread phase reads from shared memory is fetched while the product before it runs.
//     TMEM: S hi/lo [0,128) | P, U [128,192) | dS [192,320) | R hi/lo [320,384) | U hi/lo, then R M2 [384,448) | S Q [448,512)
// Every mbarrier wait is bounded; on expiry a CTA frees its TMEM, returns and leaves a status word for the host.
#include "delta_rule.cuh"
#include "mma_sync.cuh"
#include "sm100.cuh"

namespace atma {

using namespace sm100;

namespace {

__device__ int g_delta_status = 0;

constexpr int kC = 64, kD = 128;
constexpr int kRecBytes = 4 * kC * kC * 2;          // M1 hi, M2 hi, M1 lo, M2 lo: [64 p][64 s] 16-bit each
constexpr int kScal = 256;                          // floats per record: a k_inv [64] | a q_inv [64] | (a_C/a) k_inv [64] | a_C
constexpr int kThreads = 320;

// One walk of the recurrence over chunks [first, last) of a sequence, for every head and block of 128 value channels.
// Planes are [head and block][128 k][128 v] fp32 in the scratch; -1 = none.
enum { kWalk = 0, kOffset = 1, kTransfer = 2 };     // from the true state, with outputs | from zero | from the identity with v = 0
struct Item {
  int seq, first, last, kind;
  int from;                                          // plane of the state before (kWalk; -1 = the state table or zero)
  int to;                                            // plane of the state after (-1 = the state table where `last` ends the sequence)
  int middle, at;                                    // plane of the state before chunk `at` (kOffset, kTransfer)
};
// A cut (a segment's first chunk that is not its sequence's) e owns planes 6 e ..: the true state before it and in its
// middle, its offset and transfer to its end, its offset and transfer to its middle.
enum { kPlaneState = 0, kPlaneMiddle = 1, kPlaneOffset = 2, kPlaneTransfer = 3, kPlaneOffsetMid = 4, kPlaneTransferMid = 5, kPlanes = 6 };
struct Plan {
  int n_first, n_second, n_chains, pad;              // items of the two launches, sequences that are cut
};
struct Chain { int first_cut, n_cuts; };

struct Params {
  const float *q_inv, *k_inv, *log_decay, *beta;
  const int32_t *cu_rows, *start_pos, *cu_chunks;
  const int64_t* slots;
  uint8_t* recs; float* scal;
  float* state; int64_t state_ss;
  void* o;
  const Plan* plan; const Item* items; const Chain* chains; float* planes;
  int second;                                        // which launch of the recurrence: 0, or 1 = from the composed states
  int max_items;
  int n_seqs, NC, H, G, vdim;
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
// two fp32 values as a pair of rounded 16-bit values and the pair of their remainders
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(x, y);
  lo = pack_bf16(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
}
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void worker_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// ---- chunk offsets of the sequences, and how the recurrence walks them ---------------------------------------------------
// A walk is a serial chain of about 3.2 us a chunk on one SM per head and value block, so few long sequences leave most of the
// machine idle.  They are then cut into segments that are walked side by side: S' = T S + B over a segment, T from the identity
// with v = 0, B from zero (first launch, without outputs; a sequence's first segment is walked for real), the true states at the
// cuts in fp32 (delta_compose_kernel), and the later segments again from them, with outputs, each as two halves (second launch:
// their middles' T and B are kept on the way).  `room` walks fit the machine at a time.  The segment length is the shortest whose
// 2 s - 1 walks per sequence of s segments fit; it is taken if one and a half segments and the composition (about ten chunks'
// time, with the launches) are shorter than the longest sequence.  Measured, 8 heads of 128: one sequence of 32768 rows 1634 us
// uncut, cut into nine 339 us (197 + 34 for the states + 105, plan 3); sequences of 3001 and 1876 rows 154 -> 87 us.
constexpr int kComposeChunks = 10;

__device__ __forceinline__ int n_chunks_of(const int32_t* cu_chunks, int s) { return cu_chunks[s + 1] - cu_chunks[s]; }

__global__ void plan_kernel(const int32_t* __restrict__ cu_rows, const int32_t* __restrict__ start_pos, int n_seqs, int room,
                            int32_t* cu_chunks, Plan* plan, Item* items, int max_items, Chain* chains) {
  const int lane = threadIdx.x;
  if (lane == 0) {
    int at = 0;
    cu_chunks[0] = 0;
    for (int s = 0; s < n_seqs; ++s) {
      if (start_pos[s] >= 0) at += (cu_rows[s + 1] - cu_rows[s] + kC - 1) / kC;
      cu_chunks[s + 1] = at;
    }
  }
  __syncwarp();
  if (items == nullptr) return;
  int length = 1 << 30;                              // chunks of a segment
  if (n_seqs + 2 <= room) {
    int longest = 0;
    for (int s = 0; s < n_seqs; ++s) longest = max(longest, n_chunks_of(cu_chunks, s));
    for (int base = 4; base < longest; base += 32) {
      int walks = 0;
      for (int s = 0; s < n_seqs; ++s) {
        const int n = n_chunks_of(cu_chunks, s);
        if (n > 0) walks += 2 * ((n + base + lane - 1) / (base + lane)) - 1;
      }
      const unsigned fits = __ballot_sync(0xffffffffu, walks <= room);
      if (fits) {
        const int l = base + __ffs(fits) - 1;
        if (l + (l + 1) / 2 + kComposeChunks < longest) length = l;
        break;
      }
    }
  }
  if (length == 1 << 30) {                           // every sequence in one walk
    for (int s = lane; s < n_seqs; s += 32) items[s] = Item{s, 0, n_chunks_of(cu_chunks, s), kWalk, -1, -1, -1, 0};
    if (lane == 0) *plan = Plan{n_seqs, 0, 0, 0};
    return;
  }
  int first = 0, cuts = 0, n_chains = 0;
  Item* after = items + max_items;
  for (int s = 0; s < n_seqs; ++s) {
    const int n = n_chunks_of(cu_chunks, s);
    if (n == 0) continue;
    const int parts = (n + length - 1) / length, longer = n % parts, base = n / parts;      // the first `longer` segments are a chunk longer
    if (lane == 0 && parts > 1) chains[n_chains] = Chain{cuts, parts - 1};
    for (int j = lane; j < parts; j += 32) {
      const int a = j * base + min(j, longer), b = a + base + (j < longer ? 1 : 0), mid = (a + b + 1) / 2;
      if (j == 0) {
        items[first] = Item{s, a, b, kWalk, -1, parts > 1 ? cuts * kPlanes + kPlaneState : -1, -1, 0};
        continue;
      }
      const int cut = cuts + j - 1, e = cut * kPlanes;
      Item* two = items + first + 2 * j - 1;
      if (j + 1 < parts) {                             // the last segment's end is reached by its own walk
        two[0] = Item{s, a, b, kOffset, -1, e + kPlaneOffset, e + kPlaneOffsetMid, mid};
        two[1] = Item{s, a, b, kTransfer, -1, e + kPlaneTransfer, e + kPlaneTransferMid, mid};
      } else {                                         // only its middle is asked for
        two[0] = Item{s, a, mid, kOffset, -1, e + kPlaneOffsetMid, -1, 0};
        two[1] = Item{s, a, mid, kTransfer, -1, e + kPlaneTransferMid, -1, 0};
      }
      after[2 * cut] = Item{s, a, mid, kWalk, e + kPlaneState, -1, -1, 0};
      after[2 * cut + 1] = Item{s, mid, b, kWalk, e + kPlaneMiddle, -1, -1, 0};             // may be empty
    }
    first += 2 * parts - 1;
    cuts += parts - 1;
    n_chains += parts > 1 ? 1 : 0;
  }
  if (lane == 0) *plan = Plan{first, 2 * cuts, n_chains, 0};
}

// ======================================= factors =========================================================================
constexpr int kLd = 68;                              // fp32 row stride of A, T and Rq
constexpr int kMat = 128 * kLd * 4;
constexpr int kOffQ = 32768, kOffT = 0, kOffR = kMat, kOffA = 2 * kMat, kFactorSmem = 3 * kMat + 1024;   // T and Rq over the K, Q tiles

struct FactorBarriers { uint64_t kq_full, g_done, tile_free; };
struct Meta { int64_t t0[2]; int rows[2]; int64_t rec[2]; int h, g; };

__device__ __forceinline__ void tile_meta(const Params& p, int64_t tile, Meta& m) {
  m.h = (int)(tile % p.H);
  m.g = m.h / (p.H / p.G);
  const int j = (int)(tile / p.H);
  const int total = p.cu_chunks[p.n_seqs];
#pragma unroll
  for (int ci = 0; ci < 2; ++ci) {
    const int c = 2 * j + ci;
    m.t0[ci] = 0; m.rows[ci] = 0; m.rec[ci] = -1;
    if (c < total) {
      int lo = 0, hi = p.n_seqs;                     // largest s with cu_chunks[s] <= c
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (p.cu_chunks[mid] <= c) lo = mid; else hi = mid;
      }
      m.t0[ci] = (int64_t)p.cu_rows[lo] + (int64_t)(c - p.cu_chunks[lo]) * kC;
      m.rows[ci] = (int)min((int64_t)kC, (int64_t)p.cu_rows[lo + 1] - m.t0[ci]);
      m.rec[ci] = (int64_t)m.h * p.NC + c;
    }
  }
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  hi = __float_as_uint(x) & 0xffffe000u;
  lo = __float_as_uint(x - __uint_as_float(hi));
}
// acc (16 x 16 as two 8-column tiles) += A (16 x 16) * B (16 x 16), both row-major with stride kLd, operands split in two
__device__ __forceinline__ void block_mma(float (&acc)[2][4], const float* A, const float* B, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) {
    uint32_t ah[4], al[4];
    split_tf32(A[g * kLd + 8 * ks + t], ah[0], al[0]);
    split_tf32(A[(g + 8) * kLd + 8 * ks + t], ah[1], al[1]);
    split_tf32(A[g * kLd + 8 * ks + t + 4], ah[2], al[2]);
    split_tf32(A[(g + 8) * kLd + 8 * ks + t + 4], ah[3], al[3]);
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      uint32_t bh[2], bl[2];
      split_tf32(B[(8 * ks + t) * kLd + 8 * nt + g], bh[0], bl[0]);
      split_tf32(B[(8 * ks + t + 4) * kLd + 8 * nt + g], bh[1], bl[1]);
      mma_tf32(acc[nt], al, bh[0], bh[1]);
      mma_tf32(acc[nt], ah, bl[0], bl[1]);
      mma_tf32(acc[nt], ah, bh[0], bh[1]);
    }
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

__global__ void __launch_bounds__(kThreads, 2)
delta_factors_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* Ks = smem;
  uint8_t* Qs = smem + kOffQ;
  float* Tf = reinterpret_cast<float*>(smem + kOffT);
  float* Rf = reinterpret_cast<float*>(smem + kOffR);
  float* Af = reinterpret_cast<float*>(smem + kOffA);
  __shared__ FactorBarriers bar;
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  __shared__ float s_lg[128], s_bt[128], s_kinv[128], s_wsum[4];

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
  const int64_t n_tiles = (int64_t)((p.cu_chunks[p.n_seqs] + 1) / 2) * p.H;

  if (warp == 0) {
    // ---- TMA producer ------------------------------------------------------------------------------------------
    if (elect_one()) {
      uint32_t it = 0;
      for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++it) {
        if (it > 0 && !mbar_wait(&bar.tile_free, (it - 1) & 1u, abort_flag)) break;
        Meta m;
        tile_meta(p, tile, m);
        mbar_arrive_expect_tx(&bar.kq_full, 4 * 16384);
#pragma unroll
        for (int ci = 0; ci < 2; ++ci)
#pragma unroll
          for (int cb = 0; cb < 2; ++cb) {
            const int t0 = (int)(ci ? m.t0[1] : m.t0[0]);
            tma_load_4d(Ks + cb * 16384 + ci * 8192, &tmap_k, &bar.kq_full, cb * 64, m.g, t0, 0);
            tma_load_4d(Qs + cb * 16384 + ci * 8192, &tmap_q, &bar.kq_full, cb * 64, m.g, t0, 0);
          }
        // the tiles' place is taken until the end of this one; meanwhile the next inputs come into L2
        if (tile + gridDim.x < n_tiles) {
          Meta mn;
          tile_meta(p, tile + gridDim.x, mn);
#pragma unroll
          for (int ci = 0; ci < 2; ++ci)
#pragma unroll
            for (int cb = 0; cb < 2; ++cb) {
              tma_prefetch_l2_4d(&tmap_k, cb * 64, mn.g, (int)mn.t0[ci], 0);
              tma_prefetch_l2_4d(&tmap_q, cb * 64, mn.g, (int)mn.t0[ci], 0);
            }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---- MMA issuer --------------------------------------------------------------------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc(128, 128, 1, 0, 0);
      const uint64_t hi_k = (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61) | (uint64_t(16 >> 4) << 16);
      const uint64_t kd = hi_k | uint64_t((smem_u32(Ks) >> 4) & 0x3FFFu), qd = hi_k | uint64_t((smem_u32(Qs) >> 4) & 0x3FFFu);
      uint32_t it = 0;
      for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++it) {
        if (!mbar_wait(&bar.kq_full, it & 1u, abort_flag)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint64_t off = uint64_t(((kk >> 2) * 16384 + (kk & 3) * 32) >> 4);
          mma_ss(tbase, kd + off, kd + off, idesc, kk > 0);
        }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint64_t off = uint64_t(((kk >> 2) * 16384 + (kk & 3) * 32) >> 4);
          mma_ss(tbase + 128, qd + off, kd + off, idesc, kk > 0);
        }
        tc_commit(&bar.g_done);
      }
    }
    __syncwarp();
  } else {
    // ---- workers -----------------------------------------------------------------------------------------------
    const int wtid = tid - 64, w = warp - 2;
    const int quad = warp & 3, half = w >> 2;
    const int row = 32 * quad + lane;                  // tile row (and TMEM lane)
    const int ci = row >> 6, pr = row & 63;            // chunk of the tile, row inside the chunk
    const uint32_t lane_base = tbase + (uint32_t(32 * quad) << 16);
    uint32_t it = 0;
    // a tile's coordinates and its row scalars are fetched a tile ahead
    Meta m_next{};
    float bt_next = 0.f, kinv_next = 0.f, qinv_next = 0.f, decay_next = 0.f;
    int sees_next = 0;                                 // columns s < sees of A, s <= sees of Rq; a row behind the sequence's end: none
    auto fetch_tile = [&](int64_t tile) {
      if (tile >= n_tiles) return;
      tile_meta(p, tile, m_next);
      const bool valid = pr < (ci ? m_next.rows[1] : m_next.rows[0]);
      const int64_t t = (ci ? m_next.t0[1] : m_next.t0[0]) + pr;
      sees_next = valid ? pr : -1;
      bt_next = valid ? p.beta[t * p.H + m_next.h] : 0.f;
      kinv_next = valid ? p.k_inv[t * p.G + m_next.g] : 0.f;
      qinv_next = valid ? p.q_inv[t * p.G + m_next.g] : 0.f;
      decay_next = valid ? p.log_decay[t * p.H + m_next.h] : 0.f;
    };
    fetch_tile(blockIdx.x);
    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++it) {
      const Meta m = m_next;
      const int64_t rec = ci ? m.rec[1] : m.rec[0];
      const float bt_p = bt_next, kinv_p = kinv_next, qinv_p = qinv_next;
      const int sees = sees_next;
      float run = decay_next;
      // decay prefix over the chunk's 64 rows (two warps)
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
      }
      worker_sync();                                   // every warp is done with the previous tile's arrays
      if (half == 0 && lane == 31) s_wsum[quad] = run;
      worker_sync();
      if (quad & 1) run += s_wsum[quad - 1];
      if (half == 0) { s_lg[row] = run; s_bt[row] = bt_p; s_kinv[row] = kinv_p; }
      worker_sync();
      const float lg_p = run, lg_C = s_lg[64 * ci + 63];
      if (half == 0 && rec >= 0) {
        float* sc = p.scal + rec * kScal;
        sc[pr] = expf(lg_p) * kinv_p;
        sc[64 + pr] = expf(lg_p) * qinv_p;
        sc[128 + pr] = expf(lg_C - lg_p) * kinv_p;
        if (pr == kC - 1) sc[192] = expf(lg_C);
      }
      // ---- A and Rq from the Gram matrices ----
      mbar_wait(&bar.g_done, it & 1u, abort_flag);      // after a timeout every later wait returns at once
      __syncwarp();
      tc_fence_after();
      if (half == 1 && (quad & 1) == 0) {               // rows 0-31 see no column of the second half
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          *reinterpret_cast<float4*>(Af + row * kLd + 32 + j) = make_float4(0.f, 0.f, 0.f, 0.f);
          *reinterpret_cast<float4*>(Rf + row * kLd + 32 + j) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      } else {
#pragma unroll 1
        for (int which = 0; which < 2; ++which) {
          uint32_t gm[32];
          tmem_ld32(lane_base + 128 * which + 64 * ci + 32 * half, gm);
          float* dst = (which ? Rf : Af) + row * kLd + 32 * half;
          const float f = which ? qinv_p : bt_p * kinv_p;
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            float x[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int s = 32 * half + j + e;
              // chosen after it is computed: as a condition around the exponential it is a branch for every element
              const float value = f * (__expf(lg_p - s_lg[64 * ci + s]) * s_kinv[64 * ci + s]) * __uint_as_float(gm[j + e]);
              x[e] = (which ? s <= sees : s < sees) ? value : 0.f;
            }
            *reinterpret_cast<float4*>(dst + j) = make_float4(x[0], x[1], x[2], x[3]);
          }
        }
      }
      tc_fence_before();
      worker_sync();
      // ---- T = (I + A)^-1: diagonal 16 x 16 blocks by substitution ----
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
      // G_il = -T_ii A_il below the diagonal (in place over A_il), then T_ij = sum_l G_il T_lj level by level
      for (int blk = w; blk < 12; blk += 8) {
        const int cc = blk / 6, e = blk % 6;
        const int bi = (e == 0) ? 1 : (e < 3 ? 2 : 3), bl = (e == 0) ? 0 : (e < 3 ? e - 1 : e - 3);
        float acc[2][4] = {};
        float* Ail = Af + (64 * cc + 16 * bi) * kLd + 16 * bl;
        block_mma(acc, Tf + (64 * cc + 16 * bi) * kLd + 16 * bi, Ail, lane);
        __syncwarp();
        block_store(Ail, acc, lane, -1.f);
      }
      worker_sync();
#pragma unroll 1
      for (int d = 1; d <= 3; ++d) {
        const int per = 4 - d;
        for (int blk = w; blk < 2 * per; blk += 8) {
          const int cc = blk / per, bj = blk % per, bi = bj + d;
          float acc[2][4] = {};
          for (int l = bj; l < bi; ++l)
            block_mma(acc, Af + (64 * cc + 16 * bi) * kLd + 16 * l, Tf + (64 * cc + 16 * l) * kLd + 16 * bj, lane);
          block_store(Tf + (64 * cc + 16 * bi) * kLd + 16 * bj, acc, lane, 1.f);
        }
        worker_sync();
      }
      fetch_tile(tile + gridDim.x);
      // ---- M1 = T diag(beta) as two terms, and zeros of M2 above the diagonal blocks: eight threads per 128-byte row ----
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int idx = wtid + 256 * i, r = idx >> 3, ch = idx & 7, rp = r & 63, rc = r >> 6;
        const int64_t to = rc ? m.rec[1] : m.rec[0];
        const bool above = (ch >> 1) > (rp >> 4);
        uint32_t hi[4] = {}, lo[4] = {};
        if (!above) {
          float x[8];
          *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(Tf + r * kLd + 8 * ch);
          *reinterpret_cast<float4*>(x + 4) = *reinterpret_cast<const float4*>(Tf + r * kLd + 8 * ch + 4);
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = 8 * ch + e <= rp ? x[e] * s_bt[64 * rc + 8 * ch + e] : 0.f;
#pragma unroll
          for (int e = 0; e < 4; ++e) split2(x[2 * e], x[2 * e + 1], hi[e], lo[e]);
        }
        if (to >= 0) {
          uint8_t* r1 = p.recs + to * (int64_t)kRecBytes + rp * 128 + ch * 16;
          *reinterpret_cast<uint4*>(r1) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(r1 + 16384) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          if (above) {
            *reinterpret_cast<uint4*>(r1 + 8192) = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4*>(r1 + 24576) = make_uint4(0u, 0u, 0u, 0u);
          }
        }
      }
      // ---- M2 = Rq T diag(beta): ten blocks per chunk, five block products per warp ----
      {
        const int cc = w >> 2, q = w & 3;
        const int64_t rc = cc ? m.rec[1] : m.rec[0];
        const int n_blk = q == 0 || q == 1 || q == 2 ? 2 : 4;
#pragma unroll 1
        for (int b = 0; b < n_blk; ++b) {
          int bi, bj;                                  // q=0: (3,0) (0,0)   1: (2,0) (1,0)   2: (3,1) (2,1)   3: (3,2) (1,1) (2,2) (3,3)
          if (q == 0) { bi = b ? 0 : 3; bj = 0; }
          else if (q == 1) { bi = b ? 1 : 2; bj = 0; }
          else if (q == 2) { bi = b ? 2 : 3; bj = 1; }
          else { bi = b == 0 ? 3 : b; bj = b == 0 ? 2 : b; }
          float acc[2][4] = {};
          for (int l = bj; l <= bi; ++l)
            block_mma(acc, Rf + (64 * cc + 16 * bi) * kLd + 16 * l, Tf + (64 * cc + 16 * l) * kLd + 16 * bj, lane);
          if (rc >= 0) {
            const int g = lane >> 2, t2 = 2 * (lane & 3);
            uint8_t* r2 = p.recs + rc * (int64_t)kRecBytes + 8192;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
              const int s = 16 * bj + 8 * nt + t2;
              const float b0 = s_bt[64 * cc + s], b1 = s_bt[64 * cc + s + 1];
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                uint32_t hi, lo;
                split2(acc[nt][2 * e] * b0, acc[nt][2 * e + 1] * b1, hi, lo);
                uint8_t* dst = r2 + (16 * bi + g + 8 * e) * 128 + s * 2;
                *reinterpret_cast<uint32_t*>(dst) = hi;
                *reinterpret_cast<uint32_t*>(dst + 16384) = lo;
              }
            }
          }
        }
      }
      fence_proxy_async();                             // the next tile's TMA writes over T and Rq
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.tile_free);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && s_abort) atomicExch(&g_delta_status, 1);
  if (warp == 1) tmem_dealloc(tbase, 256);
}

// ======================================= recurrence =======================================================================
constexpr int kStages = 2, kStateWarps = 16, kRecurThreads = 64 + 32 * kStateWarps;
// a stage: [K rows; Q rows] as two boxes of 64 channels x 128 rows | V, two boxes of 64 channels x 64 rows | [M1; M2] rounded,
// [M1; M2] remainders | scalars
constexpr int kOffKQ = 0, kOffRV = 32768, kOffRM = 49152, kOffRS = 81920, kStageBytes = 82944;
constexpr int kRecurSmem = kStages * kStageBytes + 1024;
constexpr uint32_t kColS = 0, kColP = 128, kColQ = 192, kColD = 128, kColX = 256, kColX2 = 320, kColR = 384, kColU = 448;

struct RecurBarriers {
  uint64_t in_full[kStages], m_full[kStages], empty[kStages];
  uint64_t s_ready, pq_full, r_ready, uo_full, us_ready, s_done;
};

// kCuts: the walks may be offsets and transfers (the first launch where sequences can be cut); without them the state warps' loop
// needs fewer registers than the 96 that eighteen warps leave a thread.
template <bool kCuts>
__global__ void __launch_bounds__(kRecurThreads, 1)
delta_recur_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                   const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_m, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ RecurBarriers bar;
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int vblocks = p.vdim / kD;
  const int hv = blockIdx.x, h = hv / vblocks, g = h / (p.H / p.G);
  Item entry{(int)blockIdx.y, 0, 0, kWalk, -1, -1, -1, 0};
  if (p.items == nullptr) {
    entry.last = n_chunks_of(p.cu_chunks, blockIdx.y);
  } else {
    if ((int)blockIdx.y >= (p.second ? p.plan->n_second : p.plan->n_first)) return;    // the whole CTA, before anything is allocated
    entry = p.items[(p.second ? p.max_items : 0) + blockIdx.y];
  }
  const int b = entry.seq, n_chunks = entry.last - entry.first;
  if (n_chunks <= 0 || p.slots[b] < 0 || (kCuts && entry.kind == kTransfer && hv % vblocks != 0)) return;
  const int row_begin = p.cu_rows[b] + entry.first * kC, row_end = p.cu_rows[b + 1];
  const int64_t rec0 = (int64_t)h * p.NC + p.cu_chunks[b] + entry.first;
  __shared__ Item s_item;
  const volatile Item& item = s_item;                 // read where it is needed: the loop's registers are all taken

  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) { mbar_init(&bar.in_full[i], 1); mbar_init(&bar.m_full[i], 1); mbar_init(&bar.empty[i], 1 + kStateWarps); }
    mbar_init(&bar.s_ready, kStateWarps); mbar_init(&bar.r_ready, kStateWarps); mbar_init(&bar.us_ready, kStateWarps);
    mbar_init(&bar.pq_full, 1); mbar_init(&bar.uo_full, 1); mbar_init(&bar.s_done, 1);
    s_abort = 0;
    s_item = entry;
    s_item.at = entry.middle >= 0 ? entry.at - entry.first : -1;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(&s_tmem_base, 512);
  if (warp == 0 && lane == 0) { prefetch_tensormap(&tmap_q); prefetch_tensormap(&tmap_k); prefetch_tensormap(&tmap_v); prefetch_tensormap(&tmap_m); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = s_tmem_base;
  volatile int* abort_flag = &s_abort;

  if (warp == 0) {
    // ---- TMA producer ------------------------------------------------------------------------------------------
    if (elect_one()) {
      for (int i = 0; i < n_chunks; ++i) {
        const int s = i % kStages;
        uint8_t* st = smem + s * kStageBytes;
        const int t0 = row_begin + i * kC;
        const int64_t rec = rec0 + i;
        if (!mbar_wait(&bar.empty[s], ((uint32_t)(i / kStages) & 1u) ^ 1u, abort_flag)) break;
        mbar_arrive_expect_tx(&bar.in_full[s], 3 * 16384 + 1024);
#pragma unroll
        for (int cb = 0; cb < 2; ++cb) {
          tma_load_4d(st + kOffKQ + cb * 16384, &tmap_k, &bar.in_full[s], cb * 64, g, t0, 0);
          tma_load_4d(st + kOffKQ + cb * 16384 + 8192, &tmap_q, &bar.in_full[s], cb * 64, g, t0, 0);
          tma_load_4d(st + kOffRV + cb * 8192, &tmap_v, &bar.in_full[s], cb * 64, hv, t0, 0);
        }
        bulk_load(st + kOffRS, p.scal + rec * kScal, kScal * 4, &bar.in_full[s]);
        mbar_arrive_expect_tx(&bar.m_full[s], kRecBytes);
#pragma unroll
        for (int q = 0; q < 4; ++q) tma_load_4d(st + kOffRM + q * 8192, &tmap_m, &bar.m_full[s], 0, (int)(rec * 256) + q * 64, 0, 0);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---- MMA issuer --------------------------------------------------------------------------------------------
    if (elect_one()) {
      // B rows as they lie: [K; Q] or [M1; M2]; without outputs only the first half
      const uint32_t idesc_k = !kCuts || item.kind == kWalk ? make_idesc(128, 128, 1, 0, 0) : make_idesc(128, 64, 1, 0, 0);
      constexpr uint32_t idesc_ds = make_idesc(128, 128, 1, 0, 1);     // B = K [s][k], MN-major
      const uint64_t hi_k = (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61) | (uint64_t(16 >> 4) << 16);
      const uint64_t hi_mn = (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61) | (uint64_t(16384 >> 4) << 16);
      bool ok = true;
      for (int i = 0; i < n_chunks && ok; ++i) {
        const int s = i % kStages;
        const uint32_t ph = (uint32_t)(i / kStages) & 1u, pi = (uint32_t)i & 1u;
        const uint32_t st = smem_u32(smem + s * kStageBytes);
        const uint64_t kq = hi_k | uint64_t(((st + kOffKQ) >> 4) & 0x3FFFu), kmn = hi_mn | uint64_t(((st + kOffKQ) >> 4) & 0x3FFFu);
        const uint64_t md = hi_k | uint64_t(((st + kOffRM) >> 4) & 0x3FFFu);
        ok = mbar_wait(&bar.s_ready, pi, abort_flag) && mbar_wait(&bar.in_full[s], ph, abort_flag);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int term = 0; term < 2; ++term)
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            mma_ts(tbase + kColP, tbase + kColS + term * 64 + kk * 8, kq + uint64_t(((kk >> 2) * 16384 + (kk & 3) * 32) >> 4), idesc_k,
                   (term > 0 || kk > 0) ? 1u : 0u);
        tc_commit(&bar.pq_full);
        ok = mbar_wait(&bar.r_ready, pi, abort_flag) && mbar_wait(&bar.m_full[s], ph, abort_flag);
        if (!ok) break;
        tc_fence_after();
        // (rounded, rounded), (remainder, rounded), (rounded, remainder)
#pragma unroll
        for (int term = 0; term < 3; ++term)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_ts(tbase + kColX, tbase + kColR + (term == 1 ? 32 : 0) + kk * 8, md + uint64_t(((term == 2 ? 16384 : 0) + kk * 32) >> 4), idesc_k,
                   (term > 0 || kk > 0) ? 1u : 0u);
        tc_commit(&bar.uo_full);
        ok = mbar_wait(&bar.us_ready, pi, abort_flag);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int term = 0; term < 2; ++term)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_ts(tbase + kColD, tbase + kColU + term * 32 + kk * 8, kmn + uint64_t((kk * 2048) >> 4), idesc_ds, (term > 0 || kk > 0) ? 1u : 0u);
        tc_commit(&bar.s_done);
        tc_commit(&bar.empty[s]);
      }
    }
    __syncwarp();
  } else {
    // ---- state warps -------------------------------------------------------------------------------------------
    const int quad = warp & 3, qt = (warp - 2) >> 2;   // qt: 32 of the 128 state columns, 16 of a chunk's 64 rows
    const int v = 32 * quad + lane;                    // TMEM lane = value channel of this CTA's block
    const uint32_t lane_base = tbase + (uint32_t(32 * quad) << 16);
    const int vcol = (hv % vblocks) * kD + v;
    auto table = [&] { return p.state + p.slots[b] * p.state_ss + ((int64_t)h * kD + 32 * qt) * p.vdim + vcol; };   // element (k = 32 qt + j, v)
    auto plane_of = [&](int i) {
      int unit = hv;
      asm volatile("" : "+r"(unit));                    // no part of the address is kept through the loop
      return p.planes + ((int64_t)i * gridDim.x + unit) * (kD * kD) + 32 * qt * kD + v;
    };
    float S[32];
    if (kCuts && item.kind != kWalk) {
      const bool identity = item.kind == kTransfer;
#pragma unroll
      for (int j = 0; j < 32; ++j) S[j] = identity && 32 * qt + j == v ? 1.f : 0.f;
    } else {
      const int from = item.from;
      const bool fresh = from < 0 && p.start_pos[b] == 0;
      const float* src = from < 0 ? table() : plane_of(from);
      int64_t step = from < 0 ? p.vdim : kD;
      asm volatile("" : "+l"(step));                    // not a loop invariant: its multiples would be kept in registers
#pragma unroll
      for (int j = 0; j < 32; ++j) { S[j] = fresh ? 0.f : *src; src += step; }
    }
    auto put = [&](float* dst, int64_t step) {
      asm volatile("" : "+l"(step));
#pragma unroll
      for (int j = 0; j < 32; ++j) { *dst = S[j]; dst += step; }
    };
    float gC = 0.f;                                    // decay over the chunk before
    bool ok = true;
    for (int i = 0; i <= n_chunks; ++i) {
      if (i > 0) {                                     // the state after chunk i - 1
        ok = mbar_wait(&bar.s_done, (uint32_t)(i - 1) & 1u, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        uint32_t d[32];
        tmem_ld32(lane_base + kColD + 32 * qt, d);
#pragma unroll
        for (int j = 0; j < 32; ++j) S[j] = fmaf(gC, S[j], __uint_as_float(d[j]));
      }
      if (i == n_chunks) break;
      if (kCuts && i == item.at) put(plane_of(item.middle), kD);
      // ---- S^T as two 16-bit terms (the dS columns have been read: the next products may overwrite them) ----
      {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) split2(S[2 * j], S[2 * j + 1], hi[j], lo[j]);
        tmem_st16(lane_base + kColS + 16 * qt, hi);
        tmem_st16(lane_base + kColS + 64 + 16 * qt, lo);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.s_ready);

      const int s = i % kStages;
      const uint8_t* st = smem + s * kStageBytes;
      const float* sc = reinterpret_cast<const float*>(st + kOffRS) + 16 * qt;
      // ---- R^T = V^T - (a k_inv) P: this thread's value channel, rows 16 qt .. + 15 ----
      ok = mbar_wait(&bar.in_full[s], (uint32_t)(i / kStages) & 1u, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      float vv[16], ek[16];
      {
        const uint8_t* vb = st + kOffRV + (v >> 6) * 8192 + (v & 7) * 2;
        const int ch = (v & 63) >> 3;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int t = 16 * qt + j;
          vv[j] = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(vb + t * 128 + ((ch ^ (t & 7)) << 4)));
        }
        if (kCuts && item.kind == kTransfer) {
#pragma unroll
          for (int j = 0; j < 16; ++j) vv[j] = 0.f;
        }
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const float4 e = *reinterpret_cast<const float4*>(sc + j);
          ek[j] = e.x; ek[j + 1] = e.y; ek[j + 2] = e.z; ek[j + 3] = e.w;
        }
      }
      ok = mbar_wait(&bar.pq_full, (uint32_t)i & 1u, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      {
        uint32_t pr[16], hi[8], lo[8];
        tmem_ld16(lane_base + kColP + 16 * qt, pr);
#pragma unroll
        for (int j = 0; j < 16; j += 2)
          split2(fmaf(-ek[j], __uint_as_float(pr[j]), vv[j]), fmaf(-ek[j + 1], __uint_as_float(pr[j + 1]), vv[j + 1]), hi[j >> 1], lo[j >> 1]);
        if (i == n_chunks - 1 && row_end - (row_begin + i * kC) < kC) {
          // Rows behind the sequence's end are another's.  Their factors are zero, but they may be infinite or no numbers: no R, and
          // zeros for K, whose product with S has been read, in front of the product with U
          const int left = row_end - (row_begin + i * kC);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const uint32_t keep = 16 * qt + j < left ? 0xffffffffu : j & 1 ? 0x0000ffffu : 0xffff0000u;
            hi[j >> 1] &= keep; lo[j >> 1] &= keep;
          }
          uint8_t* kr = smem + s * kStageBytes + kOffKQ;
          for (int at = tid - 64 + left * 16; at < kC * 16; at += 32 * kStateWarps)      // 16 pieces of 16 bytes a row, eight in each box
            *reinterpret_cast<uint4*>(kr + ((at & 8) << 11) + (at >> 4) * 128 + ((at & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
          fence_proxy_async();
        }
        tmem_st8(lane_base + kColR + 8 * qt, hi);
        tmem_st8(lane_base + kColR + 32 + 8 * qt, lo);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.r_ready);
      }
      // ---- U^T scaled by (a_C / a) k_inv; S^T Q^T leaves the columns that dS will take ----
      float ed[16];
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const float4 e = *reinterpret_cast<const float4*>(sc + 128 + j);
        ed[j] = e.x; ed[j + 1] = e.y; ed[j + 2] = e.z; ed[j + 3] = e.w;
      }
      uint32_t sq[16];
      tmem_ld16(lane_base + kColQ + 16 * qt, sq);
      ok = mbar_wait(&bar.uo_full, (uint32_t)i & 1u, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      {
        uint32_t u[16], hi[8], lo[8];
        tmem_ld16(lane_base + kColX + 16 * qt, u);
#pragma unroll
        for (int j = 0; j < 16; j += 2) split2(__uint_as_float(u[j]) * ed[j], __uint_as_float(u[j + 1]) * ed[j + 1], hi[j >> 1], lo[j >> 1]);
        tmem_st8(lane_base + kColU + 8 * qt, hi);
        tmem_st8(lane_base + kColU + 32 + 8 * qt, lo);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.us_ready);
      }
      // ---- O = (a q_inv) S Q + R M2, under the last product ----
      {
        gC = reinterpret_cast<const float*>(st + kOffRS)[192];
        const int t0 = row_begin + i * kC + 16 * qt;
        const int n_ok = !kCuts || item.kind == kWalk ? min(16, row_end - t0) : 0;      // without outputs whatever the columns hold stays here
        uint16_t* oc = static_cast<uint16_t*>(p.o) + ((int64_t)t0 * p.H + h) * p.vdim + vcol;
        int64_t orow = (int64_t)p.H * p.vdim;
        asm volatile("" : "+l"(orow));
        uint32_t r[16];
        tmem_ld16(lane_base + kColX2 + 16 * qt, r);
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const float2 e = *reinterpret_cast<const float2*>(sc + 64 + j);
          const uint32_t w = pack_bf16(fmaf(e.x, __uint_as_float(sq[j]), __uint_as_float(r[j])), fmaf(e.y, __uint_as_float(sq[j + 1]), __uint_as_float(r[j + 1])));
          if (j < n_ok) *oc = (uint16_t)(w & 0xffffu);
          oc += orow;
          if (j + 1 < n_ok) *oc = (uint16_t)(w >> 16);
          oc += orow;
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.empty[s]);
      }
    }
    if (ok) {
      if (kCuts && item.to >= 0) put(plane_of(item.to), kD);
      else if (item.last == n_chunks_of(p.cu_chunks, b)) put(table(), p.vdim);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && s_abort) atomicExch(&g_delta_status, 1);
  if (warp == 1) tmem_dealloc(tbase, 512);
}

// ---- the true states at the cuts ------------------------------------------------------------------------------------------
// S_next = T S + B along a sequence's cuts, and the state in the middle of every segment beside it, in fp32.  A CTA owns eight
// value channels of a head (columns are independent): 128 threads hold two rows of T x four channels each, the other 128 the
// middle's.  The matrices do not depend on the states, so their quarters (32 columns; row stride 36: sixteen-byte reads of
// neighbouring rows hit different banks) stream through six stages of shared memory ahead of the chain.
constexpr int kComposeCols = 8, kComposeLd = 36, kComposePart = kD * kComposeLd, kComposeStages = 6;
constexpr int kComposeSmem = 2 * kComposeStages * kComposePart * 4;

__global__ void __launch_bounds__(256, 1) delta_compose_kernel(const Params p) {
  extern __shared__ __align__(16) float parts[];
  __shared__ __align__(16) float S[2][kD][kComposeCols];
  if ((int)blockIdx.y >= p.plan->n_chains) return;
  const Chain chain = p.chains[blockIdx.y];
  const int vblocks = p.vdim / kD, HV = p.H * vblocks;
  const int hv = blockIdx.x / (kD / kComposeCols), v0 = blockIdx.x % (kD / kComposeCols) * kComposeCols;
  const int tid = threadIdx.x & 127, side = threadIdx.x >> 7, k = tid >> 1, half = tid & 1;      // side 1: the middle's matrix
  auto plane = [&](int i, int unit) { return p.planes + ((int64_t)(chain.first_cut * kPlanes + i) * HV + unit) * (kD * kD); };
  float* mine = parts + side * kComposeStages * kComposePart;
  const int64_t at = (int64_t)k * kD + v0 + 4 * half;                                            // rows k and k + 64
  const int units = 4 * chain.n_cuts;
  auto active = [&](int c) { return side == 1 || c + 1 < chain.n_cuts; };                        // the last segment's end is not composed
  auto request = [&](int u) {
    if (u < units && active(u >> 2)) {
      const float* T = plane((u >> 2) * kPlanes + (side ? kPlaneTransferMid : kPlaneTransfer), hv - hv % vblocks) + (u & 3) * 32;
      float* dst = mine + u % kComposeStages * kComposePart;
#pragma unroll
      for (int i = tid; i < kD * 8; i += 128)
        mma::cp_async16(mma::smem_u32(dst + (i >> 3) * kComposeLd + (i & 7) * 4), T + (i >> 3) * kD + (i & 7) * 4);
    }
    mma::cp_async_commit();
  };

  for (int u = 0; u < kComposeStages - 1; ++u) request(u);
#pragma unroll
  for (int r = 0; r < 2; ++r)                          // both sides write the same
    *reinterpret_cast<float4*>(&S[0][k + 64 * r][4 * half]) = *reinterpret_cast<const float4*>(plane(kPlaneState, hv) + at + 64 * r * kD);
  float2 acc[2][2];
  float4 off[2];
  for (int u = 0; u < units; ++u) {
    const int c = u >> 2, base = c * kPlanes;
    mma::cp_async_wait<kComposeStages - 2>();
    __syncthreads();                                   // the part has landed for everyone, and the stage asked for below is free
    request(u + kComposeStages - 1);
    if (!active(c)) continue;
    if ((u & 3) == 0) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        acc[r][0] = acc[r][1] = make_float2(0.f, 0.f);
        off[r] = *reinterpret_cast<const float4*>(plane(base + (side ? kPlaneOffsetMid : kPlaneOffset), hv) + at + 64 * r * kD);
      }
    }
    const float* row = mine + u % kComposeStages * kComposePart + k * kComposeLd;
    const float* s = &S[c & 1][32 * (u & 3)][4 * half];
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      const float4 t0 = *reinterpret_cast<const float4*>(row + j), t1 = *reinterpret_cast<const float4*>(row + 64 * kComposeLd + j);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float w0 = e == 0 ? t0.x : e == 1 ? t0.y : e == 2 ? t0.z : t0.w, w1 = e == 0 ? t1.x : e == 1 ? t1.y : e == 2 ? t1.z : t1.w;
        const float4 x = *reinterpret_cast<const float4*>(s + (j + e) * kComposeCols);
        const float2 lo = make_float2(x.x, x.y), hi = make_float2(x.z, x.w);
        acc[0][0] = __ffma2_rn(make_float2(w0, w0), lo, acc[0][0]); acc[0][1] = __ffma2_rn(make_float2(w0, w0), hi, acc[0][1]);
        acc[1][0] = __ffma2_rn(make_float2(w1, w1), lo, acc[1][0]); acc[1][1] = __ffma2_rn(make_float2(w1, w1), hi, acc[1][1]);
      }
    }
    if ((u & 3) == 3) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float4 x = make_float4(acc[r][0].x + off[r].x, acc[r][0].y + off[r].y, acc[r][1].x + off[r].z, acc[r][1].y + off[r].w);
        *reinterpret_cast<float4*>(plane(side ? base + kPlaneMiddle : base + kPlanes + kPlaneState, hv) + at + 64 * r * kD) = x;
        if (side == 0) *reinterpret_cast<float4*>(&S[(c & 1) ^ 1][k + 64 * r][4 * half]) = x;
      }
    }
  }
  mma::cp_async_wait<0>();
}

// (channel, head, row) view of a (rows, heads, 128) tensor; boxes of 64 channels x 64 rows of one head
int heads_map(CUtensorMap* out, const void* base, int heads, int64_t rows) {
  const uint64_t dims[4] = {128, (uint64_t)heads, (uint64_t)rows, 1};
  const int64_t strides[3] = {128, (int64_t)heads * 128, (int64_t)heads * 128 * rows};
  const uint32_t box[4] = {64, 1, 64, 1};
  return make_tmap_16bit_4d(out, base, 1, dims, strides, box);
}

int64_t max_chunks(const atma_delta_args& a) { return a.total_rows / kC + a.n_seqs; }
int64_t align_up(int64_t n) { return (n + 1023) & ~int64_t(1023); }

// Where the scratch's parts lie, from launch-time sizes only.
struct Layout {
  int room, max_items;                                // walks that fit the machine at a time; items of either launch
  bool cuts;                                          // whether a sequence may be cut
  int64_t cu, plan, items, chains, scal, recs, planes, bytes;
};
Layout layout_of(const atma_delta_args& a, int64_t longest_rows) {
  Layout l{};
  const int64_t n = max_chunks(a) * a.H;
  const int walks = a.H * (a.vdim / kD);
  l.room = sm_count_of_current_device() / walks;
  // what plan_kernel decides, if every other sequence takes one walk: where it cannot cut, two launches and the plan are left
  // out (4 x 500 rows 56 -> 51 us, one after another; 8 x 200 44 -> 38)
  const bool space = a.n_seqs + 2 <= l.room && (a.total_rows + kC - 1) / kC > 6 + kComposeChunks;      // whatever the longest is
  if (space) {
    const int64_t longest = (longest_rows + kC - 1) / kC, parts = (l.room - a.n_seqs + 2) / 2, least = (longest + parts - 1) / parts;
    const int64_t length = least > 4 ? least : 4;
    l.cuts = length + (length + 1) / 2 + kComposeChunks < longest;
  }
  l.max_items = space ? l.room : a.n_seqs;
  l.plan = align_up(4 * ((int64_t)a.n_seqs + 1));
  l.items = l.plan + align_up(sizeof(Plan));
  l.chains = l.items + align_up(2 * (int64_t)l.max_items * sizeof(Item));
  l.scal = l.chains + align_up((int64_t)a.n_seqs * sizeof(Chain));
  l.recs = l.scal + n * kScal * 4;
  l.planes = l.recs + n * kRecBytes;
  l.bytes = l.planes + (space ? (int64_t)(l.room / 2) * kPlanes * walks * kD * kD * 4 : 0);
  return l;
}

}  // namespace

bool delta_scan_sm100_supported(const atma_delta_args& a) {
  return a.dtype == ATMA_BF16 && a.dim == kD && a.vdim > 0 && a.vdim % kD == 0 && a.G > 0 && a.H > 0 &&
         max_chunks(a) * a.H * 256 < (int64_t(1) << 31);
}

int64_t delta_scan_sm100_scratch_bytes(const atma_delta_args& a) { return layout_of(a, a.total_rows).bytes + 1024; }

int delta_scan_sm100(const atma_delta_args& a, int longest, const void* q, const void* k, const void* v, const float* q_inv, const float* k_inv,
                     const float* log_decay, const float* beta, void* o, void* scratch, cudaStream_t st) {
  ATMA_REQUIRE(scratch != nullptr, "delta_scan: scratch is required for this shape");
  auto al = [](const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0; };
  ATMA_REQUIRE(al(q) && al(k) && al(v), "delta_scan: q, k and v must be 16-byte aligned");
  const int64_t NC = max_chunks(a);
  Params p{};
  uint8_t* base = reinterpret_cast<uint8_t*>(align_up((int64_t)reinterpret_cast<uintptr_t>(scratch)));
  const Layout l = layout_of(a, longest < a.total_rows ? longest : a.total_rows);
  int32_t* cu_chunks = reinterpret_cast<int32_t*>(base);
  Plan* plan = reinterpret_cast<Plan*>(base + l.plan);
  Item* items = reinterpret_cast<Item*>(base + l.items);
  Chain* chains = reinterpret_cast<Chain*>(base + l.chains);
  p.plan = plan; p.items = l.cuts ? items : nullptr; p.chains = chains; p.max_items = l.max_items;
  p.planes = reinterpret_cast<float*>(base + l.planes);
  p.scal = reinterpret_cast<float*>(base + l.scal);
  p.recs = base + l.recs;
  p.q_inv = q_inv; p.k_inv = k_inv; p.log_decay = log_decay; p.beta = beta;
  p.cu_rows = a.cu_rows; p.start_pos = a.start_pos; p.cu_chunks = cu_chunks; p.slots = a.slots;
  p.state = a.state_table; p.state_ss = a.state_ss; p.o = o;
  p.n_seqs = a.n_seqs; p.NC = (int)NC; p.H = a.H; p.G = a.G; p.vdim = a.vdim;
  CUtensorMap mq, mk, mv, mm;
  int rc = heads_map(&mq, q, a.G, a.total_rows);
  if (rc == ATMA_OK) rc = heads_map(&mk, k, a.G, a.total_rows);
  if (rc == ATMA_OK) rc = heads_map(&mv, v, a.H * (a.vdim / kD), a.total_rows);
  if (rc == ATMA_OK) {
    const int64_t rows = NC * a.H * 256;
    const uint64_t dims[4] = {64, (uint64_t)rows, 1, 1};
    const int64_t strides[3] = {64, rows * 64, rows * 64};
    const uint32_t box[4] = {64, 64, 1, 1};
    rc = make_tmap_16bit_4d(&mm, p.recs, 1, dims, strides, box);
  }
  if (rc != ATMA_OK) return rc;
  plan_kernel<<<1, 32, 0, st>>>(a.cu_rows, a.start_pos, a.n_seqs, l.room, cu_chunks, plan, l.cuts ? items : nullptr, l.max_items, chains);
  const int64_t tiles = (NC + 1) / 2 * a.H;
  const int sms = sm_count_of_current_device();
  ATMA_CUDA_OK(cudaFuncSetAttribute(delta_factors_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFactorSmem));
  delta_factors_kernel<<<(unsigned)(tiles < 2 * sms ? tiles : 2 * sms), kThreads, kFactorSmem, st>>>(mq, mk, p);
  ATMA_CUDA_OK(cudaFuncSetAttribute(delta_recur_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRecurSmem));
  const int walks = a.H * (a.vdim / kD);
  const dim3 grid(walks, l.cuts ? l.max_items : a.n_seqs);
  if (l.cuts) {                                       // whether one is cut is decided on the device: the last two may find nothing to do
    ATMA_CUDA_OK(cudaFuncSetAttribute(delta_recur_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRecurSmem));
    ATMA_CUDA_OK(cudaFuncSetAttribute(delta_compose_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kComposeSmem));
    delta_recur_kernel<true><<<grid, kRecurThreads, kRecurSmem, st>>>(mq, mk, mv, mm, p);
    delta_compose_kernel<<<dim3(walks * (kD / kComposeCols), a.n_seqs), 256, kComposeSmem, st>>>(p);
    p.second = 1;
  }
  delta_recur_kernel<false><<<grid, kRecurThreads, kRecurSmem, st>>>(mq, mk, mv, mm, p);
  return launch_status("delta_scan (tcgen05)");
}

int delta_sm100_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  ATMA_CUDA_OK(cudaMemcpyFromSymbol(&v, g_delta_status, sizeof(int)));
  if (v != 0) ATMA_CUDA_OK(cudaMemcpyToSymbol(g_delta_status, &zero, sizeof(int)));
  *out = v;
  return ATMA_OK;
}

}  // namespace atma
