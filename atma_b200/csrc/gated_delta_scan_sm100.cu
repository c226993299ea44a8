// Gated-delta scan, the recurrence over chunks, on the 5th-generation tensor cores (sm_100a):
// tcgen05.mma with TMEM accumulators, per-chunk factor records and the rows of q, k, v brought in by TMA.
//
// One CTA owns one (recurrence, head) and the whole state S [dk][dv], held TRANSPOSED: every
// thread of the eight state warps keeps 64 fp32 values of one row of S^T [v][k] in registers for
// the whole sequence.  Per 64-token chunk, with Tw, Tu, Rq and the row scalars of gated_delta_scan.cuh
// (s, p = rows of the chunk; k, v = key / value channel):
//
//   the chain
//     MMA   U^T += S^T (-W)^T                 K=128 (k);   state warps: U^T -> 16 bits, times (g_C / g) k_inv, then as it is
//     MMA   dS^T = (U (g_C / g) k_inv)^T K    N=128 (k);   state warps: S^T = g_C S^T + dS^T
//   under the thread phase of U, for the next chunk
//     MMA  -W^T = K^T Tw^T   M=128 (k) N=64 (p) K=64 (s);  W warps: -> 16 bits, shared memory (B operand)
//   under the thread phase of S, issued by a warp of its own so that the chain's never waits for what these wait for
//     MMA   U^T = V^T Tu^T of the next chunk; stays in TMEM
//     MMA   O1^T = S^T Q^T,  O2^T = U^T Rq^T;  O warps: o = g q_inv O1 + O2
//
// Q, K, V and the record tiles are operands exactly as TMA delivers them; scalars per row are applied to fp32
// accumulators.  fp16 has no room for an unbounded 1 / |k|, neither in Tw nor in U, so in chunks with very short or long
// rows a warp brings the K rows in shared memory to a length between 1 and 2 by a power of two, which loses nothing, ahead of
// the first product that reads them, and k_inv stands for what is left, a factor between 1/2 and 1.  The rows arrive shortly before
// that product, so this costs such a chunk 2000 clocks.  Behind the last rows of a sequence a chunk holds another's, whose
// factors are zero; they may be infinite or no numbers, so the same warp clears them.  The A operands of the chain (16-bit
// copies of S^T and U^T) are read from TMEM.  All accumulators have a channel on the 128 TMEM lanes, which spreads the thread
// phases over all four schedulers.
//
// What bounds it is the latency of the chain: 3000 to 3300 clocks a chunk, 1000 for the state's phase and its hand-over, 420 for U's
// products, 850 for U's phase, up to 600 of waiting for the next -W to leave dS^T's columns, 450 to 640 for dS's products; 2750
// without outputs, where -W has columns of its own.  Measured with the chunk-local stage, which no longer writes W, U0, Qg and
// Kt: 8 sequences of 16384 tokens, 8 heads, 330 + 412 us (617 + 385 with those in 72 KB records; fp16 995 -> 753 in all), 8 of 300
// 44 -> 36 us.  Context-parallel walks, 2 x 16384: state only 333 -> 349 us, with outputs 382 -> 412, factors 164 -> 93.
//
//   warp 0       TMA producer: V, Tw, Tu and K three chunks ahead, Q and Rq two
//   warp 1       issues the chain's products and -W^T; owns the TMEM allocation
//   warp 2       issues the other products
//   warp 3       K and V rows in place, where they need it
//   warps 4-11   state warps; warp w works on TMEM lanes 32 (w % 4) .. +31 and on column half
//                (w - 4) / 4 of whatever it reads (k for S^T, p for U^T); with sixteen of them a phase
//                takes longer, their waits and arrivals cost more than the shorter rows save
//   warps 12-15  W warps, warps 16-19 O warps: TMEM lanes 32 (w % 4) .. +31
// TMEM (512 columns allocated): 16-bit S^T [0,64) and, every other chunk, [64,128) | 16-bit U^T [128,160), scaled
// [160,192) | U^T fp32 [192,256) | O1^T [256,320) | O2^T [320,384) | dS^T [384,512), where -W^T of the next chunk passes
// through between the state's reading and the next dS^T; without outputs in O1^T's place.
// Every mbarrier wait is bounded; on expiry the CTA frees its TMEM, returns and leaves a status
// word for the host.
#include "common.cuh"
#include "sm100.cuh"
#include "gated_delta_scan.cuh"

namespace atma {

using namespace sm100;
using namespace scan;

namespace {

__device__ int g_scan_status = 0;

constexpr int kStateWarps = 8, kHelpWarps = 4, kThreads = 32 * (4 + kStateWarps + 2 * kHelpWarps);
// 640 threads are launched with 96 registers each, 61440; then 256 of them take 136 and 384 keep 64, together 59392
constexpr int kStateRegs = 136, kOtherRegs = 64;
constexpr int kRowBytes = kC * kD * 2;            // 64 rows of 128 channels: two boxes of 64 channels, 8 KiB each
// rings: [V | Tw | Tu], [K], [Q | Rq], scalars; then -W^T [128 k][64 p]
constexpr int kVts = 3, kVtBytes = kRowBytes + 2 * kTile64, kKs = 3, kQrs = 2, kQrBytes = kRowBytes + kTile64, kScs = 4, kScBytes = kScal * 4;
constexpr int kOffK = kVts * kVtBytes, kOffQr = kOffK + kKs * kRowBytes, kOffW = kOffQr + kQrs * kQrBytes, kOffSc = kOffW + kD * 128,
              kSmemBytes = kOffSc + kScs * kScBytes + 1024;
constexpr uint32_t kColSb = 0, kColUb = 128, kColUs = 160, kColU = 192, kColO1 = 256, kColO2 = 320, kColS = 384;

struct Barriers {
  uint64_t vt_full[kVts], vt_empty[kVts], k_full[kKs], k_empty[kKs], qr_full[kQrs], qr_empty[kQrs], sc_full[kScs], sc_empty[kScs];
  uint64_t last_sent, k_ready[kKs], v_ready, w_done, w_read, w_ready, u0_done, sb_ready, u_full, us_ready, ub_ready, s_done, o_done, o_free;
};

struct Params {
  const float* scal;
  const float* initial_state;
  void* o;
  float* final_state;
  int Tlen, H, Hkv, NC;
  RecMap map;
  VarLen var;
};

__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// shared-memory descriptors of tiles with 128-byte rows: K-major, and MN-major in boxes of 8 KiB
__device__ __forceinline__ uint64_t desc_k(uint32_t addr) {
  return (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61) | (uint64_t(16 >> 4) << 16) | uint64_t((addr >> 4) & 0x3FFFu);
}
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr) {
  return (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61) | (uint64_t(8192 >> 4) << 16) | uint64_t((addr >> 4) & 0x3FFFu);
}
template <int kRegs, bool kMore>
__device__ __forceinline__ void set_registers() {       // of every warp of a warpgroup
  if constexpr (kMore) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs));
  else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs));
}

// kWide: o is 4-byte aligned, two channels are stored at a time
template <bool kBf16, bool kWide>
__global__ void __launch_bounds__(kThreads, 1)
scan_recur_sm100_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                        const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_rec, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ Barriers bar;
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.x, b = blockIdx.y;
  const bool packed = p.var.cu_seqlens != nullptr;
  const int rb = packed ? 0 : p.map.rec[b];
  const bool zero_u0 = packed ? false : p.map.zero_u0[b] != 0;
  int c_begin, c_end;
  int64_t tok_in, tok_base, tok_end;                     // first token of the inputs; first and past-the-end token of o
  if (packed) {
    c_begin = p.var.cu_chunks[b]; c_end = p.var.cu_chunks[b + 1];
    tok_in = tok_base = p.var.cu_seqlens[b]; tok_end = p.var.cu_seqlens[b + 1];
  } else {
    c_begin = p.map.c_begin[b]; c_end = p.map.c_end[b] > 0 ? p.map.c_end[b] : p.NC;
    const int64_t orow0 = (int64_t)max(p.map.o_row[b], 0) * p.Tlen;  // the batch row of o this recurrence writes
    tok_in = (int64_t)rb * p.Tlen + (int64_t)c_begin * kC;
    tok_base = orow0 + (int64_t)c_begin * kC;
    tok_end = orow0 + min((int64_t)p.Tlen, (int64_t)c_end * kC);
  }
  const int n_chunks = max(c_end - c_begin, 0);
  const int last_rows = (int)(tok_end - tok_base - (int64_t)(n_chunks - 1) * kC);    // of the last chunk
  const bool want_o = p.o != nullptr && (packed || p.map.o_row[b] >= 0);   // a negative row: this recurrence only carries state
  const uint32_t col_w = want_o ? kColS : kColO1;                    // without outputs the chain need not wait for its reading
  auto partial = [&](int c) { return c == n_chunks - 1 && last_rows < kC; };
  auto prepared = [&](int c) { return !kBf16 || partial(c); };       // chunks whose K rows warp 3 works on first
  const int64_t rec0 = ((int64_t)rb * p.H + h) * p.NC + c_begin;     // first record of this recurrence

  if (tid == 0) {
    for (int i = 0; i < kVts; ++i) { mbar_init(&bar.vt_full[i], 1); mbar_init(&bar.vt_empty[i], 2); }
    for (int i = 0; i < kKs; ++i) { mbar_init(&bar.k_full[i], 1); mbar_init(&bar.k_empty[i], 1); mbar_init(&bar.k_ready[i], 1); }
    for (int i = 0; i < kQrs; ++i) { mbar_init(&bar.qr_full[i], 1); mbar_init(&bar.qr_empty[i], 1); }
    for (int i = 0; i < kScs; ++i) { mbar_init(&bar.sc_full[i], 1); mbar_init(&bar.sc_empty[i], kStateWarps + kHelpWarps + (kBf16 ? 0 : 1)); }
    mbar_init(&bar.sb_ready, kStateWarps); mbar_init(&bar.us_ready, kStateWarps); mbar_init(&bar.ub_ready, kStateWarps);
    mbar_init(&bar.last_sent, 1); mbar_init(&bar.v_ready, 1); mbar_init(&bar.w_read, kHelpWarps); mbar_init(&bar.w_ready, kHelpWarps); mbar_init(&bar.u0_done, 1); mbar_init(&bar.o_free, kHelpWarps);
    mbar_init(&bar.w_done, 1); mbar_init(&bar.u_full, 1); mbar_init(&bar.s_done, 1); mbar_init(&bar.o_done, 1);
    s_abort = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(&s_tmem_base, 512);
  if (warp == 0 && lane == 0) { prefetch_tensormap(&tmap_q); prefetch_tensormap(&tmap_k); prefetch_tensormap(&tmap_v); prefetch_tensormap(&tmap_rec); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = s_tmem_base;
  volatile int* abort_flag = &s_abort;

  if (warp < 4) {
    set_registers<kOtherRegs, false>();
    if (warp == 0) {
      // =============================== TMA producer ================================================
      if (elect_one()) {
        const int hk = h / (p.H / p.Hkv);
        for (int i = 0; i <= n_chunks; ++i) {
          if (i < n_chunks) {
            const int t0 = (int)(tok_in + (int64_t)i * kC), row = (int)((rec0 + i) * (3 * kC));
            uint8_t* st = smem + i % kVts * kVtBytes;
            uint64_t* full = &bar.vt_full[i % kVts];
            if (!mbar_wait(&bar.vt_empty[i % kVts], ((uint32_t)(i / kVts) & 1u) ^ 1u, abort_flag)) break;
            mbar_arrive_expect_tx(full, kVtBytes);
            tma_load_4d(st + kRowBytes, &tmap_rec, full, 0, row, 0, 0);
            tma_load_4d(st + kRowBytes + kTile64, &tmap_rec, full, 0, row + kC, 0, 0);
            tma_load_4d(st, &tmap_v, full, 0, hk, t0, 0);
            tma_load_4d(st + 8192, &tmap_v, full, 64, hk, t0, 0);
            st = smem + kOffK + i % kKs * kRowBytes;
            full = &bar.k_full[i % kKs];
            if (!mbar_wait(&bar.k_empty[i % kKs], ((uint32_t)(i / kKs) & 1u) ^ 1u, abort_flag)) break;
            mbar_arrive_expect_tx(full, kRowBytes);
            tma_load_4d(st, &tmap_k, full, 0, hk, t0, 0);
            tma_load_4d(st + 8192, &tmap_k, full, 64, hk, t0, 0);
            full = &bar.sc_full[i % kScs];
            if (!mbar_wait(&bar.sc_empty[i % kScs], ((uint32_t)(i / kScs) & 1u) ^ 1u, abort_flag)) break;
            mbar_arrive_expect_tx(full, kScBytes);
            bulk_load(smem + kOffSc + i % kScs * kScBytes, p.scal + (rec0 + i) * kScal, kScBytes, full);
            if (kBf16 && i == n_chunks - 1) mbar_arrive(&bar.last_sent);
          }
          const int c = i - 1;                           // what o needs comes a chunk behind
          if (want_o && c >= 0) {
            const int t0 = (int)(tok_in + (int64_t)c * kC), row = (int)((rec0 + c) * (3 * kC));
            uint8_t* st = smem + kOffQr + c % kQrs * kQrBytes;
            uint64_t* full = &bar.qr_full[c % kQrs];
            if (!mbar_wait(&bar.qr_empty[c % kQrs], ((uint32_t)(c / kQrs) & 1u) ^ 1u, abort_flag)) break;
            mbar_arrive_expect_tx(full, kQrBytes);
            tma_load_4d(st, &tmap_q, full, 0, h, t0, 0);
            tma_load_4d(st + 8192, &tmap_q, full, 64, h, t0, 0);
            tma_load_4d(st + kRowBytes, &tmap_rec, full, 0, row + 2 * kC, 0, 0);
          }
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      // =============================== the chain's products =======================================
      if (elect_one()) {
        constexpr int fmt = kBf16 ? 1 : 0;
        constexpr uint32_t idesc_w = make_idesc(128, 64, fmt, 0, 1);       // B = -W^T [k][p], MN-major
        constexpr uint32_t idesc_s = make_idesc(128, 128, fmt, 0, 1);      // B = K [s][k], MN-major
        constexpr uint32_t idesc_kt = make_idesc(128, 64, fmt, 1, 0);      // A = K rows [s][k], MN-major; B = Tw, K-major
        const uint32_t base = smem_u32(smem);
        const uint64_t wt = desc_mn(base + kOffW);
        bool ok = true;
        for (int i = -1; i < n_chunks && ok; ++i) {
          const uint32_t pi = (uint32_t)i & 1u;
          if (i >= 0) {
            ok = mbar_wait(&bar.w_ready, pi, abort_flag) && mbar_wait(&bar.u0_done, pi, abort_flag) && mbar_wait(&bar.sb_ready, pi, abort_flag);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              mma_ts(tbase + kColU, tbase + kColSb + 64 * pi + kk * 8, wt + uint64_t((kk * 2048) >> 4), idesc_w, (kk > 0 || !zero_u0) ? 1u : 0u);
            tc_commit(&bar.u_full);
          }
          const int n = i + 1;                           // -W^T of the next chunk, over dS^T, which has been read (sb_ready)
          if (n < n_chunks) {
            const uint32_t vt = base + n % kVts * kVtBytes, nkr = base + kOffK + n % kKs * kRowBytes;
            ok = mbar_wait(&bar.vt_full[n % kVts], (uint32_t)(n / kVts) & 1u, abort_flag) && mbar_wait(&bar.k_full[n % kKs], (uint32_t)(n / kKs) & 1u, abort_flag) &&
                 (!prepared(n) || mbar_wait(&bar.k_ready[n % kKs], kBf16 ? 0u : (uint32_t)(n / kKs) & 1u, abort_flag));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              mma_ss(tbase + col_w, desc_mn(nkr) + uint64_t((kk * 2048) >> 4), desc_k(vt + kRowBytes) + uint64_t((kk * 32) >> 4), idesc_kt, kk > 0);
            tc_commit(&bar.w_done);
            tc_commit(&bar.vt_empty[n % kVts]);
          }
          if (i < 0) continue;
          ok = mbar_wait(&bar.us_ready, pi, abort_flag) && (!want_o || n == n_chunks || mbar_wait(&bar.w_read, pi ^ 1u, abort_flag));
          if (!ok) break;
          tc_fence_after();
          const uint64_t kr = desc_mn(base + kOffK + i % kKs * kRowBytes);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_ts(tbase + kColS, tbase + kColUs + kk * 8, kr + uint64_t((kk * 2048) >> 4), idesc_s, kk > 0);
          tc_commit(&bar.s_done);
          tc_commit(&bar.k_empty[i % kKs]);
        }
      }
    } else if (warp == 2) {
      // =============================== the other products =========================================
      if (elect_one()) {
        constexpr int fmt = kBf16 ? 1 : 0;
        constexpr uint32_t idesc_vt = make_idesc(128, 64, fmt, 1, 0);      // A = V rows [s][v], MN-major; B = Tu, K-major
        constexpr uint32_t idesc_n64 = make_idesc(128, 64, fmt, 0, 0);     // B = Q or Rq rows, K-major
        const uint32_t base = smem_u32(smem);
        bool ok = true;
        for (int i = -1; i < n_chunks && ok; ++i) {
          const int n = i + 1;                           // U0^T of the next chunk, once U^T of this one has been read
          if (n < n_chunks) {
            const uint32_t vt = base + n % kVts * kVtBytes;
            ok = mbar_wait(&bar.vt_full[n % kVts], (uint32_t)(n / kVts) & 1u, abort_flag) && (i < 0 || mbar_wait(&bar.ub_ready, (uint32_t)i & 1u, abort_flag)) &&
                 (!partial(n) || mbar_wait(&bar.v_ready, 0, abort_flag));
            if (!ok) break;
            tc_fence_after();
            if (!zero_u0) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                mma_ss(tbase + kColU, desc_mn(vt) + uint64_t((kk * 2048) >> 4), desc_k(vt + kRowBytes + kTile64) + uint64_t((kk * 32) >> 4), idesc_vt, kk > 0);
            }
            tc_commit(&bar.u0_done);
            tc_commit(&bar.vt_empty[n % kVts]);
          }
          if (i >= 0 && want_o) {
            const uint32_t qr = base + kOffQr + i % kQrs * kQrBytes;
            ok = mbar_wait(&bar.ub_ready, (uint32_t)i & 1u, abort_flag) && mbar_wait(&bar.qr_full[i % kQrs], (uint32_t)(i / kQrs) & 1u, abort_flag) &&
                 (i == 0 || mbar_wait(&bar.o_free, (uint32_t)(i - 1) & 1u, abort_flag));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              mma_ts(tbase + kColO1, tbase + kColSb + 64 * (i & 1) + kk * 8, desc_k(qr) + uint64_t(((kk >> 2) * 8192 + (kk & 3) * 32) >> 4), idesc_n64, kk > 0);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              mma_ts(tbase + kColO2, tbase + kColUb + kk * 8, desc_k(qr + kRowBytes) + uint64_t((kk * 32) >> 4), idesc_n64, kk > 0);
            tc_commit(&bar.o_done);
            tc_commit(&bar.qr_empty[i % kQrs]);
          }
        }
      }
    } else {
      // =============================== rows in place ==============================================
      // zeros for what is not the sequence's; in fp16 K rows times their powers of two, if a chunk has any: eight lanes a row
      for (int c = kBf16 ? max(n_chunks - 1, 0) : 0; c < n_chunks; ++c) {
        if (!prepared(c)) break;
        // K and V have been asked for before either of these, so their barriers are in this chunk's phase
        if (!(kBf16 ? mbar_wait_warp(&bar.last_sent, 0, abort_flag) : mbar_wait_warp(&bar.sc_full[c % kScs], (uint32_t)(c / kScs) & 1u, abort_flag))) break;
        const float* sc = reinterpret_cast<const float*>(smem + kOffSc + c % kScs * kScBytes);
        const bool scaled = !kBf16 && sc[kScalFar] != 0.f;
        const int rows = partial(c) ? last_rows : kC;
        if (scaled || rows < kC) {
          if (!mbar_wait_warp(&bar.k_full[c % kKs], (uint32_t)(c / kKs) & 1u, abort_flag)) break;
          uint8_t* kr = smem + kOffK + c % kKs * kRowBytes;
#pragma unroll 8
          for (int i = 0; i < 32; ++i) {                 // both boxes of a row one after the other
            const int r = 4 * (i >> 1) + (lane >> 3);
            uint4* at = reinterpret_cast<uint4*>(kr + (i & 1) * 8192 + box_off(r, lane & 7));
            if (r >= rows) {
              *at = make_uint4(0u, 0u, 0u, 0u);
            } else if (scaled) {
              uint4 u = *at;
              const __half2 f = reinterpret_cast<const __half2*>(sc)[kScalP + r], f1 = __low2half2(f), f2 = __high2half2(f);
              __half2* v = reinterpret_cast<__half2*>(&u);
#pragma unroll
              for (int e = 0; e < 4; ++e) v[e] = __hmul2(__hmul2(v[e], f1), f2);
              *at = u;
            }
          }
          fence_proxy_async();
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&bar.k_ready[c % kKs]);
          if constexpr (!kBf16) mbar_arrive(&bar.sc_empty[c % kScs]);
        }
        if (rows < kC) {
          if (!mbar_wait_warp(&bar.vt_full[c % kVts], (uint32_t)(c / kVts) & 1u, abort_flag)) break;
          uint8_t* vr = smem + c % kVts * kVtBytes;
#pragma unroll 4
          for (int i = 0; i < 32; ++i) {
            const int r = 4 * (i >> 1) + (lane >> 3);
            if (r >= rows) *reinterpret_cast<uint4*>(vr + (i & 1) * 8192 + box_off(r, lane & 7)) = make_uint4(0u, 0u, 0u, 0u);
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar.v_ready);
        }
      }
    }
  } else if (warp < 4 + kStateWarps) {
    set_registers<kStateRegs, true>();
    // =============================== state warps ==================================================
    const int quad = warp & 3, half = (warp - 4) >> 2;
    const int row = 32 * quad + lane;                    // TMEM lane = value channel v
    const uint32_t lane_base = tbase + (uint32_t(32 * quad) << 16);

    // where the state comes from and goes to: element (k, v) of the [dk][dv] plane, k = 64*half + j
    const int64_t plane = ((int64_t)h * kD + 64 * half) * kD + row;
    auto table = [&] { return p.var.state_table + p.var.slots[b] * p.var.slot_stride + plane; };
    const bool tabled = packed && p.var.state_table != nullptr;
    const int64_t sbase = (int64_t)(packed ? b : p.map.state_row[b]) * p.H * kD * kD + plane;

    float2 S[32];                                         // S^T[v = row][k = 64*half + j], fp32 master
    {
      const float* s_in = p.initial_state ? p.initial_state + sbase : nullptr;
      if (tabled) s_in = (p.var.has_initial == nullptr || p.var.has_initial[b] != 0) ? table() : nullptr;
#pragma unroll
      for (int j = 0; j < 32; ++j) S[j] = s_in ? make_float2(s_in[2 * j * kD], s_in[(2 * j + 1) * kD]) : make_float2(0.f, 0.f);
    }
    auto put = [&](float* dst) {
#pragma unroll
      for (int j = 0; j < 32; ++j) { dst[2 * j * kD] = S[j].x; dst[(2 * j + 1) * kD] = S[j].y; }
    };
    bool ok = true;
    float gC = 0.f;                                       // decay over the chunk before
    for (int i = 0; i <= n_chunks; ++i) {
      const uint32_t sb = lane_base + kColSb + 64 * (i & 1) + 32 * half;
      // ---- state phase: after this block S is the state before chunk i, its 16-bit copy the A operand of U and O1 ------
      if (i > 0) {
        ok = mbar_wait_warp(&bar.s_done, (uint32_t)(i - 1) & 1u, abort_flag);
        if (!ok) break;
        tc_fence_after();
        uint32_t d[2][16];
        tmem_ld16_nowait(lane_base + kColS + 64 * half, d[0]);
#pragma unroll
        for (int part = 0; part < 4; ++part) {            // the next 16 columns are on their way while these are added
          uint32_t(&x)[16] = d[part & 1];
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) reg_fence(x[j]);
          if (part < 3) tmem_ld16_nowait(lane_base + kColS + 64 * half + 16 * (part + 1), d[(part + 1) & 1]);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            S[8 * part + j] = __ffma2_rn(make_float2(gC, gC), S[8 * part + j], make_float2(__uint_as_float(x[2 * j]), __uint_as_float(x[2 * j + 1])));
          uint32_t w[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) w[j] = pack2<kBf16>(S[8 * part + j].x, S[8 * part + j].y);
          tmem_st8(sb + 8 * part, w);
        }
      } else {
#pragma unroll
        for (int part = 0; part < 4; ++part) {
          uint32_t w[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) w[j] = pack2<kBf16>(S[8 * part + j].x, S[8 * part + j].y);
          tmem_st8(sb + 8 * part, w);
        }
      }
      tmem_st_wait();
      tc_fence_before();                                  // also: the dS^T columns have been read, the next may overwrite them
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.sb_ready);          // nobody waits for the last one
      // snapshot: the state after i chunks
      if (packed && p.var.snapshots != nullptr && i > 0 && (i % p.var.snap_chunks) == 0 && tok_base + (int64_t)i * kC <= tok_end)
        put(p.var.snapshots + ((int64_t)p.var.snap_offsets[b] + i / p.var.snap_chunks - 1) * p.H * kD * kD + plane);
      if (i == n_chunks) break;

      // ---- U^T of this chunk: chunk rows 32*half .. +31, as it is and scaled ------------------------------
      const float* sc = reinterpret_cast<const float*>(smem + kOffSc + i % kScs * kScBytes);
      ok = mbar_wait_warp(&bar.sc_full[i % kScs], (uint32_t)(i / kScs) & 1u, abort_flag);
      if (!ok) break;
      gC = sc[kScalG];
      ok = mbar_wait_warp(&bar.u_full, (uint32_t)i & 1u, abort_flag);
      if (!ok) break;
      tc_fence_after();
      {
        uint32_t r[32];
        tmem_ld32(lane_base + kColU + 32 * half, r);
        {
          uint32_t w[16];
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float4 ks = *reinterpret_cast<const float4*>(sc + kScalK + 32 * half + 2 * j);
            const float2 x = __fmul2_rn(make_float2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])), make_float2(ks.x, ks.y));
            const float2 y = __fmul2_rn(make_float2(__uint_as_float(r[2 * j + 2]), __uint_as_float(r[2 * j + 3])), make_float2(ks.z, ks.w));
            w[j] = pack2<kBf16>(x.x, x.y);
            w[j + 1] = pack2<kBf16>(y.x, y.y);
          }
          tmem_st16(lane_base + kColUs + 16 * half, w);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar.us_ready);
        }
        // the products of o one chunk back have read the plain copy, and the S^T that the next one will take the place of
        if (want_o && i > 0 && !(ok = mbar_wait_warp(&bar.o_done, (uint32_t)(i - 1) & 1u, abort_flag))) break;
        uint32_t w[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) w[j] = pack2<kBf16>(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
        tmem_st16(lane_base + kColUb + 16 * half, w);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&bar.ub_ready);
          mbar_arrive(&bar.sc_empty[i % kScs]);
        }
      }
    }
    if (ok) {
      if (tabled) put(table());
      else if (p.final_state != nullptr) put(p.final_state + sbase);
    }
  } else if (warp < 4 + kStateWarps + kHelpWarps) {
    set_registers<kOtherRegs, false>();
    // =============================== W warps ======================================================
    const int row = 32 * (warp & 3) + lane;              // TMEM lane: key channel
    const uint32_t lane_base = tbase + (uint32_t(32 * (warp & 3)) << 16);
    for (int i = 0; i < n_chunks; ++i) {
      if (!mbar_wait_warp(&bar.w_done, (uint32_t)i & 1u, abort_flag)) break;       // the chain's product with the one before is done, too
      tc_fence_after();
      uint32_t w[32];
#pragma unroll
      for (int hh = 0; hh < 4; ++hh) {
        uint32_t r[16];
        tmem_ld16(lane_base + col_w + 16 * hh, r);
#pragma unroll
        for (int e = 0; e < 8; ++e) w[8 * hh + e] = pack2<kBf16>(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.w_read);
      uint8_t* wt = smem + kOffW;
#pragma unroll
      for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(wt + box_off(row, c)) = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.w_ready);
    }
  } else {
    set_registers<kOtherRegs, false>();
    // =============================== O warps ======================================================
    const int row = 32 * (warp & 3) + lane;              // TMEM lane: value channel
    const uint32_t lane_base = tbase + (uint32_t(32 * (warp & 3)) << 16);
    const int64_t orow = (int64_t)p.H * kD;
    for (int i = 0; i < n_chunks; ++i) {
      if (!mbar_wait_warp(&bar.sc_full[i % kScs], (uint32_t)(i / kScs) & 1u, abort_flag)) break;
      if (!want_o) {                                     // not before the scalars are there: an arrival belongs to one use of their place
        if (lane == 0) mbar_arrive(&bar.sc_empty[i % kScs]);
        continue;
      }
      if (!mbar_wait_warp(&bar.o_done, (uint32_t)i & 1u, abort_flag)) break;
      tc_fence_after();
      const float* qs = reinterpret_cast<const float*>(smem + kOffSc + i % kScs * kScBytes) + kScalQ;
      const int n_ok = (int)min((int64_t)kC, tok_end - (tok_base + (int64_t)i * kC));
      uint16_t* first = static_cast<uint16_t*>(p.o) + ((tok_base + (int64_t)i * kC) * p.H + h) * kD + row;
#pragma unroll 1
      for (int hh = 0; hh < 4; ++hh) {
        uint32_t x[16], y[16], w[8];                     // w: rows 2 j and 2 j + 1
        tmem_ld16_nowait(lane_base + kColO1 + 16 * hh, x);
        tmem_ld16_nowait(lane_base + kColO2 + 16 * hh, y);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          const float4 f = *reinterpret_cast<const float4*>(qs + 16 * hh + 2 * j);
#pragma unroll
          for (int e = 0; e < 4; ++e) { reg_fence(x[2 * j + e]); reg_fence(y[2 * j + e]); }
          const float2 a = __ffma2_rn(make_float2(f.x, f.y), make_float2(__uint_as_float(x[2 * j]), __uint_as_float(x[2 * j + 1])),
                                      make_float2(__uint_as_float(y[2 * j]), __uint_as_float(y[2 * j + 1])));
          const float2 b2 = __ffma2_rn(make_float2(f.z, f.w), make_float2(__uint_as_float(x[2 * j + 2]), __uint_as_float(x[2 * j + 3])),
                                       make_float2(__uint_as_float(y[2 * j + 2]), __uint_as_float(y[2 * j + 3])));
          w[j] = pack2<kBf16>(a.x, a.y);
          w[j + 1] = pack2<kBf16>(b2.x, b2.y);
        }
        if (hh == 3) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) { mbar_arrive(&bar.o_free); mbar_arrive(&bar.sc_empty[i % kScs]); }
        }
        if constexpr (kWide) {
          // two lanes swap halves, so that an even one stores two channels of the even row, an odd one of the odd row
          uint32_t* dst = reinterpret_cast<uint32_t*>(first - (lane & 1) + ((lane & 1) + 16 * hh) * orow);
          const uint32_t pick = lane & 1 ? 0x3276u : 0x5410u;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t other = __shfl_xor_sync(0xffffffffu, w[j], 1);
            if (16 * hh + 2 * j + (lane & 1) < n_ok) *dst = __byte_perm(w[j], other, pick);
            dst += orow;
          }
        } else {
          uint16_t* dst = first + 16 * hh * orow;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (16 * hh + j < n_ok) *dst = (uint16_t)(w[j >> 1] >> (16 * (j & 1)));
            dst += orow;
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0 && s_abort) atomicExch(&g_scan_status, 1);
  if (warp == 1) tmem_dealloc(tbase, 512);
}

}  // namespace

int gated_delta_recur_sm100(const Rows& rows, const uint8_t* recs, const float* scal, int64_t n_records, const float* initial_state,
                            void* o, float* final_state, int Tlen, int NC, int n_rec, const RecMap& map, const VarLen& var,
                            cudaStream_t st) {
  if (n_rec <= 0 || n_records <= 0) return ATMA_OK;
  if (n_records * 3 * kC >= (int64_t(1) << 31))
    return fail(ATMA_ERR_INVALID, "gated_delta_scan: %lld chunk records exceed the tensor-map row range", (long long)n_records);
  if (rows.tokens >= (int64_t(1) << 31)) return fail(ATMA_ERR_INVALID, "gated_delta_scan: %lld tokens exceed the tensor-map range", (long long)rows.tokens);
  CUtensorMap mq, mk, mv, mr;
  int rc = make_rows_map(&mq, rows.q, rows.is_bf16, rows.H, rows.tokens);
  if (rc == ATMA_OK) rc = make_rows_map(&mk, rows.k, rows.is_bf16, rows.Hkv, rows.tokens);
  if (rc == ATMA_OK) rc = make_rows_map(&mv, rows.v, rows.is_bf16, rows.Hkv, rows.tokens);
  if (rc == ATMA_OK) {
    const uint64_t n = (uint64_t)n_records * 3 * kC;                 // a record as rows of 64 values
    const uint64_t dims[4] = {64, n, 1, 1};
    const int64_t strides[3] = {64, (int64_t)n * 64, (int64_t)n * 64};
    const uint32_t box[4] = {64, 64, 1, 1};
    rc = make_tmap_16bit_4d(&mr, recs, rows.is_bf16, dims, strides, box);
  }
  if (rc != ATMA_OK) return rc;
  Params p{};
  p.scal = scal; p.initial_state = initial_state; p.o = o; p.final_state = final_state;
  p.Tlen = Tlen; p.H = rows.H; p.Hkv = rows.Hkv; p.NC = NC; p.map = map; p.var = var;
  const bool wide = (reinterpret_cast<uintptr_t>(o) & 3) == 0;
  auto kernel = rows.is_bf16 ? (wide ? scan_recur_sm100_kernel<true, true> : scan_recur_sm100_kernel<true, false>)
                             : (wide ? scan_recur_sm100_kernel<false, true> : scan_recur_sm100_kernel<false, false>);
  ATMA_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
  kernel<<<dim3(rows.H, n_rec), kThreads, kSmemBytes, st>>>(mq, mk, mv, mr, p);
  return launch_status("gated_delta_scan (recurrence, tcgen05)");
}

int scan_sm100_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  ATMA_CUDA_OK(cudaMemcpyFromSymbol(&v, g_scan_status, sizeof(int)));
  if (v != 0) ATMA_CUDA_OK(cudaMemcpyToSymbol(g_scan_status, &zero, sizeof(int)));
  *out = v;
  return ATMA_OK;
}

}  // namespace atma
