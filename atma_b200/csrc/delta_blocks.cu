// Gated delta rule in fp32 arithmetic, eight rows at a time.
//
// Row by row, S <- g S + k (beta (v - g S^T k))^T is a chain of two sums over the keys per row, each ending in shuffles:
// 0.58 us a row, whatever the rest of the chip does.  Over a block of eight rows the eight corrections are linear in the
// state in front of the block, so their products with it do not wait for one another.  With e_i = g_0 .. g_i and
// P_ij = g_{j+1} .. g_i inside the block:
//   rhs_i = beta_i (v_i - e_i S^T k_i)     A_ij = beta_i P_ij k_i.k_j (j < i)     T = (I + A)^-1
//   o_i   = e_i S^T q_i + sum_{j<=i} R'_ij rhs_j        R' = (P_ij q_i.k_j, j <= i) T
//   S     <- e_7 S + sum_j k'_j rhs_j^T                 k'_j = sum_{i>=j} P_7i T_ij k_i
// Kernel 1 makes T's products R' and k' of every block, side by side; kernel 2 walks the blocks.  Records take 1.6 KB per row and
// head of 128, so inputs whose records would take over 1 GB (85000 rows of 8 heads) go in portions, and the one sequence that a
// portion's end cuts hands its state on in the scratch.  Smaller portions would put sequences one behind the other that
// can be walked side by side (128 MB: 4 x 8192 rows 3.3 ms instead of 1.6).  In kernel 2 a warp owns four
// state columns, 16 lanes x DK / 16 rows for two of them; of the 16 products with k_i and q_i each lane ends up with one
// (halving exchange), the right sides go round once, and the update needs nothing else.  Bound by issue slots: about 60
// per row and warp, FMAs in pairs (f32x2).  Blocks of 16 rows would double the exchange and the factor work per row.
// Products of decays, not differences of logarithms, so a decay of zero stays one; terms of later rows are left out, not
// multiplied by zero, so an infinity does not reach rows in front of it.
// Measured (8 heads of 128 x 128, one sequence, both kernels): 1500 rows 866 -> 153 us
// against row by row, 2048 rows 1117 -> 216 us against chunks of 64 in fp32; errors against 64 bits unchanged (4.8e-6 of a
// whole model, 8.5e-7 of a block).
#include "delta_blocks.cuh"
#include "f32x2.cuh"

namespace atma {

namespace {

constexpr int kN = 8;                       // rows of a block
constexpr int kExtra = 96;                  // floats behind a record's vectors: R' [8][8] | e [8] | beta [8] | pad
constexpr int kAtE = kN * kN, kAtBeta = kAtE + kN;
constexpr int kStages = 4;
constexpr int64_t kMostBytes = 1 << 30;      // of the records that are there at a time

__host__ __device__ constexpr int record_floats(int DK) { return 3 * kN * DK + kExtra; }
// records in front of sequence s, whose first row is r0: enough for every sequence before it, without counting them
__device__ __forceinline__ int64_t first_record(int64_t r0, int s) { return r0 / kN + s; }

struct Rows { int64_t r0; int n; };
__device__ __forceinline__ Rows rows_of(const DeltaBlocks& a, int s) {
  if (a.cu_rows == nullptr) return {(int64_t)s * a.len, a.len};
  const int r0 = a.cu_rows[s];
  return {r0, a.cu_rows[s + 1] - r0};
}

// A portion's first record, and the states [H][dk][dv] that come in and go out where a sequence is cut.
struct Cut {
  int64_t first;
  const float* carry_in;
  float* carry_out;
};

template <typename T, int DK>
__global__ void __launch_bounds__(128)
delta_blocks_factors_kernel(const DeltaBlocks a, float* __restrict__ recs, int64_t n_records, int64_t first) {
  __shared__ __align__(16) float K[kN][DK + 4], Q[kN][DK + 4];
  __shared__ float g[kN], bt[kN], A[kN][kN], Rq[kN][kN], Tm[kN][kN];
  const int64_t idx = first + blockIdx.x;
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int lo = 0, hi = a.n_seqs - 1;            // the last sequence whose records begin at or before idx
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (first_record(rows_of(a, mid).r0, mid) <= idx) lo = mid; else hi = mid - 1;
  }
  const Rows seq = rows_of(a, lo);
  const int64_t at = (idx - first_record(seq.r0, lo)) * kN;
  if (at < 0 || at >= seq.n) return;
  const int valid = min((int64_t)kN, seq.n - at);
  const int64_t row0 = seq.r0 + at;
  float* rec = recs + ((int64_t)h * n_records + blockIdx.x) * record_floats(DK);
  const int hq = h / (a.H / a.Hq), hk = h / (a.H / a.G);

#pragma unroll
  for (int i = warp; i < kN; i += 4) {
    const bool ok = i < valid;
    const int64_t r = row0 + i;
    const T* qr = static_cast<const T*>(a.q) + (r * a.Hq + hq) * a.dk;
    const T* kr = static_cast<const T*>(a.k) + (r * a.G + hk) * a.dk;
    float qx[DK / 32], kx[DK / 32], qs = 0.f, ks = 0.f;
#pragma unroll
    for (int c = 0; c < DK / 32; ++c) {
      const int d = lane + 32 * c;
      qx[c] = ok && d < a.dk ? to_f32(qr[d]) : 0.f;
      kx[c] = ok && d < a.dk ? to_f32(kr[d]) : 0.f;
      qs = fmaf(qx[c], qx[c], qs);
      ks = fmaf(kx[c], kx[c], ks);
    }
    float qi = a.q_scale, ki = 1.f;
    if (a.q_inv != nullptr) {
      if (ok) { qi *= a.q_inv[r * a.Hq + hq]; ki = a.k_inv[r * a.G + hk]; }
    } else if (a.normalize) {
      qi *= 1.0f / fmaxf(sqrtf(warp_sum(qs)), 1e-12f);
      ki = 1.0f / fmaxf(sqrtf(warp_sum(ks)), 1e-12f);
    }
#pragma unroll
    for (int c = 0; c < DK / 32; ++c) {
      const int d = lane + 32 * c;
      const float kv = kx[c] * ki, qv = qx[c] * qi;
      K[i][d] = kv; Q[i][d] = qv;
      rec[i * DK + d] = kv; rec[(kN + i) * DK + d] = qv;
    }
    if (lane == 0) {
      g[i] = ok ? expf(a.log_decay[r * a.H + h]) : 1.f;
      bt[i] = ok ? a.beta[r * a.H + h] : 0.f;
    }
  }
  __syncthreads();

  const int i = (tid >> 3) & 7, j = tid & 7;
  if (j <= i) {                             // threads 0..63: A, 64..127: q.k
    const float4* x = reinterpret_cast<const float4*>(tid < 64 ? K[i] : Q[i]);
    const float4* y = reinterpret_cast<const float4*>(K[j]);
    float4 s = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int d = 0; d < DK / 4; ++d) {
      const float4 u = x[d], w = y[d];
      s.x = fmaf(u.x, w.x, s.x); s.y = fmaf(u.y, w.y, s.y); s.z = fmaf(u.z, w.z, s.z); s.w = fmaf(u.w, w.w, s.w);
    }
    float p = (s.x + s.y) + (s.z + s.w);
    for (int l = j + 1; l <= i; ++l) p *= g[l];
    if (tid < 64) A[i][j] = bt[i] * p; else Rq[i][j] = p;
  }
  __syncthreads();
  if (tid < kN) {                           // column tid of T
    float col[kN];
#pragma unroll
    for (int p = 0; p < kN; ++p) {
      float acc = p == tid ? 1.f : 0.f;
#pragma unroll
      for (int s = 0; s < p; ++s)
        if (s >= tid) acc = fmaf(-A[p][s], col[s], acc);
      col[p] = acc;
      Tm[p][tid] = acc;
    }
  }
  __syncthreads();
  float* extra = rec + 3 * kN * DK;
  if (tid < kN * kN) {
    float acc = 0.f;
    for (int s = j; s <= i; ++s) acc = fmaf(Rq[i][s], Tm[s][j], acc);
    extra[tid] = acc;
    if (j == 0) {
      float e = 1.f;
      for (int l = 0; l <= i; ++l) e *= g[l];
      extra[kAtE + i] = e;
      extra[kAtBeta + i] = bt[i];
    }
  }
  float left[kN];                           // P_7i
  left[kN - 1] = 1.f;
#pragma unroll
  for (int l = kN - 1; l > 0; --l) left[l - 1] = left[l] * g[l];
  for (int d = tid; d < DK; d += 128) {
    float kc[kN];
#pragma unroll
    for (int l = 0; l < kN; ++l) kc[l] = left[l] * K[l][d];
#pragma unroll
    for (int c = 0; c < kN; ++c) {
      float acc = 0.f;
#pragma unroll
      for (int l = c; l < kN; ++l) acc = fmaf(Tm[l][c], kc[l], acc);
      rec[(2 * kN + c) * DK + d] = acc;
    }
  }
}

// CUT: one of several portions (5% slower, so not where there is one only).
template <typename T, int DK, int W, bool CUT>
__global__ void __launch_bounds__(W * 32)
delta_blocks_walk_kernel(const DeltaBlocks a, const float* __restrict__ recs, int64_t n_records, const Cut p) {
  extern __shared__ __align__(16) float ring[];
  constexpr int R4 = DK / 64, kRec = record_floats(DK);        // quadruples of rows per lane
  const int tid = threadIdx.x, lane = tid & 31, l = lane & 15, half = lane >> 4;
  const int h = blockIdx.y, s = blockIdx.z;
  const int col = (blockIdx.x * W + (tid >> 5)) * 4 + half * 2;
  const bool c0 = col < a.dv, c1 = col + 1 < a.dv;
  Rows seq = rows_of(a, s);
  int64_t record = first_record(seq.r0, s);            // that it begins with in this portion
  int blocks = (seq.n + kN - 1) / kN;                  // it has there
  bool begun = false, ends = true;                     // portions in front have rows of it; there are none behind
  if constexpr (CUT) {
    const int64_t ahead = record - p.first;
    const int b0 = (int)max(-ahead, (int64_t)0), b1 = (int)min(n_records - ahead, (int64_t)blocks);
    if (blocks == 0 ? ahead < 0 || ahead >= n_records : b0 >= b1) return;
    begun = b0 > 0; ends = b1 == blocks;
    blocks = b1 - b0;
    record = ahead + b0;
    seq.r0 += (int64_t)b0 * kN; seq.n -= b0 * kN;
  }
  const int start = a.start_pos ? a.start_pos[s] : 1;
  const int64_t slot = a.slots ? a.slots[s] : s;
  T* o = static_cast<T*>(a.o) + (seq.r0 * a.H + h) * a.dv + col;
  const int64_t o_rs = (int64_t)a.H * a.dv;
  if (start < 0 || slot < 0) {
    for (int r = l; r < (CUT ? min(blocks * kN, seq.n) : seq.n); r += 16) {
      if (c0) o[r * o_rs] = from_f32<T>(0.f);
      if (c1) o[r * o_rs + 1] = from_f32<T>(0.f);
    }
    return;
  }
  const int64_t carry = (int64_t)h * a.dk * a.dv + col, plane = slot * a.state_ss + carry;
  uint64_t S[2][2 * R4];                    // [column][pair of rows]: rows 64 m + 4 l .. + 3
#pragma unroll
  for (int m = 0; m < 2 * R4; ++m) {
    float x[2][2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int row = 64 * (m >> 1) + 4 * l + 2 * (m & 1) + e;
      const float* src = (begun ? p.carry_in + carry : a.state_in + plane) + (int64_t)row * a.dv;
      const bool ok = (begun || (a.state_in != nullptr && start > 0)) && row < a.dk;
      x[0][e] = ok && c0 ? src[0] : 0.f;
      x[1][e] = ok && c1 ? src[1] : 0.f;
    }
    S[0][m] = pack2(x[0][0], x[0][1]);
    S[1][m] = pack2(x[1][0], x[1][1]);
  }

  const float* rec = recs + ((int64_t)h * n_records + record) * kRec;
  const int NB = CUT ? blocks : (seq.n + kN - 1) / kN;
  auto stage = [&](int b) {
    if (b < NB) {
      const float* src = rec + (int64_t)b * kRec;
      const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(ring + (b % kStages) * kRec));
      for (int i = tid; i < kRec / 4; i += W * 32)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * i), "l"(src + 4 * i) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int hv = h / (a.H / a.Hv);
  const T* v = static_cast<const T*>(a.v) + (seq.r0 * a.Hv + hv) * a.dv + col;
  const int64_t v_rs = (int64_t)a.Hv * a.dv;
  auto value = [&](int b) {
    const int r = b * kN + l;
    const bool ok = l < kN && r < seq.n;
    return float2{ok && c0 ? to_f32(v[r * v_rs]) : 0.f, ok && c1 ? to_f32(v[r * v_rs + 1]) : 0.f};
  };
#pragma unroll
  for (int b = 0; b < kStages - 1; ++b) stage(b);
  float2 v_now = value(0), v_next = value(1);

  for (int b = 0; b < NB; ++b) {
    const float2 v_after = value(b + 2);
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();                        // block b is there, and everyone is done with block b - 1
    stage(b + kStages - 1);
    const float* now = ring + (b % kStages) * kRec;
    const float* extra = now + 3 * kN * DK;
    const float e = extra[kAtE + (l & 7)], bt = extra[kAtBeta + (l & 7)], e_all = extra[kAtE + kN - 1];

    float d[2][2 * kN];                     // this lane's part of S^T k_i, S^T q_i
#pragma unroll
    for (int i = 0; i < 2 * kN; ++i) {
      uint64_t t0 = 0, t1 = 0;
#pragma unroll
      for (int m = 0; m < R4; ++m) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(now + i * DK + 64 * m + 4 * l);
        t0 = m ? fma2(x.x, S[0][2 * m], t0) : mul2(x.x, S[0][0]);
        t1 = m ? fma2(x.x, S[1][2 * m], t1) : mul2(x.x, S[1][0]);
        t0 = fma2(x.y, S[0][2 * m + 1], t0);
        t1 = fma2(x.y, S[1][2 * m + 1], t1);
      }
      const float2 f0 = unpack2(t0), f1 = unpack2(t1);
      d[0][i] = f0.x + f0.y;
      d[1][i] = f1.x + f1.y;
    }
#pragma unroll
    for (int off = kN; off > 0; off >>= 1) {
      const bool up = l & off;
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < off; ++i) {
          const float keep = up ? d[c][i + off] : d[c][i], send = up ? d[c][i] : d[c][i + off];
          d[c][i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    // lane l < 8: S^T k_l, lane l >= 8: S^T q_(l-8)
    const bool real = b * kN + (l & 7) < seq.n;
    const float rhs0 = real ? bt * (v_now.x - e * d[0][0]) : 0.f, rhs1 = real ? bt * (v_now.y - e * d[1][0]) : 0.f;
    float r0[kN], r1[kN];
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      r0[j] = __shfl_sync(0xffffffffu, rhs0, j, 16);
      r1[j] = __shfl_sync(0xffffffffu, rhs1, j, 16);
    }
    const uint64_t fade = pack2(e_all, e_all);
#pragma unroll
    for (int m = 0; m < 2 * R4; ++m) { S[0][m] = mul2(S[0][m], fade); S[1][m] = mul2(S[1][m], fade); }
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      const uint64_t p0 = pack2(r0[j], r0[j]), p1 = pack2(r1[j], r1[j]);
#pragma unroll
      for (int m = 0; m < R4; ++m) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(now + (2 * kN + j) * DK + 64 * m + 4 * l);
        S[0][2 * m] = fma2(x.x, p0, S[0][2 * m]);
        S[1][2 * m] = fma2(x.x, p1, S[1][2 * m]);
        S[0][2 * m + 1] = fma2(x.y, p0, S[0][2 * m + 1]);
        S[1][2 * m + 1] = fma2(x.y, p1, S[1][2 * m + 1]);
      }
    }
    if (l >= kN) {
      const int i = l - kN;
      const float4 ra = *reinterpret_cast<const float4*>(extra + i * kN), rb = *reinterpret_cast<const float4*>(extra + i * kN + 4);
      const float rr[kN] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
      float o0 = e * d[0][0], o1 = e * d[1][0];
#pragma unroll
      for (int j = 0; j < kN; ++j)
        if (j <= i) { o0 = fmaf(rr[j], r0[j], o0); o1 = fmaf(rr[j], r1[j], o1); }
      if (real) {
        T* at = o + (int64_t)(b * kN + i) * o_rs;
        if (c0) at[0] = from_f32<T>(o0);
        if (c1) at[1] = from_f32<T>(o1);
      }
    }
    v_now = v_next; v_next = v_after;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (ends && a.state_out == nullptr) return;
  float* to = ends ? a.state_out + plane : p.carry_out + carry;
#pragma unroll
  for (int m = 0; m < 2 * R4; ++m) {
    const float2 f0 = unpack2(S[0][m]), f1 = unpack2(S[1][m]);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int row = 64 * (m >> 1) + 4 * l + 2 * (m & 1) + e;
      float* dst = to + (int64_t)row * a.dv;
      if (row < a.dk && c0) dst[0] = e ? f0.y : f0.x;
      if (row < a.dk && c1) dst[1] = e ? f1.y : f1.x;
    }
  }
}

int padded(int dk) { return dk <= 64 ? 64 : (dk <= 128 ? 128 : 256); }
int64_t records(int64_t total_rows, int n_seqs) { return total_rows / kN + n_seqs; }
int64_t portion(int64_t n_records, int H, int dk) {
  const int64_t fit = kMostBytes / ((int64_t)H * record_floats(padded(dk)) * 4);
  return n_records <= fit ? n_records : (fit > 16 ? fit : 16);
}

template <typename T, int DK>
int launch(const DeltaBlocks& a, float* recs, cudaStream_t st) {
  const int64_t all = records(a.total_rows, a.n_seqs), n = portion(all, a.H, a.dk);
  float* carry = recs + n * a.H * record_floats(DK);
  const int64_t state = (int64_t)a.H * a.dk * a.dv;
  const int smem = kStages * record_floats(DK) * 4;
  // Every CTA reads its head's records again, so wide CTAs are better as long as they fill the chip.
#define ATMA_WALK(W, CUT)                                                                                                  \
  do {                                                                                                                     \
    auto kern = delta_blocks_walk_kernel<T, DK, W, CUT>;                                                                   \
    ATMA_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));                           \
    kern<<<dim3((a.dv + 4 * W - 1) / (4 * W), a.H, a.n_seqs), W * 32, smem, st>>>(a, recs, m, cut);                        \
  } while (0)
  for (int64_t first = 0, i = 0; first < all; first += n, ++i) {
    // two planes in turn: the state that comes in may be another sequence's than the one that goes out
    const Cut cut{first, carry + (i & 1) * state, carry + (~i & 1) * state};
    const int64_t m = first + n < all ? n : all - first;
    delta_blocks_factors_kernel<T, DK><<<dim3((unsigned)m, a.H), 128, 0, st>>>(a, recs, m, first);
    const bool wide = (int64_t)((a.dv + 31) / 32) * a.H * a.n_seqs >= sm_count_of_current_device();
    if (n < all) { if (wide) ATMA_WALK(8, true); else ATMA_WALK(2, true); }
    else { if (wide) ATMA_WALK(8, false); else ATMA_WALK(2, false); }
  }
#undef ATMA_WALK
  return launch_status("delta rule (fp32 arithmetic)");
}

}  // namespace

bool delta_blocks_supported(int64_t total_rows, int n_seqs, int H, int dk) {
  return dk > 0 && dk <= 256 && H > 0 && H <= 65535 && n_seqs > 0 && n_seqs <= 65535 && records(total_rows, n_seqs) < (int64_t(1) << 31);
}

int64_t delta_blocks_scratch_bytes(int64_t total_rows, int n_seqs, int H, int dk, int dv) {
  if (!delta_blocks_supported(total_rows, n_seqs, H, dk)) return 0;
  const int64_t all = records(total_rows, n_seqs), n = portion(all, H, dk);
  return n * H * record_floats(padded(dk)) * 4 + (n < all ? 2 * (int64_t)H * dk * dv * 4 : 0) + 16;
}

int delta_blocks_scan(const DeltaBlocks& a, void* scratch, cudaStream_t st) {
  ATMA_REQUIRE(scratch != nullptr, "delta rule: scratch is required");
  float* recs = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(scratch) + 15) & ~(uintptr_t)15);
  ATMA_DISPATCH_DTYPE(a.dtype, T, {
    if (a.dk <= 64) return launch<T, 64>(a, recs, st);
    if (a.dk <= 128) return launch<T, 128>(a, recs, st);
    return launch<T, 256>(a, recs, st);
  });
  return ATMA_OK;
}

}  // namespace atma
