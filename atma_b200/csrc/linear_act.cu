// The first product of an MLP with its activation, 16-bit, over many rows: out = act(x w^T + bias), where w holds two halves of
// features and the activation joins them (1: second * relu(first)^2, 2: gelu_tanh(first) * second) or one (3: relu(.)^2).
//
// As a library product and a kernel behind it, the product's result goes to memory and comes back, which is a third of the
// product's time again: 12000 x 8192 x 1024 136 us and 49 for the gate.  Here two SMs share a tile of 256 rows x 256 features
// (cta_group::2: each holds its 128 rows of x and half of the features, so that a stage of 64 columns is 32 KB a CTA for 512
// clocks of products; a CTA by itself would have to fetch 48 KB for them).  With two halves the tile is 128 features of each: the
// first CTA of the pair loads the first half's, its neighbour the second half's, and in either one's TMEM the two values that
// meet lie 128 columns apart in the same lane.  Pairs take tiles in turn, eight tiles of rows beside one another; the
// accumulators of one tile are read, joined and stored (32 rows x 64 columns a warp, through swizzled shared memory and TMA)
// while the next tile's products go to the other half of TMEM.
//   warp 0 TMA (both CTAs), warp 1 MMA (the first CTA's, for both), warps 2-9 activation and stores.
// Bound by the products: the same takes 125 us with the gate, 1609 TFLOP/s; 32768 x 8192 x 1024 337 us (form 2 352, 3 362) against 502
// (482, 583); 4096 x 16384 x 2048 164 against 195, 1677 TFLOP/s.  Few rows pay for a tile's latency (launch to end 19 us for one): see
// the rule where it is called.
// Rounding: forms 1 and 2 round what the product would have written and, in bf16, relu^2 before the gate, as the separate calls
// do; form 3 adds the bias to the fp32 sum and rounds once.
// Every mbarrier wait is bounded; on expiry the CTAs free their TMEM, return and leave a status word for the host.
#include "common.cuh"
#include "gelu.cuh"
#include "linear_act.cuh"
#include "sm100.cuh"

namespace atma {

namespace {

using namespace sm100;

constexpr int kBM = 128, kBK = 64, kBN = 128;              // a CTA's rows, columns of a stage, its share of the features
constexpr int kStages = 5;
constexpr int kPlane = kBM * kBK * 2, kStageBytes = 2 * kPlane;
constexpr int kOutWarps = 8, kThreads = 64 + 32 * kOutWarps;
constexpr int kStaging = 32 * 128;                          // bytes of a warp's 32 rows x 64 results
constexpr int kSmem = kStages * kStageBytes + kOutWarps * kStaging + 1024;
constexpr int kGroup = 8;                                   // tiles of rows beside one another

static_assert(kBM == kBN, "planes of x and w have one size");

__device__ int g_linear_act_status = 0;

struct Args {
  const void* bias;                         // [N] or null
  int M, N, K, width;                       // width: features of the result
};

__device__ __forceinline__ uint32_t in_first(uint32_t addr) {                      // the same place in the pair's first CTA
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// a tile into this CTA's memory, counted on a barrier of either
__device__ __forceinline__ void tma_load_pair(void* dst, const CUtensorMap* m, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(0), "r"(0)
      : "memory");
}
__device__ __forceinline__ void tma_store(const CUtensorMap* m, const void* src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(0), "r"(0)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void stores_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier at this place in both CTAs
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}


template <typename T, int kForm>
__device__ __forceinline__ float joined(float a, float b) {
  if constexpr (kForm == 3) {
    const float p = fmaxf(a, 0.f);
    return p * p;
  } else {
    a = round_through<T>(a); b = round_through<T>(b);
    if constexpr (kForm == 2) return gelu_tanh_16(a) * b;
    const float p = fmaxf(a, 0.f);
    float sq = p * p;
    if constexpr (std::is_same<T, __nv_bfloat16>::value) sq = round_through<T>(sq);
    return b * sq;
  }
}

template <typename T, int kForm>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
linear_act_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                  const __grid_constant__ CUtensorMap tm_out, const __grid_constant__ Args a) {
  constexpr bool kHalves = kForm != 3;
  constexpr int kTileN = kHalves ? kBN : 2 * kBN;           // results of a tile's row
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2];      // full and acc_empty: the first CTA's are used
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort_v;
  __shared__ __align__(16) float s_bias[kOutWarps][kHalves ? 2 : 1][64];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int m_tiles = (a.M + 2 * kBM - 1) / (2 * kBM), n_tiles = (a.width + kTileN - 1) / kTileN, tiles = m_tiles * n_tiles;
  auto place = [&](int tile, int& m0, int& n0) {            // the pair's first row, the first result of a row
    const int group = tile / (kGroup * n_tiles), in = tile - group * kGroup * n_tiles, tall = min(kGroup, m_tiles - group * kGroup);
    m0 = (group * kGroup + in % tall) * 2 * kBM;
    n0 = in / tall * kTileN;
  };

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
    for (int i = 0; i < kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 2 * kOutWarps); }
    s_abort_v = 0;
    fence_barrier_init();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                           // the neighbour's barriers are there
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const int NK = (a.K + kBK - 1) / kBK;
  volatile int* abort = &s_abort_v;

  if (warp == 0) {
    if (elect_one()) {
      uint32_t n = 0;                       // stages so far, over all tiles
      bool ok = true;
      for (int tile = pair; tile < tiles && ok; tile += pairs) {
        int m0, n0;
        place(tile, m0, n0);
        const int xr = m0 + (int)rank * kBM, wr = kHalves ? n0 + (int)rank * a.width : n0 + (int)rank * kBN;
        for (int it = 0; it < NK; ++it, ++n) {
          const uint32_t st = n % kStages;
          if (n >= kStages && !(ok = mbar_wait(&empty[st], (n / kStages - 1) & 1, abort))) break;
          uint8_t* to = smem + st * kStageBytes;
          if (rank == 0) mbar_arrive_expect_tx(&full[st], 2 * kStageBytes);
          const uint32_t bar = in_first(smem_u32(&full[st]));
          tma_load_pair(to, &tm_x, bar, it * kBK, xr);
          tma_load_pair(to + kPlane, &tm_w, bar, it * kBK, wr);
        }
      }
      // whatever the others do, the CTA does not end before its copies have landed and the products that read them are done
      volatile int alone = 0;
      for (uint32_t i = n > kStages ? n - kStages : 0; i < n; ++i)
        if (!mbar_wait(&empty[i % kStages], (i / kStages) & 1, &alone)) { *abort = 1; break; }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc(2 * kBM, 2 * kBN, std::is_same<T, __nv_bfloat16>::value ? 1 : 0, 0, 0);
      uint32_t n = 0, t = 0;
      bool ok = true;
      for (int tile = pair; tile < tiles && ok; tile += pairs, ++t) {
        const uint32_t buf = t & 1, d = tmem + buf * 2 * kBN;
        if (t >= 2 && !(ok = mbar_wait(&acc_empty[buf], (t / 2 - 1) & 1, abort))) break;
        tc_fence_after();
        for (int it = 0; it < NK; ++it, ++n) {
          const uint32_t st = n % kStages;
          if (!(ok = mbar_wait(&full[st], (n / kStages) & 1, abort))) break;
          tc_fence_after();
          const uint32_t at = smem_u32(smem + st * kStageBytes);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)
            mma_pair(d, make_sdesc_sw128(at + 32 * k, 16, 1024), make_sdesc_sw128(at + kPlane + 32 * k, 16, 1024), idesc, it > 0 || k > 0);
          commit_pair(&empty[st]);
        }
        if (ok) commit_pair(&acc_full[buf]);
      }
    }
  } else {
    const int w = warp - 2, quarter = warp & 3, side = w >> 2;
    uint8_t* s = smem + kStages * kStageBytes + w * kStaging;
    const T* bias = static_cast<const T*>(a.bias);
    uint32_t t = 0;
    for (int tile = pair; tile < tiles; tile += pairs, ++t) {
      const uint32_t buf = t & 1;
      int m0, n0;
      place(tile, m0, n0);
      const int row0 = m0 + (int)rank * kBM + 32 * quarter;
      if (!mbar_wait_warp(&acc_full[buf], (t / 2) & 1, abort)) break;
      tc_fence_after();
      const uint32_t at = tmem + (uint32_t(32 * quarter) << 16) + buf * 2 * kBN;
#pragma unroll 1
      for (int chunk = side; chunk < kTileN / 64; chunk += 2) {
        const int c0 = n0 + 64 * chunk;
        __syncwarp();
        if (lane == 0) stores_read();       // of the chunk in front, by the lane that asked for them
#pragma unroll
        for (int h = 0; h < (kHalves ? 2 : 1); ++h)
#pragma unroll
          for (int i = 0; i < 64; i += 32)
            s_bias[w][h][i + lane] = bias != nullptr && c0 + i + lane < a.width ? to_f32(bias[h * a.width + c0 + i + lane]) : 0.f;
        __syncwarp();
#pragma unroll 1
        for (int c = 0; c < 64; c += 32) {
          uint32_t y[kHalves ? 2 : 1][32];
          tmem_ld32_nowait(at + 64 * chunk + c, y[0]);
          if constexpr (kHalves) tmem_ld32_nowait(at + kBN + 64 * chunk + c, y[kHalves ? 1 : 0]);
          tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < (kHalves ? 2 : 1); ++h)
#pragma unroll
            for (int i = 0; i < 32; ++i) reg_fence(y[h][i]);
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
              const float4 b0 = *reinterpret_cast<const float4*>(&s_bias[w][0][c + i + j]);
              const float4 b1 = *reinterpret_cast<const float4*>(&s_bias[w][kHalves ? 1 : 0][c + i + j]);
              const float p[4] = {b0.x, b0.y, b0.z, b0.w}, q[4] = {b1.x, b1.y, b1.z, b1.w};
#pragma unroll
              for (int e = 0; e < 4; ++e)
                v[j + e] = joined<T, kForm>(__uint_as_float(y[0][i + j + e]) + p[e], __uint_as_float(y[kHalves ? 1 : 0][i + j + e]) + q[e]);
            }
            alignas(16) T o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = from_f32<T>(v[j]);
            *reinterpret_cast<uint4*>(s + lane * 128 + ((((c + i) >> 3) ^ (lane & 7)) << 4)) = *reinterpret_cast<const uint4*>(o);
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0 && row0 < a.M && c0 < a.width) tma_store(&tm_out, s, c0, row0);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_cluster(in_first(smem_u32(&acc_empty[buf])));
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync();                           // nobody signals a CTA that is gone
  tc_fence_after();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  if (tid == 0 && s_abort_v) atomicExch(&g_linear_act_status, 1);
}

int make_map(CUtensorMap* out, const void* base, bool bf16, int64_t rows, int64_t rs, int cols, int box_rows) {
  const uint64_t dims[4] = {(uint64_t)cols, (uint64_t)rows, 1, 1};
  const int64_t strides[3] = {rs, rs, rs};
  const uint32_t box[4] = {64, (uint32_t)box_rows, 1, 1};
  return make_tmap_16bit_4d(out, base, bf16, dims, strides, box);
}

template <typename T, int kForm>
int launch(const CUtensorMap& x, const CUtensorMap& w, const CUtensorMap& out, const Args& a, cudaStream_t st) {
  auto kern = linear_act_kernel<T, kForm>;
  ATMA_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  const int tile_n = kForm == 3 ? 2 * kBN : kBN;
  const int64_t tiles = (int64_t)((a.M + 2 * kBM - 1) / (2 * kBM)) * ((a.width + tile_n - 1) / tile_n);
  ATMA_REQUIRE(tiles < INT32_MAX / 2, "linear_act: too many tiles");
  const int pairs = sm_count_of_current_device() / 2;
  kern<<<2 * (unsigned)(tiles < pairs ? tiles : pairs), kThreads, kSmem, st>>>(x, w, out, a);
  return launch_status("linear_act (tcgen05)");
}

}  // namespace

int linear_act_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  ATMA_CUDA_OK(cudaMemcpyFromSymbol(&v, g_linear_act_status, sizeof(int)));
  if (v != 0) ATMA_CUDA_OK(cudaMemcpyToSymbol(g_linear_act_status, &zero, sizeof(int)));
  *out = v;
  return ATMA_OK;
}

}  // namespace atma

using namespace atma;

extern "C" int atma_linear_act(const void* x, int64_t x_rs, const void* weight, const void* bias, void* out, int64_t out_rs, int M, int N,
                               int K, int form, int dtype, void* stream) {
  ATMA_REQUIRE(dtype == ATMA_BF16 || dtype == ATMA_F16, "linear_act: 16-bit activations and weights only (dtype %d)", dtype);
  ATMA_REQUIRE(form >= 1 && form <= 3, "linear_act: unknown form %d", form);
  ATMA_REQUIRE(M >= 0 && M <= (1 << 29) && K > 0 && K <= (1 << 24) && K % 8 == 0, "linear_act: bad shape (%d, %d, %d)", M, N, K);
  ATMA_REQUIRE(N > 0 && N <= (1 << 24) && N % (form == 3 ? 8 : 16) == 0, "linear_act: N=%d must be a multiple of %d", N, form == 3 ? 8 : 16);
  if (M == 0) return ATMA_OK;
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const Args a{bias, M, N, K, form == 3 ? N : N / 2};
  ATMA_REQUIRE(x != nullptr && weight != nullptr && out != nullptr && al16(x) && al16(weight) && al16(out) && x_rs % 8 == 0 && out_rs % 8 == 0 &&
                   x_rs >= K && out_rs >= a.width,
               "linear_act: x, weight and out must be 16-byte aligned with row strides that are multiples of 8 elements");
  const bool bf16 = dtype == ATMA_BF16;
  CUtensorMap mx, mw, mo;
  int rc = make_map(&mx, x, bf16, M, x_rs, K, kBM);
  if (rc == ATMA_OK) rc = make_map(&mw, weight, bf16, N, K, K, kBN);
  if (rc == ATMA_OK) rc = make_map(&mo, out, bf16, M, out_rs, a.width, 32);
  if (rc != ATMA_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;
#define ATMA_ACT(T) (form == 1 ? launch<T, 1>(mx, mw, mo, a, st) : form == 2 ? launch<T, 2>(mx, mw, mo, a, st) : launch<T, 3>(mx, mw, mo, a, st))
  return bf16 ? ATMA_ACT(__nv_bfloat16) : ATMA_ACT(__half);
#undef ATMA_ACT
}
