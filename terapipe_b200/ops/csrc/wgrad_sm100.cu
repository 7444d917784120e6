// Weight gradients of all layers of a stage in one launch per kind of weight, for sm_100a:
//   g[l] = dY[l]^T X[l]    (dY [K][M], X [K][N], K = all rows of the stage's batch, M and N contiguous)
// and what becomes of g: straight into Adam (it is never stored), or into the fp32 gradient matrix.
//
// One launch for all layers: a layer's product is often 1.3 to 3.5 waves of tiles (2048 x 6144: 192
// tiles of 256 x 256 on 74 CTA pairs), each with an empty part of a wave, a start and an exposed last
// epilogue of its own; the tiles of all layers fill whole waves but for one.  The layers' buffers lie a
// constant distance apart, so one 3-D tensor map reaches all of them.
//
// 256 rows of 256 columns, 24 layers: 18 us for the products of a layer one by one, 1.6 in these launches;
// 8192 x 768, 10 layers: 131 and 87.
//
// Adam in the epilogue: 26 bytes a parameter move (12 read, 12 written, the 16-bit copy) instead of the 8
// of an accumulating gradient and the 34 of a pass over flat buffers, and they move under the main loop of
// the next tile.  us for the four weights of a layer, rows x width: product + pass / this kernel (of which the
// bare product):
//   256 x 256 22.6 / 4.5 (1.6), 8192 x 768 170 / 105 (87), 16384 x 2048 1804 / 1433 (1254), 6144 x 2560
//   1232 / 844 (658), 16384 x 5120 10653 / 9057 (8271), 4096 x 12288 26125 / 16440 (12678).
//
// The product is the CTA-pair GEMM (two CTAs of a cluster, one 256 x BN tile, see gemm_sm100.cu).
#include "adam.cuh"
#include "common.cuh"
#include "ptx.cuh"
#include "tile_choice.h"
#include "tile_order.h"

namespace tp {

struct WgradParams {
  int M, N, K;
  int num_m_tiles, num_tiles, layers;   // tiles of one layer
  int num_n_tiles, m_major, m_first, order_split, order_group, order_first_only, order_pipelined;  // TileOrder
  long long ldo, layer_stride;          // of the output matrices, in elements
  float* grad;                          // gradient kernels
  int accumulate;                       // 1: fetched ahead and added here, 2: added in L2
  AdamBuffers adam;                     // ADAM kernels: the optimizer's matrices
  int follows;                          // the launch before this one is another of these products
  int* err;
};

constexpr int kWgBM = 128, kWgBK = 64;
constexpr int kWgThreads = 320, kWgEpiWarps = 8;
constexpr int kWgEpiBytes = 8192;       // a 32 x 64 fp32 chunk per epilogue warp

template <int BN> struct WgradCfg {
  static constexpr int kABytes = kWgBM * kWgBK * 2;
  static constexpr int kBChunks = (BN / 2 + 63) / 64;   // a CTA's half of B comes in 64-column chunks
  static constexpr int kStageBytes = kABytes + kBChunks * 64 * kWgBK * 2;
  static constexpr int kStages = BN > 128 ? 5 : 6;
  static constexpr int kAccCols = BN > 128 ? 256 : 128;
  static constexpr int kTmemCols = 2 * kAccCols;
  static constexpr int kSmemBytes = kStages * kStageBytes + kWgEpiWarps * kWgEpiBytes + 1024 + 256;
};

// What the epilogue needs from memory for 8 rows of a 32 x 64 chunk: four rows a lane, 16 bytes of each.  A
// thread holds a row of the accumulator, but the matrices in memory are wanted in long pieces of a row, so
// the chunk turns round in the warp's shared memory.  256 bytes a row, 512 with the chunk of the quarter's
// other warp beside it, keep DRAM rows open: with 128 and 256, 4096 x 12288 over 4096 rows took 443 us
// instead of 422.  One set (48 registers with Adam) is fetched ahead of its use; the epilogue warps of an SM have
// 48 KB in flight.
template <bool ADAM> struct WgradRegs { float4 p[4], m[ADAM ? 4 : 1], v[ADAM ? 4 : 1]; };

template <bool ADAM>
__device__ __forceinline__ void wgrad_fetch(const WgradParams& p, WgradRegs<ADAM>& a, long long base, int row0, int n,
                                            int q, int lane) {
  if (!ADAM && p.accumulate != 1) return;
  const int col = n + (lane & 15) * 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int row = row0 + q * 8 + k * 2 + (lane >> 4);
    if (row < p.M && col < p.N) {
      const long long i = base + row * p.ldo + col;
      if (ADAM) {
        a.p[k] = __ldcs(reinterpret_cast<const float4*>(p.adam.p + i));
        a.m[k] = __ldcs(reinterpret_cast<const float4*>(p.adam.m + i));
        a.v[k] = __ldcs(reinterpret_cast<const float4*>(p.adam.v + i));
      } else {
        a.p[k] = __ldcs(reinterpret_cast<const float4*>(p.grad + i));
      }
    }
  }
}

template <typename T, bool ADAM>
__device__ __forceinline__ void wgrad_finish(const WgradParams& p, const AdamCoef& co, WgradRegs<ADAM>& a,
                                             const uint8_t* sb, long long base, int row0, int n, int q, int lane) {
  const int col = n + (lane & 15) * 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int rr = q * 8 + k * 2 + (lane >> 4), row = row0 + rr;
    if (row < p.M && col < p.N) {
      float4 g = *reinterpret_cast<const float4*>(sb + rr * 256 + (((lane & 15) ^ (rr & 7)) << 4));
      const long long i = base + row * p.ldo + col;
      if (ADAM) {
        adam_update(g, a.p[k], a.m[k], a.v[k], co);
        __stcs(reinterpret_cast<float4*>(p.adam.p + i), a.p[k]);
        __stcs(reinterpret_cast<float4*>(p.adam.m + i), a.m[k]);
        __stcs(reinterpret_cast<float4*>(p.adam.v + i), a.v[k]);
        uint2 w;
        w.x = Elem<T>::pack2(a.p[k].x, a.p[k].y);
        w.y = Elem<T>::pack2(a.p[k].z, a.p[k].w);
        __stcs(reinterpret_cast<uint2*>(static_cast<T*>(p.adam.model) + i), w);
      } else {
        if (p.accumulate == 1) { g.x += a.p[k].x; g.y += a.p[k].y; g.z += a.p[k].z; g.w += a.p[k].w; }
        // (in L2: one addition an element a launch, so the order is the launches')
        if (p.accumulate == 2) atomicAdd(reinterpret_cast<float4*>(p.grad + i), g);
        else __stcs(reinterpret_cast<float4*>(p.grad + i), g);
      }
    }
  }
}

// The optimizer's values of a 32 x 64 chunk on their way to L2: two lines a row and matrix.  Where the main loop
// is shorter than the epilogue, the epilogue's latency is what a tile waits for; under a longer one the lines
// only get in the operands' way.  4096 x 12288, us without / with, over 512 rows 377 / 299, 1536 382 / 323, 2048
// 386 / 341, 3072 408 / 403, 4096 415 / 436.
constexpr int kWgPrefetchK = 3072;
// Gradients that are added to, the other way round: under a longer main loop the values fetched ahead come for nothing,
// under a short one that chain is what a tile waits for, and nobody waits for what L2 adds up.  us fetched / added in L2,
// the four weights of one layer: 1600 wide over 32 rows 73.7 / 50.8, 2048 over 256 114 / 92, 4096 over 256 413 / 332; one
// weight, four times as high: 2048 wide over 1024 41.5 / 32.5, 4096 over 1024 155 / 144, over 2048 216 / 222, over 4096 467 / 482.
constexpr int kWgAddInL2K = 1024;
__device__ __forceinline__ void wgrad_prefetch(const WgradParams& p, long long base, int row0, int n, int lane) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int row = row0 + h * 16 + (lane >> 1), col = n + (lane & 1) * 32;
    if (row < p.M && col < p.N) {
      const long long i = base + row * p.ldo + col;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.adam.p + i));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.adam.m + i));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.adam.v + i));
    }
  }
}

template <typename T, int BN, bool ADAM>
__global__ void __launch_bounds__(kWgThreads, 1)
wgrad_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const WgradParams p) {
  using Cfg = WgradCfg<BN>;
  constexpr int S = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* epi_smem = smem + S * Cfg::kStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi_smem + kWgEpiWarps * kWgEpiBytes);
  uint64_t* full = bars;               // in the leader: both CTAs' loads count their bytes on it
  uint64_t* empty = bars + S;
  uint64_t* tfull = bars + 2 * S;
  uint64_t* tempty = bars + 2 * S + 2; // in the leader: the epilogue warps of both CTAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();   // 0 = leader
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const WaitCtx wctx{abort_flag, p.err};

  if (threadIdx.x == 0) {
    for (int i = 0; i < S; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 2 * kWgEpiWarps);
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers are initialised before any remote arrival
  if (p.follows) pdl_trigger();
  else pdl_wait();     // set-up done; from here on the predecessor's results are read
  uint32_t tmem_base = 0;
  if (warp >= 1) {     // (the producer warp starts loading at once)
    if (warp == 1) {
      tmem_alloc_pair(tmem_slot, Cfg::kTmemCols);
      tmem_relinquish_pair();
    }
    tc_fence_before();
    asm volatile("bar.sync 1, 288;" ::: "memory");
    tc_fence_after();
    tmem_base = *tmem_slot;
  }
  const int num_kb = (p.K + kWgBK - 1) / kWgBK;
  const int total = p.num_tiles * p.layers;
  auto coords = [&](int tile, int& layer, int& m_idx, int& n_idx) {
    layer = tile / p.num_tiles;
    pair_tile_coords(p, tile - layer * p.num_tiles, m_idx, n_idx);
  };

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < total && ok; tile += npairs) {
        int layer, m_idx, n_idx;
        coords(tile, layer, m_idx, n_idx);
        const int m0 = m_idx * (2 * kWgBM) + static_cast<int>(cta) * kWgBM;
        const int n0 = n_idx * BN + static_cast<int>(cta) * (BN / 2);
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait(&empty[stage], phase ^ 1, wctx, kErrWaitProducer);
          if (!ok) break;
          uint8_t* sA = smem + stage * Cfg::kStageBytes;
          uint8_t* sB = sA + Cfg::kABytes;
          if (cta == 0) mbar_expect_tx(&full[stage], 2 * Cfg::kStageBytes);
          const uint32_t bar = mapa_u32(smem_u32(&full[stage]), 0);
#pragma unroll
          for (int c = 0; c < kWgBM / 64; ++c)
            tma_load_3d_pair(sA + c * (kWgBK * 128), &tmA, bar, m0 + c * 64, kb * kWgBK, layer);
#pragma unroll
          for (int c = 0; c < Cfg::kBChunks; ++c)
            tma_load_3d_pair(sB + c * (kWgBK * 128), &tmB, bar, n0 + c * 64, kb * kWgBK, layer);
          if (++stage == S) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (cta == 0 && elect_one()) {
      constexpr uint32_t idesc = umma_idesc_f16(Elem<T>::fmt, 1, 1, 2 * kWgBM, BN);
      int stage = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < total && ok; tile += npairs, ++it) {
        const int acc = it & 1;
        ok = mbar_wait(&tempty[acc], ((it >> 1) & 1) ^ 1, wctx, kErrWaitTmemEmpty);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * Cfg::kAccCols;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait(&full[stage], phase, wctx, kErrWaitMma);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_base = smem_u32(smem + stage * Cfg::kStageBytes), b_base = a_base + Cfg::kABytes;
#pragma unroll
          for (int k = 0; k < kWgBK / 16; ++k)
            umma_f16_pair(d_tmem, umma_desc_sw128(a_base + k * 2048, kWgBK * 128, 1024),
                          umma_desc_sw128(b_base + k * 2048, kWgBK * 128, 1024), idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit_pair(&empty[stage], 3);
          if (++stage == S) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit_pair(&tfull[acc], 3);
      }
    }
  } else {
    const int quarter = warp & 3;      // TMEM lane quarter this warp may access
    const int half = (warp - 2) >> 2;  // which of the two warps of that quarter: alternate chunks
    uint8_t* sb = epi_smem + (warp - 2) * kWgEpiBytes;
    AdamCoef co = {};
    if (ADAM) co = adam_coef(p.adam);
    int it = 0;
    bool ok = true;
    for (int tile = pair; tile < total && ok; tile += npairs, ++it) {
      const int acc = it & 1;
      int layer, m_idx, n_idx;
      coords(tile, layer, m_idx, n_idx);
      const int row0 = m_idx * (2 * kWgBM) + static_cast<int>(cta) * kWgBM + quarter * 32, n0 = n_idx * BN;
      // checked build: the tile lies inside the grid (rows and columns past the matrix are skipped below)
      const bool tile_ok = TP_CHECK(layer >= 0 && layer < p.layers && m_idx >= 0 && m_idx < p.num_m_tiles &&
                                        n_idx >= 0 && n_idx < p.num_n_tiles, p.err, kErrCheckTile);
      const int nc = tile_ok && row0 < p.M ? (min(BN, p.N - n0) + 63) / 64 : 0;
      const long long base = layer * p.layer_stride;
      WgradRegs<ADAM> a, b;
      if (half < nc) wgrad_fetch<ADAM>(p, a, base, row0, n0 + half * 64, 0, lane);   // under this tile's main loop
      if (ADAM && p.K <= kWgPrefetchK)
        for (int c = half; c < nc; c += 2) wgrad_prefetch(p, base, row0, n0 + c * 64, lane);
      ok = mbar_wait(&tfull[acc], (it >> 1) & 1, wctx, kErrWaitEpilogue);
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * Cfg::kAccCols;
#pragma unroll 1
      for (int c = half; c < nc; c += 2) {
        const int n = n0 + c * 64;
        uint32_t r[32];
        __syncwarp();      // (and the last chunk has been read)
        wgrad_fetch<ADAM>(p, b, base, row0, n, 1, lane);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          tmem_ld_32x32(t_acc + c * 64 + h * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int g = 0; g < 8; ++g)   // 16-byte pieces turned by the row: no bank conflicts either way
            *reinterpret_cast<uint4*>(sb + lane * 256 + ((((h << 3) | g) ^ (lane & 7)) << 4)) =
                make_uint4(r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
        }
        __syncwarp();
        wgrad_finish<T, ADAM>(p, co, a, sb, base, row0, n, 0, lane);
        wgrad_fetch<ADAM>(p, a, base, row0, n, 2, lane);
        wgrad_finish<T, ADAM>(p, co, b, sb, base, row0, n, 1, lane);
        wgrad_fetch<ADAM>(p, b, base, row0, n, 3, lane);
        wgrad_finish<T, ADAM>(p, co, a, sb, base, row0, n, 2, lane);
        if (c + 2 < nc) wgrad_fetch<ADAM>(p, a, base, row0, n + 128, 0, lane);
        wgrad_finish<T, ADAM>(p, co, b, sb, base, row0, n, 3, lane);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&tempty[acc]), 0));
    }
  }

  // nobody leaves (or frees TMEM) while the peer may still read this CTA's shared memory or signal its
  // barriers.  On an aborted run give in-flight copies time to land first.
  __syncthreads();
  if (*abort_flag) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmem_base, Cfg::kTmemCols);
  if (p.follows && blockIdx.x == 0 && threadIdx.x == 0) pdl_wait(false);
}

template <typename T, int BN, bool ADAM>
static int launch_wgrad(const CUtensorMap& tmA, const CUtensorMap& tmB, const WgradParams& p, cudaStream_t s) {
  using Cfg = WgradCfg<BN>;
  static_assert(Cfg::kSmemBytes + kTmemKernelMinSmem > kSmemPerSm, "allocates TMEM after pdl_wait");
  auto kern = wgrad_kernel<T, BN, ADAM>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess)
      return kErrLaunch;
    configured = true;
  }
  const int tiles = p.num_tiles * p.layers, pairs = tiles < num_sms() / 2 ? tiles : num_sms() / 2;
  return launch_pdl(kern, dim3(2 * pairs), dim3(kWgThreads), Cfg::kSmemBytes, s, 2, tmA, tmB, p) == cudaSuccess
             ? kOk
             : kErrLaunch;
}

// [layers][K][cols], columns contiguous: boxes of 64 columns x 64 rows of one layer.  (One layer: any stride.)
static bool wgrad_tmap(CUtensorMap* out, const void* x, long long ld, long long layer_stride, int layers, int cols,
                       int K, bool bf16) {
  const uint64_t dims[3] = {static_cast<uint64_t>(cols), static_cast<uint64_t>(K), static_cast<uint64_t>(layers)};
  const uint64_t strides[2] = {static_cast<uint64_t>(ld) * 2,
                               static_cast<uint64_t>(layers > 1 ? layer_stride : ld * K) * 2};
  const uint32_t box[3] = {64, kWgBK, 1};
  return make_tmap_16b(out, x, 3, dims, strides, box, bf16);
}

template <bool ADAM>
static int wgrad(int dtype, const void* A, long long lda, long long a_stride, const void* B, long long ldb,
                 long long b_stride, WgradParams p, cudaStream_t s) {
  if (p.M <= 0 || p.N <= 0 || p.K <= 0 || p.layers <= 0) return kErrBadArgument;
  if ((p.M % 8) || (p.N % 8) || (lda % 8) || (ldb % 8) || (p.ldo % 8) || (a_stride % 8) || (b_stride % 8) ||
      (p.layer_stride % 8) || lda < p.M || ldb < p.N || p.ldo < p.N)
    return kErrBadArgument;
  if (p.layers > 1 && (a_stride < p.M || b_stride < p.N)) return kErrBadArgument;
  // no two layers write the same element: whole matrices apart, or side by side in the rows of a wider one
  const long long ends = (p.M - 1) * p.ldo + p.N;
  if (p.layers > 1 && p.layer_stride < ends &&
      (p.layer_stride < p.N || (p.layers - 1) * p.layer_stride + p.N > p.ldo))
    return kErrBadArgument;
  const uintptr_t out = ADAM ? reinterpret_cast<uintptr_t>(p.adam.p) | reinterpret_cast<uintptr_t>(p.adam.m) |
                                   reinterpret_cast<uintptr_t>(p.adam.v) | reinterpret_cast<uintptr_t>(p.adam.model)
                             : reinterpret_cast<uintptr_t>(p.grad);
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | out) & 15) return kErrBadArgument;
  const bool bf16 = dtype == 1;
  CUtensorMap tmA, tmB;
  if (!wgrad_tmap(&tmA, A, lda, a_stride, p.layers, p.M, p.K, bf16) ||
      !wgrad_tmap(&tmB, B, ldb, b_stride, p.layers, p.N, p.K, bf16))
    return kErrDriver;
  const int BN = choose_wgrad_tile(p.M, p.N, p.K, p.layers, ADAM, num_sms());
  if (p.accumulate) p.accumulate = p.K <= kWgAddInL2K ? 2 : 1;
  p.num_m_tiles = (p.M + 255) / 256;
  p.num_n_tiles = (p.N + BN - 1) / BN;
  const long long tiles = static_cast<long long>(p.num_m_tiles) * p.num_n_tiles;
  if (tiles * p.layers > 0x3fffffffLL) return kErrTooLarge;
  p.num_tiles = static_cast<int>(tiles);
  apply_tile_order(p, dram_tile_order(p.num_m_tiles, p.num_n_tiles, 256, BN, p.K, num_sms() / 2));
#define TP_DISPATCH(T)                                                                                   \
  (BN == 256 ? launch_wgrad<T, 256, ADAM>(tmA, tmB, p, s) : BN == 192 ? launch_wgrad<T, 192, ADAM>(tmA, tmB, p, s) \
                                                                      : launch_wgrad<T, 128, ADAM>(tmA, tmB, p, s))
  return bf16 ? TP_DISPATCH(__nv_bfloat16) : TP_DISPATCH(__half);
#undef TP_DISPATCH
}

}  // namespace tp

using namespace tp;

// Layer l's operands are A + l * a_stride ([K][M], leading dimension lda) and B + l * b_stride ([K][N]);
// its output matrices [M][N] (leading dimension ldo) lie layer_stride apart.
//   tp_wgrad: grad (fp32) = or += the product
//   tp_wgrad_adam: tp_fused_adam of the matrices w, m, v (fp32) and model (16 bits) with the product as gradient
// follows: the call before on this stream was one of these too, and neither's outputs are the other's; the CTAs then
// start in the last wave of that launch, as its SMs become free: the four launches of 24 layers of 256 columns over 256
// rows took 125 us one after the other and take 106.
extern "C" int tp_wgrad(int dtype, const void* A, long long lda, long long a_stride, const void* B, long long ldb,
                        long long b_stride, float* grad, long long ldo, long long layer_stride, int layers, int M,
                        int N, int K, int accumulate, int follows, int* err_flag, void* stream) {
  WgradParams p = {};
  p.M = M; p.N = N; p.K = K; p.layers = layers;
  p.ldo = ldo; p.layer_stride = layer_stride;
  p.grad = grad; p.accumulate = accumulate; p.follows = follows;
  p.err = err_flag;
  return wgrad<false>(dtype, A, lda, a_stride, B, ldb, b_stride, p, static_cast<cudaStream_t>(stream));
}

extern "C" int tp_wgrad_adam(int dtype, const void* A, long long lda, long long a_stride, const void* B,
                             long long ldb, long long b_stride, float* w, float* m, float* v, void* model,
                             long long ldo, long long layer_stride, int layers, int M, int N, int K,
                             const float* state, float lr, float beta1, float beta2, float eps,
                             float weight_decay, float grad_scale, int follows, int* err_flag,
                             void* stream) {
  WgradParams p = {};
  p.M = M; p.N = N; p.K = K; p.layers = layers;
  p.ldo = ldo; p.layer_stride = layer_stride; p.follows = follows;
  p.adam = AdamBuffers{w, m, v, model, state, lr, beta1, beta2, eps, weight_decay, grad_scale};
  p.err = err_flag;
  return wgrad<true>(dtype, A, lda, a_stride, B, ldb, b_stride, p, static_cast<cudaStream_t>(stream));
}

TP_DEFINE_WAIT_LIMIT_SETTER(tp_set_wait_limit_ns_wgrad)
