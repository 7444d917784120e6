// Memory-bound kernels of the training step: LayerNorm forward/backward, bias-gradient
// column sums, the fused mixed-precision Adam update and small helpers.  All use 16-byte
// vector accesses; statistics and reductions are fp32.
#include "adam.cuh"
#include "common.cuh"
#include "ln_geometry.h"
#include "ptx.cuh"

namespace tp {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Output fan-out of the LayerNorm kernels under sequence-parallel tensor parallelism: the kernel
// runs on this rank's token shard and stores each output row at the same offset into the buffer
// of EVERY rank of the group (dst[0..n); plain peer stores over NVLink for the others), which is
// the all-gather the following column-parallel GEMM needs.  When all CTAs are done, the last one
// raises flags[r][rank] = epoch + *epoch_base at every other rank r; the consumer (tp_gemm_ag)
// waits for that value.  n == 1 and flags unset: an ordinary single-destination kernel.
constexpr int kMaxPush = 8;
struct PushDst {
  void* dst[kMaxPush];
  int* flags[kMaxPush];
  int n, rank, epoch;
  const int* epoch_base;
  int* counter;   // zero between launches; counts finished CTAs
};

__device__ __forceinline__ void push_signal(const PushDst& pd) {
  if (pd.n <= 1 || pd.counter == nullptr) return;
  __threadfence_system();   // this thread's peer stores are visible system-wide
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned total = gridDim.x * gridDim.y;
    if (atomicAdd(reinterpret_cast<unsigned*>(pd.counter), 1u) == total - 1) {
      *pd.counter = 0;
      const int epoch = pd.epoch + (pd.epoch_base ? *pd.epoch_base : 0);
      __threadfence_system();
      for (int r = 0; r < pd.n; ++r)
        if (r != pd.rank)
          asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(pd.flags[r] + pd.rank), "r"(epoch) : "memory");
    }
  }
}

// Sum over the CTA; every thread gets the result.  `red` holds >= 33 floats.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < nw ? red[lane] : 0.0f;
    t = warp_sum(t);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

template <typename T> __device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = Elem<T>::unpack2(w[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}
template <typename T> __device__ __forceinline__ void load8(const T* p, float (&f)[8]) {
  unpack8<T>(*reinterpret_cast<const uint4*>(p), f);
}
template <typename T> __device__ __forceinline__ void store8(T* p, const float (&f)[8]) {
  uint4 u;
  u.x = Elem<T>::pack2(f[0], f[1]);
  u.y = Elem<T>::pack2(f[2], f[3]);
  u.z = Elem<T>::pack2(f[4], f[5]);
  u.w = Elem<T>::pack2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}

// ------------------------------------------------------------------ LayerNorm
// A row is handled by WPR warps; each lane keeps NV vectors of 8 consecutive elements, vector i
// of lane l of warp w at column ((i * WPR + w) * 32 + l) * 8, so a warp reads 512 contiguous
// bytes per vector.  A CTA of 8 warps (16 when WPR = 16) holds RPC = max(1, 8 / WPR) rows.
template <int WPR> struct LnGeom {
  static constexpr int kWarps = WPR > 8 ? WPR : 8;
  static constexpr int kRowsPerCta = kWarps / WPR;
  static constexpr int kThreads = kWarps * 32;
};

// Sum over the WPR warps of a row group; `red` is [slots][RPC][WPR] (ping-pong by `slot`).  Only
// the warps of the group meet (named barrier 1 + grp), so the row groups of a CTA run
// independently.  RPC = row groups per CTA (at most 15 named barriers are free).
template <int WPR, int RPC>
__device__ __forceinline__ float group_sum_named(float v, float* red, int slot, int grp, int wr, int lane) {
  v = warp_sum(v);
  if (WPR == 1) return v;
  float* r = red + (slot * RPC + grp) * WPR;
  if (lane == 0) r[wr] = v;
  asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(WPR * 32) : "memory");
  float t = 0.0f;
#pragma unroll
  for (int i = 0; i < WPR; ++i) t += r[i];
  return t;
}

// Forward.  Memory bound: what counts is how many rows an SM has in flight.  The row stays in its 16-bit
// form (NV registers of 16 bytes; unpacked again for each of the three passes over it), which lets four
// CTAs of 8 warps share an SM; with the row in fp32 only two fitted and 16384 x 2048 took 52 us.
template <typename T, int NV, int WPR>
__global__ void __launch_bounds__(LnGeom<WPR>::kThreads, 1024 / LnGeom<WPR>::kThreads)
layernorm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ gamma,
                     const T* __restrict__ beta, const PushDst pd, float* __restrict__ mean_out,
                     float* __restrict__ rstd_out, int rows, int H, float eps) {
  using G = LnGeom<WPR>;
  __shared__ float red[2 * G::kRowsPerCta * WPR + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grp = warp / WPR, wr = warp % WPR;
  pdl_wait(pd.n <= 1);
  const long long row = static_cast<long long>(blockIdx.x) * G::kRowsPerCta + grp;
  const bool row_ok = row < rows;
  uint4 xq[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = ((i * WPR + wr) * 32 + lane) * 8;
    xq[i] = row_ok && col < H ? *reinterpret_cast<const uint4*>(x + row * H + col) : make_uint4(0, 0, 0, 0);
  }
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float v[8];
    unpack8<T>(xq[i], v);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += v[j];
  }
  const float mean = group_sum_named<WPR, G::kRowsPerCta>(s, red, 0, grp, wr, lane) / H;
  float q = 0.0f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = ((i * WPR + wr) * 32 + lane) * 8;
    if (col < H) {
      float v[8];
      unpack8<T>(xq[i], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float d = v[j] - mean;
        q += d * d;
      }
    }
  }
  const float rstd = rsqrtf(group_sum_named<WPR, G::kRowsPerCta>(q, red, 1, grp, wr, lane) / H + eps);
  if (row_ok) {
    if (wr == 0 && lane == 0) {
      mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = ((i * WPR + wr) * 32 + lane) * 8;
      if (col < H) {
        float v[8], g[8], b[8], o[8];
        unpack8<T>(xq[i], v);
        load8(gamma + col, g);
        load8(beta + col, b);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (v[j] - mean) * rstd * g[j] + b[j];
        for (int d = 0; d < pd.n; ++d) store8(static_cast<T*>(pd.dst[d]) + row * H + col, o);
      }
    }
  }
  push_signal(pd);
}

// Backward geometry (ln_geometry.h): one CTA per SM, so an SM holds kRowsPerCta rows at a time, each with
// its three inputs in flight.
template <int NV, int WPR> struct LnBwdGeom {
  static constexpr int kWarps = ln_bwd_warps(NV, WPR);
  static constexpr int kRowsPerCta = ln_bwd_rows(NV, WPR);
  static constexpr int kThreads = kWarps * 32;
};

// dx = rstd * (g - mean(g) - xhat * mean(g * xhat)) (+ dres), g = dy * gamma.
// Persistent CTAs stride over rows.  The partial sums of dgamma = sum dy*xhat and dbeta = sum dy
// live in shared memory, one [2][H] region per row group, each lane adding to its own columns
// (no synchronisation inside the loop).  Inside a region the two 16-byte halves of a lane's 8
// columns lie in two planes, [array][half][H / 8][4], so that neighbouring lanes touch neighbouring
// 16 bytes (no bank conflicts).  At the end the regions are added in a fixed order and the CTA
// writes (or adds to) one slot of scratch[gridDim.x][2][H]; a second kernel adds the slots into
// the fp32 gradients.  x, dy and dres of a row are loaded together and stay in their 16-bit form (xhat
// and g are computed twice), which fits 16 to 24 warps; 16 that fetched dres after the row's
// reductions took 98 us for 16384 x 2048.
template <typename T, int NV, int WPR>
__global__ void __launch_bounds__(LnBwdGeom<NV, WPR>::kThreads, 1)
layernorm_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                     const float* __restrict__ mean, const float* __restrict__ rstd,
                     const T* __restrict__ gamma, const T* __restrict__ dres, const PushDst pd,
                     float* __restrict__ scratch, int rows, int H, int accumulate_slots) {
  using G = LnBwdGeom<NV, WPR>;
  extern __shared__ __align__(16) float part_smem[];  // [kRowsPerCta][2][H]
  __shared__ float red[2 * 2 * G::kRowsPerCta * WPR + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grp = warp / WPR, wr = warp % WPR;
  float* my_part = part_smem + static_cast<long long>(grp) * 2 * H;
  pdl_wait(pd.n <= 1);
  int parity = 0;
  bool fresh = true;      // the group's region holds nothing yet
  const uint4 zero4 = make_uint4(0, 0, 0, 0);
  for (long long base = static_cast<long long>(blockIdx.x) * G::kRowsPerCta; base < rows;
       base += static_cast<long long>(gridDim.x) * G::kRowsPerCta, parity ^= 1, fresh = false) {
    const long long row = base + grp;
    const bool row_ok = row < rows;
    uint4 xq[NV], dq[NV], rq[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = ((i * WPR + wr) * 32 + lane) * 8;
      const bool in = row_ok && col < H;
      xq[i] = in ? *reinterpret_cast<const uint4*>(x + row * H + col) : zero4;
      dq[i] = in ? *reinterpret_cast<const uint4*>(dy + row * H + col) : zero4;
      rq[i] = in && dres ? *reinterpret_cast<const uint4*>(dres + row * H + col) : zero4;
    }
    const float mu = row_ok ? mean[row] : 0.0f, rs = row_ok ? rstd[row] : 0.0f;
    float s1 = 0.0f, s2 = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = ((i * WPR + wr) * 32 + lane) * 8;
      if (col < H) {
        float xv[8], dyv[8], gam[8], pg[8];
        unpack8<T>(xq[i], xv);
        unpack8<T>(dq[i], dyv);
        load8(gamma + col, gam);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = (xv[j] - mu) * rs, g = dyv[j] * gam[j];
          s1 += g;
          s2 += g * xh;
          pg[j] = dyv[j] * xh;
        }
        float4* sgam = reinterpret_cast<float4*>(my_part + (col >> 1));      // half 0; half 1 is
        float4* sbet = reinterpret_cast<float4*>(my_part + H + (col >> 1));  // H / 2 floats further
#pragma unroll
        for (int hlf = 0; hlf < 2; ++hlf) {
          float4 a = make_float4(pg[4 * hlf], pg[4 * hlf + 1], pg[4 * hlf + 2], pg[4 * hlf + 3]);
          float4 c = make_float4(dyv[4 * hlf], dyv[4 * hlf + 1], dyv[4 * hlf + 2], dyv[4 * hlf + 3]);
          if (!fresh) {
            const float4 a0 = sgam[hlf * (H >> 3)], c0 = sbet[hlf * (H >> 3)];
            a.x += a0.x; a.y += a0.y; a.z += a0.z; a.w += a0.w;
            c.x += c0.x; c.y += c0.y; c.z += c0.z; c.w += c0.w;
          }
          sgam[hlf * (H >> 3)] = a;
          sbet[hlf * (H >> 3)] = c;
        }
      }
    }
    const float m1 = group_sum_named<WPR, G::kRowsPerCta>(s1, red, 2 * parity, grp, wr, lane) / H;
    const float m2 = group_sum_named<WPR, G::kRowsPerCta>(s2, red, 2 * parity + 1, grp, wr, lane) / H;
    if (row_ok) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int col = ((i * WPR + wr) * 32 + lane) * 8;
        if (col < H) {
          float xv[8], dyv[8], gam[8], r[8], o[8];
          unpack8<T>(xq[i], xv);
          unpack8<T>(dq[i], dyv);
          unpack8<T>(rq[i], r);
          load8(gamma + col, gam);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            o[j] = rs * (dyv[j] * gam[j] - m1 - (xv[j] - mu) * rs * m2) + r[j];
          for (int d = 0; d < pd.n; ++d) store8(static_cast<T*>(pd.dst[d]) + row * H + col, o);
        }
      }
    }
  }
  // add the row groups' regions in a fixed order (16-byte accesses), then write the CTA's sums
  // to (or add them into) its slot of the persistent partial buffer
  __syncthreads();
  float* sg = scratch + static_cast<long long>(blockIdx.x) * 2 * H;
  for (int c = threadIdx.x * 4; c < 2 * H; c += blockDim.x * 4) {
    // columns [q, q + 4) of array c / H: half (q / 4) & 1 of the 8-column group q / 8
    const int arr = c >= H ? 1 : 0, q = c - arr * H;
    const int sidx = arr * H + ((q >> 2) & 1) * (H >> 1) + (q >> 3) * 4;
    float4 v = *reinterpret_cast<const float4*>(part_smem + sidx);
#pragma unroll
    for (int gsel = 1; gsel < G::kRowsPerCta; ++gsel) {
      const float4 o = *reinterpret_cast<const float4*>(part_smem + static_cast<long long>(gsel) * 2 * H + sidx);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    if (accumulate_slots) {
      const float4 o = __ldcg(reinterpret_cast<const float4*>(sg + c));
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    __stcg(reinterpret_cast<float4*>(sg + c), v);
  }
  push_signal(pd);
}

// ------------------------------------------------------------------ bias and LayerNorm gradients
// All column sums of a layer, or of all layers, in one launch: db[n] += sum_rows dy[row][n] for up to kMaxColsums
// matrices of the same number of rows, and the fold of up to kMaxFolds sets of LayerNorm partial
// slots (as layernorm_bwd_reduce_kernel, clearing the slots).  Each is a handful of CTAs or a few
// microseconds long, so separate launches cost more than the sums.  A CTA of 256 threads takes 8 V
// columns of a chunk of rows, 8 rows of 16 bytes per thread in flight.  The (at most 8) chunks of a
// column block form a cluster whose first CTA adds them up in order through distributed shared
// memory, so the sums do not depend on timing.  V = 32 reads longer pieces of a row and V = 8 makes four
// times as many CTAs of them; layer_sums_launch has the line between them.  (One launch per matrix with
// one load in flight per thread ran on 64 of 148 SMs: 16384 x 2048 alone took 63 us.)
//
// LAYERS: several layers, blockIdx.y; a single one does without their strides, which cost it 0.1 us.  The chunk's
// address is hidden from the compiler: left to fold it into the loads' own it took 72 registers for bf16 layers, three
// CTAs an SM where the launch counts on four, and slower loops for the others.  us folded / hidden: one matrix of
// 16384 x 8192 51.7 / 48.6 (bf16 58.3 / 48.4), 8192 x 768 5.8 / 5.3; all four of 5 layers of 2048 columns, 16384 rows,
// 515 / 438 (bf16 500 / 439), 4 of 1600, 5120 rows, 110 / 102 (bf16 145 / 103).
constexpr int kMaxColsums = 4, kMaxFolds = 2;
struct SumJobs {
  const void* dy[kMaxColsums];
  float* db[kMaxColsums];
  long long ld[kMaxColsums];
  int N[kMaxColsums];
  int cta_end[kMaxColsums];      // CTAs [cta_end[i - 1], cta_end[i]) work on matrix i
  int n, rows, chunks, rows_per_chunk;   // chunks = cluster size
  float* slots[kMaxFolds];
  float* dgamma[kMaxFolds];
  float* dbeta[kMaxFolds];
  int folds, parts, H;           // the CTAs behind the matrices' fold 32 columns each
  // LAYERS: elements from a layer's matrices, slots and sums to the next's
  long long dy_stride[kMaxColsums], slot_stride, out_stride;
  int overwrite;                 // the sums replace what the gradients hold
};

// Fold 32 columns, from column c0 on, of slots [parts][2][H]; thread (tx, ty) of (32, 8), 4 loads in
// flight each, fixed-order tree in shared memory.
// clear bit 0: zero the slots afterwards; bit 1: overwrite dgamma/dbeta instead of adding.
__device__ __forceinline__ void fold_slots(float* __restrict__ slots, int parts, int H, int c0,
                                           float* __restrict__ dgamma, float* __restrict__ dbeta,
                                           int tx, int ty, int clear, float (&sm)[8][33]) {
  const int c = c0 + tx;
  const long long stride = 2ll * H;
  float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
  if (c < 2 * H) {
    int p = ty;
    for (; p + 24 < parts; p += 32) {
      s0 += __ldcg(slots + p * stride + c);
      s1 += __ldcg(slots + (p + 8) * stride + c);
      s2 += __ldcg(slots + (p + 16) * stride + c);
      s3 += __ldcg(slots + (p + 24) * stride + c);
    }
    for (; p < parts; p += 8) s0 += __ldcg(slots + p * stride + c);
    if (clear & 1)
      for (int q = ty; q < parts; q += 8) slots[q * stride + c] = 0.0f;
  }
  sm[ty][tx] = (s0 + s1) + (s2 + s3);
  __syncthreads();
  if (ty == 0 && c < 2 * H) {
    float t = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += sm[i][tx];
    float* dst = c < H ? dgamma + c : dbeta + (c - H);
    *dst = (clear & 2) ? t : *dst + t;
  }
}

// dgamma[c] += sum_p scratch[p][0][c]; dbeta[c] += sum_p scratch[p][1][c]; blockDim = (32, 8), 32
// columns per CTA; `clear` as in fold_slots.
__global__ void layernorm_bwd_reduce_kernel(float* __restrict__ scratch, int parts, int H,
                                            float* __restrict__ dgamma, float* __restrict__ dbeta,
                                            int clear) {
  __shared__ float sm[8][33];
  pdl_wait();
  fold_slots(scratch, parts, H, blockIdx.x * 32, dgamma, dbeta, threadIdx.x, threadIdx.y, clear, sm);
}

// PER: chunks of a CTA, one after the other (their sums are folded in the same order).
template <typename T, int V, bool LAYERS, int PER>
__global__ void __launch_bounds__(256)
layer_sums_kernel(const SumJobs j) {
  constexpr int kCols = 8 * V, kRows = 256 / V;   // columns of a CTA, rows of one load
  __shared__ union { float col[kRows][kCols + 1]; float fold[8][33]; } sm;
  __shared__ float chunk_sum[PER][kCols];
  const int tid = threadIdx.x, vec = tid % V, lane_row = tid / V;
  const int cta = blockIdx.x;
  const long long layer = LAYERS ? blockIdx.y : 0;
  pdl_wait();
  int first = 0;
#pragma unroll
  for (int i = 0; i < kMaxColsums; ++i) {
    if (i >= j.n) break;
    if (cta < j.cta_end[i]) {
      const int ctas = j.chunks / PER, rank = (cta - first) % ctas;   // of a column block: a cluster
      const int col0 = (cta - first) / ctas * kCols, col = col0 + vec * 8;
      float s = 0.0f;
#pragma unroll 1
      for (int u = 0; u < PER; ++u) {
        const int chunk = rank * PER + u;
        const int r_end = min(j.rows, (chunk + 1) * j.rows_per_chunk);
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (col < j.N[i]) {
          const T* src = static_cast<const T*>(j.dy[i]) + layer * j.dy_stride[i] + col;
          asm("" : "+l"(src));
          for (int r = chunk * j.rows_per_chunk + lane_row; r < r_end; r += 8 * kRows) {
            uint4 v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
              v[k] = r + kRows * k < r_end ? *reinterpret_cast<const uint4*>(src + (r + kRows * k) * j.ld[i])
                                           : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              float f[8];
              unpack8<T>(v[k], f);
#pragma unroll
              for (int q = 0; q < 8; ++q) acc[q] += f[q];
            }
          }
        }
        if (u > 0) __syncthreads();      // the last chunk's values have been added up
#pragma unroll
        for (int q = 0; q < 8; ++q) sm.col[lane_row][vec * 8 + q] = acc[q];
        __syncthreads();
        if (tid < kCols) {
          float t = 0.0f;
#pragma unroll
          for (int r = 0; r < kRows; ++r) t += sm.col[r][tid];
          if (PER > 1 || ctas > 1) chunk_sum[u][tid] = t;
          s = u == 0 ? t : s + t;
        }
      }
      if (ctas > 1) {
        cluster_sync_all();
        if (rank == 0 && tid < kCols) {
          for (int q = 1; q < ctas; ++q) {
#pragma unroll
            for (int u = 0; u < PER; ++u) {
              float v;
              asm volatile("ld.shared::cluster.f32 %0, [%1];"
                           : "=f"(v) : "r"(mapa_u32(smem_u32(&chunk_sum[u][tid]), q)) : "memory");
              s += v;
            }
          }
        }
        cluster_sync_all();   // nobody leaves while its sums may be read
        if (rank != 0) return;
      }
      if (tid < kCols && col0 + tid < j.N[i]) {
        float* db = j.db[i] + layer * j.out_stride + col0 + tid;
        *db = j.overwrite ? s : *db + s;
      }
      return;
    }
    first = j.cta_end[i];
  }
  const int per_fold = (2 * j.H + 31) / 32;
  const int f = (cta - first) / per_fold;
  if (f >= j.folds) return;        // (the grid is a whole number of clusters)
  fold_slots(j.slots[f] + layer * j.slot_stride, j.parts, j.H, (cta - first) % per_fold * 32,
             j.dgamma[f] + layer * j.out_stride, j.dbeta[f] + layer * j.out_stride,
             tid & 31, tid >> 5, j.overwrite ? 3 : 1, sm.fold);
}

// ------------------------------------------------------------------ fused Adam
// state[0] = step count (as float), state[1] = 1 - beta1^t, state[2] = 1 - beta2^t.
__global__ void adam_tick_kernel(float* state, float beta1, float beta2) {
  const float t = state[0] + 1.0f;
  state[0] = t;
  state[1] = 1.0f - powf(beta1, t);
  state[2] = 1.0f - powf(beta2, t);
}

// One pass over flat buffers: g = grad * grad_scale; m, v, p (fp32 master) updated in place;
// the 16-bit model copy is rewritten and the gradient accumulator is zeroed.
template <typename T>
__device__ __forceinline__ void adam_vec4(float4* grad, const AdamBuffers& a, const AdamCoef& co, long long i) {
  float4 p4 = reinterpret_cast<float4*>(a.p)[i];
  float4 m4 = reinterpret_cast<float4*>(a.m)[i];
  float4 v4 = reinterpret_cast<float4*>(a.v)[i];
  adam_update(grad[i], p4, m4, v4, co);
  reinterpret_cast<float4*>(a.p)[i] = p4;
  reinterpret_cast<float4*>(a.m)[i] = m4;
  reinterpret_cast<float4*>(a.v)[i] = v4;
  grad[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  uint2 o;
  o.x = Elem<T>::pack2(p4.x, p4.y);
  o.y = Elem<T>::pack2(p4.z, p4.w);
  reinterpret_cast<uint2*>(a.model)[i] = o;
}

template <typename T>
__global__ void fused_adam_kernel(float* __restrict__ grad, const AdamBuffers a, long long n4) {
  const AdamCoef co = adam_coef(a);
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n4;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    adam_vec4<T>(reinterpret_cast<float4*>(grad), a, co, i);
}

// The same for a few ranges of every layer (what the weight-gradient products have not updated
// already: biases and LayerNorm parameters).  blockIdx.y = layer; offsets and lengths in float4.
constexpr int kMaxAdamRanges = 8;
struct AdamRanges {
  long long begin[kMaxAdamRanges], layer_stride;
  int len[kMaxAdamRanges];
  int n;
};
template <typename T>
__global__ void adam_ranges_kernel(float* __restrict__ grad, const AdamBuffers a, const AdamRanges r) {
  pdl_wait();
  const AdamCoef co = adam_coef(a);
  int i = blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll 1
  for (int k = 0; k < r.n; ++k) {
    if (i < r.len[k]) {
      adam_vec4<T>(reinterpret_cast<float4*>(grad), a, co, r.begin[k] + blockIdx.y * r.layer_stride + i);
      return;
    }
    i -= r.len[k];
  }
}

template <typename T>
__global__ void fill_kernel(T* p, long long n, float value) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    p[i] = Elem<T>::from_f(value);
}

}  // namespace tp

using namespace tp;

#define TP_LN_DISPATCH_WPR(T, NV, CALL)                  \
  switch (wpr) {                                          \
    case 1: CALL(T, NV, 1); break;                        \
    case 2: CALL(T, NV, 2); break;                        \
    case 4: CALL(T, NV, 4); break;                        \
    case 8: CALL(T, NV, 8); break;                        \
    default: CALL(T, NV, 16); break;                      \
  }
#define TP_LN_DISPATCH(T, CALL)                           \
  switch (nv) {                                           \
    case 1: TP_LN_DISPATCH_WPR(T, 1, CALL) break;         \
    case 2: TP_LN_DISPATCH_WPR(T, 2, CALL) break;         \
    case 3: TP_LN_DISPATCH_WPR(T, 3, CALL) break;         \
    default: TP_LN_DISPATCH_WPR(T, 4, CALL) break;        \
  }

namespace tp {
static PushDst single_dst(void* y) {
  PushDst pd;
  for (int i = 0; i < kMaxPush; ++i) { pd.dst[i] = nullptr; pd.flags[i] = nullptr; }
  pd.dst[0] = y;
  pd.n = 1; pd.rank = 0; pd.epoch = 0; pd.epoch_base = nullptr; pd.counter = nullptr;
  return pd;
}

static bool make_push(PushDst* pd, void* const* dst_ptrs, int* const* flag_ptrs, int n, int rank,
                      int epoch, const int* epoch_base, int* counter) {
  if (n < 1 || n > kMaxPush || rank < 0 || rank >= n || !dst_ptrs || !flag_ptrs || !counter) return false;
  for (int i = 0; i < kMaxPush; ++i) {
    pd->dst[i] = i < n ? dst_ptrs[i] : nullptr;
    pd->flags[i] = i < n ? flag_ptrs[i] : nullptr;
  }
  pd->n = n; pd->rank = rank; pd->epoch = epoch; pd->epoch_base = epoch_base; pd->counter = counter;
  return true;
}

static int layernorm_fwd_launch(int dtype, const void* x, const void* gamma, const void* beta,
                                const PushDst& pd, float* mean, float* rstd, int rows, int H,
                                float eps, cudaStream_t s) {
  if (rows <= 0) return kOk;
  int nv, wpr;
  if (!ln_geometry(H, &nv, &wpr, 4)) return kErrBadArgument;
#define LN_FWD(T, NV, WPR)                                                                       \
  launch_pdl(layernorm_fwd_kernel<T, NV, WPR>,                                                   \
             dim3((rows + LnGeom<WPR>::kRowsPerCta - 1) / LnGeom<WPR>::kRowsPerCta),             \
             dim3(LnGeom<WPR>::kThreads), 0, s, 1, static_cast<const T*>(x),                     \
             static_cast<const T*>(gamma), static_cast<const T*>(beta), pd, mean, rstd, rows, H, eps)
  if (dtype == 1) { TP_LN_DISPATCH(__nv_bfloat16, LN_FWD) }
  else { TP_LN_DISPATCH(__half, LN_FWD) }
#undef LN_FWD
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}
}  // namespace tp

extern "C" int tp_layernorm_fwd(int dtype, const void* x, const void* gamma, const void* beta,
                                void* y, float* mean, float* rstd, int rows, int H, float eps,
                                void* stream) {
  return layernorm_fwd_launch(dtype, x, gamma, beta, single_dst(y), mean, rstd, rows, H, eps,
                              static_cast<cudaStream_t>(stream));
}

// LayerNorm forward of this rank's token shard whose output rows go to the same place in the
// buffer of every rank of a tensor-parallel group (`y_ptrs[r]`, r < n; entry `rank` is the local
// buffer), followed by a flag at every peer: flag_ptrs[r][rank] = epoch + *epoch_base.
// `counter` is a zero-initialised device int used to find the last CTA.  The consumer is
// tp_gemm_ag with the same epoch.
extern "C" int tp_layernorm_fwd_push(int dtype, const void* x, const void* gamma, const void* beta,
                                     void* const* y_ptrs, float* mean, float* rstd, int rows, int H,
                                     float eps, int n, int rank, int* const* flag_ptrs, int epoch,
                                     const int* epoch_base, int* counter, void* stream) {
  PushDst pd;
  if (!make_push(&pd, y_ptrs, flag_ptrs, n, rank, epoch, epoch_base, counter)) return kErrBadArgument;
  return layernorm_fwd_launch(dtype, x, gamma, beta, pd, mean, rstd, rows, H, eps,
                              static_cast<cudaStream_t>(stream));
}

// Number of CTA slots the backward writes; scratch must hold parts * 2 * H floats.
extern "C" int tp_layernorm_bwd_parts(int rows) {
  const int cap = num_sms();
  return rows < cap ? rows : cap;
}

namespace tp {
// Opt the kernel in to more than 48 KB of shared memory, once per instantiation (the first,
// eager launch; never inside a stream capture).
template <typename K> static void ln_allow_smem(K kern) {
  // (instantiations of one element type share the function-pointer type K, so the kernels
  // already handled are remembered by address)
  static const void* seen[64];
  static int n_seen = 0;
  const void* key = reinterpret_cast<const void*>(kern);
  for (int i = 0; i < n_seen; ++i)
    if (seen[i] == key) return;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 192 * 1024);
  if (n_seen < 64) seen[n_seen++] = key;
}

static int ln_parts(int rows, int rows_per_cta) {
  int parts = (rows + rows_per_cta - 1) / rows_per_cta;
  const int cap = tp_layernorm_bwd_parts(rows);
  return parts > cap ? cap : parts;
}

// mode 0: write the CTA partials into `scratch` and fold them into dgamma/dbeta right away.
// mode 1: ADD the CTA partials into the persistent slots `scratch` (zero-initialised by the
//         caller) and leave dgamma/dbeta alone; tp_layernorm_bwd_finish folds them later.
static int layernorm_bwd_launch(int dtype, const void* dy, const void* x, const float* mean,
                                const float* rstd, const void* gamma, const void* dres,
                                const PushDst& pd, float* dgamma, float* dbeta, float* scratch,
                                int rows, int H, int mode, cudaStream_t s) {
  if (rows <= 0) return kOk;
  int nv, wpr;
  if (!ln_bwd_geometry(H, rows, num_sms(), &nv, &wpr)) return kErrBadArgument;
  const int rows_per_cta = ln_bwd_rows(nv, wpr);
  const int parts = ln_parts(rows, rows_per_cta);
  // one [2][H] fp32 region per row group of the CTA: at most 192 KB (H <= 1024 * WPR)
  const size_t smem = static_cast<size_t>(rows_per_cta) * 2 * H * sizeof(float);
#define LN_BWD(T, NV, WPR)                                                                      \
  {                                                                                             \
    auto kern = layernorm_bwd_kernel<T, NV, WPR>;                                               \
    if (smem > 40 * 1024) ln_allow_smem(kern); /* dynamic + static must stay under 48 KB */    \
    launch_pdl(kern, dim3(parts), dim3(LnBwdGeom<NV, WPR>::kThreads), smem, s, 1,                   \
               static_cast<const T*>(dy), static_cast<const T*>(x), mean, rstd,                 \
               static_cast<const T*>(gamma), static_cast<const T*>(dres), pd, scratch,           \
               rows, H, mode);                                                                  \
  }
  if (dtype == 1) { TP_LN_DISPATCH(__nv_bfloat16, LN_BWD) }
  else { TP_LN_DISPATCH(__half, LN_BWD) }
#undef LN_BWD
  if (mode == 0)
    launch_pdl(layernorm_bwd_reduce_kernel, dim3((2 * H + 31) / 32), dim3(32, 8), 0, s, 1, scratch, parts, H,
               dgamma, dbeta, 0);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}
}  // namespace tp

extern "C" int tp_layernorm_bwd(int dtype, const void* dy, const void* x, const float* mean,
                                const float* rstd, const void* gamma, const void* dres, void* dx,
                                float* dgamma, float* dbeta, float* scratch, int rows, int H,
                                void* stream) {
  return layernorm_bwd_launch(dtype, dy, x, mean, rstd, gamma, dres, single_dst(dx), dgamma, dbeta,
                              scratch, rows, H, 0, static_cast<cudaStream_t>(stream));
}

// Variant that only accumulates into persistent partial slots (tp_layernorm_bwd_parts(rows)
// slots of 2*H floats, zero before the first call of a backward pass).
extern "C" int tp_layernorm_bwd_accum(int dtype, const void* dy, const void* x, const float* mean,
                                      const float* rstd, const void* gamma, const void* dres,
                                      void* dx, float* slots, int rows, int H, void* stream) {
  return layernorm_bwd_launch(dtype, dy, x, mean, rstd, gamma, dres, single_dst(dx), nullptr, nullptr,
                              slots, rows, H, 1, static_cast<cudaStream_t>(stream));
}

// tp_layernorm_bwd_accum on this rank's token shard with the input gradient rows stored into the
// buffer of every rank of the group and a flag raised at every peer (see tp_layernorm_fwd_push).
extern "C" int tp_layernorm_bwd_accum_push(int dtype, const void* dy, const void* x, const float* mean,
                                           const float* rstd, const void* gamma, const void* dres,
                                           void* const* dx_ptrs, float* slots, int rows, int H, int n,
                                           int rank, int* const* flag_ptrs, int epoch,
                                           const int* epoch_base, int* counter, void* stream) {
  PushDst pd;
  if (!make_push(&pd, dx_ptrs, flag_ptrs, n, rank, epoch, epoch_base, counter)) return kErrBadArgument;
  return layernorm_bwd_launch(dtype, dy, x, mean, rstd, gamma, dres, pd, nullptr, nullptr, slots, rows,
                              H, 1, static_cast<cudaStream_t>(stream));
}

// Fold `parts` slots into dgamma/dbeta (+=) and clear them for the next backward pass.
extern "C" int tp_layernorm_bwd_finish(float* slots, int parts, int H, float* dgamma, float* dbeta,
                                       void* stream) {
  launch_pdl(layernorm_bwd_reduce_kernel, dim3((2 * H + 31) / 32), dim3(32, 8), 0,
             static_cast<cudaStream_t>(stream), 1, slots, parts, H, dgamma, dbeta, 1);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

// As tp_layernorm_bwd_finish, but dgamma/dbeta are overwritten with the folded sums (used when the
// sums of several ranks are added up afterwards, see tp_peer_sum).
extern "C" int tp_layernorm_bwd_finish_assign(float* slots, int parts, int H, float* dgamma,
                                              float* dbeta, void* stream) {
  launch_pdl(layernorm_bwd_reduce_kernel, dim3((2 * H + 31) / 32), dim3(32, 8), 0,
             static_cast<cudaStream_t>(stream), 1, slots, parts, H, dgamma, dbeta, 3);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

namespace tp {
static int layer_sums_launch(int dtype, SumJobs& j, int layers, cudaStream_t s) {
  long long blocks = 0;           // of 256 columns
  for (int i = 0; i < j.n; ++i) blocks += (j.N[i] + 255) / 256;
  blocks *= layers;
  // V = 32 once its CTAs fill the chip, us V = 8 / V = 32:
  //   one layer's four matrices of width  768 (27 blocks)   2048 (72)     4096 (144)
  //     rows    256                         3.8 / 5.0       5.3 / 6.3     7.8 / 10.2
  //     rows   1024                         6.0 / 6.6      11.0 / 10.4   21.7 / 14.3
  //     rows  16384                        49.1 / 60.3      108 / 93.6    203 / 182
  const bool wide = blocks >= 128 || (blocks >= 48 && blocks * j.rows >= 48 * 1024);
  const int cols = wide ? 256 : 64, round = 8 * 256 / (cols / 8);   // rows of one round of loads
  // Chunks of at least one round, a portable cluster of them at most; with V = 32 no more than 4 CTAs per
  // SM, which run at once (2560-wide layer, 16384 rows: 156 us with 8 chunks a block, 131 with 4;
  // 5120-wide, 1024 rows: 28.6 with 8, 21.8 with 2), unless even two chunks take several rounds: four then, of which
  // a CTA takes two where pairs of CTAs are few enough for five per SM, which still run at once (360 blocks of 16384
  // rows: 435 us instead of 477).
  int most = 8;
  if (wide) {
    while (most > 2 && blocks * most > 4 * num_sms()) most /= 2;
    if (blocks * most > 4 * num_sms()) most = 4;
  }
  j.chunks = 1;
  while (j.n > 0 && j.chunks < most && j.rows >= 2 * round * j.chunks) j.chunks *= 2;
  const bool twice = wide && j.chunks == 4 && blocks * 4 > 5 * num_sms() && blocks * 2 <= 5 * num_sms();
  const int cluster = twice ? 2 : j.chunks;      // CTAs of a block
  j.rows_per_chunk = (j.rows + j.chunks - 1) / j.chunks;
  long long ctas = 0;
  for (int i = 0; i < j.n; ++i) {
    ctas += (j.N[i] + cols - 1) / cols * static_cast<long long>(cluster);
    j.cta_end[i] = static_cast<int>(ctas);
  }
  ctas += static_cast<long long>(j.folds) * ((2 * j.H + 31) / 32);
  if (ctas == 0) return kOk;
  ctas = (ctas + cluster - 1) / cluster * cluster;
  if (ctas > 0x7fffffffLL) return kErrTooLarge;
  const dim3 grid(static_cast<unsigned>(ctas), static_cast<unsigned>(layers)), block(256);
#define TP_SUMS(T, LAYERS)                                                                     \
  (twice  ? launch_pdl(layer_sums_kernel<T, 32, LAYERS, 2>, grid, block, 0, s, cluster, j)     \
   : wide ? launch_pdl(layer_sums_kernel<T, 32, LAYERS, 1>, grid, block, 0, s, cluster, j)     \
          : launch_pdl(layer_sums_kernel<T, 8, LAYERS, 1>, grid, block, 0, s, cluster, j))
  const cudaError_t e = dtype == 1 ? (layers > 1 ? TP_SUMS(__nv_bfloat16, true) : TP_SUMS(__nv_bfloat16, false))
                                   : (layers > 1 ? TP_SUMS(__half, true) : TP_SUMS(__half, false));
#undef TP_SUMS
  return e == cudaSuccess ? kOk : kErrLaunch;
}
}  // namespace tp

extern "C" int tp_colsum(int dtype, const void* dy, long long ld, int rows, int N, float* db,
                         void* stream) {
  if (rows <= 0) return kOk;
  if (N <= 0 || N % 8 || ld % 8) return kErrBadArgument;
  SumJobs j = {};
  j.dy[0] = dy; j.ld[0] = ld; j.N[0] = N; j.db[0] = db;
  j.n = 1; j.rows = rows;
  return layer_sums_launch(dtype, j, 1, static_cast<cudaStream_t>(stream));
}

// The bias gradients (`n` <= 4 matrices dy[i] [rows][N[i]], added to db[i]) and LayerNorm parameter
// gradients (`folds` <= 2 sets of slots as for tp_layernorm_bwd_finish) of `layers` layers in one launch; the
// layers' matrices lie dy_stride[i], slots slot_stride and sums out_stride elements apart.
// overwrite: the sums replace what db, dgamma and dbeta hold.
extern "C" int tp_stage_sums(int dtype, int n, const void* const* dy, const long long* ld, const int* N,
                             float* const* db, int rows, int folds, float* const* slots, int parts, int H,
                             float* const* dgamma, float* const* dbeta, int layers, const long long* dy_stride,
                             long long slot_stride, long long out_stride, int overwrite, void* stream) {
  if (n < 0 || n > kMaxColsums || folds < 0 || folds > kMaxFolds || rows < 0 ||
      (folds > 0 && (H <= 0 || parts <= 0)) || layers < 1 || layers > 65535)
    return kErrBadArgument;
  SumJobs j = {};
  j.n = n; j.rows = rows;
  for (int i = 0; i < n; ++i) {
    j.dy_stride[i] = layers > 1 ? dy_stride[i] : 0;
    if (N[i] <= 0 || N[i] % 8 || ld[i] % 8 || j.dy_stride[i] % 8) return kErrBadArgument;
    j.dy[i] = dy[i]; j.ld[i] = ld[i]; j.N[i] = N[i]; j.db[i] = db[i];
  }
  j.folds = folds; j.parts = parts; j.H = H;
  j.slot_stride = slot_stride; j.out_stride = out_stride; j.overwrite = overwrite;
  for (int f = 0; f < folds; ++f) { j.slots[f] = slots[f]; j.dgamma[f] = dgamma[f]; j.dbeta[f] = dbeta[f]; }
  return layer_sums_launch(dtype, j, layers, static_cast<cudaStream_t>(stream));
}

// The same for one layer, added to the gradients (for callers that have the layers' matrices in buffers of their own).
extern "C" int tp_layer_sums(int dtype, int n, const void* const* dy, const long long* ld, const int* N,
                             float* const* db, int rows, int folds, float* const* slots, int parts, int H,
                             float* const* dgamma, float* const* dbeta, void* stream) {
  return tp_stage_sums(dtype, n, dy, ld, N, db, rows, folds, slots, parts, H, dgamma, dbeta, 1, nullptr, 0, 0, 0,
                       stream);
}

extern "C" int tp_adam_tick(float* state, float beta1, float beta2, void* stream) {
  adam_tick_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(state, beta1, beta2);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

extern "C" int tp_fused_adam(int dtype, float* grad, float* p, float* m, float* v, void* model,
                             long long n, const float* state, float lr, float beta1, float beta2,
                             float eps, float weight_decay, float grad_scale, void* stream) {
  if (n % 4) return kErrBadArgument;
  if (n == 0) return kOk;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const long long n4 = n / 4;
  long long blocks = (n4 + 255) / 256;
  const long long cap = 8ll * num_sms();
  if (blocks > cap) blocks = cap;
  const AdamBuffers a{p, m, v, model, state, lr, beta1, beta2, eps, weight_decay, grad_scale};
  if (dtype == 1) fused_adam_kernel<__nv_bfloat16><<<static_cast<int>(blocks), 256, 0, s>>>(grad, a, n4);
  else fused_adam_kernel<__half><<<static_cast<int>(blocks), 256, 0, s>>>(grad, a, n4);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

// tp_fused_adam over `n` <= 8 ranges [begin[k], begin[k] + len[k]) of each of `layers` layers, whose flat
// ranges lie `layer_stride` apart (elements; all multiples of 4).
extern "C" int tp_fused_adam_ranges(int dtype, float* grad, float* p, float* m, float* v, void* model, int n,
                                    const long long* begin, const long long* len, int layers,
                                    long long layer_stride, const float* state, float lr, float beta1,
                                    float beta2, float eps, float weight_decay, float grad_scale, void* stream) {
  if (n < 0 || n > kMaxAdamRanges || layers < 0 || layers > 65535 || layer_stride % 4) return kErrBadArgument;
  AdamRanges r = {};
  long long total = 0;
  for (int k = 0; k < n; ++k) {
    if (begin[k] < 0 || len[k] < 0 || begin[k] % 4 || len[k] % 4) return kErrBadArgument;
    r.begin[k] = begin[k] / 4;
    r.len[k] = static_cast<int>(len[k] / 4);
    total += len[k] / 4;
    if (total > 0x3fffffffLL) return kErrTooLarge;
  }
  r.n = n;
  r.layer_stride = layer_stride / 4;
  if (total == 0 || layers == 0) return kOk;
  const AdamBuffers a{p, m, v, model, state, lr, beta1, beta2, eps, weight_decay, grad_scale};
  const dim3 grid(static_cast<unsigned>((total + 255) / 256), static_cast<unsigned>(layers));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = dtype == 1 ? launch_pdl(adam_ranges_kernel<__nv_bfloat16>, grid, dim3(256), 0, s, 1, grad, a, r)
                                   : launch_pdl(adam_ranges_kernel<__half>, grid, dim3(256), 0, s, 1, grad, a, r);
  return e == cudaSuccess ? kOk : kErrLaunch;
}

extern "C" int tp_fill(int dtype, void* p, long long n, float value, void* stream) {
  if (n <= 0) return kOk;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  long long blocks = (n + 255) / 256;
  if (blocks > 8ll * num_sms()) blocks = 8ll * num_sms();
  if (dtype == 1) fill_kernel<__nv_bfloat16><<<static_cast<int>(blocks), 256, 0, s>>>(static_cast<__nv_bfloat16*>(p), n, value);
  else fill_kernel<__half><<<static_cast<int>(blocks), 256, 0, s>>>(static_cast<__half*>(p), n, value);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

// ------------------------------------------------------------------ allocation-free variant
// LayerNorm backward for callers that cannot allocate: the per-CTA partial sums go to a fixed
// array inside the library image instead of a caller-provided buffer (see terapipe_noalloc.h).
#include "terapipe_noalloc.h"

namespace tp {
constexpr int kStaticSlots = 160;
constexpr int kStaticMaxH = 4096;
constexpr long long kStaticScratchFloats = static_cast<long long>(kStaticSlots) * 2 * kStaticMaxH;
// In host code this name is only a handle for cudaGetSymbolAddress; kernels get the address.
static __device__ __align__(256) float g_ln_static_scratch[kStaticScratchFloats];
}  // namespace tp

extern "C" long long tp_layernorm_bwd_noalloc_capacity(void) { return tp::kStaticScratchFloats; }

extern "C" int tp_layernorm_bwd_noalloc(int dtype, const void* dy, const void* x, const float* mean,
                                        const float* rstd, const void* gamma, const void* dres,
                                        void* dx, float* dgamma, float* dbeta, int rows, int H,
                                        void* stream) {
  constexpr int kMaxDevices = 64;
  static float* scratch_of_device[kMaxDevices] = {nullptr};
  if (rows <= 0) return kOk;
  if (H <= 0 || H % 8) return kErrBadArgument;
  if (H > kStaticMaxH) return kErrTooLarge;
  const int parts = tp_layernorm_bwd_parts(rows);
  if (static_cast<long long>(parts) * 2 * H > kStaticScratchFloats) return kErrTooLarge;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return kErrDriver;
  if (!scratch_of_device[dev]) {
    // once per device, with that device current: resolve the array's device address
    float* p = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_ln_static_scratch) != cudaSuccess || !p) {
      cudaGetLastError();
      return kErrDriver;
    }
    scratch_of_device[dev] = p;
  }
  // mode 0 writes every slot it later reads, so stale contents of the shared array are harmless
  return layernorm_bwd_launch(dtype, dy, x, mean, rstd, gamma, dres, single_dst(dx), dgamma, dbeta,
                              scratch_of_device[dev], rows, H, 0, static_cast<cudaStream_t>(stream));
}

// Programmatic dependent launch of the GEMM, attention and LayerNorm kernels (on by default;
// TERAPIPE_PDL=0 in the environment or tp_set_pdl(0) turns it off).
extern "C" int tp_set_pdl(int enabled) {
  tp::pdl_enabled() = enabled ? 1 : 0;
  return kOk;
}
// 1 or 0, so that a caller who changes it can put it back.
extern "C" int tp_pdl_enabled(void) { return tp::pdl_enabled(); }
