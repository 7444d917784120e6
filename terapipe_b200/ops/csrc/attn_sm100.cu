// Slice-causal attention over a cached prefix for sm_100a (tcgen05 + TMEM + TMA).
//
// One token slice of `t` positions attends to the `c` positions cached by earlier slices plus
// itself; only the last `t` key columns carry a causal mask.  Q, K and V are read in place
// from the stage's full-length projection buffer
//     qkv[L][b][h][3][D]          (position, batch, local head, {q,k,v}, head dim)
// through 3-D tensor maps, so "appending to the KV cache" is just the QKV GEMM writing its
// rows; no gather/scatter kernels exist.  Scores never reach memory: S lives in TMEM, P (and dS)
// take its place there as 16-bit values and are the next MMA's A operand, the running output
// stays in TMEM and is rescaled lazily (only when the row maximum grows by more than 2^8).
//
// Backward recomputes P from Q, K and the saved log-sum-exp (base 2); see the comment above
// attn_bwd_kernel.  No gradient accumulator crosses slices: the backward pass walks the
// slices in reverse, so when slice j is processed the attention-output gradients dO of all
// later slices already sit in a full-length buffer, and dK/dV of slice j's keys are computed
// in one go by streaming over those later queries.
//
// Every kernel has two groups of 4 softmax warps (one TMEM lane quarter each, one row per thread,
// so row reductions need no shuffles), a warp for the TMA copies and one or two for the MMAs.
#include <math.h>
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"

namespace tp {

constexpr int kAttnThreads = 352;   // forward: 8 softmax warps, TMA, two MMA warps

struct AttnParams {
  int t, c, b, h;
  float scale, scale2;  // d^-0.5 and d^-0.5 * log2(e)
  void* o;              // fwd out: [t*b][ld_o], column = head*D + e
  long long ld_o;
  float* lse2;          // [b*h][lse_stride], indexed by absolute position
  long long lse_stride;
  float* delta;         // bwd: [b*h][lse_stride] = rowsum(dO * O), indexed by absolute position
  int q_end;            // bwd: end (absolute position) of the rows already back-propagated
  void* dqkv;           // [t*b][ld_dqkv], same column order as qkv
  long long ld_dqkv;
  int* err;
};

// One arrival per warp (after the warp's lanes have finished their part): far cheaper than 32
// contending shared-memory atomics on the same barrier word.
__device__ __forceinline__ void warp_arrive(uint64_t* bar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

__device__ __forceinline__ void named_bar_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// A descriptor's low word is the address / 16 and the leading offset / 16; the high word is the same
// for every tile here (umma_desc_sw128).
constexpr uint32_t kDescHi = (1024 >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_k(uint32_t addr) { return (addr >> 4) | (1u << 16); }   // K-major
__device__ __forceinline__ uint32_t desc_n(uint32_t addr, uint32_t chunk) {                       // N-major
  return (addr >> 4) | ((chunk >> 4) << 16);
}
__device__ __forceinline__ uint64_t desc64(uint32_t lo) {
  return (static_cast<uint64_t>(kDescHi) << 32) | lo;
}

// D[tmem] = A * B^T with both operands K-major, K = DH*64 split in DH sub-tiles.
template <int DH>
__device__ __forceinline__ void mma_kk(uint32_t tmem_d, uint32_t a, uint32_t a_sub, uint32_t b,
                                       uint32_t b_sub, uint32_t idesc) {
#pragma unroll
  for (int hh = 0; hh < DH; ++hh)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      umma_f16(tmem_d, desc64(a + hh * (a_sub >> 4) + k * 2), desc64(b + hh * (b_sub >> 4) + k * 2), idesc,
               (hh | k) != 0 ? 1u : 0u);
}

// D[tmem] (+)= A * B: A = [128 x 64] 16-bit values in TMEM (two per column), B = [64 (k) x N] N-major.
__device__ __forceinline__ void mma_tn(uint32_t tmem_d, uint32_t tmem_a, uint32_t b, uint32_t idesc,
                                       bool accumulate) {
#pragma unroll
  for (int k = 0; k < 4; ++k)
    umma_f16_ta(tmem_d, tmem_a + k * 8, desc64(b + k * 128), idesc, (accumulate || k != 0) ? 1u : 0u);
}

// Which tile of which head a CTA takes.  CTAs start in the order of their index.  Heads go in
// chunks of kHeadChunk whose operands stay in L2 together (2 MB a head at 2048 x 128), and inside a
// chunk the tiles with the longest streams come first, so that what is left at the end is short.
constexpr int kHeadChunk = 16;
__device__ __forceinline__ void tile_of_cta(int idx, int tiles, int heads, int& rank, int& bh) {
  const int chunk = idx / (tiles * kHeadChunk);
  const int in = idx - chunk * (tiles * kHeadChunk);
  const int width = min(kHeadChunk, heads - chunk * kHeadChunk);
  rank = in / width;                 // 0 = longest stream
  bh = chunk * kHeadChunk + in % width;
}

// ============================================================================ forward
// A CTA owns 256 queries of one head, 128 per softmax group, and streams the keys in blocks of
// 64: both groups use every K/V tile.  Where only one tile of queries is left (short slices, the
// end of a long one) and it has at least kSplitBlocks key blocks, the two groups take alternate
// blocks of that tile, and their partial outputs are merged at the end.
//
// Each group has two S buffers and an MMA warp of its own.  P overwrites the S it came from, and
// the scores of block k + 2 overwrite that P: they are issued right after P V of block k (MMAs of one
// thread execute in order, so nobody waits in between), and a group finds the scores of its next
// block ready when it has handed in P.  With O that is 4 x 64 + 2 x D columns of TMEM, all 512 at
// D = 128.  One MMA warp for both groups spent 185 cycles on each of six waits and as much on
// commits per pair of blocks, 2700 cycles at either D.
//
// What bounds it: 128 queries x 64 keys take 512 cycles of the exponential unit; S takes 384 cycles
// (6 KB of operands through shared memory per 32 cycles of tensor work) and P V 256 at D = 128,
// half of that at D = 64.  Over a whole kernel the exponential unit is busy half of the time and the tensor
// pipe 44 % (D = 128) or 25 %: a CTA's start and end overlap nothing, for it holds all of TMEM.  With P
// through shared memory and one group of 128 queries per CTA, 8 x 16 heads of 2048 x 128 took 302 us, now
// 161; 48 heads of 2048 x 64 113 and 67.
struct FwdShared {
  uint64_t bar_q[2], bar_k[4], bar_kfree[4], bar_v[4], bar_vfree[4], bar_s[2][2], bar_p[2][2], bar_o[2],
      bar_fin[2];
  float m[2][128], l[2][128];   // split mode: row statistics of the two groups
  uint32_t tmem_slot;
  int abort_flag;
};

constexpr int kFwdStages = 4;   // depth of the K and of the V ring
// A split saves a part of every block and pays for the merge, which has more columns to move at D = 128.
// 128 queries, us split / not split, at 8 heads and at 256:
//   key blocks         5          8          12         32
//   D = 64, 8       6.0/6.1    7.5/7.9    9.2/10.3   17.8/22.4
//   D = 64, 256   12.8/12.7  15.6/16.5   19.4/21.5   38.7/48.0
//   D = 128, 8      7.8/7.0    9.2/8.9   11.1/11.4   20.0/23.7
//   D = 128, 256  16.6/15.1  20.4/19.6   27.7/27.5   54.4/55.0
// 8 lies between the two widths' even points, 5 and 10 to 12.
constexpr int kSplitBlocks = 8;

template <typename T, int D>
__global__ void __launch_bounds__(kAttnThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV,
                const AttnParams p) {
  constexpr int DH = D / 64;
  constexpr int kQSub = 128 * 128, kKSub = 64 * 128;   // [rows][64 columns] 16-bit, 128-byte swizzle
  constexpr int kQTile = DH * kQSub, kKTile = DH * kKSub;
  constexpr int KS = kFwdStages;
  static_assert(kSplitBlocks >= 2, "both groups of a split tile have blocks");
  static_assert(D * 128 * 4 <= KS * kKTile, "the groups of a split tile exchange their halves through the K ring");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;                      // [2][kQTile]
  uint8_t* sK = sQ + 2 * kQTile;           // [KS][kKTile]
  uint8_t* sV = sK + KS * kKTile;          // [KS][kKTile]
  FwdShared* sh = reinterpret_cast<FwdShared*>(sV + KS * kKTile);

  const int warp = threadIdx.x >> 5;
  const WaitCtx wctx{&sh->abort_flag, p.err};
  const int tiles = (p.t + 255) / 256;
  int rank, bh;
  tile_of_cta(blockIdx.x, tiles, p.b * p.h, rank, bh);
  const int bi = bh / p.h, hi = bh % p.h;
  const int q0 = (tiles - 1 - rank) * 256;
  // key blocks of the first tile and of the last
  const int nb0 = (p.c + min(p.t, q0 + 128) + 63) / 64;
  const int n = (p.c + min(p.t, q0 + 256) + 63) / 64;   // blocks that are loaded
  const bool single = q0 + 128 >= p.t;                  // one tile of queries (n = nb0)
  const bool split = single && nb0 >= kSplitBlocks;     // the groups share its key blocks
  // blocks of the two groups: the k-th block of group w is blk(w, k)
  const int n_it0 = split ? (nb0 + 1) / 2 : nb0, n_it1 = split ? nb0 / 2 : single ? 0 : n;
  auto blk = [&](int w, int k) { return split ? 2 * k + w : k; };

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh->bar_q[i], 1);
      mbar_init(&sh->bar_o[i], 1);
      mbar_init(&sh->bar_fin[i], 1);
      for (int k = 0; k < 2; ++k) {
        mbar_init(&sh->bar_s[i][k], 1);
        mbar_init(&sh->bar_p[i][k], 4);
      }
    }
    for (int i = 0; i < KS; ++i) {
      mbar_init(&sh->bar_k[i], 1);
      mbar_init(&sh->bar_kfree[i], single ? 1 : 2);   // users of a block
      mbar_init(&sh->bar_v[i], 1);
      mbar_init(&sh->bar_vfree[i], single ? 1 : 2);
    }
    sh->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 9) {
    tmem_alloc(&sh->tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();  // set-up done; from here on the predecessor's results are read
  const uint32_t tmem = sh->tmem_slot;
  // columns: S / P of group w at 128 w (+ 64 for the odd blocks), O of group w at 256 + D w

  if (warp == 8) {
    if (elect_one()) {
      auto load_q = [&](int w) {
        mbar_expect_tx(&sh->bar_q[w], kQTile);
        for (int hh = 0; hh < DH; ++hh)
          tma_load_3d(sQ + w * kQTile + hh * kQSub, &tmQ, &sh->bar_q[w], hh * 64, bh, p.c + q0 + w * 128);
      };
      auto load_kv = [&](uint8_t* ring, uint64_t* full, uint64_t* freed, int col, int j) -> bool {
        const int st = j % KS;
        if (!mbar_wait(&freed[st], ((j / KS) & 1) ^ 1, wctx, kErrWaitAttn)) return false;
        mbar_expect_tx(&full[st], kKTile);
        for (int hh = 0; hh < DH; ++hh)
          tma_load_3d(ring + st * kKTile + hh * kKSub, &tmKV, &full[st], col + hh * 64, bh, j * 64);
        return true;
      };
      // in the order of use: each group has the scores of two blocks ahead of P V
      const int ahead = split ? 4 : 2;
      load_q(0);
      bool ok = load_kv(sK, sh->bar_k, sh->bar_kfree, D, 0);
      if (!single) load_q(1);
      for (int j = 1; j < ahead && j < n && ok; ++j) ok = load_kv(sK, sh->bar_k, sh->bar_kfree, D, j);
      for (int j = 0; j < n && ok; ++j) {
        // (the groups differ by at most two blocks, which are the last ones: their tiles, which
        // group 1 alone uses, are not waited for)
        ok = load_kv(sV, sh->bar_v, sh->bar_vfree, 2 * D, j);
        if (ok && j + ahead < n) ok = load_kv(sK, sh->bar_k, sh->bar_kfree, D, j + ahead);
      }
    }
  } else if (warp >= 9) {
    const int w = warp - 9;
    const int n_it = w == 0 ? n_it0 : n_it1;
    if (n_it > 0 && elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_f16(Elem<T>::fmt, 0, 0, 128, 64);
      constexpr uint32_t idesc_pv = umma_idesc_f16(Elem<T>::fmt, 0, 1, 128, D);
      const uint32_t dQ = desc_k(smem_u32(sQ + (single ? 0 : w * kQTile))), dK = desc_k(smem_u32(sK)),
                     dV = desc_n(smem_u32(sV), kKSub);
      const uint32_t tSw = tmem + w * 128, tOw = tmem + 256 + w * D;
      auto issue_s = [&](int k) {
        const int st = blk(w, k) % KS;
        mma_kk<DH>(tSw + (k & 1) * 64, dQ, kQSub, dK + st * (kKTile >> 4), kKSub, idesc_s);
        umma_commit(&sh->bar_s[w][k & 1]);
        umma_commit(&sh->bar_kfree[st]);
      };
      bool ok = mbar_wait(&sh->bar_q[single ? 0 : w], 0, wctx, kErrWaitAttn);
      for (int k = 0; k < 2 && k < n_it && ok; ++k) {
        const int j = blk(w, k);
        ok = mbar_wait(&sh->bar_k[j % KS], (j / KS) & 1, wctx, kErrWaitAttn);
        tc_fence_after();
        if (ok) issue_s(k);
      }
      for (int k = 0; k < n_it && ok; ++k) {
        const int j = blk(w, k), j2 = blk(w, k + 2);
        const bool more = k + 2 < n_it;
        uint64_t *bp = &sh->bar_p[w][k & 1], *bv = &sh->bar_v[j % KS], *bk = &sh->bar_k[j2 % KS];
        ok = more ? mbar_wait_all(bp, (k >> 1) & 1, bv, (j / KS) & 1, bk, (j2 / KS) & 1, wctx, kErrWaitAttn)
                  : mbar_wait_all(bp, (k >> 1) & 1, bv, (j / KS) & 1, wctx, kErrWaitAttn);
        if (!ok) break;
        tc_fence_after();
        mma_tn(tOw, tSw + (k & 1) * 64, dV + (j % KS) * (kKTile >> 4), idesc_pv, k > 0);
        umma_commit(&sh->bar_o[w]);
        umma_commit(&sh->bar_vfree[j % KS]);
        if (more) issue_s(k + 2);
      }
      if (ok) umma_commit(&sh->bar_fin[w]);
    }
  } else {
    const int w = warp >> 2;               // softmax group
    const int r = threadIdx.x & 127;       // row of the tile = TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + w * 128 + lane_base, tO = tmem + 256 + w * D + lane_base;
    const int qt = q0 + (single ? 0 : w * 128);   // first query of the tile
    const int qi = qt + r;
    const int qpos = p.c + qi;
    const int n_it = w == 0 ? n_it0 : n_it1;
    float m = -INFINITY;
    float2 l2 = make_float2(0.0f, 0.0f);
    bool ok = true;
    for (int k = 0; k < n_it; ++k) {
      ok = mbar_wait(&sh->bar_s[w][k & 1], (k >> 1) & 1, wctx, kErrWaitAttn);
      if (!ok) break;
      tc_fence_after();
      const int kbase = blk(w, k) * 64;
      const uint32_t tSk = tS + (k & 1) * 64;
      uint32_t s[2][32];
      __syncwarp();
      tmem_ld_32x32(tSk, s[0]);
      tmem_ld_32x32(tSk + 32, s[1]);
      tmem_ld_wait();
      if (kbase + 63 > p.c + qt) {         // the causal edge runs through this block
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (kbase + g * 32 + i > qpos) s[g][i] = 0xff800000u;   // -inf
      }
      float mx4[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const uint32_t* sg = &s[g >> 1][(g & 1) * 16];
        mx4[g] = fmaxf(__uint_as_float(sg[0]), __uint_as_float(sg[1]));
#pragma unroll
        for (int i = 2; i < 16; i += 2) mx4[g] = max3(mx4[g], __uint_as_float(sg[i]), __uint_as_float(sg[i + 1]));
      }
      const float mx = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]) * p.scale2;
      bool need = false;
      float alpha = 1.0f;
      if (k == 0) {
        m = mx;
      } else if (mx > m + 8.0f) {
        need = true;
        alpha = exp2f(m - mx);
        m = mx;
        l2 = mul2(l2, dup2(alpha));
      }
      if (__any_sync(0xffffffffu, need)) {
        // O may only be touched once P V of the group's previous block has been added to it
        ok = mbar_wait(&sh->bar_o[w], (k - 1) & 1, wctx, kErrWaitAttn);
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int ch = 0; ch < D / 32; ++ch) {
          uint32_t raw[32];
          tmem_ld_32x32(tO + ch * 32, raw);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) raw[i] = __float_as_uint(__uint_as_float(raw[i]) * alpha);
          tmem_st_32x32(tO + ch * 32, raw);
        }
      }
      // m = -inf: every score so far has overflowed (a row sees keys in its group's first block)
      const float2 nm = dup2(m == -INFINITY ? 0.0f : -m), sc = dup2(p.scale2);
      float2 sum = make_float2(0.0f, 0.0f);   // of this block first: shorter chains of additions
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float2 e = fma2(make_float2(__uint_as_float(s[g][2 * i]), __uint_as_float(s[g][2 * i + 1])), sc, nm);
          e.x = exp2f(e.x);
          e.y = exp2f(e.y);
          sum = add2(sum, e);
          pk[i] = Elem<T>::pack2(e.x, e.y);
        }
        tmem_st_32x16(tSk + g * 16, pk);
      }
      l2 = add2(l2, sum);
      tmem_st_wait();
      tc_fence_before();
      warp_arrive(&sh->bar_p[w][k & 1]);
    }
    float l = l2.x + l2.y;
    // checked build: the row's statistics slot and its columns of the output exist
    const bool row_ok = qi < p.t && TP_CHECK(qpos >= 0 && qpos < p.lse_stride && (hi + 1) * D <= p.ld_o,
                                             p.err, kErrCheckAttn);
    T* orow = static_cast<T*>(p.o) + (static_cast<long long>(qi) * p.b + bi) * p.ld_o + hi * D;
    float* lse_slot = p.lse2 + static_cast<long long>(bh) * p.lse_stride + qpos;
    auto store32 = [&](int col, const float (&v)[32], float mul) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        uint4 u;
        u.x = Elem<T>::pack2(v[g * 8 + 0] * mul, v[g * 8 + 1] * mul);
        u.y = Elem<T>::pack2(v[g * 8 + 2] * mul, v[g * 8 + 3] * mul);
        u.z = Elem<T>::pack2(v[g * 8 + 4] * mul, v[g * 8 + 5] * mul);
        u.w = Elem<T>::pack2(v[g * 8 + 6] * mul, v[g * 8 + 7] * mul);
        *reinterpret_cast<uint4*>(orow + col + g * 8) = u;
      }
    };
    auto load32 = [&](int col, float (&v)[32]) {
      uint32_t raw[32];
      __syncwarp();
      tmem_ld_32x32(tO + col, raw);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(raw[i]);
    };
    if (!split) {
      ok = ok && n_it > 0;     // (the second group of a short single tile has nothing)
      if (ok) ok = mbar_wait(&sh->bar_fin[w], 0, wctx, kErrWaitAttn);
      if (ok) {
        tc_fence_after();
        const float inv_l = 1.0f / l;
#pragma unroll 1
        for (int ch = 0; ch < D / 32; ++ch) {
          float v[32];
          load32(ch * 32, v);
          if (row_ok) store32(ch * 32, v, inv_l);
        }
        if (row_ok) *lse_slot = m + log2f(l);
      }
    } else {
      // Each group finishes half of the columns and hands the other half over through the K ring
      // (every tile has been used once both groups' last products are done).
      if (ok) ok = mbar_wait(&sh->bar_fin[0], 0, wctx, kErrWaitAttn);
      if (ok) ok = mbar_wait(&sh->bar_fin[1], 0, wctx, kErrWaitAttn);
      tc_fence_after();
      float* give = reinterpret_cast<float*>(sK) + w * (D / 2) * 128;        // [D / 2][128 rows]
      const float* take = reinterpret_cast<const float*>(sK) + (w ^ 1) * (D / 2) * 128;
      sh->m[w][r] = m;
      sh->l[w][r] = l;
      if (ok) {
#pragma unroll 1
        for (int ch = 0; ch < D / 64; ++ch) {
          float v[32];
          load32((w ^ 1) * (D / 2) + ch * 32, v);
#pragma unroll
          for (int i = 0; i < 32; ++i) give[(ch * 32 + i) * 128 + r] = v[i];
        }
      }
      named_bar_sync(1, 256);
      if (ok) {
        const float m_o = sh->m[w ^ 1][r], l_o = sh->l[w ^ 1][r];
        const float mm = fmaxf(m, m_o);
        // (both groups see keys of every row; m = -inf are scores that overflowed)
        const float a = m == -INFINITY ? 0.0f : exp2f(m - mm);
        const float a_o = m_o == -INFINITY ? 0.0f : exp2f(m_o - mm);
        l = l * a + l_o * a_o;
        const float inv_l = 1.0f / l;
#pragma unroll 1
        for (int ch = 0; ch < D / 64; ++ch) {
          const int col = w * (D / 2) + ch * 32;
          float v[32];
          load32(col, v);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = fmaf(take[(ch * 32 + i) * 128 + r], a_o, v[i] * a);
          if (row_ok) store32(col, v, inv_l);
        }
        if (row_ok && w == 0) *lse_slot = mm + log2f(l);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (sh->abort_flag) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_after();
  if (warp == 9) tmem_dealloc(tmem, 512);
}

// ============================================================================ delta = rowsum(dO * O)
// A row (one position of one head) is D / 8 lanes of 16 bytes each, and every lane has four rows in
// flight: memory bound.  (One warp per row with 4-byte loads kept 256 bytes per warp in flight:
// 16384 x 2048 took 67 us.)  o_vec = 0: `o` is only 4-byte aligned.
constexpr int kDeltaThreads = 256, kDeltaUnroll = 4;
template <int D> struct DeltaRows { static constexpr int value = kDeltaThreads / (D / 8) * kDeltaUnroll; };

template <typename T, int D>
__global__ void __launch_bounds__(kDeltaThreads)
attn_delta_kernel(const T* __restrict__ o, long long ld_o, const T* __restrict__ d_o, long long ld_do,
                  float* __restrict__ delta, long long delta_stride, int c, int t, int b, int h, int o_vec) {
  constexpr int kLanes = D / 8, kGroups = kDeltaThreads / kLanes;
  const int lane = threadIdx.x % kLanes;
  const long long row0 = static_cast<long long>(blockIdx.x) * DeltaRows<D>::value + threadIdx.x / kLanes;
  const long long rows = static_cast<long long>(t) * b * h;
  pdl_wait();
  uint4 vo[kDeltaUnroll], vd[kDeltaUnroll];
#pragma unroll
  for (int k = 0; k < kDeltaUnroll; ++k) {
    const long long row = row0 + k * kGroups;
    vo[k] = vd[k] = make_uint4(0, 0, 0, 0);
    if (row < rows) {
      const long long pos = row / h;          // position * b + batch
      const int col = static_cast<int>(row - pos * h) * D + lane * 8;
      const T* po = o + pos * ld_o + col;
      if (o_vec) {
        vo[k] = *reinterpret_cast<const uint4*>(po);
      } else {
        const uint32_t* p4 = reinterpret_cast<const uint32_t*>(po);
        vo[k] = make_uint4(p4[0], p4[1], p4[2], p4[3]);
      }
      vd[k] = *reinterpret_cast<const uint4*>(d_o + pos * ld_do + col);
    }
  }
#pragma unroll
  for (int k = 0; k < kDeltaUnroll; ++k) {
    const uint32_t wo[4] = {vo[k].x, vo[k].y, vo[k].z, vo[k].w};
    const uint32_t wd[4] = {vd[k].x, vd[k].y, vd[k].z, vd[k].w};
    float acc = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 x = Elem<T>::unpack2(wo[q]), g = Elem<T>::unpack2(wd[q]);
      acc += x.x * g.x + x.y * g.y;
    }
#pragma unroll
    for (int m = kLanes / 2; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    const long long row = row0 + k * kGroups;
    if (lane == 0 && row < rows) {
      const int bh = static_cast<int>(row % (static_cast<long long>(b) * h));   // batch * h + head
      delta[bh * delta_stride + c + row / (static_cast<long long>(b) * h)] = acc;
    }
  }
}

// ============================================================================ backward
// One streaming kernel, two modes (both deterministic, no floating-point atomics):
//   MODE 0 (dK/dV): stationary = 128 keys of the current slice (K, V tiles); streams, in
//     blocks of 64, the queries q >= k of this slice and of every later slice (Q and dO rows,
//     which later slices left in the full-length buffers).  dK/dV of a key block are therefore
//     complete when the CTA ends and are written once, as 16-bit values.
//   MODE 1 (dQ): stationary = 128 queries of the current slice (Q, dO tiles); streams the keys
//     k <= q (K, V tiles of 64 rows).
// Per streamed block:  S = X1 Y1^T, dP = X2 Y2^T (TMEM, double buffered);
//   P = exp2(S*scale2 - lse), dS = P (dP - delta)  -> 16-bit, into the columns of S and dP;
//   MODE 0: dV += P * dO, dK += dS * Q;   MODE 1: dQ += dS * K   (P, dS are A operands from TMEM).
// 10 warps: two worker groups of 4 warps alternate over the streamed blocks (each owns one
// S/dP buffer), warp 8 brings the streamed tiles, warp 9 elects the MMA thread.
//
// What bounds it: shared memory.  A 128 x 64 block of S reads 6 KB of operands for 32 cycles of
// tensor work (48 cycles of shared memory), so at D = 128 a block takes 1280 cycles in MODE 0
// and 1024 in MODE 1.  P and dS used to go through shared memory as well, single buffered: each
// block's store waited for the previous block's products and these for the store, and a block took
// 4000 cycles.  The MMA thread now issues the products of block i and then the scores of block
// i + 2, which overwrite the same columns: MMAs of one thread execute in order, so only the
// workers' arrival is waited for.  8 x 16 heads of 2048 x 128, both modes and delta: 858 us before, 566 now.
constexpr int kBwdThreads = 320;
constexpr int kBwdStages = 4;   // ring depth of the streamed tiles

struct BwdShared {
  uint64_t bar_x, bar_y[kBwdStages], bar_yfree[kBwdStages], bar_s[2], bar_p[2], bar_done;
  alignas(16) float nlse[kBwdStages][64];   // MODE 0: per streamed block, negated, by the producer warp
  alignas(16) float ndelta[kBwdStages][64];
  uint32_t tmem_slot;
  int abort_flag;
};

template <typename T, int D, int MODE>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQKV128,
                const __grid_constant__ CUtensorMap tmQKV64,
                const __grid_constant__ CUtensorMap tmDO128,
                const __grid_constant__ CUtensorMap tmDO64, const AttnParams p) {
  constexpr int DH = D / 64;
  constexpr int kXSub = 128 * 128, kYSub = 64 * 128;
  constexpr int kStageBytes = 2 * DH * kYSub;
  constexpr uint32_t kTmemCols = 512;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sX1 = smem;
  uint8_t* sX2 = sX1 + DH * kXSub;
  uint8_t* sY = sX2 + DH * kXSub;                 // [stages][Y1 | Y2][DH][kYSub]
  BwdShared* sh = reinterpret_cast<BwdShared*>(sY + kBwdStages * kStageBytes);

  const int warp = threadIdx.x >> 5;
  const WaitCtx wctx{&sh->abort_flag, p.err};
  const int tiles = (p.t + 127) / 128;
  int rank, bh;
  tile_of_cta(blockIdx.x, tiles, p.b * p.h, rank, bh);
  const int bi = bh / p.h, hi = bh % p.h;
  // dK/dV: the first keys have the most queries; dQ: the last queries have the most keys
  const int xt = (MODE == 0 ? rank : tiles - 1 - rank) * 128;
  const int x0 = p.c + xt;                // first stationary row (absolute position)
  int ystart, n_iter;
  if (MODE == 0) {
    ystart = x0;
    n_iter = (p.q_end - x0 + 63) / 64;
  } else {
    ystart = 0;
    n_iter = (p.c + min(p.t, xt + 128) + 63) / 64;
  }

  if (threadIdx.x == 0) {
    mbar_init(&sh->bar_x, 1);
    for (int i = 0; i < kBwdStages; ++i) {
      mbar_init(&sh->bar_y[i], MODE == 0 ? 2 : 1);   // the tiles, and in MODE 0 the statistics
      mbar_init(&sh->bar_yfree[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh->bar_s[i], 1);
      mbar_init(&sh->bar_p[i], 4);
    }
    mbar_init(&sh->bar_done, 1);
    sh->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 9) {
    tmem_alloc(&sh->tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Set-up done; from here on the predecessor's results are read.  dQ follows dK/dV, of which it reads nothing: it
  // starts once all CTAs of dK/dV run, which they do when everything before them is done, and waits for them
  // at its own end, so that whoever waits for dQ waits for both.
  if (MODE == 0) pdl_wait();
  else pdl_trigger();
  const uint32_t tmem = sh->tmem_slot;
  // columns: S / P of buffer 0 at 0, of 1 at 64, dP / dS at 128 and 192, Acc1 256, Acc2 256 + D
  const uint32_t tA1 = tmem + 256, tA2 = tmem + 256 + D;

  if (warp == 8) {
    // Producer.  Lane 0 issues every tile copy.  In MODE 0 the whole warp brings the streamed
    // queries' lse and delta (64 floats each): two of each per lane, loaded a block ahead so that
    // their latency passes while the ring is full, whatever the block's alignment in the row and
    // wherever the sequence ends.  (They used to be bulk copies, which need a 16-byte boundary;
    // blocks without one, or with the sequence's end in them, went through 128 plain loads of a
    // single thread, and a head's 2048 keys at an odd slice start took 434 us instead of 36.)
    const int lane = threadIdx.x & 31;
    const float* lse_row = MODE == 0 ? p.lse2 + static_cast<long long>(bh) * p.lse_stride : nullptr;
    const float* delta_row = MODE == 0 ? p.delta + static_cast<long long>(bh) * p.lse_stride : nullptr;
    float nl[2] = {0.0f, 0.0f}, nd[2] = {0.0f, 0.0f};
    auto fetch_stats = [&](int y0) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int y = y0 + lane + 32 * k;
        const bool in = y < p.q_end && TP_CHECK(y >= 0 && y < p.lse_stride, p.err, kErrCheckAttn);
        nl[k] = in ? __ldcg(lse_row + y) : 0.0f;
        nd[k] = in ? __ldcg(delta_row + y) : 0.0f;
      }
    };
    if (lane == 0) {
      mbar_expect_tx(&sh->bar_x, 2 * DH * kXSub);
      for (int hh = 0; hh < DH; ++hh) {
        if (MODE == 0) {
          tma_load_3d(sX1 + hh * kXSub, &tmQKV128, &sh->bar_x, D + hh * 64, bh, x0);
          tma_load_3d(sX2 + hh * kXSub, &tmQKV128, &sh->bar_x, 2 * D + hh * 64, bh, x0);
        } else {
          tma_load_3d(sX1 + hh * kXSub, &tmQKV128, &sh->bar_x, hh * 64, bh, x0);
          tma_load_3d(sX2 + hh * kXSub, &tmDO128, &sh->bar_x, hi * D + hh * 64, bi, x0);
        }
      }
    }
    if (MODE == 0 && n_iter > 0) fetch_stats(ystart);
    for (int i = 0; i < n_iter; ++i) {
      const int st = i % kBwdStages;
      int ok = 1;
      if (lane == 0) ok = mbar_wait(&sh->bar_yfree[st], ((i / kBwdStages) & 1) ^ 1, wctx, kErrWaitAttn);
      if (!__shfl_sync(0xffffffffu, ok, 0)) break;
      uint8_t* y1 = sY + st * kStageBytes;
      uint8_t* y2 = y1 + DH * kYSub;
      const int y0 = ystart + i * 64;
      if (lane == 0) {
        mbar_expect_tx(&sh->bar_y[st], kStageBytes);
        for (int hh = 0; hh < DH; ++hh) {
          if (MODE == 0) {
            tma_load_3d(y1 + hh * kYSub, &tmQKV64, &sh->bar_y[st], hh * 64, bh, y0);
            tma_load_3d(y2 + hh * kYSub, &tmDO64, &sh->bar_y[st], hi * D + hh * 64, bi, y0);
          } else {
            tma_load_3d(y1 + hh * kYSub, &tmQKV64, &sh->bar_y[st], D + hh * 64, bh, y0);
            tma_load_3d(y2 + hh * kYSub, &tmQKV64, &sh->bar_y[st], 2 * D + hh * 64, bh, y0);
          }
        }
      }
      if (MODE == 0) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          sh->nlse[st][lane + 32 * k] = -nl[k];
          sh->ndelta[st][lane + 32 * k] = -nd[k];
        }
        warp_arrive(&sh->bar_y[st]);
        if (i + 1 < n_iter) fetch_stats(y0 + 64);
      }
    }
  } else if (warp == 9) {
    if (elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_f16(Elem<T>::fmt, 0, 0, 128, 64);
      constexpr uint32_t idesc_g = umma_idesc_f16(Elem<T>::fmt, 0, 1, 128, D);
      const uint32_t dX1 = desc_k(smem_u32(sX1)), dX2 = desc_k(smem_u32(sX2)), dY = desc_k(smem_u32(sY)),
                     dYn = desc_n(smem_u32(sY), kYSub);
      constexpr uint32_t kStage16 = kStageBytes >> 4, kY2 = (DH * kYSub) >> 4;   // descriptor steps
      auto issue_s = [&](int i) {
        const uint32_t y = dY + (i % kBwdStages) * kStage16;
        mma_kk<DH>(tmem + (i & 1) * 64, dX1, kXSub, y, kYSub, idesc_s);
        mma_kk<DH>(tmem + 128 + (i & 1) * 64, dX2, kXSub, y + kY2, kYSub, idesc_s);
        umma_commit(&sh->bar_s[i & 1]);
      };
      bool ok = mbar_wait(&sh->bar_x, 0, wctx, kErrWaitAttn);
      for (int i = 0; i < 2 && i < n_iter && ok; ++i) {
        ok = mbar_wait(&sh->bar_y[i], 0, wctx, kErrWaitAttn);
        tc_fence_after();
        if (ok) issue_s(i);
      }
      for (int i = 0; i < n_iter && ok; ++i) {
        const int st = i % kBwdStages;
        const bool more = i + 2 < n_iter;
        uint64_t *bp = &sh->bar_p[i & 1], *by = &sh->bar_y[(i + 2) % kBwdStages];
        ok = more ? mbar_wait_all(bp, (i >> 1) & 1, by, ((i + 2) / kBwdStages) & 1, wctx, kErrWaitAttn)
                  : mbar_wait(bp, (i >> 1) & 1, wctx, kErrWaitAttn);
        if (!ok) break;
        tc_fence_after();
        const uint32_t buf = (i & 1) * 64;
        if (MODE == 0) mma_tn(tA1, tmem + buf, dYn + st * kStage16 + kY2, idesc_g, i > 0);
        mma_tn(tA2, tmem + 128 + buf, dYn + st * kStage16, idesc_g, i > 0);
        umma_commit(&sh->bar_yfree[st]);
        if (more) issue_s(i + 2);
      }
      if (ok) umma_commit(&sh->bar_done);
    }
  } else {
    const int grp = warp >> 2;                 // worker group 0 / 1
    const int r = threadIdx.x & 127;           // row of the stationary tile = TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int xabs = x0 + r;                   // absolute position of this thread's row
    // checked build: the row's statistics slot and its columns of the gradient exist
    const bool x_ok = xabs < p.c + p.t &&
                      TP_CHECK(xabs >= p.c && xabs < p.lse_stride && (hi + 1) * 3 * D <= p.ld_dqkv, p.err,
                               kErrCheckAttn);
    float2 nlse_r = make_float2(0.0f, 0.0f), ndelta_r = make_float2(0.0f, 0.0f);
    if (MODE == 1 && x_ok) {
      nlse_r = dup2(-p.lse2[static_cast<long long>(bh) * p.lse_stride + xabs]);
      ndelta_r = dup2(-p.delta[static_cast<long long>(bh) * p.lse_stride + xabs]);
    }
    const uint32_t tS = tmem + grp * 64 + lane_base, tP = tmem + 128 + grp * 64 + lane_base;
    const float2 sc = dup2(p.scale2);
    bool ok = true;
    for (int i = grp; i < n_iter; i += 2) {
      const int y0 = ystart + i * 64;
      const int st = i % kBwdStages;
      // blocks strictly inside the causal region need no per-element mask
      const bool full = MODE == 0 ? (y0 >= x0 + 127 && y0 + 64 <= p.q_end) : (y0 + 63 <= x0);
      if (MODE == 0) {
        // The statistics belong to columns here.  With a row per thread each thread read all 64 of
        // both (32 16-byte loads a warp and block, under the MMAs' operand traffic: half of the
        // block's time).  As MMA fragments, 16 lanes at a time, a thread has 16 columns of four rows.
        const int lane = threadIdx.x & 31;
        ok = mbar_wait(&sh->bar_y[st], (i / kBwdStages) & 1, wctx, kErrWaitAttn);
        if (!ok) break;
        float2 nl[8], nd[8];     // columns 8 k + 2 (lane % 4) and the next
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          nl[k] = *reinterpret_cast<const float2*>(&sh->nlse[st][8 * k + 2 * (lane & 3)]);
          nd[k] = *reinterpret_cast<const float2*>(&sh->ndelta[st][8 * k + 2 * (lane & 3)]);
        }
        ok = mbar_wait(&sh->bar_s[grp], (i >> 1) & 1, wctx, kErrWaitAttn);
        if (!ok) break;
        tc_fence_after();
        // (one copy of the loop per case: with the mask inside, its tests cost as much as the rest)
        auto halves = [&](auto masked) {
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {     // lanes 0-15, 16-31 of the warp's quarter
            const uint32_t half = static_cast<uint32_t>(hf * 16) << 16;
            uint32_t s[32], d[32], pk[16], dk[16];
            __syncwarp();
            tmem_ld_16x64(tS + half, s);
            tmem_ld_16x64(tP + half, d);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 8; ++k) {
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                const int e = 4 * k + 2 * q;
                float2 pr = fma2(make_float2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), sc, nl[k]);
                pr.x = exp2f(pr.x);
                pr.y = exp2f(pr.y);
                if (decltype(masked)::value) {
                  const int row = x0 + (warp & 3) * 32 + hf * 16 + q * 8 + (lane >> 2);
                  const int yabs = y0 + 8 * k + 2 * (lane & 3);
                  pr.x = yabs < p.q_end && row <= yabs ? pr.x : 0.0f;
                  pr.y = yabs + 1 < p.q_end && row <= yabs + 1 ? pr.y : 0.0f;
                }
                const float2 ds = mul2(pr, add2(make_float2(__uint_as_float(d[e]), __uint_as_float(d[e + 1])), nd[k]));
                pk[2 * k + q] = Elem<T>::pack2(pr.x, pr.y);
                dk[2 * k + q] = Elem<T>::pack2(ds.x, ds.y);
              }
            }
            // (these lanes' scores have all been read)
            tmem_st_16x32(tS + half, pk);
            tmem_st_16x32(tP + half, dk);
          }
        };
        if (full) halves(std::false_type());
        else halves(std::true_type());
      } else {
        ok = mbar_wait(&sh->bar_s[grp], (i >> 1) & 1, wctx, kErrWaitAttn);
        if (!ok) break;
        tc_fence_after();
        // dS into the columns of dP, 32 columns at a time.  The first half's results take 16 columns that
        // were read already; the second half's values lie beyond them.
        auto halves = [&](auto masked) {
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            uint32_t s[32], d[32], dk[16];
            __syncwarp();
            tmem_ld_32x32(tS + g * 32, s);
            tmem_ld_32x32(tP + g * 32, d);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              const int e = 2 * k;             // column within the half
              float2 pr = fma2(make_float2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), sc, nlse_r);
              pr.x = exp2f(pr.x);
              pr.y = exp2f(pr.y);
              if (decltype(masked)::value) {
                const int yabs = y0 + g * 32 + e;
                pr.x = x_ok && yabs <= xabs ? pr.x : 0.0f;
                pr.y = x_ok && yabs + 1 <= xabs ? pr.y : 0.0f;
              }
              const float2 ds = mul2(pr, add2(make_float2(__uint_as_float(d[e]), __uint_as_float(d[e + 1])), ndelta_r));
              dk[k] = Elem<T>::pack2(ds.x, ds.y);
            }
            tmem_st_32x16(tP + g * 16, dk);
          }
        };
        if (full) halves(std::false_type());
        else halves(std::true_type());
      }
      tmem_st_wait();
      tc_fence_before();
      warp_arrive(&sh->bar_p[grp]);
    }
    if (ok && n_iter > 0) ok = mbar_wait(&sh->bar_done, 0, wctx, kErrWaitAttn);
    if (ok && n_iter > 0) {
      tc_fence_after();
      const long long out_row = (static_cast<long long>(xabs - p.c) * p.b + bi) * p.ld_dqkv + hi * 3 * D;
      T* drow = static_cast<T*>(p.dqkv) + out_row;
      uint32_t tsrc;
      int col0, ncols, slot;
      float mul;
      if (MODE == 0) {   // group 0: dV (Acc1) -> v slot; group 1: dK (Acc2) * scale -> k slot
        tsrc = grp == 0 ? tA1 : tA2;
        col0 = 0; ncols = D; slot = grp == 0 ? 2 * D : D;
        mul = grp == 0 ? 1.0f : p.scale;
      } else {           // dQ (Acc2) * scale -> q slot, each group writes half of the columns
        tsrc = tA2;
        col0 = grp * (D / 2); ncols = D / 2; slot = 0;
        mul = p.scale;
      }
#pragma unroll 1
      for (int cc = col0; cc < col0 + ncols; cc += 32) {
        uint32_t raw[32];
        __syncwarp();
        tmem_ld_32x32(tsrc + lane_base + cc, raw);
        tmem_ld_wait();
        if (x_ok) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 u;
            u.x = Elem<T>::pack2(__uint_as_float(raw[g * 8 + 0]) * mul, __uint_as_float(raw[g * 8 + 1]) * mul);
            u.y = Elem<T>::pack2(__uint_as_float(raw[g * 8 + 2]) * mul, __uint_as_float(raw[g * 8 + 3]) * mul);
            u.z = Elem<T>::pack2(__uint_as_float(raw[g * 8 + 4]) * mul, __uint_as_float(raw[g * 8 + 5]) * mul);
            u.w = Elem<T>::pack2(__uint_as_float(raw[g * 8 + 6]) * mul, __uint_as_float(raw[g * 8 + 7]) * mul);
            __stcg(reinterpret_cast<uint4*>(drow + slot + cc + g * 8), u);
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (sh->abort_flag) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_after();
  if (warp == 9) tmem_dealloc(tmem, kTmemCols);
  if (MODE == 1) pdl_wait(false);
}

// ---------------------------------------------------------------------------- host side
static bool qkv_tmap(CUtensorMap* out, const void* qkv, int D, int b, int h, int rows_valid,
                     int box_rows, bool bf16) {
  uint64_t dims[3] = {static_cast<uint64_t>(3 * D), static_cast<uint64_t>(b * h),
                      static_cast<uint64_t>(rows_valid)};
  uint64_t strides[2] = {static_cast<uint64_t>(3 * D) * 2, static_cast<uint64_t>(b) * h * 3 * D * 2};
  uint32_t box[3] = {64, 1, static_cast<uint32_t>(box_rows)};
  return make_tmap_16b(out, qkv, 3, dims, strides, box, bf16);
}

static bool do_tmap(CUtensorMap* out, const void* d_o, long long ld, int D, int b, int h, int t,
                    int box_rows, bool bf16) {
  uint64_t dims[3] = {static_cast<uint64_t>(h * D), static_cast<uint64_t>(b), static_cast<uint64_t>(t)};
  uint64_t strides[2] = {static_cast<uint64_t>(ld) * 2, static_cast<uint64_t>(b) * ld * 2};
  uint32_t box[3] = {64, 1, static_cast<uint32_t>(box_rows)};
  return make_tmap_16b(out, d_o, 3, dims, strides, box, bf16);
}

template <typename K> static bool set_smem(K kern, int bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}

template <int D> constexpr int fwd_smem() {
  return (D / 64) * (2 * 128 * 128 + 2 * kFwdStages * 64 * 128) + 1024 + static_cast<int>(sizeof(FwdShared)) + 64;
}
template <int D> constexpr int bwd_smem() {
  return (D / 64) * (2 * 128 * 128 + kBwdStages * 2 * 64 * 128) + 1024 + static_cast<int>(sizeof(BwdShared)) + 64;
}

static_assert(fwd_smem<64>() >= kTmemKernelMinSmem && bwd_smem<64>() >= kTmemKernelMinSmem,
              "allocate TMEM before pdl_wait");

template <typename T, int D>
static int attn_fwd_launch(const void* qkv, const AttnParams& p, bool bf16, cudaStream_t s) {
  CUtensorMap tmQ, tmKV;
  if (!qkv_tmap(&tmQ, qkv, D, p.b, p.h, p.c + p.t, 128, bf16) ||
      !qkv_tmap(&tmKV, qkv, D, p.b, p.h, p.c + p.t, 64, bf16))
    return kErrDriver;
  auto kern = attn_fwd_kernel<T, D>;
  static bool cfg = false;
  if (!cfg) { if (!set_smem(kern, fwd_smem<D>())) return kErrLaunch; cfg = true; }
  const long long ctas = static_cast<long long>((p.t + 255) / 256) * p.b * p.h;
  if (ctas > 0x7fffffffLL) return kErrTooLarge;
  return launch_pdl(kern, dim3(static_cast<unsigned>(ctas)), dim3(kAttnThreads), fwd_smem<D>(), s, 1, tmQ, tmKV,
                    p) == cudaSuccess
             ? kOk
             : kErrLaunch;
}

template <typename T, int D>
static int attn_bwd_launch(const void* qkv, const void* o, const void* do_full, long long ld_do,
                           const AttnParams& p, bool bf16, cudaStream_t s) {
  CUtensorMap tm128, tm64, tmdO64, tmdO128;
  if (!qkv_tmap(&tm128, qkv, D, p.b, p.h, p.q_end, 128, bf16) ||
      !qkv_tmap(&tm64, qkv, D, p.b, p.h, p.q_end, 64, bf16) ||
      !do_tmap(&tmdO64, do_full, ld_do, D, p.b, p.h, p.q_end, 64, bf16) ||
      !do_tmap(&tmdO128, do_full, ld_do, D, p.b, p.h, p.q_end, 128, bf16))
    return kErrDriver;
  const long long ctas = static_cast<long long>((p.t + 127) / 128) * p.b * p.h;
  if (ctas > 0x7fffffffLL) return kErrTooLarge;
  {
    const long long rows = static_cast<long long>(p.t) * p.b * p.h;
    const long long blocks = (rows + DeltaRows<D>::value - 1) / DeltaRows<D>::value;
    const T* do_slice = static_cast<const T*>(do_full) + static_cast<long long>(p.c) * p.b * ld_do;
    const int o_vec = (reinterpret_cast<uintptr_t>(o) & 15) == 0 ? 1 : 0;
    if (launch_pdl(attn_delta_kernel<T, D>, dim3(static_cast<unsigned>(blocks)), dim3(kDeltaThreads), 0, s, 1,
                   static_cast<const T*>(o), p.ld_o, do_slice, ld_do, p.delta, p.lse_stride, p.c, p.t, p.b,
                   p.h, o_vec) != cudaSuccess)
      return kErrLaunch;
  }
  auto k0 = attn_bwd_kernel<T, D, 0>;
  auto k1 = attn_bwd_kernel<T, D, 1>;
  static bool cfg = false;
  if (!cfg) {
    if (!set_smem(k0, bwd_smem<D>()) || !set_smem(k1, bwd_smem<D>())) return kErrLaunch;
    cfg = true;
  }
  const dim3 grid(static_cast<unsigned>(ctas));
  if (launch_pdl(k0, grid, dim3(kBwdThreads), bwd_smem<D>(), s, 1, tm128, tm64, tmdO128, tmdO64, p) !=
      cudaSuccess)
    return kErrLaunch;
  return launch_pdl(k1, grid, dim3(kBwdThreads), bwd_smem<D>(), s, 1, tm128, tm64, tmdO128, tmdO64, p) ==
                 cudaSuccess
             ? kOk
             : kErrLaunch;
}

}  // namespace tp

using namespace tp;

// `scale` multiplies q.k before the softmax; <= 0 selects D^-0.5.  A caller whose heads are narrower
// than the kernel's D (zero-padded columns) passes the scale of the real width.
static AttnParams base_params(int D, float scale, int b, int h, int t, int c, int* err) {
  AttnParams p;
  memset(&p, 0, sizeof(p));
  p.t = t; p.c = c; p.b = b; p.h = h;
  p.scale = scale > 0.0f ? scale : 1.0f / sqrtf(static_cast<float>(D));
  p.scale2 = p.scale * 1.4426950408889634f;
  p.err = err;
  return p;
}

// qkv: base of the full-length [L][b][h][3][D] buffer; rows [0, c+t) must be valid.
extern "C" int tp_attn_fwd_scaled(int dtype, int D, float scale, const void* qkv, int b, int h, int t,
                                  int c, void* o, long long ld_o, float* lse2, long long lse_stride,
                                  int* err, void* stream) {
  if ((D != 64 && D != 128) || t <= 0 || c < 0 || b <= 0 || h <= 0) return kErrBadArgument;
  if (ld_o % 8) return kErrBadArgument;
  AttnParams p = base_params(D, scale, b, h, t, c, err);
  p.o = o; p.ld_o = ld_o; p.lse2 = lse2; p.lse_stride = lse_stride;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool bf16 = dtype == 1;
  if (D == 128) return bf16 ? attn_fwd_launch<__nv_bfloat16, 128>(qkv, p, true, s)
                            : attn_fwd_launch<__half, 128>(qkv, p, false, s);
  return bf16 ? attn_fwd_launch<__nv_bfloat16, 64>(qkv, p, true, s)
              : attn_fwd_launch<__half, 64>(qkv, p, false, s);
}

extern "C" int tp_attn_fwd(int dtype, int D, const void* qkv, int b, int h, int t, int c, void* o,
                           long long ld_o, float* lse2, long long lse_stride, int* err,
                           void* stream) {
  return tp_attn_fwd_scaled(dtype, D, 0.0f, qkv, b, h, t, c, o, ld_o, lse2, lse_stride, err, stream);
}

// Backward of the slice [c, c+t).  The slices after it must already have been processed:
//   o        this slice's attention output, [t*b][ld_o]
//   do_full  full-length gradient of the attention output, [L*b][ld_do]; rows [c*b, q_end*b)
//            are read (this slice's rows must have been written by the caller)
//   lse2, delta   fp32 [b*h][lse_stride], indexed by absolute position; delta rows [c, c+t) are
//            written here, rows [c+t, q_end) were written by the calls for the later slices
//   dqkv     this slice's [t*b][ld_dqkv] output (same column order as qkv)
extern "C" int tp_attn_bwd_scaled(int dtype, int D, float scale, const void* qkv, int b, int h, int t,
                                  int c, int q_end, const void* o, long long ld_o, const void* do_full,
                                  long long ld_do, const float* lse2, long long lse_stride,
                                  float* delta, void* dqkv, long long ld_dqkv, int* err,
                                  void* stream) {
  if ((D != 64 && D != 128) || t <= 0 || c < 0 || b <= 0 || h <= 0 || q_end < c + t)
    return kErrBadArgument;
  if (ld_o % 8 || ld_do % 8 || ld_dqkv % 8) return kErrBadArgument;
  AttnParams p = base_params(D, scale, b, h, t, c, err);
  p.o = const_cast<void*>(o); p.ld_o = ld_o;
  p.lse2 = const_cast<float*>(lse2); p.lse_stride = lse_stride;
  p.delta = delta; p.q_end = q_end; p.dqkv = dqkv; p.ld_dqkv = ld_dqkv;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool bf16 = dtype == 1;
  if (D == 128) return bf16 ? attn_bwd_launch<__nv_bfloat16, 128>(qkv, o, do_full, ld_do, p, true, s)
                            : attn_bwd_launch<__half, 128>(qkv, o, do_full, ld_do, p, false, s);
  return bf16 ? attn_bwd_launch<__nv_bfloat16, 64>(qkv, o, do_full, ld_do, p, true, s)
              : attn_bwd_launch<__half, 64>(qkv, o, do_full, ld_do, p, false, s);
}

extern "C" int tp_attn_bwd(int dtype, int D, const void* qkv, int b, int h, int t, int c, int q_end,
                           const void* o, long long ld_o, const void* do_full, long long ld_do,
                           const float* lse2, long long lse_stride, float* delta, void* dqkv,
                           long long ld_dqkv, int* err, void* stream) {
  return tp_attn_bwd_scaled(dtype, D, 0.0f, qkv, b, h, t, c, q_end, o, ld_o, do_full, ld_do, lse2,
                            lse_stride, delta, dqkv, ld_dqkv, err, stream);
}

TP_DEFINE_WAIT_LIMIT_SETTER(tp_set_wait_limit_ns_attn)
