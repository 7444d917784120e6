// Which output tile an ordinary product runs on: plain C++, shared by the launch code and the host
// harness of the CPU tests.
#pragma once

namespace tp {

// Codes: 32 / 64 / 128 / 256 = one CTA, 128 x BN tile; 512 = one CTA, 256 x 256; 1000 + BN = CTA pair,
// 256 x BN (BN = 128, 192, 224, 256).  Measured model of one launch, in kilo-cycles: waves x (main
// loop of one tile, proportional to K, + epilogue where it does not overlap the next tile) + exposed
// epilogue of the last tile.  Wave quantisation matters because M is only ~1024 rows per token slice.
// `loop` is per 2048 of K: the CTA-pair tiles run at 80-98 % of the MMA rate, the one-CTA tiles
// at 50-67 % (L2 -> shared-memory feed of one SM).
// kSplitCode * parts + BN = one CTA, 128 x BN tile (BN = 64, 128), K shared by `parts` CTAs of a cluster.
constexpr int kSplitCode = 10000;
struct TileCand {
  int code, bm, bn;
  bool pair;
  float loop, epi_each, tail;
};
constexpr TileCand kTileCands[6] = {
    {1256, 256, 256, true, 16.7f, 0.0f, 8.5f}, {1128, 256, 128, true, 10.0f, 0.0f, 5.5f},
    {512, 256, 256, false, 36.0f, 18.0f, 0.0f}, {256, 128, 256, false, 24.7f, 0.0f, 10.0f},
    {128, 128, 128, false, 16.4f, 0.0f, 5.4f}, {64, 128, 64, false, 9.5f, 0.0f, 3.0f}};
// 192 and 224 columns are for products of a few waves, whose last one is nearly empty with 256: 2048 x
// 5120 is 160 tiles of 256 columns on 74 pairs (3 waves of 16.7) or 216 of 192 (3 waves of 13.2).
// 2048 x 5120 x 10240 took 201 us with 256 columns and takes 163 with 192, 2048 x 7680 x 5120 121 and
// 110 with 224.
constexpr TileCand kCutCands[2] = {{1224, 256, 224, true, 15.0f, 0.0f, 7.8f},
                                   {1192, 256, 192, true, 13.2f, 0.0f, 7.0f}};

inline float tile_waves(const TileCand& c, int M, int N, int sms) {
  const long long tiles = static_cast<long long>((M + c.bm - 1) / c.bm) * ((N + c.bn - 1) / c.bn);
  const int slots = c.pair ? sms / 2 : sms;
  return static_cast<float>((tiles + slots - 1) / slots);
}

// second: the epilogue reads or writes a second matrix of the output's size (residual, pre-activation).
// allow_cut: an all-gather -> GEMM product keeps the full widths, with which its order of tiles (this
// rank's row blocks first) was built and measured on several GPUs.
// time: the model's estimate.
inline int choose_tile(int M, int N, int K, bool b_mn, bool second, bool allow_256x256, bool allow_pair,
                       bool allow_cut, int sms, float* time = nullptr) {
  int best = 128;
  float best_t = 1e30f;
  for (const TileCand& c : kTileCands) {
    if ((c.code == 512 && !allow_256x256) || (c.pair && !allow_pair)) continue;
    const float t = tile_waves(c, M, N, sms) * (c.loop * static_cast<float>(K) / 2048.0f + c.epi_each) + c.tail;
    if (t < best_t) { best_t = t; best = c.code; }
  }
  if (time) *time = best_t;
  // A one-CTA tile of 128 or 256 columns wins where the rows are an odd number of 128-row blocks, few
  // of them: the second CTA of the last pair row has no rows.  The model puts such a tile too slow by
  // up to a third, so a cut pair tile may not take its place: 77 x 12288 x 4096 takes 21.8 us on
  // 128 columns and 27.0 on a pair's 192, 300 x 12288 x 3072 26.3 on 256 columns and 34.7; of 47 such
  // products between 16 and 800 rows, 45 took longer with the cut tile.
  if (!allow_pair || !allow_cut || best == 128 || best == 256) return best;
  for (const TileCand& c : kCutCands) {
    const float waves = tile_waves(c, M, N, sms);
    // Where N is contiguous, B comes in 64-column chunks: a CTA's 96 or 112 columns take the loads of
    // 128.  In a long row of waves each costs 4 % and 0.3 more than the model says: 10240 x 3840 x
    // 1280 took 71 us with 256 columns and 79 with 192, 8192 x 3072 x 768 32.7 and 35.4.  Not where a
    // short K and a second matrix leave the epilogue to bound a wave: with an activation's derivative or a
    // residual the latter product takes 8 % less with 192 columns, 5120 x 4096 x 1024 6 % less;
    // 5120 x 4096 x 2048 takes 2 to 6 % more.
    const bool chunks = b_mn && waves > 4.0f && !(second && K <= 1600);
    const float loop = c.loop * (chunks ? 1.04f : 1.0f) * static_cast<float>(K) / 2048.0f;
    const float t = waves * (loop + c.epi_each + (chunks ? 0.3f : 0.0f)) + c.tail;
    if (t < 0.97f * best_t) { best_t = t; best = c.code; }   // near ties go to the full widths
  }
  if (time) *time = best_t;
  return best;
}

// 32 columns a tile where the tiles of 64 or more leave SMs idle and those of 32 still run at once: a warp's
// epilogue then is one chunk, and it is most of such a product's time.  us with 64 / 32: 256 x 768 x 256 4.0 / 3.2,
// 256 x 1024 x 256 with GeLU 5.3 / 3.9, 77 x 3072 x 768 5.5 / 4.8, 128 x 4096 x 1024 6.5 / 5.6; in two rounds
// 154 x 3072 x 768 takes 7.2 instead of 5.8.  A long K is better shared where it can be (640 x 768 x 3072 9.5, 11.8
// on 32 columns), so `time` stays what it was there.
inline bool choose_narrow(int M, int N, int K, int code, int sms, float* time) {
  if (code != 64 && code != 128) return false;
  if (static_cast<long long>((M + 127) / 128) * ((N + 31) / 32) > sms) return false;
  const float t = 8.96f * static_cast<float>(K) / 2048.0f + 1.9f;
  if (K <= 1024 && t < *time) *time = t;
  return true;
}

// Whether a product is better off with K shared by a cluster (gemm_split_kernel): the code, or 0.  `time` is the
// estimate of choose_tile; the same units here.  A step of 64 of K takes what the MMA needs to read its operands
// from shared memory, all of them together at least their bytes at 13 TB/s out of L2; what a split pays for is the
// exchange of the partial sums, which grows with the rows and, where they are many, with the CTAs.  All clusters
// have to run at once, and an SM group holds few large ones: 36 clusters of 4 take two rounds (16 x 2304 x 768 7.9 us
// instead of 4.3 in 36 pairs), 16 of 8 as well (32 x 1024 x 4096 10.0, 16 of 4 6.3).  us without / with:
//   77 x 768 x 3072 12.3 / 5.9 (8 parts of 64 columns), 16 x 768 x 768 4.7 / 4.1 (4),
//   128 x 1024 x 4096 15.4 / 7.7 (4), 128 x 2048 x 8192 27.6 / 11.4 (4), 16 x 8192 x 2048 16.5 / 7.5 (2 of 128
//   columns), 64 x 4096 x 16384 52.6 / 27.9 (4 of 128), 256 x 2048 x 8192 27.9 / 16.3 (2 of 64).
// (Above 80 rows the ring of a 128-column split is shallow; with weights out of DRAM it is 2 to 10 % slower there than whole K
// on 64 columns: 80 x 6144 x 8192 30.6 / 27.0, but 104 x 6144 x 8192 31.0 / 34.0.)
inline int choose_split(int M, int N, int K, float time, int sms) {
  struct Cand { int bn, parts; float ctas, step, base, rows; };   // share of the SMs; per 64 of K; per 128 rows
  constexpr Cand cands[5] = {{64, 2, 1.0f, 0.254f, 4.0f, 1.5f}, {64, 4, 0.87f, 0.254f, 3.3f, 2.5f},
                             {64, 8, 0.65f, 0.254f, 3.4f, 3.8f}, {128, 2, 1.0f, 0.287f, 3.2f, 6.2f},
                             {128, 4, 0.87f, 0.287f, 3.4f, 5.8f}};
  const int rows = M < 128 ? M : 128;
  const float r = static_cast<float>(rows) / 128.0f;
  int best = 0;
  float best_t = 0.9f * time;
  for (const Cand& c : cands) {
    const long long tiles = static_cast<long long>((M + 127) / 128) * ((N + c.bn - 1) / c.bn), ctas = tiles * c.parts;
    if (static_cast<float>(ctas) > c.ctas * static_cast<float>(sms) || (K + 127) / 128 < c.parts) continue;
    const float crowd = ctas > 64 ? 0.025f * static_cast<float>(ctas - 64) : 0.0f;
    const float mma = (c.bn == 128 && M > 96 ? 0.4f : c.step) * static_cast<float>(K) / (64.0f * c.parts);
    const float feed = 2.4e-7f * static_cast<float>(tiles) * static_cast<float>(rows + c.bn) * static_cast<float>(K);
    const float t = (mma > feed ? mma : feed) + c.base + r * (c.rows + crowd);
    if (t < best_t) { best_t = t; best = kSplitCode * c.parts + c.bn; }
  }
  return best;
}

// What an ordinary forward or data-gradient product takes instead of choose_tile's `code`, whose estimate is `time`.
inline int choose_small(int M, int N, int K, int code, float time, int sms) {
  const bool narrow = choose_narrow(M, N, K, code, sms, &time);
  const int split = choose_split(M, N, K, time, sms);
  return split ? split : narrow ? 32 : code;
}

// Columns of a CTA pair's tile for the weight gradients of `layers` layers in one launch (wgrad_sm100.cu).
// A wave takes its main loop or, where that is shorter, what its epilogue moves at the copy bandwidth
// (kilo-cycles of 1.8 GHz: 26 bytes an element with Adam, else the staged stores); the last wave's epilogue is
// exposed.
inline int choose_wgrad_tile(int M, int N, int K, int layers, bool adam, int sms) {
  struct Cand { int bn; float loop, adam, store; };
  constexpr Cand cands[3] = {{256, 16.7f, 35.0f, 8.5f}, {192, 13.7f, 26.2f, 7.0f}, {128, 10.0f, 17.5f, 5.5f}};
  int best = 256;
  float best_t = 1e30f;
  for (const Cand& c : cands) {
    const long long tiles = static_cast<long long>((M + 255) / 256) * ((N + c.bn - 1) / c.bn) * layers;
    const float waves = static_cast<float>((tiles + sms / 2 - 1) / (sms / 2));
    const float loop = c.loop * static_cast<float>(K) / 2048.0f, epi = adam ? c.adam : c.store;
    const float t = waves * (loop > epi ? loop : epi) + epi;
    if (t < 0.97f * best_t) { best_t = t; best = c.bn; }
  }
  return best;
}

}  // namespace tp
