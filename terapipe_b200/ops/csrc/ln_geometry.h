// Thread geometry of the LayerNorm kernels: plain C++, shared by the launch code and the host harness
// of the CPU tests.  A row is handled by `wpr` warps (a power of two up to 16) whose lanes hold `nv`
// vectors of 8 elements each.
#pragma once

namespace tp {

// The smallest warps-per-row that keeps at most `most` vectors per lane.
inline bool ln_geometry(int H, int* nv, int* wpr, int most) {
  if (H % 8 || H <= 0) return false;
  const int vecs = H / 8;
  for (int w = 1; w <= 16; w *= 2) {
    const int n = (vecs + 32 * w - 1) / (32 * w);
    if (n <= most) { *nv = n; *wpr = w; return true; }
  }
  return false;
}

// Backward: warps of a CTA, of which there is one per SM.  24 leave 80 registers a thread, too few for four
// vectors of each of the three inputs; 16 hold these, and with the fewer warps a row takes then 4 / 3
// as many rows as 24 warps of two vectors.  16384 x 2048: two vectors 63.2 us, four on 24 warps
// 65.3, four on 16 warps 57.8.  (Eight warps a row stay with 24, three rows, whatever it costs in
// registers: 16384 x 8192 takes 242 us, 16 warps of two vectors and one row take 290.)
constexpr int ln_bwd_warps(int nv, int wpr) { return wpr == 16 || (nv == 4 && wpr < 8) ? 16 : 24; }
constexpr int ln_bwd_rows(int nv, int wpr) { return ln_bwd_warps(nv, wpr) / wpr; }   // of a CTA

// Few rows: the geometry with the fewest vectors that takes all rows in one round of the CTAs, for the
// lanes then have the least to do one after the other.  1024 x 2048 takes 6.7 us in one round of
// four vectors, 8.4 in two of two; 77 x 768 3.9 us with one vector, 6.2 with three.  (Not four
// vectors on 24 warps: 256 x 8192 takes 8.4 us in two rounds and 10.0 in one of these.)
// Many rows: three vectors at most, unless four on 16 warps, whose rounds take 5 / 4 as long (57.8 us / 14
// against 63.2 / 19 above), need so many fewer (2048 x 1024 6.3 us against 8.1; 6144 x 1600 stays
// at 20.0 us, it would take 21.0), or rows of eight warps are at least 2048 (2048 x 8192 43.2 us
// against 45.6, but 1024 rows 21.7 against 19.4).
inline bool ln_bwd_geometry(int H, int rows, int sms, int* nv, int* wpr) {
  const auto rounds = [&](int n, int w) { return (rows - 1) / (sms * ln_bwd_rows(n, w)) + 1; };
  for (int most = 1; most <= 4; ++most)
    if (ln_geometry(H, nv, wpr, most) && rounds(*nv, *wpr) == 1 && (*nv < 4 || ln_bwd_warps(*nv, *wpr) == 16))
      return true;
  int n4, w4;
  if (!ln_geometry(H, &n4, &w4, 4)) return false;
  const bool upto3 = ln_geometry(H, nv, wpr, 3);
  const bool four = upto3 && n4 == 4 && (w4 < 8 ? rounds(n4, w4) * 5ll < rounds(*nv, *wpr) * 4ll
                                                      : w4 == 8 && rows >= 2048);
  if (!upto3 || four) {
    *nv = n4;
    *wpr = w4;
  }
  return true;
}

}  // namespace tp
