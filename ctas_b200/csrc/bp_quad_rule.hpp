// bp_quad_rule.hpp -- which slices of a stack go through the four-slice kernel
// (bp_quad.cu), from estimates of both ways' device time (host code).
//
// Both kernels fill the device in waves of CTAs, and a stack of a few small slices is
// mostly last waves: three slices of 612 x 612 take 212 us as one group and 168 one at a
// time, four 212 and 256.  A rule by the number of tiles alone cost up to 1.37 times the
// time of one slice at a time (3 x 600 x 600; 5 x 600 x 600 1.25, 9 x 408 x 408 1.20).
// Times measured at 720 projections over 51 widths from 192 to 2600 and 1 to 12 slices,
// in microseconds by x = tiles with pixels in the disc over SMs: steps up to x = 4, then
// a line.  Singles with the tile that ran fastest for each.  With the allowances in
// quad_slices() no choice was more than 1.5 % slower than one slice at a time, and the
// mean over all was 1.30 times as fast (with the best choice for each 1.34).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

namespace ctas {

// Whether the sharing patterns' margin, (W + 256) 2^-19 = (32 W + 8192) 2^-24, covers the
// rounding of an output geometry.  Two values of t in the disc differ from exact ones by
// at most 12 W 2^-24; a pixel coordinate o + p k by half an ulp of p k and one of the
// sum, which two pixels and two axes make 2.84 (p k + W) 2^-24: within the margin up to
// p k = 4 W + 1024.  Beyond (65536 rows with a disc at their far end) pixels were off by
// a sample, about one in 10^6.
inline bool quad_sharing_exact(int64_t W, int64_t rows, int64_t cols, double p) {
  return p * (double)std::max(rows, cols) <= 4.0 * (double)W + 1024.0;
}

// Tiles of one slice: all of 64 x 64, and those of 64 x 64 and of 32 x 64 that hold a
// pixel of the reconstruction disc (centre offset 0).
struct SliceTiles {
  int64_t all64 = 0, in64 = 0, in32 = 0;
};

inline SliceTiles slice_tiles(int64_t W, int64_t rows, int64_t cols, double oj, double oi, double p) {
  const double hp = (double)(W / 2);
  // distance of the disc's centre from the coordinates of pixels a .. b of an axis
  auto apart = [&](double o, int64_t a, int64_t b) {
    const double lo = o + p * (double)a, hi = o + p * (double)b;
    return hp < lo ? lo - hp : hp > hi ? hp - hi : 0.0;
  };
  std::vector<double> di2;
  for (int64_t i = 0; i < cols; i += 64) {
    const double d = apart(oi, i, std::min(cols, i + 64) - 1);
    di2.push_back(d * d);
  }
  auto count = [&](int64_t ty) {
    int64_t n = 0;
    for (int64_t j = 0; j < rows; j += ty) {
      const double d = apart(oj, j, std::min(rows, j + ty) - 1), room = hp * hp - d * d;
      for (const double v : di2) n += v < room;
    }
    return n;
  };
  SliceTiles t;
  t.all64 = ((rows + 63) / 64) * ((cols + 63) / 64);
  t.in64 = count(64);
  t.in32 = count(32);
  return t;
}

// kernel forms: truncation, truncation on the wide layout, linear interpolation
enum QuadForm { kQuadTrunc = 0, kQuadWide = 1, kQuadLinear = 2 };

struct FillTime {
  double step[4], off, slope;
  double at(double x) const {
    return x <= 0 ? 0 : x <= 4 ? step[(int)std::ceil(x) - 1] : std::max(step[3], off + slope * x);
  }
};
struct FormTimes {
  FillTime single, small, large;  // one slice at a time; groups on 32 x 64 and 64 x 64 tiles
};
inline const FormTimes &quad_times(QuadForm f) {
  static const FormTimes t[3] = {
      {{{99, 167, 255, 316}, 65, 71.8}, {{158, 213, 371, 426}, 0, 107}, {{342, 342, 613, 678}, 69, 169}},
      {{{127, 190, 327, 362}, 82, 81.2}, {{191, 250, 441, 500}, 0, 125}, {{430, 430, 720, 850}, -34, 245}},
      {{{240, 474, 706, 940}, 104, 231}, {{240, 365, 605, 730}, 0, 183}, {{654, 654, 1165, 1300}, -141, 385}}};
  return t[f];
}

// Groups on the small tile: below one and a half 64 x 64 tiles per SM (4 slices of
// 1023 x 1023: 104 us per slice on the large tile, 115 on the small one).
inline bool quad_small_tile(int64_t tiles64, int sms) { return 2 * tiles64 < 3 * (int64_t)sms; }

inline double singles_us(QuadForm f, const SliceTiles &t, int64_t slices, int sms, double more = 1.0) {
  return quad_times(f).single.at(more * (double)(t.in64 * slices) / sms);
}
inline double groups_us(QuadForm f, const SliceTiles &t, int64_t groups, int sms, double more = 1.0) {
  const FormTimes &m = quad_times(f);
  return quad_small_tile(t.all64 * groups, sms) ? m.small.at(more * (double)(t.in32 * groups) / sms)
                                                : m.large.at(more * (double)(t.in64 * groups) / sms);
}
// The first n slices in groups, the others one at a time.  more: tiles are taken so many
// times as many; single slices just below a step run at the next (x = 0.92: 133 us).
inline double stack_us(QuadForm f, const SliceTiles &t, int64_t slices, int64_t n, int sms,
                       double more = 1.0) {
  return groups_us(f, t, (n + 3) / 4, sms) + singles_us(f, t, slices - n, sms, more);
}

// Slices from which groups always pay (a dozen 64 x 64 tiles per SM): no estimate of
// singles is taken there, so that buffers sized up to here serve every count.
inline int64_t quad_always(const SliceTiles &t, int sms) {
  return 12 * (int64_t)sms / std::max<int64_t>(1, t.in64) + 4;
}

// How many of `slices` slices (the first ones) go through groups: 0, all, or all but a
// rest below four, whichever is estimated fastest.  One slice at a time is preferred
// within 6 %, on tiles taken a tenth fewer, and groups are taken on 3 % more: the steps
// lie that near to one another, and a shifted disc moves a few tiles.
inline int64_t quad_slices(QuadForm f, const SliceTiles &t, int64_t slices, int sms) {
  if (slices < 3 || t.in64 < 1) return 0;
  double best = 0.94 * quad_times(f).single.at(0.9 * (double)(t.in64 * slices) / sms);
  if (slices > quad_always(t, sms)) best = HUGE_VAL;
  int64_t n = 0;
  for (const int64_t c : {slices - slices % 4, slices}) {
    if (c < 3) continue;
    const double us = groups_us(f, t, (c + 3) / 4, sms, 1.03) + singles_us(f, t, slices - c, sms);
    if (us < best) {
      best = us;
      n = c;
    }
  }
  return n;
}

}  // namespace ctas
