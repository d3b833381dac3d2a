// pp_tables.h -- bin categories on the host: the category of a distance, the
// thresholds of d^2 the kernels compare with, the lookup table over its bits and
// the rule for the approximate guess.  Plain C++, no CUDA.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

namespace pp_tables {

constexpr double kEpsilon = 1.0e-6;  // src/PARAPROBE_Numerics.h:44

struct Tables {
  // histogram
  float rmin = 0.f, rincr = 0.1f, rmax = 2.f;  // reference defaults, src/PARAPROBE_Settings.cpp:106-108
  uint32_t nbins = 0;
  double hstart = 0, hend = 0, hscale = 0;
};

// Category of one float distance under histogram::add
// (src/PARAPROBE_Histogram.h:97-117): 0 lowest, 1 + b bin b, nbins + 1 highest.
inline int category_of_distance(const Tables& t, float x) {
  const double xx = x;
  if (xx >= t.hstart && xx <= t.hend) {
    const float rb = (float)((xx - t.hstart) * t.hscale);
    const uint32_t b = (uint32_t)std::floor(rb);
    return b < t.nbins ? (int)(1 + b) : (int)(t.nbins + 1);
  }
  if (xx < t.hstart) return 0;
  return (int)(t.nbins + 1);
}

inline int category_of_d2(const Tables& t, float d2) { return category_of_distance(t, std::sqrt(d2)); }

inline void set_tables(Tables& t, float rmin, float rincr, float rmax) {
  t.rmin = rmin; t.rincr = rincr; t.rmax = rmax;
  t.hstart = rmin; t.hend = rmax;
  size_t nb = 0;
  if ((double)rincr > kEpsilon) nb = (size_t)(((double)rmax - (double)rmin) / (double)rincr);
  t.nbins = (uint32_t)nb;
  t.hscale = nb ? 1.0 / (t.hend - t.hstart) * (double)nb : 0.0;
}

// T[k] = smallest non-negative float d^2 whose category is >= k (k = 1..H-1),
// +inf when no finite d^2 reaches k.  The category is monotone in d^2, so a
// search over the ordered bit patterns of non-negative floats finds it: outward
// from the bin's edge in doubling steps, then by bisection -- seven categories
// evaluated where bisecting all patterns takes 31.  Every pass builds these
// tables: 100 bins 102 -> 12 us, 400 bins 265 -> 18 us with build_lut.
inline std::vector<float> threshold_table(const Tables& t) {
  const int H = (int)t.nbins + 2;
  constexpr uint32_t top = 0x7f7fffffu;  // the largest finite float
  std::vector<float> T(H, 0.f);
  for (int k = 1; k < H; ++k) {
    auto cat = [&](uint32_t u) {
      float f;
      std::memcpy(&f, &u, 4);
      return category_of_d2(t, f);
    };
    if (cat(top) < k) { T[k] = INFINITY; continue; }
    const double edge = t.hstart + (t.hscale > 0.0 ? (double)(k - 1) / t.hscale : 0.0);
    const float guess = (float)(edge * edge);
    uint32_t at = 0;
    if (guess > 0.f && guess < INFINITY) std::memcpy(&at, &guess, 4);
    // lo: everything below is of a lower category; hi: of category k or more
    uint32_t lo = 0, hi = top;
    if (cat(at) >= k) {
      hi = at;
      for (uint64_t step = 2; step <= hi; step *= 2) {
        const uint32_t u = hi - (uint32_t)step;
        if (cat(u) < k) { lo = u + 1; break; }
        hi = u;
      }
    } else {
      lo = at + 1;
      for (uint64_t step = 2; step <= top - lo; step *= 2) {
        const uint32_t u = lo + (uint32_t)step;
        if (cat(u) >= k) { hi = u; break; }
        lo = u + 1;
      }
    }
    while (lo < hi) {
      const uint32_t mid = lo + (hi - lo) / 2;
      if (cat(mid) >= k) hi = mid; else lo = mid + 1;
    }
    std::memcpy(&T[k], &lo, 4);
  }
  return T;
}

// Category lookup table over the ordered bit patterns of d^2 in [0, R^2]:
// cell c covers the patterns with (bits >> shift) == base + c and holds the
// category of its smallest d^2 (cell 0 also takes every smaller d^2, all of
// category T-count-at-0).  The device starts there and steps up through T, so
// the result equals the threshold search for any shift; the shift is the
// finest that keeps the table within max_cells, so a cell rarely spans more
// than one threshold.
inline void build_lut(const std::vector<float>& T, float r2, int max_cells, std::vector<uint16_t>& lut, int& shift,
                      uint32_t& base, bool* one_step = nullptr) {
  const int H = (int)T.size();
  auto bits = [](float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; };
  auto cat = [&](float d2) {
    int k = 0;
    while (k + 1 < H && T[k + 1] <= d2) ++k;
    return k;
  };
  float tmin = r2;
  for (int k = 1; k < H; ++k)
    if (T[k] > 0.f && T[k] < tmin) tmin = T[k];
  const uint32_t top = bits(std::max(r2, 0.f));
  for (shift = 0; shift < 31; ++shift) {
    base = bits(tmin) >> shift;
    if ((int64_t)(top >> shift) - (int64_t)base + 1 <= max_cells) break;
  }
  base = bits(tmin) >> shift;
  const int n = (int)((top >> shift) - base + 1);
  lut.assign(n, 0);
  int k = cat(0.f);
  lut[0] = (uint16_t)k;
  for (int c = 1; c < n; ++c) {  // cells ascend, and so do their categories
    const uint32_t u = (base + (uint32_t)c) << shift;
    float f;
    std::memcpy(&f, &u, 4);
    while (k + 1 < H && T[k + 1] <= f) ++k;
    lut[c] = (uint16_t)k;
  }
  if (one_step) {
    // categories rise with d^2, so within cell c they run from lut[c] to at
    // most lut[c + 1] (cell 0 also takes every d^2 below it: no positive
    // threshold lies there); the last cell holds r2, and only d^2 <= r2 count
    bool one = true;
    for (int c = 0; c + 1 < n && one; ++c) one = lut[c + 1] <= lut[c] + 1;
    *one_step = one && cat(std::max(r2, 0.f)) <= lut[n - 1] + 1;
  }
}

// Whether floor(sqrt(d^2) * scale + 1/2), to within an eighth of a bin, is the
// category of d^2 or one less for every d^2 in [0, R^2]: the bins start at 0
// and every threshold lies within 1/256 of a bin of its edge.  The float
// evaluation takes little of the margin of 3/8: sqrt.approx is within 2^-23 of
// the root, and the scale, its quotient and the product each round by 2^-24,
// together below 2^-21 of at most 16382 bins.
inline bool category_fast_ok(const std::vector<float>& T, const Tables& t) {
  if (t.rmin != 0.f) return false;
  const double scale = (double)(float)t.hscale;
  for (size_t k = 1; k < T.size(); ++k)
    if (!(std::fabs(std::sqrt((double)T[k]) * scale - (double)(k - 1)) < 1.0 / 256)) return false;
  return true;
}

}  // namespace pp_tables
