// quant_table.h — decision thresholds of the phased re-quantiser, found on the host
// (fxc_device.cuh, quantise_many, applies them).
#pragma once

#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>

namespace fxc {

enum : int32_t { QUANT_SEARCH = 0, QUANT_COMPARE = 1, QUANT_STEP = 2 };

struct QuantTable {
  int32_t kind = QUANT_SEARCH;
  float hi = 0.0f, step = 0.0f, offset = 0.0f;
};

// Thresholds of the nearest-level rule (first index wins ties) for strictly
// ascending levels: thr[i], i = 1..n-1, is the least f32 x whose rounded distance
// to level i is below that to level i - 1.  Between two levels both rounded
// distances are monotonic in x, so that is a step, found by bisection; and no
// other level can be nearer or tie as long as the spacing does not vanish in the
// rounding: levels no closer than 2^-20 of their range, |x| up to 2^20
// spacings beyond them; nor in the overflow: levels and |x| up to 2^126, so that
// an infinite x, which is as far from every level, is the search's.  Other tables
// keep the search.
inline QuantTable quant_thresholds(const float* lv, uint32_t n, bool ascending, float* thr) {
  QuantTable q;
  for (int i = 0; i < 257; ++i) thr[i] = std::numeric_limits<float>::infinity();
  thr[0] = -thr[256];
  if (!ascending || n < 2) return q;
  double gap = 1e300;
  for (uint32_t i = 1; i < n; ++i) gap = std::min(gap, (double)lv[i] - (double)lv[i - 1]);
  const double top = std::max(std::fabs((double)lv[0]), std::fabs((double)lv[n - 1]));
  if (!(top <= 0x1p+126) || !(gap > 0x1p-100) || gap < top * 0x1p-20) return q;
  // f32 values in order as integers
  auto key = [](float x) {
    int32_t b;
    std::memcpy(&b, &x, 4);
    return b < 0 ? (int64_t)INT32_MIN - b : (int64_t)b;
  };
  auto val = [](int64_t k) {
    const int32_t b = k < 0 ? (int32_t)((int64_t)INT32_MIN - k) : (int32_t)k;
    float x;
    std::memcpy(&x, &b, 4);
    return x;
  };
  for (uint32_t i = 1; i < n; ++i) {
    int64_t lo = key(lv[i - 1]), hi = key(lv[i]);  // not past, past
    while (hi - lo > 1) {
      const int64_t m = lo + (hi - lo) / 2;
      const float x = val(m);
      const float below = std::fabs(x - lv[i - 1]), above = std::fabs(x - lv[i]);
      if (above < below) hi = m;
      else lo = m;
    }
    thr[i] = val(hi);
  }
  q.hi = (float)std::min(gap * 0x1p+20, 0x1p+126);
  if (n <= 4) {
    q.kind = QUANT_COMPARE;
    return q;
  }
  // a uniform table: the guess is right but next to a threshold
  const double step = ((double)lv[n - 1] - (double)lv[0]) / (n - 1);
  for (uint32_t i = 0; i < n; ++i)
    if (std::fabs((double)lv[i] - ((double)lv[0] + i * step)) > 0.01 * step) return q;
  q.kind = QUANT_STEP;
  q.step = (float)(1.0 / step);
  q.offset = (float)(0.5 - (double)lv[0] / step);
  return q;
}

}  // namespace fxc
