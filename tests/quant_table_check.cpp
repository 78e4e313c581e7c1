// quant_table_check.cpp — the re-quantiser's thresholds (quant_table.h) against the
// nearest-level search, over level tables and samples where they could part: every
// threshold and its neighbours, the levels, the ends of the thresholds' range,
// infinities and NaN.  The decision and the search are those of fxc_device.cuh.
// Prints the tables by kind and the samples that differ.
#include "quant_table.h"

#include <cfloat>
#include <cstdio>
#include <random>
#include <vector>

using namespace fxc;

static uint32_t search(float x, const std::vector<float>& lv) {
  const int n = (int)lv.size();
  int lo = 0, hi = n;
  if (n > 16) {
    int a = 0, b = n;
    while (a < b) {
      const int m = (a + b) >> 1;
      if (lv[m] > x) b = m;
      else a = m + 1;
    }
    lo = std::max(0, a - 2);
    hi = std::min(n, a + 2);
  }
  uint32_t best = (uint32_t)lo;
  float least = FLT_MAX;
  for (int i = lo; i < hi; ++i) {
    const float err = std::fabs(x - lv[i]);
    if (err < least) {
      least = err;
      best = (uint32_t)i;
    }
  }
  return best;
}

static uint32_t decide(float x, const std::vector<float>& lv, const QuantTable& q, const float* thr) {
  const int n = (int)lv.size();
  if (!(std::fabs(x) <= q.hi) || q.kind == QUANT_SEARCH) return search(x, lv);
  if (q.kind == QUANT_COMPARE)
    return ((uint32_t)(x >= thr[1]) + (uint32_t)(x >= thr[2]) + (uint32_t)(x >= thr[3])) &
           (uint32_t)(n - 1);
  const float f = std::floor(std::fmaf(x, q.step, q.offset));
  int g = f < 0.0f ? 0 : (f > (float)(n - 1) ? n - 1 : (int)f);
  g += (x >= thr[g + 1] ? 1 : 0) - (x < thr[g] ? 1 : 0);
  return (uint32_t)g;
}

int main() {
  std::mt19937 rng(7);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  int kinds[3] = {0, 0, 0};
  long differ = 0, samples = 0;
  for (int bits : {1, 2, 4, 8}) {
    const int n = 1 << bits;
    for (double scale : {1e-40, 1e-31, 1e-6, 1.0, 3.7, 1e9, 1e30, 1e32, 1e33, 1e36, 1e38, 3e38})
      for (double offset : {0.0, 0.3, 50.0, 1e5})
        for (double uneven : {0.0, 0.004, 0.4}) {
          std::vector<float> lv(n);
          for (int i = 0; i < n; ++i) {
            const double x = 2.0 * i / (n - 1) - 1.0;  // -1 .. 1
            lv[i] = (float)(scale * (x + uneven * x * x * x / n + offset) / (1.0 + offset));
          }
          bool up = true;
          for (int i = 1; i < n; ++i) up = up && lv[i] > lv[i - 1];
          float thr[257];
          const QuantTable q = quant_thresholds(lv.data(), n, up, thr);
          kinds[q.kind] += 1;
          std::vector<float> x = {0.0f, -0.0f, FLT_MAX, -FLT_MAX, INFINITY, -INFINITY, NAN,
                                  FLT_MIN, 1e-45f, q.hi, -q.hi, 0x1p+126f, -0x1p+126f, 0x1p+127f};
          for (int i = 0; i < n; ++i) {
            x.push_back(lv[i]);
            if (i) x.push_back(thr[i]);
            if (i) x.push_back(0.5f * lv[i - 1] + 0.5f * lv[i]);
          }
          for (int k = 0; k < 2000; ++k)
            x.push_back((float)(lv[n - 1] * u(rng) * std::exp2(k % 5 * 6)));
          for (float x0 : x)
            for (int d = -3; d <= 3; ++d) {
              float v = x0;
              for (int s = 0; s < std::abs(d); ++s) v = std::nextafter(v, d < 0 ? -INFINITY : INFINITY);
              samples += 1;
              // the search leaves descending and repeated tables their own order
              if (up && decide(v, lv, q, thr) != search(v, lv)) differ += 1;
            }
        }
  }
  std::printf("%d %d %d %ld %ld\n", kinds[0], kinds[1], kinds[2], samples, differ);
  return 0;
}
