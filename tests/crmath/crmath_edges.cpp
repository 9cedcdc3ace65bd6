// Edges of the tables and argument reductions of bpl_crmath.cuh: the floats
// beside every boundary between log table entries (all exponents) and
// between exp reduction integers, checked against the reference expressions;
// and the exactness the reductions rely on.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <initializer_list>

#include "../../bp-layers_gb300/csrc/bpl_crmath.cuh"

using namespace bpl::crm;

int main() {
  long bad = 0, n = 0;
  auto chk_e = [&](float x) {
    float y;
    ++n;
    if (exp_fast(x, y) && y != static_cast<float>(std::exp(static_cast<double>(x)))) ++bad;
  };
  auto chk_l = [&](float s) {
    float y;
    ++n;
    if (log_fast(s, y) && y != static_cast<float>(std::log(static_cast<double>(s)))) ++bad;
  };
  for (int e = 1; e < 255; ++e)
    for (int j = 0; j < kLogEntries; ++j)
      for (int k = -2; k <= 2; ++k) chk_l(i2f((e << 23) + (j << 16) + k));
  for (int m = -16100; m <= 16300; ++m) {  // (m / 2) ln2/64: reduction integers and the midpoints between them
    float x = static_cast<float>(0.5 * m * 0.010830424696249145);
    for (int k = 0; k < 3; ++k, x = std::nextafter(x, 100.0f)) chk_e(x);
  }
  for (int j = 0; j < kLogEntries; ++j) {
    for (int k = 0; k < 65536; ++k) {  // mnt * c - 1 is exact
      const double r = static_cast<double>(i2f(0x3f800000 | (j << 16) | k)) * kTab.l[j].c - 1.0;
      if (static_cast<double>(static_cast<float>(r)) != r) ++bad;
    }
    for (int e = -126; e <= 127; ++e) {  // e L_hi + hi is exact, and 0 or at least as large as mnt * c - 1
      const double hi = static_cast<double>(e) * kL_hi + kTab.l[j].hi;
      if (static_cast<double>(static_cast<float>(hi)) != hi || (hi != 0.0 && std::fabs(hi) < 0.0077)) ++bad;
    }
  }
  // out of range: never decided
  float y;
  const float inf = INFINITY;
  for (float x : {-87.0f, 88.0f, -200.0f, 200.0f, inf, -inf, std::nanf("")}) bad += exp_fast(x, y) ? 1 : 0;
  for (float s : {0.0f, -0.0f, -1.0f, 1e-40f, inf, -inf, std::nanf("")}) bad += log_fast(s, y) ? 1 : 0;
  printf("%ld checked, %ld bad\n", n, bad);
  return bad ? 1 : 0;
}
