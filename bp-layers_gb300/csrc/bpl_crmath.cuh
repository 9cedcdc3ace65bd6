// Correctly rounded exp and log for the message normalisation, in FP32
// arithmetic.
//
// The reference normalises every message with exp and log evaluated in double
// precision and rounded to float (ops/lbp_stereo/src/lbp_min_sum_kernel.cu:167,
// :180-181).  GB300's FP64 rate is a small fraction of its FP32 rate, so
// evaluating one double exp per message label makes the kernel FP64-bound.
// Here exp(x) and log(s) are evaluated in float-float arithmetic (errors below
// 2^-39 relative and 2^-36 + 2^-43 |e| absolute, e the exponent of s) with
// table-driven argument reduction after
//   P. T. P. Tang, "Table-driven implementation of the exponential function
//   in IEEE floating-point arithmetic", ACM TOMS 15(2), 1989, and
//   P. T. P. Tang, "Table-driven implementation of the logarithm function in
//   IEEE floating-point arithmetic", ACM TOMS 16(4), 1990,
// then rounded to float.  When the float-float value lies so close to a
// rounding boundary that the rounding cannot be decided from it (about one
// evaluation in 10^4-10^5), the reference's own double-precision expression is
// evaluated instead (Ziv's strategy).  Either way the float result equals the
// reference's (float)exp((double)x) / (float)log((double)s).
//
// Both evaluations are short dependency chains: the reduced arguments are
// exact by construction (see kC1, LogEntry), the leading terms keep their
// rounding errors (fused multiply-adds against exact differences), and the
// rounding test adds the error bound to the correction with both signs
// (one rounding each) instead of measuring the distance to a half ulp.
// One exp and one log sit on the dependency chain of every scanline step
// (26 and 30 operations deep before, 14 and 12 now; table and log lookups in
// shared memory instead of indexed constant loads): with the sum tree's
// butterfly a forward pass at 376x1240x192 went from 2.85 to 2.48 ms, the
// semantic global pass at 2x512x1024, L = 19 from 2.95 to 2.06 ms.
//
// Tables (2^(j/64); log of the reciprocals' inverses) are computed at
// compile time from power series in double precision.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define BPL_HD __device__ __forceinline__
#else
#define BPL_HD inline
#include <cmath>
#include <cstring>
#endif

namespace bpl {
namespace crm {

// ---------------------------------------------------------------------------
// compile-time tables
constexpr double kLn2 = 0.69314718055994530941723212145818;

constexpr double cx_exp(double y) {
  // exp(y) for 0 <= y < 0.7 by its Taylor series (terms decrease fast)
  double term = 1.0, sum = 1.0;
  for (int k = 1; k < 30; ++k) {
    term = term * y / k;
    sum += term;
  }
  return sum;
}

constexpr double cx_log(double x) {
  // log(x) for x in [1, 2] as 2*atanh((x-1)/(x+1))
  const double z = (x - 1.0) / (x + 1.0);
  const double z2 = z * z;
  double p = z, sum = 0.0;
  for (int k = 0; k < 40; ++k) {
    sum += p / (2 * k + 1);
    p *= z2;
  }
  return 2.0 * sum;
}

// 2^(j/64) as a float pair
struct alignas(8) ExpEntry {
  float hi, lo;
};
// For a mantissa mnt in [1 + j/128, 1 + (j+1)/128): c close to 1/mnt with
// eight bits after the point (1 for j = 0, 1/2 for j = 127), so that
// mnt * c - 1 is exact in a float (below 2^-7 with its last bit at 2^-31),
// and log(1/c) as hi + lo, hi a multiple of 2^-16.
struct alignas(16) LogEntry {
  float c, hi, lo, pad;
};
constexpr int kExpEntries = 64, kLogEntries = 128;
struct Tables {
  ExpEntry e[kExpEntries];
  LogEntry l[kLogEntries];
};

constexpr Tables make_tables() {
  Tables t{};
  for (int j = 0; j < kExpEntries; ++j) {
    const double v = cx_exp(kLn2 * j / 64.0);
    t.e[j].hi = static_cast<float>(v);
    t.e[j].lo = static_cast<float>(v - static_cast<double>(t.e[j].hi));
  }
  for (int j = 0; j < kLogEntries; ++j) {
    const double mid = 1.0 + (j + 0.5) / 128.0;
    const int k = (j == 0) ? 256 : (j == kLogEntries - 1) ? 128 : static_cast<int>(256.0 / mid + 0.5);
    const double v = cx_log(256.0 / k);
    const double hi = static_cast<int>(v * 65536.0 + 0.5) / 65536.0;
    t.l[j].c = static_cast<float>(k / 256.0);
    t.l[j].hi = static_cast<float>(hi);
    t.l[j].lo = static_cast<float>(v - hi);
    t.l[j].pad = 0.0f;
  }
  return t;
}

// Kernels copy the table they need to shared memory (coalesced loads) and
// pass it to the evaluations.
#if defined(__CUDACC__)
static __device__ const Tables kTab = make_tables();
#else
constexpr Tables kTab = make_tables();
#endif

// ln2/64 = C1 + C2 + C3: C1 = 1420 * 2^-17, C2 = -7120 * 2^-31, so that
// x - N*C1 and then - N*C2 are exact (below); ln2 = L_hi + L_mid + L_lo with
// 16 significant bits in L_hi (a multiple of 2^-16) and L_mid.  Values from a
// 60-digit evaluation of ln 2.
constexpr float kC1 = 0.010833740234375f;
constexpr float kC2 = -3.3155083656311035e-06f;
constexpr float kC3 = -2.9760223436840126e-11f;
constexpr float kL_hi = 0.693145751953125f;
constexpr float kL_mid = 1.4286197256296873e-06f;
constexpr float kL_lo = -1.2905320041778356e-11f;

// ---------------------------------------------------------------------------
// exact float transforms (explicit rounding: no contraction)
#if defined(__CUDACC__)
BPL_HD float add_(float a, float b) { return __fadd_rn(a, b); }
BPL_HD float sub_(float a, float b) { return __fsub_rn(a, b); }
BPL_HD float mul_(float a, float b) { return __fmul_rn(a, b); }
BPL_HD float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
BPL_HD int f2i(float f) { return __float_as_int(f); }
BPL_HD float i2f(int i) { return __int_as_float(i); }
#else
inline float add_(float a, float b) { volatile float r = a + b; return r; }
inline float sub_(float a, float b) { volatile float r = a - b; return r; }
inline float mul_(float a, float b) { volatile float r = a * b; return r; }
inline float fma_(float a, float b, float c) { return std::fmaf(a, b, c); }
inline int f2i(float f) { int i; std::memcpy(&i, &f, 4); return i; }
inline float i2f(int i) { float f; std::memcpy(&f, &i, 4); return f; }
#endif

// exp(x) rounded to float; returns false (ambiguous or out of the fast range)
// when the caller must evaluate the reference expression instead.  About 30
// operations, 14 deep.
BPL_HD bool exp_fast(float x, float& out, const ExpEntry* tab = kTab.e) {
  // N = rint(x * 64/ln2) by the 1.5 * 2^23 shift (|x * 64/ln2| < 2^13: the
  // float spacing there is 1), N's integer in the low bits of the sum
  const float tN = fma_(x, 92.332482616893656f, 12582912.0f);
  const float N = sub_(tN, 12582912.0f);  // exact
  const int tb = f2i(tN);
  const ExpEntry T = tab[tb & 63];
  // rh = x - N (C1 + C2), exactly: N has 13 bits and C1 11, so the first
  // product and difference fit a float; both x (|x| >= 2^-8 when N != 0) and
  // N * C2 are multiples of 2^-31 and |rh| < 2^-7, so the second does too.
  // rl = -N * C3, below 2^-19.
  const float rh = fma_(-N, kC2, fma_(-N, kC1, x));
  const float rl = mul_(-N, kC3);
  // exp(rh) - 1 = a + ae + poly: a + ae = rh + rh^2/2 (rh - a is exact)
  const float hr = mul_(0.5f, rh);
  const float a = fma_(hr, rh, rh);
  const float ae = fma_(hr, rh, sub_(rh, a));
  const float cube = mul_(mul_(rh, rh), rh);
  const float pq = fma_(rh, 0.041666666666666667f, 0.16666666666666667f);
  // exp(rh) (exp(rl) - 1) = rl (1 + a + rl/2) up to 2^-55
  const float rle = fma_(rl, fma_(0.5f, rl, a), rl);
  const float tail = fma_(cube, pq, add_(ae, rle));
  // 2^(j/64) * (1 + a + tail)
  const float y = fma_(T.hi, a, T.hi);
  const float ye = fma_(T.hi, a, sub_(T.hi, y));  // T.hi - y is exact
  const float corr = add_(fma_(T.hi, tail, ye), fma_(T.lo, a, T.lo));
  // total error below 2^-39 (y in [1, 2)): the same rounding at both ends
  // decides it
  const float z = add_(y, add_(corr, 1.8189894035458565e-12f));
  const float zl = add_(y, sub_(corr, 1.8189894035458565e-12f));
  out = i2f(f2i(z) + static_cast<int>(static_cast<unsigned>(tb & ~63) << 17));
  return x > -87.0f && x < 88.0f && z == zl;
}

// log(s) rounded to float for a positive float s; false when the caller must
// evaluate the reference expression instead.
BPL_HD bool log_fast(float s, float& out, const LogEntry* tab = kTab.l) {
  const int bits = f2i(s);
  const LogEntry T = tab[(bits >> 16) & 127];
  const float mnt = i2f((bits & 0x007fffff) | 0x3f800000);
  const float ef = sub_(i2f(((bits >> 23) & 0xff) | 0x4b000000), 8388735.0f);  // the exponent (2^23 + 127)
  const float r = fma_(mnt, T.c, -1.0f);  // exact
  // log(s) = e ln2 + log(1/c) + log1p(r); hi exact (multiples of 2^-16)
  const float hi = fma_(ef, kL_hi, T.hi);
  const float lo = fma_(ef, kL_lo, fma_(ef, kL_mid, T.lo));
  // hi is 0 or at least as large as r, so the sum's error is exact
  const float y = add_(hi, r);
  const float ye = sub_(r, sub_(y, hi));
  const float q = fma_(r, fma_(r, fma_(r, 0.2f, -0.25f), 0.33333333333333333f), -0.5f);
  const float corr = add_(fma_(mul_(r, r), q, lo), ye);
  // error below 2^-36 + 2^-43 |e|
  const float err = fma_(ef < 0.0f ? -ef : ef, 1.1368683772161603e-13f, 1.4551915228366852e-11f);
  const float z = add_(y, add_(corr, err));
  const float zl = add_(y, sub_(corr, err));
  out = z;
  // positive, normal, finite
  return static_cast<unsigned>(bits - 0x00800000) < 0x7f000000u && z == zl;
}

}  // namespace crm
}  // namespace bpl
