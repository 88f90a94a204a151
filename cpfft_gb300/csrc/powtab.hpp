// powtab.hpp -- x^y for a fixed exponent from a table: the rate exponents of the slip laws
// (stress.cu) and the annihilation exponent of the density laws (mrr.cuh).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define POWTAB_HD __host__ __device__ __forceinline__
#else
#define POWTAB_HD inline
#endif

// Table of x^y for a fixed exponent 0 < y <= 8 (tpow; filled by pow_table): x = 2^k m, c the
// midpoint of m's interval of [1, 2).
struct PowTab {
  static constexpr int NM = 256, NE = 1024, EMID = 512;
  struct alignas(16) Pair {
    double v, d;  // a value rounded to double, and what it lacks, relative to it
  };
  Pair P[NM];      // rc^-y
  // 2^(y (k - EMID)); zero where x^y isn't normal on all of that binade, and at NE (other binades)
  Pair E[NE + 1];
  double rc[NM];  // 1 / c, rounded
  double c[6];    // binomial coefficients y, y (y - 1) / 2, .. of (1 + u)^y - 1
  double y;
};

namespace powtab {
inline PowTab::Pair pair(long double x) {
  const double v = (double)x;
  return {v, (double)((x - v) / v)};
}
}  // namespace powtab

// the table, in long double
inline bool pow_table(double y, PowTab& t) {
  if (!(y > 0.0 && y <= 8.0)) return false;
  t.y = y;
  long double b = 1.0L;
  for (int k = 1; k <= 6; k++) {
    b *= ((long double)y - (k - 1)) / k;
    t.c[k - 1] = (double)b;
  }
  for (int i = 0; i < PowTab::NM; i++) {
    t.rc[i] = (double)(1.0L / (1.0L + (i + 0.5L) / PowTab::NM));
    t.P[i] = powtab::pair(powl((long double)t.rc[i], -(long double)y));
  }
  t.E[PowTab::NE] = {0.0, 0.0};
  for (int k = 0; k < PowTab::NE; k++) {
    const int e = k - PowTab::EMID;
    const bool normal = y * e >= -1022.0 && y * (e + 1) <= 1023.0;
    t.E[k] = normal ? powtab::pair(exp2l((long double)y * e)) : PowTab::Pair{0.0, 0.0};
  }
  return true;
}

namespace powtab {
POWTAB_HD double load(const double* p) {
#ifdef __CUDA_ARCH__
  return __ldg(p);
#else
  return *p;
#endif
}
POWTAB_HD PowTab::Pair load(const PowTab::Pair* p) {
#ifdef __CUDA_ARCH__
  const double2 t = __ldg(reinterpret_cast<const double2*>(p));
  return {t.x, t.y};
#else
  return *p;
#endif
}
// a double's words (the device's own 32-bit forms: through 64-bit masks the stress kernels spill
// more, 0.7 % of a fast-form pass at 128^3)
POWTAB_HD int high(double x) {
#ifdef __CUDA_ARCH__
  return __double2hiint(x);
#else
  int64_t b;
  std::memcpy(&b, &x, 8);
  return (int)(b >> 32);
#endif
}
POWTAB_HD double with_high(double x, int hi) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(hi, __double2loint(x));
#else
  int64_t b;
  std::memcpy(&b, &x, 8);
  b = (int64_t)((uint64_t)(uint32_t)hi << 32) | (b & 0xffffffff);
  std::memcpy(&x, &b, 8);
  return x;
#endif
}
}  // namespace powtab

// x^y, x >= 0, with the exponent's table: x = 2^k m, the interval's 1/c from m's leading bits,
// u = m / c - 1, w = c^y 2^(y k) with its rounding error, (1 + u)^y by its binomial series
// (|u| <= 2^-9).  Twelve FP64 instructions where CUDA's pow takes about 95; error below 0.6 ulp
// where x^y is a normal number and 2^-512 <= x < 2^512.  Other x (zeros of E) take pow.  The FP64
// pipe bounds the callers: a 32^3 pass of 48 systems takes 3.85 ms, without the three
// instructions of the error terms 3.72 (up to 2.6 ulp; pow has up to 1.3).
POWTAB_HD double tpow(const PowTab* t, double x) {
  using namespace powtab;
  const int hi = high(x);
  const unsigned k = (unsigned)((hi >> 20) - 1023 + PowTab::EMID);
  const PowTab::Pair e = load(t->E + (k < PowTab::NE ? k : PowTab::NE));
  if (high(e.v) == 0) return x == 0.0 ? 0.0 : pow(x, t->y);
  const int i = (hi >> 12) & (PowTab::NM - 1);
  const PowTab::Pair p = load(t->P + i);
  const double m = with_high(x, (hi & 0xfffff) | 0x3ff00000);
  const double u = fma(m, load(t->rc + i), -1.0);
  const double w = p.v * e.v, dw = fma(p.v, e.v, -w);
  double q = load(t->c + 5);
#pragma unroll
  for (int j = 4; j >= 0; j--) q = fma(q, u, load(t->c + j));
  return w + fma(w, fma(q, u, p.d + e.d), dw);
}
