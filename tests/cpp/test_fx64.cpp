// Host check of the fixed-point arithmetic of the FP64 hopping term
// (grid_gb300/csrc/gb_fx64.cuh, compiled here by g++): the conversion of doubles, the limbs,
// and one output site (eight legs of SU(3) x two-spinor, summed) against long double and
// beside the same site in double.
#include "gb_fx64.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

using namespace gb;
typedef long double ld;

static int failures = 0;
static void expect(bool ok, const char* what, double got, double bound) {
  if (!ok && failures++ < 10) std::printf("FAIL %s: %.3e > %.3e\n", what, got, bound);
}
static void words(double d, uint32_t& hi, uint32_t& lo) {
  uint64_t u;
  std::memcpy(&u, &d, 8);
  hi = uint32_t(u >> 32);
  lo = uint32_t(u);
}
static int exponent(double d) {
  uint32_t hi, lo;
  words(d, hi, lo);
  return int((hi & 0x7fffffffu) >> 20);
}
static long long fixed(double d, int E) {
  uint32_t hi, lo;
  words(d, hi, lo);
  return fx::from_words(hi, lo, E);
}

int main() {
  std::mt19937_64 rng(20251205);
  std::normal_distribution<double> nd(0.0, 1.0);

  // conversion: truncation in units of 2^(E - 1023 - 59), |v| < 2^60; zeros give 0
  for (int i = 0; i < 1000000; i++) {
    const double d = nd(rng) * std::ldexp(1.0, int(rng() % 140) - 120);
    const int E = std::max(exponent(d), int(rng() % 40) + 1010);
    const long long v = fixed(d, E);
    const ld unit = std::ldexp((ld)1, E - 1023 - 59);
    expect(std::fabs((ld)v * unit - (ld)d) < unit, "conversion", double(std::fabs((ld)v * unit - (ld)d) / unit), 1);
    expect(v > -(1ll << 60) && v < (1ll << 60), "range", double(v), 1);
    int hi, lo;
    fx::split(v, hi, lo);
    expect(((long long)hi * 4294967296ll) + lo == v, "limbs", 0, 0);
  }
  expect(fixed(0.0, fx::kEmin) == 0 && fixed(-0.0, fx::kEmax) == 0 && fixed(5e-324, fx::kEmin) == 0, "zero", 0, 0);
  for (long long v : {0x80000000ll, -0x80000000ll, 0x17fffffffll, 0x180000000ll, -0x180000000ll, 0x7fffffffll}) {
    int hi, lo;
    fx::split_link(v, hi, lo);
    expect(lo != INT32_MIN, "link limb", lo, 0);
    expect(std::llabs(hi * 4294967296ll + lo - v) <= 1, "link value", 0, 1);
  }
  // the dot at its bounds: |u| a row at 1.5 2^k, every |h| just below 2^61, all signs alike
  {
    const long long umax = (long long)std::ldexp(1.5 / 6, 61), hmax = (1ll << 61) - 1;
    for (int sign = -1; sign <= 1; sign += 2) {
      long long hh = fx::kStartHh, mid = fx::kStartMid;
      for (int t = 0; t < 6; t++) {
        int uh, ul, xh, xl;
        fx::split_link(sign * umax, uh, ul);
        fx::split(hmax, xh, xl);
        hh = fx::mad(uh, xh, hh);
        mid = fx::mad(uh, xl, mid);
        mid = fx::mad(ul, xh, mid);
      }
      const ld want = (ld)6 * umax * hmax * sign / std::ldexp((ld)1, 64);
      expect(std::fabs((ld)fx::join(hh, mid) - want) <= 4, "dot at its bound", double(fx::join(hh, mid)), double(want));
    }
  }
  // one output component summed over eight legs, random SU(3)-like rows (|row|^2 = 1/4) and
  // Gaussian two-spinors whose sites differ by up to 2^6 in size
  ld e_fx = 0, e_d = 0, norm = 0;
  for (int site = 0; site < 200000; site++) {
    ld want = 0;
    double dsum = 0;
    double u[8][6], f[8][12];
    int E = 0, El[8];
    for (int leg = 0; leg < 8; leg++) {
      double n = 0;
      for (int t = 0; t < 6; t++) { u[leg][t] = nd(rng); n += u[leg][t] * u[leg][t]; }
      for (int t = 0; t < 6; t++) u[leg][t] *= 0.5 / std::sqrt(n);
      const double size = std::ldexp(1.0, int(rng() % 7));
      El[leg] = 0;
      for (int t = 0; t < 12; t++) { f[leg][t] = nd(rng) * size; El[leg] = std::max(El[leg], exponent(f[leg][t])); }
      E = std::max(E, El[leg]);
    }
    long long acc = 0;
    for (int leg = 0; leg < 8; leg++) {
      ld w = 0;
      double d = 0;
      long long hh = fx::kStartHh, mid = fx::kStartMid;
      for (int t = 0; t < 6; t++) {  // h = f_t + f_{t+6}
        const ld h = (ld)f[leg][t] + (ld)f[leg][t + 6];
        w += (ld)u[leg][t] * h;
        d = std::fma(u[leg][t], f[leg][t] + f[leg][t + 6], d);
        int uh, ul, xh, xl;
        fx::split_link(std::llrint(std::ldexp(u[leg][t], 61)), uh, ul);
        fx::split((fixed(f[leg][t], El[leg]) + fixed(f[leg][t + 6], El[leg])) >> (E - El[leg]), xh, xl);
        hh = fx::mad(uh, xh, hh);
        mid = fx::mad(uh, xl, mid);
        mid = fx::mad(ul, xh, mid);
      }
      want += w;
      dsum += d;
      acc += fx::join(hh, mid);
    }
    const double got = std::ldexp(double(acc), fx::result_exponent(E, 0));
    e_fx += ((ld)got - want) * ((ld)got - want);
    e_d += ((ld)dsum - want) * ((ld)dsum - want);
    norm += want * want;
  }
  const double r_fx = double(std::sqrt(e_fx / norm)), r_d = double(std::sqrt(e_d / norm));
  std::printf("relative L2 error of a site: fixed point %.2e, double %.2e\n", r_fx, r_d);
  // the last rounding to a double alone is 2^-53 / sqrt(3) at most
  expect(r_fx < std::ldexp(1.0, -53), "site error", r_fx, std::ldexp(1.0, -53));
  expect(r_fx < r_d, "no larger than double", r_fx, r_d);
  std::printf(failures ? "FAILED %d\n" : "PASSED\n", failures);
  return failures ? 1 : 0;
}
