// gb_dhop_fx.cu -- the FP64 hopping term in 64-bit fixed-point arithmetic (gb_fx64.cuh).
//
// The same sum as gb_dhop.cu's dhop_kernel<double> (DhopEO / DhopOE and their daggers,
// WilsonKernelsImplementation.h:113-163) on the same FP64 fields.  What bounds that kernel is
// the FP64 pipe, 2 lanes per clock and SM for 860 operations per output site.  Here:
//   fx_convert_kernel     the input checkerboard as integers with one exponent per 5D site (and that of its smallest
//                         pair of spins): a
//                         pass over the field (22 us for 75 MB in, 77 MB out, at HBM rate).
//                         Converting inside the legs, eight times per site, took 1700 of 6200
//                         instructions per output site and was slower for every Moebius size
//   dhop_fx_kernel        projections, SU(3) products and sums over legs and spins in
//                         integer arithmetic, each result rounded to a double once; 1728 wide
//                         multiply-adds (32 lanes per clock and SM) of 4500 instructions per
//                         output site.  The multiply-add pipe is its bound (74 % busy); four
//                         CTAs of 128 threads at 128 registers beat three at 168
//   dhop_fx_split_kernel  the same with a site's directions over two or four warps
// DhopEO, dhop_kernel<double> -> these: 16^4 x 16 820 -> 185 us, 16^4 x 12 599 -> 144 us,
// 24^3 x 32 x 12 right-hand sides 3847 -> 931 us, Wilson 24^3 x 32 345 -> 116 us, 8^4 33 -> 8 us.
//
// A site whose values the fixed-point range does not hold (infinities, NaN, magnitudes outside
// 2^(fx::kEmin - 1023) .. 2^(fx::kEmax - 1022)) is marked, and the outputs next to it are
// computed by fx_site_fp64 in FP64; so are outputs whose terms are all small (fx_site_exponent).  With every
// output on that path, a field of one colour on unit links, DhopEO takes 847 us at 16^4 x 16.
//
// Links: fixed-point copies made at the gauge import, in one of two layouts.
//   slots in CTAs   [x_cb][leg][9] int4, staged per CTA in shared memory by TMA bulk copies, one
//                   1168-byte slot per site (the padding keeps a warp's sites on distinct
//                   banks): many slots share a site's links
//   sites in lanes  [leg][9][x_cb] int4, read coalesced by each thread, below 8 slots per site:
//                   staging 1152 bytes for each few threads would leave an SM one or two CTAs
#include <cmath>
#include <cstring>

#include "gb_dhop_site.cuh"
#include "gb_fx64.cuh"

namespace gb {
namespace {

struct FxParams {
  const void* in[2];    // [z]: the checkerboards of a full-lattice Dhop, one per blockIdx.z
  longlong2* fxin[2];   // their fixed-point copies, without padding slots: 12 planes of [x_cb][L5a]
  int* exps[2];
  void* out[2];
  const double2* z[2];  // out = c0 z + c1 Dhop when given, else the Dhop
  double c0, c1;
  const int4* links[2];
  const double* links_d[2];  // the FP64 links, for sites that leave the fixed-point range
  const int* nbr[2];
  int64_t n4h;
  size_t n5, nfx;  // 5D sites with and without padding slots
  int L5, L5a, L5c, k4;  // as DhopParams (gb_dhop.cu)
  int link_exp;          // k of gb_fx64.cuh
  int dag;
  int* err;
  longlong2* fxout[2];  // CG_FINISH_ALPHA: the fixed-point copy of out, as fxin and exps
  int* expout[2];
  double2* r[2];  // the CG forms of the split kernel: the residual, the CTAs' sums, what the last CTA does
  double* partial;
  CGFinish fin;
};

constexpr float kFxLinkRatio = 4.f;  // of the largest and smallest link row (see fx_import_links)
constexpr int kFxLinkStride = 73;  // int4 per staged site: 72 and one of padding
// Up to this many output sites in a launch the split kernel takes the slots-in-CTAs layout too.  Split against
// one thread per site, DhopEO: 16384 sites 11.8 / 15.5 us (8 slots), 24576 15.7 / 18.2 (12), 32768 18.1 / 18.9 (8) and 18.0 /
// 18.3 (16), 40960 25.1 / 25.2 (8) and 25.0 / 24.7 (20), 49152 25.9 / 25.1 (16), 65536 30.1 / 30.6 (8) and 29.9 / 30.1 (16),
// 73728 32.6 / 36.1 (12), 71680 32.2 / 29.6 (20), 124416 55.1 / 49.7 (12), 131072 58.5 / 52.0 (8), 262144 112 / 98.7 (8): within
// 4 % of one another from 32768 to 65536 but for single waves, and from there the shared staging of the links counts.
constexpr int64_t kFxSplitSites = 40000;
// Above this many CTAs of the split kernel (608 are resident with four warps each), two warps share a
// site's directions in place of four: half of the partial sums through shared memory, and no second
// wave that is nearly empty.  Four -> two warps: DhopEO 8^3 x 16 x 8 (1024 CTAs) 19.2 -> 18.4 us,
// Wilson 24^3 x 32 (6912) 125 -> 116 us, with 3 right-hand sides 319 -> 289 us, CG iteration on MpcDagMpc
// of 16^4 (1024) 133 -> 125 us; 8^4 x 12 (768) 16.1 and 16.1 us, 8^4 x 10 (640) 15.4 -> 15.8 us,
// Wilson 12^4 (324) 10.8 -> 13.2 us.
constexpr size_t kFxTwoWarps = 800;

// f of the leg's two-spinor h = (1 + S gamma_MU) f as integers
template <int MU, int S>
__device__ __forceinline__ void fx_project(const longlong2 (&f)[12], long long (&hr)[6], long long (&hi)[6]) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const longlong2 f0 = f[c], f1 = f[3 + c], f2 = f[6 + c], f3 = f[9 + c];
    if (MU == 0) {
      hr[c] = f0.x - S * f3.y; hi[c] = f0.y + S * f3.x;
      hr[3 + c] = f1.x - S * f2.y; hi[3 + c] = f1.y + S * f2.x;
    } else if (MU == 1) {
      hr[c] = f0.x - S * f3.x; hi[c] = f0.y - S * f3.y;
      hr[3 + c] = f1.x + S * f2.x; hi[3 + c] = f1.y + S * f2.y;
    } else if (MU == 2) {
      hr[c] = f0.x - S * f2.y; hi[c] = f0.y + S * f2.x;
      hr[3 + c] = f1.x + S * f3.y; hi[3 + c] = f1.y - S * f3.x;
    } else {
      hr[c] = f0.x + S * f2.x; hi[c] = f0.y + S * f2.y;
      hr[3 + c] = f1.x + S * f3.x; hi[3 + c] = f1.y + S * f3.y;
    }
  }
}

struct FxAcc {
  long long re[12], im[12];
};

// acc += u on spins 0, 1 and, on spins 2, 3, the phases of accumRecon{X,Y,Z,T}p times u
template <int MU>
__device__ __forceinline__ void fx_reconstruct(FxAcc& acc, const long long (&ur)[6], const long long (&ui)[6]) {
#pragma unroll
  for (int a = 0; a < 3; a++) {
    acc.re[a] += ur[a]; acc.im[a] += ui[a];
    acc.re[3 + a] += ur[3 + a]; acc.im[3 + a] += ui[3 + a];
    if (MU == 0) {
      acc.re[6 + a] += ui[3 + a]; acc.im[6 + a] -= ur[3 + a];
      acc.re[9 + a] += ui[a]; acc.im[9 + a] -= ur[a];
    } else if (MU == 1) {
      acc.re[6 + a] += ur[3 + a]; acc.im[6 + a] += ui[3 + a];
      acc.re[9 + a] -= ur[a]; acc.im[9 + a] -= ui[a];
    } else if (MU == 2) {
      acc.re[6 + a] += ui[a]; acc.im[6 + a] -= ur[a];
      acc.re[9 + a] -= ui[3 + a]; acc.im[9 + a] += ur[3 + a];
    } else {
      acc.re[6 + a] += ur[a]; acc.im[6 + a] += ui[a];
      acc.re[9 + a] += ur[3 + a]; acc.im[9 + a] += ui[3 + a];
    }
  }
}

// One leg; pl selects the direction and the sign S of its projector (2 mu + (S > 0)), the same
// for the whole grid, so its switches do not diverge.  The leg is a loop body: unrolled over
// the eight legs the code would not fit the instruction cache.
__device__ __forceinline__ void fx_leg(int pl, const longlong2* __restrict__ in, size_t n5, size_t i, int sh,
                                       const int4* U, size_t ustride, FxAcc& acc) {
  int hrh[6], hrl[6], hih[6], hil[6];
  {
    longlong2 f[12];
#pragma unroll
    for (int k = 0; k < 12; k++) f[k] = __ldg(in + size_t(k) * n5 + i);
    long long hr[6], hi[6];
    switch (pl) {
      case 0: fx_project<0, -1>(f, hr, hi); break;
      case 1: fx_project<0, 1>(f, hr, hi); break;
      case 2: fx_project<1, -1>(f, hr, hi); break;
      case 3: fx_project<1, 1>(f, hr, hi); break;
      case 4: fx_project<2, -1>(f, hr, hi); break;
      case 5: fx_project<2, 1>(f, hr, hi); break;
      case 6: fx_project<3, -1>(f, hr, hi); break;
      default: fx_project<3, 1>(f, hr, hi); break;
    }
#pragma unroll
    for (int k = 0; k < 6; k++) {
      fx::split(hr[k] >> sh, hrh[k], hrl[k]);
      fx::split(hi[k] >> sh, hih[k], hil[k]);
      fx::opaque(hrh[k]); fx::opaque(hrl[k]); fx::opaque(hih[k]); fx::opaque(hil[k]);
    }
  }
  long long ur[6], ui[6];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    long long rh[2], rm[2], ih[2], im[2];
#pragma unroll
    for (int b = 0; b < 3; b++) {
      const int4 w = U[size_t(a * 3 + b) * ustride];
      int nh = -w.z, nl = -w.w;
      fx::opaque(nh); fx::opaque(nl);
#pragma unroll
      for (int sp = 0; sp < 2; sp++) {
        const int k = sp * 3 + b;
        rh[sp] = fx::mad(w.x, hrh[k], b == 0 ? fx::kStartHh : rh[sp]);
        rm[sp] = fx::mad(w.x, hrl[k], b == 0 ? fx::kStartMid : rm[sp]);
        rm[sp] = fx::mad(w.y, hrh[k], rm[sp]);
        rh[sp] = fx::mad(nh, hih[k], rh[sp]);
        rm[sp] = fx::mad(nh, hil[k], rm[sp]);
        rm[sp] = fx::mad(nl, hih[k], rm[sp]);
        ih[sp] = fx::mad(w.x, hih[k], b == 0 ? fx::kStartHh : ih[sp]);
        im[sp] = fx::mad(w.x, hil[k], b == 0 ? fx::kStartMid : im[sp]);
        im[sp] = fx::mad(w.y, hih[k], im[sp]);
        ih[sp] = fx::mad(w.z, hrh[k], ih[sp]);
        im[sp] = fx::mad(w.z, hrl[k], im[sp]);
        im[sp] = fx::mad(w.w, hrh[k], im[sp]);
      }
    }
#pragma unroll
    for (int sp = 0; sp < 2; sp++) {
      ur[sp * 3 + a] = fx::join(rh[sp], rm[sp]);
      ui[sp * 3 + a] = fx::join(ih[sp], im[sp]);
    }
  }
  switch (pl >> 1) {
    case 0: fx_reconstruct<0>(acc, ur, ui); break;
    case 1: fx_reconstruct<1>(acc, ur, ui); break;
    case 2: fx_reconstruct<2>(acc, ur, ui); break;
    default: fx_reconstruct<3>(acc, ur, ui); break;
  }
}

// The FP64 sum of one site, for fx_site_fp64.
template <bool DAG, int LEG>
__device__ __forceinline__ void fp64_leg(const double2* in, const double* links, const int* nbr, size_t n5, int L5,
                                         int64_t x, int s, Spinor<double>& acc) {
  constexpr int MU = LEG & 3;
  constexpr int S = (LEG < 4 ? -1 : 1) * (DAG ? -1 : 1);
  Spinor<double> f;
  SpinorIO<double>::load(in, nullptr, n5, size_t(nbr[x * 8 + LEG]) * L5 + s, f);
  double hr[6], hi[6], ur[6], ui[6];
  project<MU, S>(f, hr, hi);
  su3_mul<double>(links + (size_t(x) * 8 + LEG) * 18, hr, hi, ur, ui);
  reconstruct<MU, S, LEG == 0>(acc, ur, ui);
}
template <bool DAG>
__device__ __forceinline__ void fp64_legs(const double2* in, const double* links, const int* nbr, size_t n5, int L5,
                                          int64_t x, int s, Spinor<double>& acc) {
  fp64_leg<DAG, 0>(in, links, nbr, n5, L5, x, s, acc);
  fp64_leg<DAG, 1>(in, links, nbr, n5, L5, x, s, acc);
  fp64_leg<DAG, 2>(in, links, nbr, n5, L5, x, s, acc);
  fp64_leg<DAG, 3>(in, links, nbr, n5, L5, x, s, acc);
  fp64_leg<DAG, 4>(in, links, nbr, n5, L5, x, s, acc);
  fp64_leg<DAG, 5>(in, links, nbr, n5, L5, x, s, acc);
  fp64_leg<DAG, 6>(in, links, nbr, n5, L5, x, s, acc);
  fp64_leg<DAG, 7>(in, links, nbr, n5, L5, x, s, acc);
}
// one output component: the Dhop's value, or (AXPY) c0 z + c1 of it
template <bool AXPY>
__device__ __forceinline__ double2 fx_result(const FxParams& p, const double2* z, size_t w, double re, double im) {
  if (AXPY) {
    const double2 v = __ldg(z + w);
    re = fma(p.c1, re, p.c0 * v.x);
    im = fma(p.c1, im, p.c0 * v.y);
  }
  return make_double2(re, im);
}

// the integer (units of 2^e) as a double, rounded once; 0 stays 0
__device__ __forceinline__ double fx_value(long long v, int e) {
  const double d = __ll2double_rn(v);
  return v == 0 ? 0.0 : __hiloint2double(__double2hiint(d) + (e << 20), __double2loint(d));
}

__device__ __noinline__ void fx_site_fp64(const double2* in, double2* out, const double2* z, double c0, double c1,
                                          const double* links, const int* nbr, size_t n5, int L5, int64_t x, int s,
                                          int dag) {
  Spinor<double> acc;
  if (dag) fp64_legs<true>(in, links, nbr, n5, L5, x, s, acc);
  else fp64_legs<false>(in, links, nbr, n5, L5, x, s, acc);
  const size_t i = size_t(x) * L5 + s;
#pragma unroll
  for (int k = 0; k < 12; k++) {
    double2 v = make_double2(acc.re[k], acc.im[k]);
    if (z) {
      const double2 w = z[size_t(k) * n5 + i];
      v = make_double2(fma(c1, v.x, c0 * w.x), fma(c1, v.y, c0 * w.y));
    }
    out[size_t(k) * n5 + i] = v;
  }
}

// The largest exponent of a site's eight neighbours, and kBad (above every other) where one is marked or where
// the output cannot be left to their common unit.  The error is a fixed part of that unit, while FP64's is one of
// the terms of each output component.  A component takes from each neighbour one pair of spins in every
// colour, and a link's row has no smaller sum than another's by more than kFxLinkRatio: its terms add up to the
// unit's size if the neighbours' smallest pairs do, to 2^-kFxSpread of it.  At that bound the error is 1.6
// times FP64's rounding (integer model on the host: 2.3e-16 against 1.4e-16 of the sum of the terms'
// magnitudes with all of it in one neighbour; eight of 2^-3 each 3e-17 against 4.5e-17; unitary links, with
// rows at kFxLinkRatio up to 2.7 times that).  Colours that the links keep
// apart and that differ in size by more than 2^4 are below it; ordinary fields are not: of a Gaussian
// field one pair of one neighbour is enough everywhere, of the smallest pole's solution on 8^3 x 16 x 8 in all but 3e-5 of the
// sites, and the sum there.  (Without the sum those few sites, 10 us each for the thread that takes them in FP64,
// made that multishift solve 52 -> 67 ms.)
constexpr int kFxSpread = 3;
__device__ __forceinline__ int fx_site_exponent(const int* exps, const int* nbr, int L5a, int64_t x, int s) {
  const int4* nb = reinterpret_cast<const int4*>(nbr + x * 8);
  const int4 a = __ldg(nb), b = __ldg(nb + 1);
  const unsigned* e = reinterpret_cast<const unsigned*>(exps) + s;
  const unsigned e0 = __vmaxu2(__ldg(e + size_t(a.x) * L5a), __ldg(e + size_t(a.y) * L5a));
  const unsigned e1 = __vmaxu2(__ldg(e + size_t(a.z) * L5a), __ldg(e + size_t(a.w) * L5a));
  const unsigned e2 = __vmaxu2(__ldg(e + size_t(b.x) * L5a), __ldg(e + size_t(b.y) * L5a));
  const unsigned e3 = __vmaxu2(__ldg(e + size_t(b.z) * L5a), __ldg(e + size_t(b.w) * L5a));
  const unsigned m = __vmaxu2(__vmaxu2(e0, e1), __vmaxu2(e2, e3));
  const int E = int(m >> 16);
  if (E - int(m & 0xffffu) <= kFxSpread || E == fx::kBad) return E;
  unsigned sum = 0;
  for (int k = 0; k < 8; k++) sum += 256u >> min(E - int(__ldg(e + size_t(__ldg(nbr + x * 8 + k)) * L5a) & 0xffffu), 31);
  return sum >= 256u >> kFxSpread ? E : fx::kBad;
}

__device__ __forceinline__ void fx_negate_lower(FxAcc& acc) {
#pragma unroll
  for (int k = 6; k < 12; k++) { acc.re[k] = -acc.re[k]; acc.im[k] = -acc.im[k]; }
}

// The legs [leg0, leg0 + n) and [leg0 + 4, leg0 + 4 + n) of one site, in units of Ea.  Spins 2,
// 3 are summed without the legs' sign S and negated after the forward legs.
__device__ __forceinline__ void fx_legs(const FxParams& p, const longlong2* in, const int* exps, const int* nbr,
                                        const int4* U, size_t ustride, int64_t x, int s, int leg0, int n, int Ea,
                                        FxAcc& acc) {
#pragma unroll
  for (int k = 0; k < 12; k++) { acc.re[k] = 0; acc.im[k] = 0; }
#pragma unroll 1
  for (int m = 0; m < 2 * n; m++) {
    if (m == n) fx_negate_lower(acc);
    const int leg = m < n ? leg0 + m : leg0 + 4 + m - n;
    const size_t j = size_t(__ldg(nbr + x * 8 + leg)) * p.L5a + s;
    fx_leg(2 * (leg & 3) + ((leg >= 4) != (p.dag != 0) ? 1 : 0), in, p.nfx, j, min(Ea - (__ldg(exps + j) >> 16), 63),
           U + size_t(leg) * 9 * ustride, ustride, acc);
  }
  if (p.dag) fx_negate_lower(acc);
}

// zeros into the padding slots of an odd right-hand-side count
__device__ __forceinline__ void fx_pad(const FxParams& p, double2* out, int64_t x, int s) {
  if (s != 0 || p.L5a == p.L5) return;
  Spinor<double> zero;
#pragma unroll
  for (int k = 0; k < 12; k++) { zero.re[k] = 0.0; zero.im[k] = 0.0; }
  for (int z = p.L5a; z < p.L5; z++) SpinorIO<double>::store(out, nullptr, p.n5, size_t(x) * p.L5 + z, zero);
}

// The upper word of the larger of a component's |re|, |im|; its lowest bit stands for the lower words.
__device__ __forceinline__ uint32_t fx_size(double2 v) {
  const uint32_t hi = max(uint32_t(__double2hiint(v.x)) & 0x7fffffffu, uint32_t(__double2hiint(v.y)) & 0x7fffffffu);
  return hi | uint32_t((__double2loint(v.x) | __double2loint(v.y)) != 0);
}

// What the exponents of a site's fixed-point copy are taken from: the sizes of its 12 components.
struct FxRange {
  uint32_t top, least;  // the largest, and the smallest over the colours and the pairs of spins that a projection adds
  // size(k): of component k = 3 spin + colour.  The pairs are those of a spin 0, 1 with a spin 2, 3.
  template <class F> __device__ __forceinline__ explicit FxRange(const F& size) : top(0), least(0xffffffffu) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const uint32_t a = size(c), b = size(3 + c), d = size(6 + c), e = size(9 + c);
      top = max(top, max(max(a, b), max(d, e)));
      least = min(least, max(min(a, b), min(d, e)));  // = the smallest of max(a, d), max(a, e), max(b, d), max(b, e)
    }
  }
  __device__ __forceinline__ bool ok() const { return int(top >> 20) >= fx::kEmin && int(top >> 20) <= fx::kEmax; }
  __device__ __forceinline__ int exponent() const { return top == 0 ? 0 : ok() ? int(top >> 20) : fx::kBad; }
  // the exponents as one word: that of the site above, that of its smallest pair below
  __device__ __forceinline__ int word() const { return exponent() << 16 | int(least >> 20); }
  // of the integers: values of zero and marked sites become zeros, or are not read
  __device__ __forceinline__ int scale() const { return ok() ? int(top >> 20) : fx::kEmax; }
};

// A site as a factor of the force: its exponent, and for each of the four pairs of spins that a projection
// adds how far (in powers of two, up to 31) the smallest colour of the pair lies below it.
__device__ __forceinline__ uint32_t fx_force_word(const Spinor<double>& f, int E) {
  int e[12];
#pragma unroll
  for (int k = 0; k < 12; k++)
    e[k] = int(max(uint32_t(__double2hiint(f.re[k])) & 0x7fffffffu, uint32_t(__double2hiint(f.im[k])) & 0x7fffffffu) >> 20);
  const auto below = [&](int i, int j) {
    const int least = min(max(e[3 * i], e[3 * j]), min(max(e[3 * i + 1], e[3 * j + 1]), max(e[3 * i + 2], e[3 * j + 2])));
    return uint32_t(min(E - least, 31));
  };
  return uint32_t(E) << 20 | below(0, 3) << 15 | below(1, 2) << 10 | below(0, 2) << 5 | below(1, 3);
}

__device__ __forceinline__ longlong2 fx_words(double2 v, int E) {
  longlong2 w;
  w.x = fx::from_words(uint32_t(__double2hiint(v.x)), uint32_t(__double2loint(v.x)), E);
  w.y = fx::from_words(uint32_t(__double2hiint(v.y)), uint32_t(__double2loint(v.y)), E);
  return w;
}

// The fixed-point copy of one checkerboard of a field (both with blockIdx.z), one thread per 5D
// site.  A pass of its own: each site is read by eight outputs, and converting it eight times
// there took more instructions than the SU(3) products.  The copies have no padding slots: with
// one right-hand side those are half of the field (DhopEO 24^3 x 32 137 -> 125 us, 16^4 22.9 -> 20.1 us,
// CG iteration on MdagM of 24^3 x 32 894 -> 840 us).
// FORCE: the exponents carry what deriv_fx_kernel asks of its factors (fx_force_word).
template <bool FORCE>
__global__ void __launch_bounds__(256) fx_convert_kernel(const __grid_constant__ FxParams p) {
  pdl_wait();
  const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= p.nfx) return;
  const double2* in = after_wait(static_cast<const double2*>(p.in[blockIdx.z]));
  longlong2* out = p.fxin[blockIdx.z];
  size_t j = i;
  if (p.L5a != p.L5) j += i / unsigned(p.L5a) * unsigned(p.L5 - p.L5a);
  Spinor<double> f;
  SpinorIO<double>::load(in, nullptr, p.n5, j, f);
  const FxRange m([&](int k) { return fx_size(make_double2(f.re[k], f.im[k])); });
  const int E = m.scale();
  p.exps[blockIdx.z][i] = FORCE ? int(fx_force_word(f, m.exponent())) : m.word();
#pragma unroll
  for (int k = 0; k < 12; k++) out[size_t(k) * p.nfx + i] = fx_words(make_double2(f.re[k], f.im[k]), E);
}

template <bool AXPY>
__global__ void __launch_bounds__(128, 4) dhop_fx_kernel(const __grid_constant__ FxParams p) {
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  int4* slink = reinterpret_cast<int4*>(dyn_smem);  // k4 * kFxLinkStride
  __shared__ __align__(8) uint64_t bar;
  const int side = blockIdx.z;
  double2* out = static_cast<double2*>(p.out[side]);
  const int* nbr = p.nbr[side];
  const int t = threadIdx.x;
  const int64_t x0 = int64_t(blockIdx.x) * p.k4;
  const int nsite = int(min(int64_t(p.k4), p.n4h - x0));
  const int j = t / p.L5c;
  const int s = int(blockIdx.y) * p.L5c + (t - j * p.L5c);
  if (t == 0) mbar_init(&bar, 1);
  __syncthreads();
  if (t == 0) {
    mbar_expect_tx(&bar, uint32_t(nsite) * 1152u);
    for (int k = 0; k < nsite; k++) bulk_g2s(slink + k * kFxLinkStride, p.links[side] + (x0 + k) * 72, 1152u, &bar);
  }
  pdl_wait();  // the field; links and neighbour tables were there before
  const double2* in = after_wait(static_cast<const double2*>(p.in[side]));
  const double2* z = after_wait(p.z[side]);
  const longlong2* fxin = after_wait(p.fxin[side]);
  const int* exps = after_wait(p.exps[side]);
  if (!mbar_wait_bounded(&bar, 0)) {  // every thread waits; the error flag as in gb_dhop.cu
    atomicExch(p.err, 1);
    return;
  }
  if (j >= nsite || s >= p.L5a) return;
  const int64_t x = x0 + j;
  fx_pad(p, out, x, s);
  const int Ea = fx_site_exponent(exps, nbr, p.L5a, x, s);
  if (Ea == fx::kBad) {
    fx_site_fp64(in, out, z, p.c0, p.c1, p.links_d[side], nbr, p.n5, p.L5, x, s, p.dag);
    return;
  }
  FxAcc acc;
  fx_legs(p, fxin, exps, nbr, slink + j * kFxLinkStride, 1, x, s, 0, 4, Ea, acc);
  const int e = fx::result_exponent(Ea, p.link_exp);
  const size_t i = size_t(x) * p.L5 + s;
#pragma unroll
  for (int k = 0; k < 12; k++) {
    const size_t w = size_t(k) * p.n5 + i;
    out[w] = fx_result<AXPY>(p, z, w, fx_value(acc.re[k], e), fx_value(acc.im[k], e));
  }
}

// |v|^2 into sum; UPDATE: of r - a v, which replaces r
template <bool UPDATE>
__device__ __forceinline__ void fx_cg_term(double2* r, double a, double2 v, double& sum) {
  if (UPDATE) {
    const double2 o = *r;
    v = make_double2(fma(-a, v.x, o.x), fma(-a, v.y, o.y));
    *r = v;
  }
  sum = fma(v.x, v.x, fma(v.y, v.y, sum));
}

// The end of a CG form for one right-hand side, by every thread of every CTA of W warps: the CTA's sum, and in
// the last CTA all of them in a fixed order and the CG's scalars from it.  The padding's scalars stay as
// cg_init_kernel set them (done, a = b = 0).
template <int W>
__device__ __forceinline__ void fx_cg_finish(const FxParams& p, double sum) {
  __shared__ double ws[W];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const auto cta_sum = [&](double v) {  // in thread 0
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) ws[warp] = v;
    __syncthreads();
    return W == 4 ? (ws[0] + ws[1]) + (ws[W - 2] + ws[W - 1]) : ws[0] + ws[1];
  };
  const int ctas = int(gridDim.x * gridDim.z);
  sum = cta_sum(sum);
  if (threadIdx.x == 0) p.partial[blockIdx.z * gridDim.x + blockIdx.x] = sum;
  if (!last_cta(p.fin.flags + kCGTicket, ctas)) return;
  sum = 0.0;
#pragma unroll 8
  for (int b = threadIdx.x; b < ctas; b += 32 * W) sum += __ldcg(p.partial + b);
  sum = cta_sum(sum);
  if (threadIdx.x != 0) return;
  CGScalars c = *p.fin.cg;
  if (p.fin.mode == CG_FINISH_ALPHA) cg_alpha_update(c, sum);
  else cg_beta_update(c, sum);
  *p.fin.cg = c;
  if (p.fin.mode != CG_FINISH_BETA) return;
  __threadfence();
  cg_set_flags(p.fin.cg, p.L5, p.fin.flags);
}

// W = 4 warps share 32 output sites, one direction (its forward and backward leg) each, or W = 2 with
// two directions each (kFxTwoWarps), and add their integer sums through shared memory: exactly, so the result does not depend on which
// kernel ran.  A site is a chain of about 4600 instructions for one thread: with few sites that
// chain is the launch's time (8^4: 12.4 us, one thread per site 20.0), and with sites in lanes
// the extra warps keep more of the links' 1152 bytes per site in flight (24^3 x 32: 138 us, one
// thread per site 153; measured with plain launches and padding in the fixed-point copies).
// SOA: the links' sites-in-lanes layout.
// CG (one right-hand side): the CG's next reduction rides on the launch.  CG_FINISH_ALPHA stores
// out, also as the fixed-point copy that the dagger's launch reads, and sums |out|^2;
// CG_FINISH_BETA applies r -= a out in place of storing out and sums |r|^2,
// and the last CTA turns the sum into the CG's a or b.  us per CG iteration on MdagM, separate passes ->
// sums here: 8^4 42.4 -> 33.7, 24^3 x 32 932 -> 894, 32^4 2137 -> 2109 (with padding in the copies);
// then with the copy left for the dagger: 8^4 33.7 -> 30.9, 24^3 x 32 840 -> 812, 32^4 1957 -> 1899; with
// two warps 24^3 x 32 753, 32^4 1753.
// With more right-hand sides the passes stay.
template <bool SOA, bool AXPY, int W, int CG = CG_FINISH_NONE>
__global__ void __launch_bounds__(32 * W, 16 / W) dhop_fx_split_kernel(const __grid_constant__ FxParams p) {
  constexpr bool LEAVE = CG == CG_FINISH_ALPHA;
  static_assert(W == 4 || W == 2, "a site's four directions over four or two warps");
  constexpr int K = 12 / W;  // components that a warp finishes
  __shared__ long long part[W][24][32];
  const int side = blockIdx.z;
  const int lane = threadIdx.x & 31, mu = threadIdx.x >> 5;
  double2* out = static_cast<double2*>(p.out[side]);
  const int* nbr = p.nbr[side];
  const int64_t g = int64_t(blockIdx.x) * 32 + lane;
  const bool active = g < p.n4h * p.L5a;
  const int64_t x = active ? g / p.L5a : 0;
  const int s = active ? int(g - x * p.L5a) : 0;
  pdl_wait();
  const double2* in = after_wait(static_cast<const double2*>(p.in[side]));
  const double2* z = after_wait(p.z[side]);
  const longlong2* fxin = after_wait(p.fxin[side]);
  const int* exps = after_wait(p.exps[side]);
  const int Ea = fx_site_exponent(exps, nbr, p.L5a, x, s);
  if (Ea != fx::kBad) {
    FxAcc acc;
    fx_legs(p, fxin, exps, nbr, SOA ? p.links[side] + x : p.links[side] + x * 72, SOA ? size_t(p.n4h) : size_t(1),
            x, s, mu * (4 / W), 4 / W, Ea, acc);
#pragma unroll
    for (int k = 0; k < 12; k++) { part[mu][2 * k][lane] = acc.re[k]; part[mu][2 * k + 1][lane] = acc.im[k]; }
  }
  __syncthreads();
  const size_t i = size_t(x) * p.L5 + s;
  double2* const r = CG == CG_FINISH_BETA ? p.r[side] + i : nullptr;
  const double a = CG == CG_FINISH_BETA ? __ldcg(&p.fin.cg->a) : 0.0;
  double sum = 0.0;
  if (active && mu == 0) {
    fx_pad(p, out, x, s);
    if (Ea == fx::kBad) {
      fx_site_fp64(in, out, z, p.c0, p.c1, p.links_d[side], nbr, p.n5, p.L5, x, s, p.dag);
      if (CG != CG_FINISH_NONE)
        for (int k = 0; k < 12; k++) fx_cg_term<CG == CG_FINISH_BETA>(r + size_t(k) * p.n5, a, out[size_t(k) * p.n5 + i], sum);
      if (LEAVE) {
        const FxRange m([&](int k) { return fx_size(out[size_t(k) * p.n5 + i]); });
        p.expout[side][g] = m.word();
        for (int k = 0; k < 12; k++) p.fxout[side][size_t(k) * p.nfx + g] = fx_words(out[size_t(k) * p.n5 + i], m.scale());
      }
    }
  }
  double2 kept[K] = {};
  if (active && Ea != fx::kBad) {
    const int e = fx::result_exponent(Ea, p.link_exp);
#pragma unroll
    for (int m = 0; m < K; m++) {  // warp mu finishes components K mu .. K mu + K - 1
      const int k = K * mu + m;
      long long v[2];
#pragma unroll
      for (int c = 0; c < 2; c++) {
        v[c] = part[0][2 * k + c][lane] + part[1][2 * k + c][lane];
        if (W == 4) v[c] += part[W - 2][2 * k + c][lane] + part[W - 1][2 * k + c][lane];
      }
      const size_t w = size_t(k) * p.n5 + i;
      const double2 d = fx_result<AXPY>(p, z, w, fx_value(v[0], e), fx_value(v[1], e));
      if (CG != CG_FINISH_BETA) out[w] = d;
      if (CG != CG_FINISH_NONE) fx_cg_term<CG == CG_FINISH_BETA>(r + size_t(k) * p.n5, a, d, sum);
      kept[m] = d;
    }
  }
  if (LEAVE) {  // the site's range is that of its warps' components
    __shared__ uint32_t size[12][32];
#pragma unroll
    for (int m = 0; m < K; m++) size[K * mu + m][lane] = fx_size(kept[m]);
    __syncthreads();
    if (active && Ea != fx::kBad) {
      const FxRange m([&](int k) { return size[k][lane]; });
      if (mu == 0) p.expout[side][g] = m.word();
#pragma unroll
      for (int k = 0; k < K; k++) p.fxout[side][size_t(K * mu + k) * p.nfx + g] = fx_words(kept[k], m.scale());
    }
  }
  if (CG != CG_FINISH_NONE) fx_cg_finish<W>(p, sum);
}

// ---- force term (gb_dhop.cu's deriv_kernel: mat = U W, W = sum_s h conj(g)^T) in fixed point ----
//
// What bounds the FP64 kernel is its 96 FP64 operations per (site, direction, s).  Here A (on the
// output's checkerboard) and B come as the fixed-point copies of fx_convert_kernel, and the sum over
// s of the two-spinors' products is exact integer arithmetic: the two-spinors are cut to b bits, b = 59
// for one slot, 58 for up to 4, 57 for up to 16 and one less for each doubling, in limbs of 29 and b - 29 bits, so
// that the sums over a lane's slots (8 products of 2^(b - 1) each in the middle, 4 of 2^(2 b - 58) on top) and over
// the two lanes stay below 2^63; products of two lower limbs, below 2^-57 of the largest, are dropped.  The sum's unit is that of its largest product, taken over s as the
// largest sum of the two exponents: B stays in the units of its own slot and A is shifted for both, so that factors
// which peak at different s (the two walls of the fifth dimension) keep their bits.  Above 64 slots b
// would fall below a double's 53 bits and more.
//
// The error is a fixed part of that unit, 2^(58 - 2 b) of it and a few 2^-59, where FP64's is one of each sum's own
// terms.  So each lane also adds up a lower bound of every colour pair's sum of |h_c| |g_b| (per slot and j, the
// smallest colour of either two-spinor's pair of spins), and where that is below 2^(2 (58 - b) - 4) of the unit, as for colours
// that the links keep apart and that differ in size, the site is summed in FP64.  At that bound the error is
// at most 4 times FP64's rounding (integer model on the host: 3.3e-16 against 8.3e-17 of the sum of the terms'
// magnitudes; with terms of one size 1e-17 to 4e-17 against 5e-17 to 7e-17).  Gaussian factors stay above it by 4 to 24:
// none of 2e5 sites falls below with up to 32 slots, 0.6 % with 33.
// U W runs in FP64.  Same lanes, warps and CTAs as deriv_kernel.  MDeriv 16^4 x 12:
// 708 -> 421 us, of which Meooe5D is 80 and the conversions 94 (two or four CTAs per SM: 466, 463; the lower
// bound of the terms 9).
constexpr int kDerivSlots = 64;

struct FxDerivParams {
  const double2* in[2];         // A, B
  const longlong2* fxin[2];
  const int* exps[2];
  const double* links;
  const int* nbr;
  double2* mat;
  size_t n5, nfx;
  int64_t n4h;
  int L5, L5a, bits;
  int half_out, dag, parity;
  int L[4];
};

// limbs of base 2^29
__device__ __forceinline__ void split29(long long v, int& hi, int& lo) {
  lo = int(uint32_t(uint64_t(v)) << 3) >> 3;
  hi = int((v - lo) >> 29);
  fx::opaque(hi);
  fx::opaque(lo);
}

template <int MU>
__device__ __forceinline__ void deriv_project(const longlong2 (&f)[12], bool plus, long long (&hr)[6], long long (&hi)[6]) {
  if (plus) fx_project<MU, 1>(f, hr, hi);
  else fx_project<MU, -1>(f, hr, hi);
}

// the limbs of the two-spinor of one site, in the site's units shifted down by sh
__device__ __forceinline__ void deriv_limbs(int mu, bool plus, const longlong2* __restrict__ in, size_t nfx, size_t i, int sh,
                                            int (&rh)[6], int (&rl)[6], int (&ih)[6], int (&il)[6]) {
  longlong2 f[12];
#pragma unroll
  for (int k = 0; k < 12; k++) f[k] = __ldg(in + size_t(k) * nfx + i);
  long long hr[6], hi[6];
  switch (mu) {
    case 0: deriv_project<0>(f, plus, hr, hi); break;
    case 1: deriv_project<1>(f, plus, hr, hi); break;
    case 2: deriv_project<2>(f, plus, hr, hi); break;
    default: deriv_project<3>(f, plus, hr, hi); break;
  }
#pragma unroll
  for (int k = 0; k < 6; k++) {
    split29(hr[k] >> sh, rh[k], rl[k]);
    split29(hi[k] >> sh, ih[k], il[k]);
  }
}

// the lane's share of W in FP64, for sites outside the fixed-point range
template <int MU, int S>
__device__ __forceinline__ void deriv_walk_fp64(const FxDerivParams& p, int64_t x, int64_t nb, int g, double (&wr)[9],
                                                double (&wi)[9]) {
  for (int s = g; s < p.L5a; s += 2) {
    double hr[6], hi[6], gr[6], gi[6];
    Spinor<double> f;
    SpinorIO<double>::load(p.in[1], nullptr, p.n5, size_t(nb) * p.L5 + s, f);
    project<MU, S>(f, hr, hi);
    SpinorIO<double>::load(p.in[0], nullptr, p.n5, size_t(x) * p.L5 + s, f);
    project<MU, S>(f, gr, gi);
    deriv_outer<double>(hr, hi, gr, gi, wr, wi);
  }
}
__device__ __noinline__ void deriv_site_fp64(const FxDerivParams& p, int64_t x, int64_t nb, int mu, int g, double (&wr)[9],
                                             double (&wi)[9]) {
  switch (2 * mu + (p.dag ? 1 : 0)) {
    case 0: deriv_walk_fp64<0, -1>(p, x, nb, g, wr, wi); break;
    case 1: deriv_walk_fp64<0, 1>(p, x, nb, g, wr, wi); break;
    case 2: deriv_walk_fp64<1, -1>(p, x, nb, g, wr, wi); break;
    case 3: deriv_walk_fp64<1, 1>(p, x, nb, g, wr, wi); break;
    case 4: deriv_walk_fp64<2, -1>(p, x, nb, g, wr, wi); break;
    case 5: deriv_walk_fp64<2, 1>(p, x, nb, g, wr, wi); break;
    case 6: deriv_walk_fp64<3, -1>(p, x, nb, g, wr, wi); break;
    default: deriv_walk_fp64<3, 1>(p, x, nb, g, wr, wi); break;
  }
}

__global__ void __launch_bounds__(128, 3) deriv_fx_kernel(const __grid_constant__ FxDerivParams p) {
  const int mu = threadIdx.y, g = threadIdx.x & 1;
  const int64_t x = int64_t(blockIdx.x) * 16 + (threadIdx.x >> 1);
  const bool active = x < p.n4h;
  const int64_t nb = active ? p.nbr[size_t(x) * 8 + mu] : 0;
  const int* ea = p.exps[0] + size_t(x) * p.L5a;
  const int* eb = p.exps[1] + size_t(nb) * p.L5a;
  int EAB = 0, worst = 0;  // of the largest product (0: all are zero), and of any factor
  if (active)
    for (int s = g; s < p.L5a; s += 2) {
      const int a = int(uint32_t(__ldg(ea + s)) >> 20), b = int(uint32_t(__ldg(eb + s)) >> 20);
      worst = max(worst, max(a, b));
      if (a != 0 && b != 0) EAB = max(EAB, a + b);
    }
  EAB = max(EAB, __shfl_xor_sync(0xffffffffu, EAB, 1));  // the same for both lanes of a site
  worst = max(worst, __shfl_xor_sync(0xffffffffu, worst, 1));
  // a factor outside the range, or a product whose double could over- or underflow
  const bool zero = EAB == 0;
  bool bad = worst == fx::kBad || (!zero && (EAB < 1146 || EAB > 2946));
  double wr[9], wi[9];
#pragma unroll
  for (int e = 0; e < 9; e++) { wr[e] = 0.0; wi[e] = 0.0; }
  if (!bad && !zero) {
    long long rh[9], rm[9], ih[9], im[9];
#pragma unroll
    for (int e = 0; e < 9; e++) { rh[e] = 0; rm[e] = 0; ih[e] = 0; im[e] = 0; }
    const int drop = 61 - p.bits;
    const bool plus = p.dag != 0;
    uint32_t least = 0;  // the lower bound of the sums' terms, 2^24 for one of the unit
#pragma unroll 1
    for (int s = g; s < p.L5a; s += 2) {
      int hrh[6], hrl[6], hih[6], hil[6], grh[6], grl[6], gih[6], gil[6];
      const uint32_t a = uint32_t(__ldg(ea + s)), b = uint32_t(__ldg(eb + s));
      if (a == 0 || b == 0) continue;
      const int sh = EAB - int(a >> 20) - int(b >> 20);
      const uint32_t ab = mu < 2 ? a >> 10 : a, bb = mu < 2 ? b >> 10 : b;
      least += ((1u << 24) >> min(uint32_t(sh) + (ab >> 5 & 31) + (bb >> 5 & 31), 31u)) +
               ((1u << 24) >> min(uint32_t(sh) + (ab & 31) + (bb & 31), 31u));
      deriv_limbs(mu, plus, p.fxin[1], p.nfx, size_t(nb) * p.L5a + s, drop, hrh, hrl, hih, hil);
      deriv_limbs(mu, plus, p.fxin[0], p.nfx, size_t(x) * p.L5a + s, min(sh + drop, 63), grh, grl, gih, gil);
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
          for (int b = 0; b < 3; b++) {
            const int h = j * 3 + c, k = j * 3 + b, e = c * 3 + b;
            const int nh = -hrh[h], nl = -hrl[h];  // limbs of base 2^29: no overflow
            rh[e] = fx::mad(hrh[h], grh[k], fx::mad(hih[h], gih[k], rh[e]));
            rm[e] = fx::mad(hrh[h], grl[k], fx::mad(hrl[h], grh[k], rm[e]));
            rm[e] = fx::mad(hih[h], gil[k], fx::mad(hil[h], gih[k], rm[e]));
            ih[e] = fx::mad(hih[h], grh[k], fx::mad(nh, gih[k], ih[e]));
            im[e] = fx::mad(hih[h], grl[k], fx::mad(hil[h], grh[k], im[e]));
            im[e] = fx::mad(nh, gil[k], fx::mad(nl, gih[k], im[e]));
          }
    }
    const int e2 = 58 + EAB - 2042 - 2 * p.bits;
    const unsigned pair = 3u << (threadIdx.x & 30);
#pragma unroll
    for (int e = 0; e < 9; e++) {
      long long re = rh[e] + ((rm[e] + (1ll << 28)) >> 29), imv = ih[e] + ((im[e] + (1ll << 28)) >> 29);
      re += __shfl_xor_sync(pair, re, 1);
      imv += __shfl_xor_sync(pair, imv, 1);
      wr[e] = fx_value(re, e2);
      wi[e] = fx_value(imv, e2);
    }
    least += __shfl_xor_sync(pair, least, 1);
    bad = least < 1u << (136 - 2 * p.bits);
    if (bad) {
#pragma unroll
      for (int e = 0; e < 9; e++) { wr[e] = 0.0; wi[e] = 0.0; }
    }
  }
  if (bad) {
    deriv_site_fp64(p, x, nb, mu, g, wr, wi);
#pragma unroll
    for (int e = 0; e < 9; e++) {  // the two lanes of a site are here together
      const unsigned pair = 3u << (threadIdx.x & 30);
      wr[e] += __shfl_xor_sync(pair, wr[e], 1);
      wi[e] += __shfl_xor_sync(pair, wi[e], 1);
    }
  }
  if (!active) return;
  double Ul[18];
  const double* src = p.links + (size_t(x) * 8 + mu) * 18;
#pragma unroll
  for (int e = 0; e < 18; e++) Ul[e] = src[e];
  const int64_t idx = p.half_out ? x : site_of_cb(p.L, p.parity, x);
  deriv_rows<2, double>(Ul, wr, wi, g, p.mat + (size_t(idx) * 4 + mu) * 9);
}

// The largest row sum of absolute values over one parity's links as the bits of a float
// rounded up (infinity for anything not finite), and the complement of the smallest's, rounded down.
__global__ void __launch_bounds__(256) fx_row_sum_kernel(const double* links, size_t rows, unsigned* out) {
  float m = 0.f, least = __int_as_float(0x7f800000);
  for (size_t r = size_t(blockIdx.x) * blockDim.x + threadIdx.x; r < rows; r += size_t(gridDim.x) * blockDim.x) {
    double s = 0.0;
#pragma unroll
    for (int e = 0; e < 6; e++) s += fabs(links[r * 6 + e]);
    const float f = __double2float_ru(s);
    m = f <= 3.0e38f ? fmaxf(m, f) : __int_as_float(0x7f800000);
    if (!(f <= 3.0e38f)) break;
    least = fminf(least, __double2float_rd(s));
  }
  m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
  least = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(least)));
  if ((threadIdx.x & 31) == 0) {
    atomicMax(out, __float_as_uint(m));
    atomicMax(out + 1, ~__float_as_uint(least));
  }
}

// fixed-point copy of one parity's links (k = exponent), AoS [x][leg][9] or SoA [leg][9][x]
__global__ void __launch_bounds__(256) fx_links_kernel(const double* links, int4* out, int64_t n4h, int k, int soa) {
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= size_t(n4h) * 72) return;
  int4 w;
  fx::split_link(__double2ll_rn(ldexp(links[2 * t], 61 - k)), w.x, w.y);
  fx::split_link(__double2ll_rn(ldexp(links[2 * t + 1], 61 - k)), w.z, w.w);
  const size_t x = t / 72, e = t - x * 72;
  out[soa ? e * size_t(n4h) + x : t] = w;
}

}  // namespace

// Operators whose FP64 hopping term runs in fixed point: the native FP64 arithmetic stays for
// 12-real links (rebuilt per CTA in FP64) and GB_FLAG_DF64 chooses its own.
bool fx_wanted(const Op* op) { return op->prec == GB_F64 && !op->recon12 && !op->df64 && !op->fx_off; }

// 5D sites of one checkerboard without padding slots
static size_t fx_sites(const Op* op) { return size_t(op->half4) * op->Ls * op->nrhs_user; }
// fixed-point copies the operator holds: the inputs of a launch, and what the CG form leaves for the next
static int fx_sets(const Op* op) { return op->Ls == 1 && op->nrhs_user == 1 ? 4 : 2; }

// The links' layout: sites in lanes below 8 slots per site (a CTA of 128 threads then stages 16
// sites at most, 18.7 KB, and four CTAs stay resident).  Wilson DhopEO, slots in CTAs against sites in lanes, us: 12^3 x 16
// with 6 / 7 / 8 / 9 slots 42.3 / 44.0 / 43.0 / 53.3 against 37.1 / 40.3 / 45.7 / 55.0; 16^4 79.5 / 94.9 / 98.9 / 118 against
// 83.5 / 99.0 / 108 / 124; 24^3 x 32 469 / 574 / 606 / 733 against 531 / 633 / 700 / 812: 4 to 7 slots on large
// lattices would be up to 12 % faster the other way, which no rule takes yet.
static bool fx_soa(const Op* op) { return op->Ls * op->nrhs_user < 8; }

// Fixed-point copies of op->links, and the scratch of fx_convert_kernel (both checkerboards of
// a field and their exponents): allocated here so that a launch allocates nothing.  Links that
// are not finite or of extreme magnitude, and a device without the memory, leave op->fx_ready off and
// the hopping term on the FP64 kernel.  So do links whose rows differ in size: they all share one unit, that
// of the largest, and an output whose own links are small would lose the bits that FP64 keeps.  The sums of
// absolute values of unitary rows differ by sqrt(6) at most, so a factor of 4 takes every gauge field of unitary
// links (also times one number, and smeared ones that have not been projected back, nearly so) and costs two bits
// of the five that the links have beyond a double's; a row of zeros is refused too.
int fx_import_links(Op* op) {
  op->fx_ready = false;
  if (!fx_wanted(op)) return GB_OK;
  unsigned* d_max = reinterpret_cast<unsigned*>(op->d_result);
  GB_CHECK_CUDA(cudaMemsetAsync(d_max, 0, 2 * sizeof(unsigned), op->stream));
  for (int p = 0; p < 2; p++)
    fx_row_sum_kernel<<<kRedBlocks, 256, 0, op->stream>>>(static_cast<const double*>(op->links[p]), size_t(op->half4) * 24,
                                                          d_max);
  GB_CHECK_CUDA(cudaGetLastError());
  GB_CHECK_CUDA(cudaMemcpyAsync(op->h_result, d_max, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, op->stream));
  GB_CHECK_CUDA(cudaStreamSynchronize(op->stream));
  unsigned sums[2];
  std::memcpy(sums, op->h_result, sizeof(sums));
  sums[1] = ~sums[1];
  float top, least;
  std::memcpy(&top, &sums[0], sizeof(top));
  std::memcpy(&least, &sums[1], sizeof(least));
  if (!(top > 1e-9f && top < 1e9f && top <= kFxLinkRatio * least)) return GB_OK;
  int k = -32;
  while (double(top) > 1.5 * std::ldexp(1.0, k)) k++;
  op->fx_exp = k;
  const size_t n = size_t(op->half4) * 72;
  const size_t field = fx_sites(op) * fx_sets(op) * (12 * sizeof(longlong2) + sizeof(int));
  if (!op->links_fx[0]) {  // (else kept from an earlier import)
    char* block = nullptr;  // one, so that it comes back as one
    if (cudaMallocAsync(reinterpret_cast<void**>(&block), 2 * n * sizeof(int4) + field, op->stream) != cudaSuccess) {
      cudaGetLastError();
      return GB_OK;
    }
    op->links_fx[0] = block;
    op->links_fx[1] = block + n * sizeof(int4);
    op->fx_field = block + 2 * n * sizeof(int4);
  }
  for (int p = 0; p < 2; p++)
    fx_links_kernel<<<unsigned((n + 255) / 256), 256, 0, op->stream>>>(static_cast<const double*>(op->links[p]),
                                                                       static_cast<int4*>(op->links_fx[p]), op->half4, k,
                                                                       fx_soa(op) ? 1 : 0);
  GB_CHECK_CUDA(cudaGetLastError());
  op->fx_ready = true;
  return GB_OK;
}

bool fx_release(Op* op) {
  if (!op->links_fx[0] || op->fx_captured || op->own_graphs > 0) return false;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (op->stream && (cudaStreamIsCapturing(op->stream, &status) != cudaSuccess || status != cudaStreamCaptureStatusNone))
    return false;
  op->fx_ready = false;
  cudaFreeAsync(op->links_fx[0], op->stream);
  op->links_fx[0] = op->links_fx[1] = op->fx_field = nullptr;
  return true;
}

// before each launch on the copies (see Op::fx_captured)
static void fx_note_capture(Op* op) {
  if (!op->stream || op->fx_captured || op->own_graphs > 0) return;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(op->stream, &status) != cudaSuccess) cudaGetLastError();
  else op->fx_captured = status != cudaStreamCaptureStatusNone;
}

static longlong2* fx_planes(const Op* op, int z) { return static_cast<longlong2*>(op->fx_field) + size_t(z) * 12 * fx_sites(op); }
static int* fx_exps(const Op* op, int z) {
  return reinterpret_cast<int*>(static_cast<longlong2*>(op->fx_field) + fx_sets(op) * 12 * fx_sites(op)) + size_t(z) * fx_sites(op);
}

// Output sites per CTA of dhop_fx_kernel for L5c slots a site: of CTAs of up to 128 and up to 96
// threads, the one that leaves fewer lanes of its warps idle, the larger one when equal (12 slots
// fill 120 of 128 lanes or 96 of 96; 16 fill both).  Measured, always 128 -> this rule: 12 slots
// 16^4 149 -> 144 us and 24^3 x 32 964 -> 931 us, 19 slots 240 -> 232 us, 22 slots 278 -> 267 us;
// 96 threads at 16 slots: 186 against 182 us.
static int fx_cta_sites(int L5c) {
  const int large = 128 / L5c, small = 96 / L5c;
  const auto lanes = [&](int sites) { return (sites * L5c + 31) / 32 * 32; };
  return small * lanes(large) > large * lanes(small) ? small : large;
}

int launch_dhop_fx(Op* op, HalfView in, HalfView out, int out_parity, const HalfView* in2, const HalfView* out2, int dag,
                   const DhopAxpy* axpy, int* parts, bool given) {
  fx_note_capture(op);
  FxParams p;
  const HalfView* ins[2] = {&in, in2};
  const HalfView* outs[2] = {&out, out2};
  for (int z = 0; z < 2; z++) {
    const int par = z ? 1 - out_parity : out_parity;
    p.in[z] = ins[z] ? ins[z]->data : nullptr;
    p.out[z] = outs[z] ? outs[z]->data : nullptr;
    p.z[z] = axpy ? static_cast<const double2*>(axpy->z[z].data) : nullptr;
    p.links[z] = static_cast<const int4*>(op->links_fx[par]);
    p.links_d[z] = static_cast<const double*>(op->links[par]);
    p.nbr[z] = op->nbr[par];
  }
  p.n4h = op->half4;
  p.n5 = op->n5();
  p.nfx = fx_sites(op);
  p.L5 = op->L5;
  p.L5a = op->Ls * op->nrhs_user;
  p.c0 = axpy ? axpy->c0 : 0.0;
  p.c1 = axpy ? axpy->c1 : 1.0;
  p.link_exp = op->fx_exp;
  p.dag = dag;
  p.err = op->d_err;
  for (int z = 0; z < 2; z++) {  // the sets 2, 3 hold what the CG form's blockIdx.z 0, 1 left
    const int set = given ? (in2 ? 3 - z : 2 + z) : z;
    p.fxin[z] = fx_planes(op, set);
    p.exps[z] = fx_exps(op, set);
  }
  if (!given)
    launch_pdl(fx_convert_kernel<false>, dim3(unsigned((p.nfx + 255) / 256), 1, in2 ? 2u : 1u), 256, 0, op->stream, p);
  const bool soa = fx_soa(op);
  void (*kernel)(const FxParams);
  const size_t ctas = size_t((p.n4h * p.L5a + 31) / 32) * (in2 ? 2 : 1);
  const bool two = ctas > kFxTwoWarps;
  if (parts && axpy && op->Ls == 1 && op->nrhs_user == 1 && ctas <= op->partial_doubles) {
    const bool beta = axpy->r[0].data != nullptr;
    for (int z = 0; z < 2; z++) {
      p.r[z] = static_cast<double2*>(axpy->r[z].data);
      p.fxout[z] = fx_planes(op, 2 + z);
      p.expout[z] = fx_exps(op, 2 + z);
    }
    p.partial = op->d_partial;
    p.fin = CGFinish{op->d_cg, op->d_all_done, beta ? CG_FINISH_BETA : CG_FINISH_ALPHA};
    *parts = -1;
    if (two) kernel = beta ? dhop_fx_split_kernel<true, true, 2, CG_FINISH_BETA> : dhop_fx_split_kernel<true, true, 2, CG_FINISH_ALPHA>;
    else kernel = beta ? dhop_fx_split_kernel<true, true, 4, CG_FINISH_BETA> : dhop_fx_split_kernel<true, true, 4, CG_FINISH_ALPHA>;
    launch_pdl(kernel, dim3(unsigned((p.n4h + 31) / 32), 1, in2 ? 2u : 1u), two ? 64u : 128u, 0, op->stream, p);
    GB_CHECK_CUDA(cudaGetLastError());
    return GB_OK;
  }
  if (soa || p.n4h * p.L5a * (in2 ? 2 : 1) <= kFxSplitSites) {
    if (soa && two) kernel = axpy ? dhop_fx_split_kernel<true, true, 2> : dhop_fx_split_kernel<true, false, 2>;
    else if (soa) kernel = axpy ? dhop_fx_split_kernel<true, true, 4> : dhop_fx_split_kernel<true, false, 4>;
    else if (two) kernel = axpy ? dhop_fx_split_kernel<false, true, 2> : dhop_fx_split_kernel<false, false, 2>;
    else kernel = axpy ? dhop_fx_split_kernel<false, true, 4> : dhop_fx_split_kernel<false, false, 4>;
    launch_pdl(kernel, dim3(unsigned((p.n4h * p.L5a + 31) / 32), 1, in2 ? 2u : 1u), two ? 64u : 128u, 0, op->stream, p);
  } else {
    kernel = axpy ? dhop_fx_kernel<true> : dhop_fx_kernel<false>;
    p.L5c = p.L5a > 128 ? 128 : p.L5a;
    p.k4 = fx_cta_sites(p.L5c);
    const dim3 grid(unsigned((p.n4h + p.k4 - 1) / p.k4), unsigned((p.L5a + p.L5c - 1) / p.L5c), in2 ? 2u : 1u);
    const unsigned threads = unsigned((p.k4 * p.L5c + 31) / 32 * 32);
    launch_pdl(kernel, grid, threads, size_t(p.k4) * kFxLinkStride * sizeof(int4), op->stream, p);
  }
  GB_CHECK_CUDA(cudaGetLastError());
  return GB_OK;
}

bool fx_deriv_ok(const Op* op) { return op->Ls * op->nrhs_user <= kDerivSlots; }

int launch_deriv_fx(Op* op, HalfView A, HalfView B, int out_parity, int dag, double* mat, int half_out) {
  fx_note_capture(op);
  FxParams c = {};  // the conversion of both factors: one launch, one per blockIdx.z
  FxDerivParams p;
  const HalfView* f[2] = {&A, &B};
  for (int z = 0; z < 2; z++) {
    c.in[z] = f[z]->data;
    c.fxin[z] = fx_planes(op, z);
    c.exps[z] = fx_exps(op, z);
    p.in[z] = static_cast<const double2*>(f[z]->data);
    p.fxin[z] = c.fxin[z];
    p.exps[z] = c.exps[z];
  }
  c.n5 = p.n5 = op->n5();
  c.nfx = p.nfx = fx_sites(op);
  c.L5 = p.L5 = op->L5;
  c.L5a = p.L5a = op->Ls * op->nrhs_user;
  launch_pdl(fx_convert_kernel<true>, dim3(unsigned((c.nfx + 255) / 256), 1, 2), 256, 0, op->stream, c);
  p.links = static_cast<const double*>(op->links[out_parity]);
  p.nbr = op->nbr[out_parity];
  p.mat = reinterpret_cast<double2*>(mat);
  p.n4h = op->half4;
  p.bits = p.L5a == 1 ? 59 : p.L5a <= 4 ? 58 : p.L5a <= 16 ? 57 : p.L5a <= 32 ? 56 : 55;
  p.half_out = half_out;
  p.dag = dag;
  p.parity = out_parity;
  for (int k = 0; k < 4; k++) p.L[k] = op->dims[k];
  deriv_fx_kernel<<<unsigned((p.n4h + 15) / 16), dim3(32, 4), 0, op->stream>>>(p);
  GB_CHECK_CUDA(cudaGetLastError());
  return GB_OK;
}

}  // namespace gb
