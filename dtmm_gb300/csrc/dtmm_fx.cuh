// Line transforms of complex128 data in 64-bit fixed point.
//
// The part issues 2 FP64 operations per clock and SM against 64 INT32 ones,
// so a complex128 FFT in FP64 arithmetic is bound by the FP64 pipe alone
// (measured: DADD / DFMA 1.6 / 1.9 lanes per clock and SM, a 64-bit integer
// add 30, a 32 x 32 + 64 multiply-add 16).  A transform only adds and
// multiplies by constants of modulus one, and its partial results are
// bounded by the sum of its inputs' moduli, so it runs in block fixed point:
// a power of two per line puts that sum below 2^60, additions are exact, and
// a product rounds at 2^-60 of full scale.  The first step of a two-step
// transform, whose DFTs sum fewer inputs, has its own finer scale, and its
// results are rounded to the second step's.  The transform's error is below
// the one of FP64 arithmetic, which rounds at every butterfly
// (tests/fx_host.cu measures both against long double).
//
// A line with an infinity or a NaN becomes NaN throughout, as an FP64
// transform makes it (every output sums every input).
#pragma once

#include "dtmm_regfft.cuh"

namespace dtmm {

// Fixed-point number: data at the line's own scale, constants in Q62.
struct fx {
  long long v;
  fx() = default;
  __host__ __device__ constexpr explicit fx(long long raw, int) : v(raw) {}
  // |c| <= 1 in Q62 (1.0 as 2^62 - 1: the high limb must fit 32 bits)
  __host__ __device__ constexpr explicit fx(double c)
      : v(c >= 1.0 ? (1LL << 62) - 1 : (long long)(c * 4611686018427387904.0)) {}
  __host__ __device__ constexpr explicit fx(int c) : v(c > 0 ? (1LL << 62) - 1 : 0) {}
};
__host__ __device__ __forceinline__ fx operator+(fx a, fx b) { return fx(a.v + b.v, 0); }
__host__ __device__ __forceinline__ fx operator-(fx a, fx b) { return fx(a.v - b.v, 0); }
__host__ __device__ __forceinline__ constexpr fx operator-(fx a) { return fx(-a.v, 0); }

// signed 32 x 32 + 64 -> 64 multiply-add (one IMAD.WIDE)
__host__ __device__ __forceinline__ long long madw(int a, int b, long long c) { return (long long)a * b + c; }
__host__ __device__ __forceinline__ int fx_hi(long long v) { return (int)(v >> 31); }
__host__ __device__ __forceinline__ int fx_lo(long long v) { return (int)(v & 0x7fffffff); }
constexpr long long kFxHalf = 1LL << 30;  // rounds the product's middle limb

// a c / 2^62, |a| below 2^62 and |c| <= 2^62: limbs of 31 bits, the low x low
// product (below the last place) left out
__host__ __device__ __forceinline__ fx operator*(fx a, fx c) {
  const long long mid = madw(fx_lo(a.v), fx_hi(c.v), madw(fx_hi(a.v), fx_lo(c.v), kFxHalf));
  return fx(madw(fx_hi(a.v), fx_hi(c.v), mid >> 31), 0);
}

// a w with the middle limbs of the two products of a component summed before
// their one shift.  |a| below 2^60: the four middle products then stay below
// sqrt(2) (1 + 1/4) 2^62 in sum.  (The data's limbs are negated: the high limb
// of the constant -1 has no negative.)
__host__ __device__ __forceinline__ cpx<fx> operator*(cpx<fx> a, cpx<fx> w) {
  const int ah = fx_hi(a.re.v), al = fx_lo(a.re.v), bh = fx_hi(a.im.v), bl = fx_lo(a.im.v);
  const int ch = fx_hi(w.re.v), cl = fx_lo(w.re.v), sh = fx_hi(w.im.v), sl = fx_lo(w.im.v);
  const long long mr = madw(-bl, sh, madw(-bh, sl, madw(al, ch, madw(ah, cl, kFxHalf))));
  const long long mi = madw(bl, ch, madw(bh, cl, madw(al, sh, madw(ah, sl, kFxHalf))));
  return mk<fx>(fx(madw(-bh, sh, madw(ah, ch, mr >> 31)), 0), fx(madw(bh, ch, madw(ah, sh, mi >> 31)), 0));
}

// Constants in Q62 from a Taylor series in 128-bit integer arithmetic (terms
// of Q62, about 20 roundings at 2^-62), after the octant reduction of ct::cos2pi.
namespace ct {
constexpr long long q62_mul(long long a, long long b) { return (long long)(((__int128)a * b + ((__int128)1 << 61)) >> 62); }
constexpr long long q62_series(long long x, bool odd) {
  const long long x2 = q62_mul(x, x), one = 1LL << 62;
  long long term = odd ? x : one, sum = term;
  for (int k = 1; k <= 12; ++k) {
    const int a = odd ? 2 * k : 2 * k - 1;
    term = -q62_mul(term, x2) / (a * (a + 1));
    sum += term;
  }
  return sum;
}
constexpr long long q62_cos2pi(long long n, long long d) {
  n %= d;
  if (n < 0) n += d;
  if (2 * n > d) n = d - n;
  long long sign = 1, num = n, den = d;
  if (4 * num > den) {
    num = den - 2 * num;
    den = 2 * den;
    sign = -1;
  }
  const __int128 two_pi_q62 = (__int128)7244019458077122842LL * 4 + 2;
  const bool high = 8 * num > den;
  if (high) {
    num = den - 4 * num;
    den = 4 * den;
  }
  // 2 pi num / den <= pi / 4 in Q62
  const long long x = (long long)((two_pi_q62 * num * 2 / den + 1) / 2);
  return sign * q62_series(x, high);
}
}  // namespace ct

template <>
struct CtConst<fx> {
  static constexpr long long below_one(long long v) { return v > (1LL << 62) - 1 ? (1LL << 62) - 1 : v; }
  static __host__ __device__ constexpr fx cos2pi(long long n, long long d) { return fx(below_one(ct::q62_cos2pi(n, d)), 0); }
  static __host__ __device__ constexpr fx sin2pi(long long n, long long d) {
    return fx(below_one(ct::q62_cos2pi(4 * n - d, 4 * d)), 0);
  }
};

// a constant turn: by odd eighths two real products, others the fused product
template <>
struct RotGeneral<fx> {
  template <bool EIGHTH>
  static __host__ __device__ __forceinline__ cpx<fx> run(cpx<fx> v, fx c, fx s) {
    if constexpr (EIGHTH) {
      // (re c - im s, re s + im c), |c| = |s|: sums first
      const bool cp = c.v > 0, sp = s.v > 0;
      const fx a = v.re + v.im, b = v.re - v.im;
      const fx h(c.v > 0 ? c.v : -c.v, 0);
      const fx p = (cp == sp ? b : a) * h, q = (cp == sp ? a : b) * h;
      // cp sp: (b, a); cp, !sp: (a, -b); !cp, sp: (-a, b); neither: (-b, -a)
      return cp ? (sp ? mk<fx>(p, q) : mk<fx>(p, -q)) : (sp ? mk<fx>(-p, q) : mk<fx>(-p, -q));
    } else {
      return v * mk<fx>(c, s);
    }
  }
};

__host__ __device__ __forceinline__ long long dbits(double x) {
#ifdef __CUDA_ARCH__
  return __double_as_longlong(x);
#else
  long long b;
  __builtin_memcpy(&b, &x, 8);
  return b;
#endif
}
__host__ __device__ __forceinline__ double bitsd(long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(b);
#else
  double x;
  __builtin_memcpy(&x, &b, 8);
  return x;
#endif
}
__host__ __device__ __forceinline__ int fx_hiword(double x) { return (int)(dbits(x) >> 32); }

// The scale of a line: every thread packs the largest biased exponent E of
// its entries and, in units of 2^(E - 1035), an upper bound of the sum of their
// |re| + |im| (fx_part; entries [lo, hi) are zeros and skipped); the line's scale follows from the words of all its
// threads (fx_scale).  Integer operations on the high words.
template <int MAXL>
__host__ __device__ __forceinline__ unsigned fx_part(const cpx<double> (&d)[MAXL], int len, int lo, int hi) {
  int m = 0;
#pragma unroll
  for (int i = 0; i < MAXL; ++i) {
    if (i >= len) break;
    if (i >= lo && i < hi) continue;
    const int a = fx_hiword(d[i].re) & 0x7fffffff, b = fx_hiword(d[i].im) & 0x7fffffff;
    m = m > a ? m : a;
    m = m > b ? m : b;
  }
  m >>= 20;
  unsigned sum = 0;
#pragma unroll
  for (int i = 0; i < MAXL; ++i) {
    if (i >= len) break;
    if (i >= lo && i < hi) continue;
    const int a = fx_hiword(d[i].re) & 0x7fffffff, b = fx_hiword(d[i].im) & 0x7fffffff;
    const int ra = m - (a >> 20), rb = m - (b >> 20);
    sum += ((unsigned)(a & 0xfffff) | 0x100000u) >> (ra < 31 ? ra : 31);
    sum += ((unsigned)(b & 0xfffff) | 0x100000u) >> (rb < 31 ? rb : 31);
  }
  // truncated bits: below one unit of 2^(E - 1043) an entry
  return (unsigned)m << 20 | ((sum + 2u * MAXL + 255u) >> 8);
}
// emax: largest biased exponent; g1, g2: guard bits of the two steps, so that
// moduli of entries scaled below 2^(60 - g) sum to less than 2^60 over one
// thread's entries and over the line
__host__ __device__ __forceinline__ void fx_scale(const unsigned* word, int n, int& emax, int& g1, int& g2) {
  int e = 0;
  for (int i = 0; i < n; ++i) {
    const int x = (int)(word[i] >> 20);
    e = e > x ? e : x;
  }
  unsigned total = 0, most = 0;
  for (int i = 0; i < n; ++i) {
    const unsigned w = word[i];
    const int r = e - (int)(w >> 20);
    const unsigned u = ((w & 0xfffffu) >> (r < 31 ? r : 31)) + 1u;
    total += u;
    most = most > u ? most : u;
  }
#ifdef __CUDA_ARCH__
  const int b1 = 32 - __clz((int)most), b2 = 32 - __clz((int)total);
#else
  int b1 = 0, b2 = 0;
  while (most >> b1) ++b1;
  while (total >> b2) ++b2;
#endif
  emax = e;
  g1 = b1 > 13 ? b1 - 13 : 0;
  g2 = b2 > 13 ? b2 - 13 : 0;
}

// a value of the first step at the second step's scale (r = g2 - g1),
// rounded to nearest
__host__ __device__ __forceinline__ fx fx_shift(fx a, int r) { return fx((a.v + ((1LL << r) >> 1)) >> r, 0); }
__host__ __device__ __forceinline__ cpx<fx> fx_shift(cpx<fx> a, int r) {
  return mk<fx>(fx_shift(a.re, r), fx_shift(a.im, r));
}

// x in the fixed point of a line whose largest biased exponent is emax, with
// g guard bits: x 2^(1082 - g - emax) rounded to nearest, below 2^(60 - g);
// integer operations (the hardware conversion issues at the FP64 rate).
// Subnormal x: the exponent of the smallest normal number, no leading one.
__host__ __device__ __forceinline__ fx to_fx(double x, int emax, int g) {
  const long long b = dbits(x);
  const int e = (int)(b >> 52) & 0x7ff;
  const int r = g + 2 + emax - (e != 0 ? e : 1);  // right shift of the 63-bit significand, less one
  const unsigned long long m = ((unsigned long long)b << 10 & 0x3fffffffffffffffULL) | (e != 0 ? 1ULL << 62 : 0ULL);
  long long t = r > 62 ? 0 : (long long)(m >> (r & 63));
  t = (t + 1) >> 1;
  return fx(b < 0 ? -t : t, 0);
}

// the double v 2^(emax + g - 1082): converted from the integer in FP64 and
// scaled through its exponent field
__host__ __device__ __forceinline__ double from_fx(fx a, int kexp) {
#ifdef __CUDA_ARCH__
  const double d = __ll2double_rn(a.v);
#else
  const double d = (double)a.v;
#endif
  return a.v == 0 ? 0.0 : bitsd(dbits(d) + ((long long)kexp << 52));
}
// kexp of from_fx for a line; results below 2^-1021 or above 2^1023 do not
// fit its exponent field arithmetic (fx_plain false): scale with ldexp
__host__ __device__ __forceinline__ int fx_kexp(int emax, int g) { return emax + g - 1082; }
__host__ __device__ __forceinline__ bool fx_plain(int emax) { return emax >= 128 && emax <= 1984; }

// ---------------------------------------------------------------------------
// exp(2 pi i u) in integer arithmetic.  The library's FP64 sincos takes about
// 40 FP64 operations; here u (turns) becomes a 64-bit fraction of a turn, its
// top 10 bits pick (cos, sin) of a table, and the remaining angle d, |d| <=
// 2 pi / 2048, turns it by 1 - cos d = d^2 / 2 - d^4 / 24 and sin d = d - (d^3 -
// d^5 / 20) / 6 (Taylor; the next terms are below 2^-59).  Error: 2^-53 of a
// component plus u's own rounding times 2 pi, as with FP64 arithmetic.
// ---------------------------------------------------------------------------
constexpr int kTurnBits = 10;
struct TurnTab {
  long long v[2 << kTurnBits];  // cos, sin in Q62
  constexpr TurnTab() : v() {
    for (int i = 0; i < (1 << kTurnBits); ++i) {
      v[2 * i] = CtConst<fx>::cos2pi(i, 1 << kTurnBits).v;
      v[2 * i + 1] = CtConst<fx>::sin2pi(i, 1 << kTurnBits).v;
    }
  }
};
#ifdef __CUDACC__
__device__ const TurnTab kTurnTab{};
#endif
static const TurnTab kTurnTabHost{};

// k / (2 pi) as the rounded product and what that lacks, relative, in units of
// 2^-83 (|rest| < 2^31): rounded alone it would turn every phase of a wavelength by
// up to 1.7e-16 of itself, the same way in every voxel and layer.
struct TurnScale {
  double k;
  int rest;
};
__host__ __device__ __forceinline__ TurnScale turn_scale(double k) {
  constexpr double c = 0.15915494309189533577, c_lo = -9.839338337591243477e-18;  // 1 / (2 pi)
  TurnScale t;
  t.k = k * c;
  const double lo = fma(k, c, -t.k) + k * c_lo, r = lo / t.k * 9671406556917033397649408.0;  // 2^83
  t.rest = fabs(r) < 2147483647.0 ? (int)r : 0;  // (zero and infinite k: none)
  return t;
}

// (cos, sin) of f / 2^64 turns in Q62
__host__ __device__ __forceinline__ cpx<fx> fx_turn_at(unsigned long long f) {
  const unsigned i = (unsigned)((f + (1ULL << (63 - kTurnBits))) >> (64 - kTurnBits)) & ((1u << kTurnBits) - 1u);
  const long long r = (long long)(f - ((unsigned long long)i << (64 - kTurnBits)));
  constexpr long long kPi4 = 3622009729038561421LL;  // pi / 4 in Q62
  const long long d = (fx(r << 7, 0) * fx(kPi4, 0)).v;   // d 2^68
  const long long z = (fx(d, 0) * fx(d, 0)).v;           // d^2 2^74
  const int zh = (int)(z >> 27), dh = (int)(d >> 30);    // d^2 2^47, d 2^38
  const int z2 = (int)(madw(zh, zh, 0) >> 32);           // d^4 2^62
  const long long cm = (z >> 7) - (madw(z2, 715827883, 0) >> 28);  // (1 - cos d) 2^68 (2^28 64 / 24)
  const int q = zh - (int)(madw(z2 >> 15, 3277, 0) >> 16);     // (d^2 - d^4 / 20) 2^47
  const long long w = madw(dh, q, 0);                          // (d^3 - d^5 / 20) 2^85
  const long long sn = d - (madw((int)(w >> 29), 715827883, 0) >> 20);  // sin d 2^68
#ifdef __CUDA_ARCH__
  const longlong2 t = ((const longlong2*)kTurnTab.v)[i];
  const cpx<fx> cs = mk<fx>(fx(t.x, 0), fx(t.y, 0));
#else
  const cpx<fx> cs = mk<fx>(fx(kTurnTabHost.v[2 * i], 0), fx(kTurnTabHost.v[2 * i + 1], 0));
#endif
  const cpx<fx> e = mk<fx>(fx(-cm, 0), fx(sn, 0)) * cs;  // 2^68
  return mk<fx>(fx(cs.re.v + ((e.re.v + 32) >> 6), 0), fx(cs.im.v + ((e.im.v + 32) >> 6), 0));
}

// (cos, sin) of u (1 + rest 2^-83) turns in Q62; u finite
__host__ __device__ __forceinline__ cpx<fx> fx_turn(double u, int rest = 0) {
  const long long b = dbits(u);
  const int sh = ((int)(b >> 52) & 0x7ff) - 1011;  // 2^64 u = significand << sh
  const unsigned long long m = ((unsigned long long)b & 0xfffffffffffffULL) | (1ULL << 52);
  unsigned long long f;
  if (sh >= 0)
    f = sh < 64 ? (m << sh) + (unsigned long long)(madw((int)(m >> 22), rest, 0) >> (sh < 61 ? 61 - sh : 0)) : 0;
  else
    f = sh > -55 ? ((m >> (-sh - 1)) + 1) >> 1 : 0;
  if (b < 0) f = 0 - f;
  return fx_turn_at(f);
}

// (cos, sin) of an angle in radians, |ang| below 2^21: its significand times
// 2^66 / (2 pi) (rounded: 2^-64 of the turns) as 128 bits, of which the fraction
// of a turn is kept, 2^-43 of a radian at the largest angle and 2^-62 at one turn
constexpr int kAngleBits = 21;
__host__ __device__ __forceinline__ bool fx_angle_ok(double ang) {
  return ((int)(dbits(ang) >> 52) & 0x7ff) < 1023 + kAngleBits;
}
__host__ __device__ __forceinline__ cpx<fx> fx_angle(double ang) {
  constexpr unsigned long long kTurns = 11743562013128004906ULL;
  const long long b = dbits(ang);
  const int sh = 1077 - ((int)(b >> 52) & 0x7ff);  // 2^64 turns = significand kTurns >> sh
  const unsigned long long m = ((unsigned long long)b & 0xfffffffffffffULL) | (1ULL << 52), lo = m * kTurns;
#ifdef __CUDA_ARCH__
  const unsigned long long hi = __umul64hi(m, kTurns);
#else
  const unsigned long long hi = (unsigned long long)(((unsigned __int128)m * kTurns) >> 64);
#endif
  unsigned long long f = sh < 64 ? hi << (64 - sh) | lo >> sh : (sh < 128 ? hi >> (sh - 64) : 0);
  if (b < 0) f = 0 - f;
  return fx_turn_at(f);
}

// exp(2 pi i u (1 + rest 2^-83)); infinite and NaN u give NaN
__host__ __device__ __forceinline__ cpx<double> turn_of(double u, int rest = 0) {
  if ((fx_hiword(u) & 0x7ff00000) == 0x7ff00000) return mk<double>(u - u, u - u);
  const cpx<fx> t = fx_turn(u, rest);
  return mk<double>(from_fx(t.re, -62), from_fx(t.im, -62));
}

// ---------------------------------------------------------------------------
// DFT over registers of a run-time length (a switch over unrolled
// transforms), forward; an inverse transform swaps the real and imaginary
// parts of its inputs and outputs.  Lengths up to MAXL.
// ---------------------------------------------------------------------------
template <typename T, int N>
struct LineDFT {
  __host__ __device__ static __forceinline__ void run(cpx<T>* v) { RegDFTg<T, N, false>::run(v); }
};

template <typename T, int MAXL>
__host__ __device__ __forceinline__ void line_dft(cpx<T> (&v)[MAXL], int n) {
#define DTMM_LINE_CASE(N) \
  case N: LineDFT<T, N>::run(v); break;
  if constexpr (MAXL <= 16) {
    switch (n) {
      DTMM_LINE_CASE(2) DTMM_LINE_CASE(3) DTMM_LINE_CASE(4) DTMM_LINE_CASE(5) DTMM_LINE_CASE(6) DTMM_LINE_CASE(7)
      DTMM_LINE_CASE(8) DTMM_LINE_CASE(9) DTMM_LINE_CASE(10) DTMM_LINE_CASE(12) DTMM_LINE_CASE(14)
      DTMM_LINE_CASE(15) DTMM_LINE_CASE(16)
      default: break;
    }
  } else {
    switch (n) {
      DTMM_LINE_CASE(5) DTMM_LINE_CASE(6) DTMM_LINE_CASE(7) DTMM_LINE_CASE(8) DTMM_LINE_CASE(9)
      DTMM_LINE_CASE(10) DTMM_LINE_CASE(11) DTMM_LINE_CASE(12) DTMM_LINE_CASE(14) DTMM_LINE_CASE(15)
      DTMM_LINE_CASE(16) DTMM_LINE_CASE(18) DTMM_LINE_CASE(20) DTMM_LINE_CASE(21) DTMM_LINE_CASE(22)
      DTMM_LINE_CASE(24) DTMM_LINE_CASE(25) DTMM_LINE_CASE(27) DTMM_LINE_CASE(28) DTMM_LINE_CASE(30)
      DTMM_LINE_CASE(32)
      default: break;
    }
  }
#undef DTMM_LINE_CASE
}

// the lengths of each class
__host__ __device__ constexpr bool line_len_ok(int n, int maxl) {
  if (maxl <= 16)
    return (n >= 1 && n <= 10) || n == 12 || (n >= 14 && n <= 16);
  return (n >= 5 && n <= 12) || n == 14 || n == 15 || n == 16 || n == 18 || n == 20 || n == 21 || n == 22 ||
         n == 24 || n == 25 || n == 27 || n == 28 || n == 30 || n == 32;
}

// Two-step shape of an n-point line, n = n1 n2: n1 lanes with n2 points each
// in the first step of the inverse transform.  The most even split of the
// smaller length class; maxl 0: none.
struct LineShape {
  int n1, n2, maxl;
};
inline LineShape line_shape(int n) {
  for (int maxl = 16; maxl <= 32; maxl += 16) {
    int best = 0;
    for (int a = 1; a * a <= n; ++a)
      if (n % a == 0 && line_len_ok(a, maxl) && line_len_ok(n / a, maxl)) best = a;
    if (best) return LineShape{best, n / best, maxl};
  }
  return LineShape{0, 0, 0};
}

}  // namespace dtmm
