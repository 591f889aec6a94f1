// Host check of the fixed-point line transforms (dtmm_gb300/csrc/dtmm_fx.cuh):
// conversions, every register DFT length of both classes, and the two-step
// transform in the slot order of dtmm_linekern.cuh, forward and inverse,
// against a direct DFT in long double.  Inputs: flat, one dominant entry,
// band-limited, 300 orders of magnitude apart, huge and tiny.  Prints
// "err <name> <n> <fixed> <fp64>" lines (relative L2; fp64: the same transform
// in FP64 arithmetic) and "OK" at the end.
#include <cmath>
#include <complex>
#include <cstdio>
#include <vector>

#include "dtmm_fx.cuh"

using namespace dtmm;
using C = std::complex<double>;
using CL = std::complex<long double>;

static int g_bad = 0;
static double g_sum[6][2];

static std::vector<CL> direct(const std::vector<C>& x, bool inv) {
  const int n = (int)x.size();
  const long double pi = acosl(-1.0L);
  std::vector<CL> w(n), X(n);
  for (int j = 0; j < n; ++j) {
    const long double a = (inv ? 2.0L : -2.0L) * pi * j / n;
    w[j] = CL(cosl(a), sinl(a));
  }
  for (int k = 0; k < n; ++k) {
    CL s = 0;
    for (int j = 0; j < n; ++j) s += CL(x[j].real(), x[j].imag()) * w[(long long)j * k % n];
    X[k] = s;
  }
  return X;
}

static double rnd(unsigned& s) {
  s = s * 1664525u + 1013904223u;
  return (s >> 8) / 16777216.0 - 0.5;
}

static std::vector<C> input(int n, int kind) {
  std::vector<C> x(n);
  unsigned s = 12345u + 104729u * n + kind;
  for (int i = 0; i < n; ++i) {
    x[i] = C(rnd(s), rnd(s));
    const int f = i < (n + 1) / 2 ? i : n - i;
    if (kind == 1) x[i] *= i == n / 3 ? 1.0 : 1e-4;
    if (kind == 2 && f > n / 5) x[i] = 0;
    if (kind == 3) x[i] *= std::pow(10.0, -300.0 * i / n);
    if (kind == 4) x[i] *= 1e280;
    if (kind == 5) x[i] *= 1e-250;
  }
  return x;
}

static double rel(const std::vector<C>& a, const std::vector<CL>& b) {
  long double num = 0, den = 0, big = 0;
  for (const CL& v : b) big = std::fmax(big, std::abs(v));
  for (size_t i = 0; i < a.size(); ++i) {
    num += std::norm((CL(a[i].real(), a[i].imag()) - b[i]) / big);
    den += std::norm(b[i] / big);
  }
  return (double)sqrtl(num / den);
}

template <typename V>
static cpx<V> tw_of(int e, int n) {
  const double a = -2.0 * M_PI * e / n;
  return mk<V>(V(std::cos(a)), V(std::sin(a)));
}

static cpx<fx> to_second(cpx<fx> a, int r) { return fx_shift(a, r); }
static cpx<double> to_second(cpx<double> a, int) { return a; }

// the two-step transform as the kernels run it, all threads of a step in turn
template <typename V>
static std::vector<cpx<V>> two_step(const std::vector<cpx<V>>& in, bool fwd, int shift) {
  const int n = (int)in.size();
  const LineShape ls = line_shape(n);
  const int n1 = ls.n1, n2 = ls.n2, P = n2 | 1;
  std::vector<cpx<V>> buf((size_t)n1 * P), out(n);
  auto dft = [&](cpx<V>(&v)[32], int len) {
    if (ls.maxl <= 16) {
      cpx<V> u[16];
      for (int i = 0; i < 16; ++i) u[i] = v[i];
      line_dft<V, 16>(u, len);
      for (int i = 0; i < 16; ++i) v[i] = u[i];
    } else {
      line_dft<V, 32>(v, len);
    }
  };
  const int a1 = fwd ? n2 : n1, l1 = fwd ? n1 : n2;
  for (int t = 0; t < a1; ++t) {
    cpx<V> v[32];
    for (int m = 0; m < l1; ++m) v[m] = in[t + a1 * m];
    dft(v, l1);
    for (int k = 0; k < l1; ++k) buf[fwd ? t + P * k : P * t + k] = to_second(k ? v[k] * tw_of<V>(t * k, n) : v[0], shift);
  }
  for (int t = 0; t < l1; ++t) {
    cpx<V> v[32];
    for (int m = 0; m < a1; ++m) v[m] = buf[fwd ? m + P * t : t + P * m];
    dft(v, a1);
    for (int m = 0; m < a1; ++m) out[t + l1 * m] = v[m];
  }
  return out;
}

static void check(int n, int kind, bool fwd, bool inv) {
  std::vector<C> x = input(n, kind);
  std::vector<cpx<double>> d(n);
  for (int i = 0; i < n; ++i)
    d[i] = inv ? mk<double>(x[i].imag(), x[i].real()) : mk<double>(x[i].real(), x[i].imag());
  // the scale as the first step's threads form it
  const LineShape ls = line_shape(n);
  const int nt = fwd ? ls.n2 : ls.n1, len = n / nt;
  unsigned part[32];
  for (int t = 0; t < nt; ++t) {
    cpx<double> v[32];
    for (int m = 0; m < len; ++m) v[m] = d[t + nt * m];
    part[t] = fx_part<32>(v, len, len, len);
  }
  int em, g1, g2;
  fx_scale(part, nt, em, g1, g2);
  const int k = fx_kexp(em, g2);
  std::vector<cpx<fx>> f(n);
  for (int i = 0; i < n; ++i) f[i] = mk<fx>(to_fx(d[i].re, em, g1), to_fx(d[i].im, em, g1));
  const std::vector<cpx<fx>> F = two_step<fx>(f, fwd, g2 - g1);
  const std::vector<cpx<double>> D = two_step<double>(d, fwd, 0);
  std::vector<C> a(n), b(n);
  for (int i = 0; i < n; ++i) {
    const double re = fx_plain(em) ? from_fx(F[i].re, k) : std::ldexp((double)F[i].re.v, k);
    const double im = fx_plain(em) ? from_fx(F[i].im, k) : std::ldexp((double)F[i].im.v, k);
    a[i] = inv ? C(im, re) : C(re, im);
    b[i] = inv ? C(D[i].im, D[i].re) : C(D[i].re, D[i].im);
  }
  const std::vector<CL> ref = direct(x, inv);
  const double ef = rel(a, ref), ed = rel(b, ref);
  std::printf("err %s%s%d %d %.3e %.3e\n", fwd ? "fwd" : "bwd", inv ? "_inv" : "", kind, n, ef, ed);
  g_sum[kind][0] += ef;
  g_sum[kind][1] += ed;
  // constants and twiddles rounded to FP64 (2^-54 in each component, about five in series) and
  // the rounding of the result (2^-53): 5e-16; and on average no worse than FP64 arithmetic
  if (!(ef <= 5e-16)) {
    std::printf("FAIL %d %d\n", n, kind);
    g_bad = 1;
  }
}

// exp(2 pi i u): 2^-53 of a component (its own rounding) and 2^-58 of the fixed-point steps
static void check_turns() {
  const long double pi = acosl(-1.0L);
  unsigned s = 99;
  long double worst = 0;
  for (int i = 0; i < 400000; ++i) {
    const double scale[8] = {1e-3, 0.1, 1.0, 7.0, 1e-9, 100.0, 1e4, 1e-17};
    double u = (rnd(s) + rnd(s) * 1e-7) * scale[i & 7];
    if (i < 4096) u = i / 2048.0 - 1.0;                      // table points and midpoints
    if (i >= 4096 && i < 8192) u = std::nextafter((i - 6144) / 2048.0, 1e3);
    const cpx<double> t = turn_of(u);
    const long double f = (long double)u - rintl((long double)u);
    worst = std::fmax(worst, std::fmax(fabsl(t.re - cosl(2 * pi * f)), fabsl(t.im - sinl(2 * pi * f))));
  }
  const double inf = HUGE_VAL;
  const bool nan = std::isnan(turn_of(inf).re) && std::isnan(turn_of(-inf).im) && std::isnan(turn_of(inf - inf).re);
  std::printf("turn_err %.3Le\n", worst);
  if (!(worst <= 1.2e-16L) || !nan) g_bad = 1;
}

// exp(i k a) through turns: the rounding of u = a k / (2 pi) alone, 2^-53 of it (and
// 2^-61, the part of the scale's rest that is cut off), beside the turn's own error
static void check_scaled_turns() {
  const long double pi = acosl(-1.0L);
  unsigned s = 7;
  long double worst = 0;
  for (int i = 0; i < 400000; ++i) {
    const double scale[4] = {0.05, 1.0, 30.0, 1e3};
    const double k = (i & 4 ? -1.0 : 1.0) * (0.1 + std::fabs(rnd(s)) * 5.0), a = rnd(s) * scale[i & 3];
    const TurnScale t = turn_scale(k);
    const cpx<double> e = turn_of(a * t.k, t.rest);
    const long double x = (long double)a * k, u = fabsl(x / (2 * pi));
    const long double bound = 1.2e-16L + 2 * pi * u * 1.01L / 9007199254740992.0L;
    worst = std::fmax(worst, std::fmax(fabsl(e.re - cosl(x)), fabsl(e.im - sinl(x))) / bound);
  }
  std::printf("scaled_turn_err %.3Lf of the bound\n", worst);
  if (!(worst <= 1.0L)) g_bad = 1;
}

int main() {
  check_turns();
  check_scaled_turns();
  for (int n = 2; n <= 1024; ++n) {
    if (line_shape(n).maxl == 0) continue;
    if (n > 400 && n % 16 && n != 405 && n != 450 && n != 500 && n != 750) continue;
    for (int kind = 0; kind < 6; ++kind) {
      check(n, kind, false, true);
      check(n, kind, true, false);
    }
  }
  for (int k = 0; k < 6; ++k)
    if (!(g_sum[k][0] <= g_sum[k][1])) g_bad = 1;
  std::printf(g_bad ? "BAD\n" : "OK\n");
  return g_bad;
}
