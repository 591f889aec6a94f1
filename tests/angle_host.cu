// Host check of the pairs of sines and cosines of the director angles
// (dtmm_gb300/csrc/dtmm_fx.cuh fx_angle, dtmm_common.cuh ff_q62) against long
// double: angles of every size that fx_angle takes, 0 and both signs.  Prints
// the largest error over its bound and "OK".
#include <cmath>
#include <cstdio>

#include "dtmm_fx.cuh"

using namespace dtmm;

static double rnd(unsigned long long& s) {
  s = s * 6364136223846793005ULL + 1442695040888963407ULL;
  return (s >> 11) / 9007199254740992.0;
}

int main() {
  unsigned long long s = 3;
  long double worst = 0;
  int bad = 0;
  for (int i = 0; i < 400000; ++i) {
    double a = (rnd(s) - 0.5) * 2.0;
    a *= std::ldexp(1.0, i % 60 - 39);  // up to 2^20, down to 2^-40
    if (i % 7 == 1) a = (rnd(s) - 0.5) * 4.0 * M_PI;
    if (i % 1000 == 2) a = (i / 1000) * (M_PI / 8);
    if (i == 0) a = 0.0;
    if (i == 1) a = std::nextafter(2097152.0, 0.0);
    if (!fx_angle_ok(a)) ++bad;
    const cpx<fx> t = fx_angle(a);
    const ff c = ff_q62(t.re.v), n = ff_q62(t.im.v);
    const long double ec = fabsl((long double)c.h + c.l - std::cos((long double)a));
    const long double en = fabsl((long double)n.h + n.l - std::sin((long double)a));
    const long double tol = fabsl((long double)a) * 0x1p-64L + 0x1p-58L + 0x1p-48L;
    worst = fmaxl(worst, fmaxl(ec, en) / tol);
    if (!(ec <= tol && en <= tol)) ++bad;
  }
  const double inf = HUGE_VAL;
  if (fx_angle_ok(2097152.0) || fx_angle_ok(-4e9) || fx_angle_ok(inf) || fx_angle_ok(inf - inf)) ++bad;
  std::printf("worst %.3Lf of its bound\n%s\n", worst, bad ? "BAD" : "OK");
  return bad != 0;
}
