// Host check of the pair-arithmetic eigenvalues (dtmm_gb300/csrc/dtmm_lean.cuh)
// against the roots in long double: random uniaxial voxels and beams (normal
// incidence, beta up to 0.8, optic axis along z and in the plane, nearly
// isotropic, index-matched to the effective medium), with and without the beam
// correction.  Prints the largest errors and "OK".
#include <cmath>
#include <cstdio>

#include "dtmm_lean.cuh"

using namespace dtmm;

static double rnd(unsigned long long& s) {
  s = s * 6364136223846793005ULL + 1442695040888963407ULL;
  return (s >> 11) / 9007199254740992.0;
}

int main() {
  unsigned long long s = 7;
  double worst = 0, worst_rec = 0;
  int bad = 0;
  for (int i = 0; i < 400000; ++i) {
    const double e0 = 1.9 + 0.7 * rnd(s);
    double dl = -0.3 + 1.1 * rnd(s);
    if (i % 7 == 1) dl = 1e-5 * (rnd(s) - 0.5);
    const double e2 = e0 + dl;
    double th = M_PI * rnd(s), az = 2 * M_PI * rnd(s), beta = 0.8 * rnd(s);
    if (i % 5 == 1) beta = 0;
    if (i % 11 == 2) th = 0;
    if (i % 11 == 3) th = M_PI / 2;
    const double phi = 2 * M_PI * rnd(s);
    const bool plain = i % 13 == 4;
    const double eps = i % 17 == 5 ? e0 : 2.0 + 0.6 * rnd(s);
    const double a = plain ? 0.0 : std::sqrt(eps - beta * beta);
    LeanVoxel v;
    v.ct = ff_of(std::cos(th));
    v.st = ff_of(std::sin(th));
    v.ca = ff_of(std::cos(az));
    v.sa = ff_of(std::sin(az));
    lean_voxel(v, ff_of(e0), ff_of(e2 - e0), ff_of(e0 * (e2 - eps)));
    const ff c2 = ff_mul(ff_of(e0), ff_sub(ff_of(e2), ff_of(beta * beta)));
    ff dp, dm;
    lean_roots<true>(v, ff_of(a), ff_of(beta * std::cos(phi)), ff_of(beta * std::sin(phi)), c2, plain ? c2 : v.cv, dp, dm);
    const long double ct = cosl(th), st = sinl(th), g = (long double)beta * cosl((long double)az - phi), d = (long double)e2 - e0;
    const long double al = plain ? 0.0L : sqrtl((long double)eps - (long double)beta * beta);
    const long double u = e0 + d * ct * ct, k = d * st * ct;
    const long double q = u * e0 * (e2 - (long double)beta * beta) - e0 * d * st * st * g * g;
    const long double p = (-k * g + sqrtl(q)) / u - al, m = (-k * g - sqrtl(q)) / u + al;
    const double ep = (double)fabsl((long double)dp.h + dp.l - p), em = (double)fabsl((long double)dm.h + dm.l - m);
    worst = std::fmax(worst, std::fmax(ep, em));
    // the FP32 record: its own rounding (2^-24) and no more than 1e-3 of that beside it, or the pair's floor
    const double rp = (double)fabsl((long double)ff_f(dp) - p), rm = (double)fabsl((long double)ff_f(dm) - m);
    const double tp = 5.97e-8 * 1.001 * fabsl(p) + 2e-13, tm = 5.97e-8 * 1.001 * fabsl(m) + 2e-13;
    worst_rec = std::fmax(worst_rec, std::fmax(rp / tp, rm / tm));
    if (!(ep < 2e-13 && em < 2e-13 && rp <= tp && rm <= tm)) ++bad;
  }
  std::printf("worst %.3e record %.4f of its bound\n%s\n", worst, worst_rec, bad ? "BAD" : "OK");
  return bad != 0;
}
