// Eigenvalues of a uniaxial voxel against the effective medium's, for FP32
// records.
//
// The records hold (alpha - a) d, a small difference between an eigenvalue of
// dtmm/tmm.py:157-278 and the effective medium's a = sqrt(eps - beta^2).  With the
// roots alpha+- = (-k gamma +- sqrt(q)) / u, q = u c2 - e0 delta sin^2 gamma^2, u = e0 +
// delta cos^2, k = delta sin cos, c2 = e0 (e2 - beta^2), gamma = beta cos(az - phi) and delta = e2 - e0,
// multiplying by the conjugate gives it without cancellation of the roots:
//   alpha+ - a = (e0 (e2 - eps) - delta (a cos + gamma sin)^2) / (sqrt(q) + a u + k gamma)
//   alpha- + a = -(the same with -gamma)
// and, for the ordinary mode, evs - a = (e0 - eps) / (evs + a).  Every factor is
// carried as a pair of FP32 numbers (about 2^-45), so that the stored FP32
// records round the same values as an FP64 solve.  Without a beam correction
// a = 0 and eps = beta^2: the first term is c2.
#pragma once

#include "dtmm_common.cuh"

namespace dtmm {

struct LeanVoxel {
  ff ca, sa, ct, st;      // cos / sin of the azimuth and of theta
  ff u, kv, qb, dl, cv;   // e0 + delta cos^2, delta sin cos, e0 delta sin^2, delta, e0 (e2 - eps)
};

__host__ __device__ __forceinline__ void lean_voxel(LeanVoxel& v, ff e0, ff dl, ff cv) {
  const ff ds = ff_mul(dl, v.st);
  v.u = ff_add(e0, ff_mul(dl, ff_mul(v.ct, v.ct)));
  v.kv = ff_mul(ds, v.ct);
  v.qb = ff_mul(e0, ff_mul(ds, v.st));
  v.dl = dl;
  v.cv = cv;
}

// dp = alpha+ - a and, with FOUR, dm = alpha- + a for the beam (a, beta cos phi, beta sin phi)
template <bool FOUR>
__host__ __device__ __forceinline__ void lean_roots(const LeanVoxel& v, ff a, ff bcp, ff bsp, ff c2, ff num, ff& dp,
                                                    ff& dm) {
  const ff gm = ff_add(ff_mul(v.ca, bcp), ff_mul(v.sa, bsp));
  const ff q = ff_sub(ff_mul(v.u, c2), ff_mul(v.qb, ff_mul(gm, gm)));
  const ff den = ff_add(ff_sqrt(q), ff_mul(a, v.u)), kg = ff_mul(v.kv, gm);
  const ff ac = ff_mul(a, v.ct), gs = ff_mul(gm, v.st);
  const ff tp = ff_add(ac, gs);
  dp = ff_div(ff_sub(num, ff_mul(v.dl, ff_mul(tp, tp))), ff_add(den, kg));
  if (FOUR) {
    const ff tm = ff_sub(ac, gs);
    dm = ff_div(ff_sub(ff_mul(v.dl, ff_mul(tm, tm)), num), ff_sub(den, kg));
  }
}

}  // namespace dtmm
