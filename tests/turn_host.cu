// Host check of the integer turns' modulus and angle (dtmm_gb300/csrc/dtmm_fx.cuh,
// fx_turn_at) against long double: random fractions of a turn and the far ends
// of the table's intervals.  An error of the modulus has the same sign in every
// phase of a transfer.  Prints the largest errors and "OK".
#include <cmath>
#include <cstdio>

#include "dtmm_fx.cuh"

using namespace dtmm;

int main() {
  unsigned long long s = 1;
  long double radial = 0, tangential = 0;
  for (int i = 0; i < 400000; ++i) {
    s = s * 6364136223846793005ULL + 1442695040888963407ULL;
    unsigned long long f = s;
    if (i < 2048) f = ((unsigned long long)i << 53) + (i & 1 ? -(1ULL << 40) : (1ULL << 40));
    const cpx<fx> t = fx_turn_at(f);
    const long double a = 2 * M_PIl * ((long double)(long long)f / 18446744073709551616.0L);
    const long double c = std::cos(a), n = std::sin(a);
    const long double dx = t.re.v / 4611686018427387904.0L - c, dy = t.im.v / 4611686018427387904.0L - n;
    radial = fmaxl(radial, fabsl(dx * c + dy * n));
    tangential = fmaxl(tangential, fabsl(dy * c - dx * n));
  }
  // radial: the next term d^6 / 720 (2^-59.6), the table (2^-60.6) and last places (2^-61); tangential:
  // the 38-bit d and 47-bit d^2 of d^3 / 6 (2^-57.3, 2^-57.9) and as much
  const bool ok = radial <= 0x1p-58L && tangential <= 0x1p-56L;
  std::printf("radial %.3Le tangential %.3Le\n%s\n", radial, tangential, ok ? "OK" : "BAD");
  return !ok;
}
