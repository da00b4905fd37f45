// Host check of the tree walk's factor for massless particles (f64emu.cuh):
// zero_mass_inv_cube(m, d, eps^2) gives m for m = +-0 exactly where mass_inv_cube takes a
// mass of 1, and refuses every other mass.
//
//   zero_mass_check <cases> <rng seed>
//
// Prints "taken refused wrong".
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include "../../gravhopper_gb300/csrc/f64emu.cuh"

static uint64_t g_rng;
static double uniform() {
  g_rng ^= g_rng << 13;
  g_rng ^= g_rng >> 7;
  g_rng ^= g_rng << 17;
  return (double)(g_rng >> 11) * 0x1p-53;
}

int main(int argc, char** argv) {
  using namespace gh::emu;
  const long long cases = atoll(argv[1]);
  g_rng = 88172645463325252ull + 2654435761ull * (uint64_t)atoll(argv[2]);
  const double special[6] = {0.0, -0.0, NAN, INFINITY, 1e-310, 1e300};
  const double other[6] = {1.0, -1.0, NAN, INFINITY, 5e-324, -1e-310};
  long long taken = 0, refused = 0, wrong = 0;
  for (long long i = 0; i < cases; i++) {
    const int e = (int)(uniform() * 340) - 170;  // beyond 2^-150 .. 2^151 at both ends
    double d[3], eps2 = 0.0;
    for (int k = 0; k < 3; k++) {
      d[k] = (uniform() < 0.5 ? -1.0 : 1.0) * ldexp(1.0 + uniform(), e - (int)(uniform() * 4));
      if (uniform() < 0.1) d[k] = special[(int)(uniform() * 6)];
    }
    if (uniform() < 0.5) eps2 = pow(ldexp(1.0 + uniform(), (int)(uniform() * 290) - 145), 2);
    int Ee;
    uint64_t W;
    if (!align_eps2(eps2, Ee, W)) return 1;
    const double m = i & 1 ? -0.0 : 0.0;
    double got = 7.0, one;
    const bool take = zero_mass_inv_cube(m, d[0], d[1], d[2], Ee, got);
    take ? taken++ : refused++;
    wrong += take != mass_inv_cube(1.0, d[0], d[1], d[2], Ee, W, one);
    wrong += take && dbits(got) != dbits(m);
    wrong += zero_mass_inv_cube(other[i % 6], d[0], d[1], d[2], Ee, got);
  }
  printf("%lld %lld %lld\n", taken, refused, wrong);
  return 0;
}
