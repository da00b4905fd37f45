// Host check of the tree walk's fixed-point interaction factor (f64emu.cuh):
// mass_inv_cube(m, d, eps^2) against m (|d|^2 + eps^2)^(-3/2) in long double.
//
//   walk_factor_check <cases> <mode> <rng seed>
//
// Prints "taken refused worst", worst = the largest relative error of a taken case in
// units of 2^-53.  Modes: 0 ordinary offsets, 1 components up to 2^100 apart, 2 softening
// from far below to far above the offset, 3 one or two zero components, 4 zero offset,
// 5 offsets and softening at the edges of the accepted range, 6 inputs to be refused.
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include "../../gravhopper_gb300/csrc/f64emu.cuh"

static uint64_t g_rng;
static double uniform() {  // [0, 1)
  g_rng ^= g_rng << 13;
  g_rng ^= g_rng >> 7;
  g_rng ^= g_rng << 17;
  return (double)(g_rng >> 11) * 0x1p-53;
}
static double sign() { return uniform() < 0.5 ? -1.0 : 1.0; }
static double mant() { return sign() * (1.0 + uniform()); }

int main(int argc, char** argv) {
  const long long cases = atoll(argv[1]);
  const int mode = atoi(argv[2]);
  g_rng = 88172645463325252ull + 2654435761ull * (uint64_t)atoll(argv[3]);
  long long taken = 0, refused = 0;
  double worst = 0.0;
  for (long long i = 0; i < cases; i++) {
    double d[3], eps = uniform() < 0.3 ? 0.0 : ldexp(1.0 + uniform(), -3), m = mant() * ldexp(1.0, (int)(uniform() * 60) - 30);
    for (int k = 0; k < 3; k++) d[k] = mant() * ldexp(1.0, (int)(uniform() * 6));
    if (mode == 1)
      for (int k = 0; k < 3; k++) d[k] = mant() * ldexp(1.0, (int)(uniform() * 200) - 100);
    if (mode == 2) eps = ldexp(1.0 + uniform(), (int)(uniform() * 200) - 100);
    if (mode == 3) {
      d[i % 3] = 0.0;
      if (i & 8) d[(i + 1) % 3] = -0.0;
    }
    if (mode == 4) {
      d[0] = d[1] = d[2] = 0.0;
      eps = ldexp(1.0 + uniform(), (int)(uniform() * 200) - 100);
    }
    if (mode == 5) {
      const int e = i & 1 ? -150 : 150;
      for (int k = 0; k < 3; k++) d[k] = mant() * ldexp(1.0, e < 0 ? e + (int)(uniform() * 2) : e - (int)(uniform() * 2));
      if (i & 2) eps = ldexp(1.0 + 0.999 * uniform(), e < 0 ? e : e - 1);
      m = mant() * ldexp(1.0, i & 4 ? -500 : 500);
    }
    if (mode == 6) {
      const double bad[6] = {NAN, INFINITY, -INFINITY, 0x1p152, 1e300, 0.0};
      const int b = (int)(i % 6);
      if (b < 5) d[i % 3] = bad[b];
      if (b == 5) {  // zero distance, no softening; or a zero, subnormal, huge or NaN mass
        eps = 0.0;
        const double bm[4] = {0.0, 1e-310, 1e200, NAN};
        const int q = (int)(i / 6 % 5);
        if (q < 4) m = bm[q];
        else d[0] = d[1] = d[2] = 0.0;
      }
    }
    const double eps2 = eps * eps;
    int Ee;
    uint64_t W;
    double got;
    if (!gh::emu::align_eps2(eps2, Ee, W) || !gh::emu::mass_inv_cube(m, d[0], d[1], d[2], Ee, W, got)) {
      refused++;
      continue;
    }
    taken++;
    long double s = eps2;
    for (int k = 0; k < 3; k++) s += (long double)d[k] * d[k];
    const long double want = (long double)m / (s * sqrtl(s));
    const double err = (double)(fabsl(((long double)got - want) / want) * 0x1p53L);
    if (!(err <= worst)) worst = err;
  }
  printf("%lld %lld %.6f\n", taken, refused, worst);
  return 0;
}
