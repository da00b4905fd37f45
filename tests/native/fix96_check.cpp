// Host check of the potential's fixed-point inverse distance (f64emu.cuh):
// inv_distance_fix96 of two positions against (|a - b|^2 + eps^2)^(-1/2) in long double.
//
//   fix96_check <cases> <mode> <rng seed>
//
// Prints "taken refused worst", worst in units of 2^-53.  Modes: 0 positions over the whole
// box, 1 one a hair from the other (down to 2^-26 of the box) beside a softening, 2 the
// same without softening (down to 2^-30: some below the reach), 3 zero, -0 and equal
// coordinates, 4 coordinates at the box's edge, 5 softening as large as the box, 6
// differences below 2^-33 of the box without softening: all to be refused.
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
  const int mode = atoi(argv[2]);
  g_rng = 88172645463325252ull + 2654435761ull * (uint64_t)atoll(argv[3]);
  long long taken = 0, refused = 0;
  double worst = 0.0;
  for (long long i = 0; i < cases; i++) {
    const int E = (int)(uniform() * 240) - 120;
    const double box = ldexp(1.0, E);
    double a[3], b[3], eps = box * ldexp(1.0 + uniform(), -1 - (int)(uniform() * 29));
    for (int k = 0; k < 3; k++) {
      a[k] = box * (2.0 * uniform() - 1.0) * 0.99;
      b[k] = box * (2.0 * uniform() - 1.0) * 0.99;
      if (mode == 1) b[k] = a[k] * (1.0 + ldexp(uniform() - 0.5, -(int)(uniform() * 26)));
      if (mode == 2) b[k] = a[k] * 0.5 + 0.49 * box * (uniform() - 0.5), b[k] = a[k] + ldexp(b[k], -(int)(uniform() * 30));
      if (mode == 4) a[k] = (uniform() < 0.5 ? -1 : 1) * nextafter(box, 0.0), b[k] = -a[k];
      if (mode == 6) b[k] = a[k] + box * ldexp(uniform(), -34);
      if (mode == 2 || mode == 4)
        if (!(fabs(b[k]) < box)) b[k] = 0.5 * a[k];
    }
    if (mode == 3) {
      a[i % 3] = 0.0;
      b[(i + 1) % 3] = -0.0;
      if (i & 4) b[i % 3] = a[i % 3];
      if (i & 8) b[(i + 2) % 3] = a[(i + 2) % 3];
    }
    if (mode == 2 || mode == 6) eps = 0.0;
    if (mode == 5) eps = box * (0.5 + 0.49 * uniform());
    int Ee;
    uint64_t W;
    double got;
    if (!align_eps2(eps * eps, Ee, W)) return 1;
    const int room = W ? E - (Ee - 1023) : 1 << 20;
    Fix96 fa[3], fb[3];
    for (int k = 0; k < 3; k++) {
      fa[k] = to_fix96(a[k], E);
      fb[k] = to_fix96(b[k], E);
    }
    if (room < 0 || !inv_distance_fix96(fa, fb, E, room, W, got)) {
      refused++;
      continue;
    }
    taken++;
    long double s = (long double)(eps * eps);
    for (int k = 0; k < 3; k++) {
      const long double d = (long double)a[k] - b[k];
      s += d * d;
    }
    const long double want = 1.0L / sqrtl(s);
    const double err = (double)(fabsl(((long double)got - want) / want) * 0x1p53L);
    if (!(err <= worst)) worst = err;
  }
  printf("%lld %lld %.6f\n", taken, refused, worst);
  return 0;
}
