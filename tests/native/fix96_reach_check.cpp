// Host check of inv_distance_fix96 (f64emu.cuh) where its fixed-point differences run out of
// bits, with the device's seed: no range check on the seed's residual, and an error of the
// FP32 approximation up to the 2^-22.9 that the instruction may have.
//
//   fix96_reach_check <cases> <mode> <rng seed>
//
// Prints "taken refused worst near", worst in units of 2^-53, near = the cases whose
// sqrt(d^2 + eps^2) is at least 2^-31 of the box (all to be taken).  sqrt(d^2 + eps^2) runs
// from 2^-33 to 2^-29 of the box: mode 0 without softening, 1 with one of any share, 2 with
// nothing else (coincident positions).
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

static uint64_t g_rng;
static double uniform() {
  g_rng ^= g_rng << 13;
  g_rng ^= g_rng >> 7;
  g_rng ^= g_rng << 17;
  return (double)(g_rng >> 11) * 0x1p-53;
}
static float device_seed(float x) {
  return (float)(1.0 / sqrt((double)x) * (1.0 + (2.0 * uniform() - 1.0) * 0x1p-22 * 0.535));
}
#define GH_EMU_HOST_RSQRT(x) device_seed(x)
#define GH_EMU_DEVICE_SEED
#include "../../gravhopper_gb300/csrc/f64emu.cuh"

int main(int argc, char** argv) {
  using namespace gh::emu;
  const long long cases = atoll(argv[1]);
  const int mode = atoi(argv[2]);
  g_rng = 88172645463325252ull + 2654435761ull * (uint64_t)atoll(argv[3]);
  long long taken = 0, refused = 0, near = 0;
  double worst = 0.0;
  for (long long i = 0; i < cases; i++) {
    const int E = (int)(uniform() * 180) - 60;
    const double box = ldexp(1.0, E), reach = box * exp2(-33.0 + 4.0 * uniform());
    const double share = mode == 0 ? 1.0 : (mode == 1 ? uniform() : 0.0);
    const double eps = reach * sqrt(1.0 - share);
    double a[3], b[3], u[3], r = 0.0;
    for (int k = 0; k < 3; k++) {
      u[k] = 2.0 * uniform() - 1.0;
      r += u[k] * u[k];
    }
    for (int k = 0; k < 3; k++) {
      a[k] = 0x1p-20 * box * (2.0 * uniform() - 1.0);
      b[k] = a[k] + reach * sqrt(share / r) * u[k];
    }
    long double s = (long double)(eps * eps);
    for (int k = 0; k < 3; k++) {
      const long double d = (long double)a[k] - b[k];
      s += d * d;
    }
    near += sqrtl(s) >= (long double)box * 0x1p-31L;
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
    if (!inv_distance_fix96(fa, fb, E, room, W, got)) {
      refused++;
      continue;
    }
    taken++;
    const long double want = 1.0L / sqrtl(s);
    const double err = (double)(fabsl(((long double)got - want) / want) * 0x1p53L);
    if (!(err <= worst)) worst = err;
  }
  printf("%lld %lld %.6f %lld\n", taken, refused, worst, near);
  return 0;
}
