// Correctly rounded FP64 reciprocal, square root and quotient on the integer
// pipes, for the softened inverse cube of the FP64 direct sum:
//
//     inv = RN( RN(1/s) / RN(sqrt(s)) )      (gravhopper/_jbgrav.c:166, :330)
//
// GB300 issues FP64 at 1/74 of the FP32 rate, and the two IEEE divisions and the
// square root take more than half of the FP64 instructions of a pair.  Here the
// three results are computed from the double's integer significand instead:
//
//   1. seed y0 ~ 1/sqrt(n) from the FP32 rsqrt approximation, n = N 2^-52 in [1, 4);
//   2. two Newton-Raphson steps for the reciprocal square root in 64-bit fixed
//      point, y' = y + y (1 - n y^2) / 2 (relative error below 2^-59);
//   3. each result from y: sqrt(n) = n y, 1/n = y^2, A/B = A y 2^-52 (one extra
//      residual correction for the quotient, whose divisor is the rounded root);
//   4. the round-to-nearest significand m of each result is confirmed by the sign of
//      exact integer remainders at the rounding boundaries 2m -+ 1 (scaled), the
//      textbook exact-rounding test for division and square root (J.-M. Muller et
//      al., Handbook of Floating-Point Arithmetic, 2nd ed., sections 4.7 and 5.4;
//      P. Markstein, IBM J. Res. Dev. 34 (1990) 111).  Quotients and square roots of
//      53-bit significands never fall on a midpoint, so no tie rule is needed.
//
// The remainders are exact modulo 2^64 and every one is proven smaller than 2^57 in
// magnitude once the first Newton residual passes its range check, so a confirmed
// result is the IEEE result.  When a check fails, or s lies outside [2^-577, 2^602)
// (zero, subnormal, negative, infinite, NaN and the far ranges included), the
// function returns false and the caller takes the native IEEE operations.
#pragma once

#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define GH_EMU_HD __host__ __device__ __forceinline__
#else
#define GH_EMU_HD inline
#endif

#ifndef __CUDA_ARCH__
#include <math.h>
// FP32 reciprocal square root used as the seed by host builds (unit tests); a test
// may define this to perturb the seed and exercise the range checks.
#ifndef GH_EMU_HOST_RSQRT
#define GH_EMU_HOST_RSQRT(x) (1.0f / sqrtf(x))
#endif
#endif

namespace gh {
namespace emu {

GH_EMU_HD uint64_t umulhi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

GH_EMU_HD uint64_t dbits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}

GH_EMU_HD double bitsd(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}

GH_EMU_HD float bitsf(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  memcpy(&x, &u, 4);
  return x;
#endif
}

GH_EMU_HD uint32_t fbits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  uint32_t u;
  memcpy(&u, &x, 4);
  return u;
#endif
}

GH_EMU_HD float rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return GH_EMU_HOST_RSQRT(x);
#endif
}

// Reciprocal square root in fixed point: for s = M 2^(E - 1075) (M in [2^52, 2^53))
// writes s = N 2^p with p even and N in [2^52, 2^54), and Y2 = 2^63 / sqrt(n),
// n = N 2^-52, to a relative error below 2^-59; false when the seed check fails.
GH_EMU_HD bool rsqrt_fixed(int E, uint64_t M, int& odd, uint64_t& N, int& p, uint64_t& Y2) {
  odd = ~E & 1;  // s = M 2^(E - 1075); E - 1075 is odd when E is even
  N = M << odd;
  p = E - 1075 - odd;

  // seed: y0 ~ 1/sqrt(n), n = N 2^-52, as Y0 = y0 2^30
  const float nf = bitsf(0x3F800000u + ((uint32_t)odd << 23) + ((uint32_t)(M >> 29) & 0x7FFFFFu));
  const uint32_t rb = fbits(rsqrt_seed(nf));
  const uint32_t ex = (rb >> 23) & 0xFFu;
  if (ex - 121u > 6u) return false;  // y0 in [2^-6, 2)
  const int32_t Y0 = (int32_t)(((rb & 0x7FFFFFu) | 0x800000u) << (ex - 120u));

  // Newton step 1: h = 1 - n y0^2 as H = h 2^60; Y1 = y1 2^63
  const uint64_t Y0sq = (uint64_t)((int64_t)Y0 * Y0);  // y0^2 2^60 <= 2^60
  const int64_t H = (int64_t)((1ull << 60) - umulhi(N << 10, Y0sq << 2));
  if ((uint64_t)(H + (1ll << 41)) >= (1ull << 42)) return false;  // |h| < 2^-19
  uint64_t Y1 = ((uint64_t)Y0 << 33) + (uint64_t)(((int64_t)Y0 * (int32_t)(H >> 10)) >> 18);
  if (Y1 >= (1ull << 63)) Y1 = (1ull << 63) - 1;

  // Newton step 2: h2 = 1 - n y1^2 as H2 = h2 2^62 (|h2| < 2^-37, fits 32 bits)
  const uint64_t Y1sq = umulhi(Y1, Y1);  // y1^2 2^62 < 2^62
  const int32_t H2 = (int32_t)(uint32_t)((1ull << 62) - umulhi(N << 10, Y1sq << 2));
  Y2 = Y1 + (uint64_t)(((int64_t)(int32_t)(Y1 >> 32) * H2) >> 31);
  if (Y2 >= (1ull << 63)) Y2 = (1ull << 63) - 1;
  return true;
}

// RN(RN(1/s) / RN(sqrt(s))) into `out` for s = M 2^(E - 1075) with M in
// [2^52, 2^53) and 446 <= E <= 1624 (the caller checks the range); false when a
// check fails (then `out` is untouched).
GH_EMU_HD bool inv_cube_core(int E, uint64_t M, double& out) {
  int odd, p;
  uint64_t N, Y2;
  if (!rsqrt_fixed(E, M, odd, N, p, Y2)) return false;

  // square root: sqrt(s) = B 2^(p/2 - 26), B = RN(sqrt(X) / 2), X = N 2^54, i.e.
  // c = 2B - 1 <= sqrt(X) < c + 2
  uint64_t B = (umulhi(N << 2, Y2) + 1) >> 1;
  {
    const uint64_t c = 2 * B - 1;
    const int64_t R = (int64_t)((N << 54) - c * c);  // X - c^2
    if (R < 0) {
      if (R + (int64_t)(4 * c) - 4 < 0) return false;
      B--;
    } else if (R >= (int64_t)(4 * c + 4)) {
      if (R >= (int64_t)(8 * c + 16)) return false;
      B++;
    }
  }

  // reciprocal: 1/s = A 2^(970 - E), A = RN(2^105 / M) in [2^52, 2^53], i.e.
  // c = 2A - 1 <= 2^106 / M < c + 2
  uint64_t A = ((umulhi(Y2, Y2) >> (8 - odd)) + 1) >> 1;
  {
    const uint64_t c = 2 * A - 1;
    const int64_t R = (int64_t)(0 - c * M);  // 2^106 - c M
    if (R < 0) {
      if (R + (int64_t)(2 * M) < 0) return false;
      A--;
    } else if (R >= (int64_t)(2 * M)) {
      if (R >= (int64_t)(4 * M)) return false;
      A++;
    }
  }

  // quotient: Qx = A 2^54 / B in (2^53, 2^55]; inv = RN(Qx 2^-sh) 2^(sh - 54 + a - b)
  const uint64_t A54 = A << 54;  // A 2^54 mod 2^64
  uint64_t Q = umulhi(A << 3, Y2);  // A 2^54 / (sqrt(n) 2^52): within 6 of Qx
  {
    const int64_t R0 = (int64_t)(A54 - Q * B);  // A 2^54 - Q B, |.| < 2^56
    Q += (uint64_t)(((int64_t)(int32_t)(R0 >> 26) * (int64_t)(int32_t)(Y2 >> 32)) >> 57);  // + R0 / B
  }
  const int sh = A >= B ? 2 : 1;
  uint64_t m = (Q + (1ull << (sh - 1))) >> sh;
  {
    const uint64_t c = (m << sh) - (1ull << (sh - 1));  // c <= Qx < c + 2^sh
    const int64_t R = (int64_t)(A54 - c * B);
    const int64_t W = (int64_t)(B << sh);
    if (R < 0) {
      if (R + W < 0) return false;
      m--;
    } else if (R >= W) {
      if (R >= 2 * W) return false;
      m++;
    }
  }
  const int k = sh - 54 + (970 - E) - (p / 2 - 26);
  out = bitsd(((uint64_t)(k + 1074) << 52) + m);  // m = 2^53 carries into the exponent
  return true;
}

// RN(RN(1/s) / RN(sqrt(s))) into `out`; false when s is out of range or a check
// fails (then `out` is untouched).
GH_EMU_HD bool inv_cube_rn(double s, double& out) {
  const uint64_t bits = dbits(s);
  const int E = (int)(bits >> 52);  // biased exponent; the sign bit makes it >= 2048
  if ((unsigned)(E - 446) > 1178u) return false;  // 2^-577 <= s < 2^602
  return inv_cube_core(E, (bits & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull, out);
}

// s^(-3/2) of a rounded s within about half an ulp (not correctly rounded); false outside
// [2^-577, 2^602).  No kernel takes this or rsqrt1 any more (the tree walk and the potential
// start from the differences, below); the host check holds rsqrt_powers to the same bounds.
GH_EMU_HD bool rsqrt_cube(double s, double& out) {
  const uint64_t bits = dbits(s);
  const int E = (int)(bits >> 52);
  if ((unsigned)(E - 446) > 1178u) return false;
  int odd, p;
  uint64_t N, Y2;
  if (!rsqrt_fixed(E, (bits & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull, odd, N, p, Y2)) return false;
  // y^3 = Y3 2^-62, y = 1/sqrt(n) in (1/2, 1]
  const uint64_t Y3 = umulhi(umulhi(Y2, Y2) << 1, Y2);
#ifdef __CUDA_ARCH__
  const int lz = __clzll((long long)Y3);
#else
  const int lz = __builtin_clzll(Y3);
#endif
  const uint64_t T = Y3 << lz;  // in [2^63, 2^64)
  const uint64_t m = (T >> 11) + ((T >> 10) & 1);  // in [2^52, 2^53]
  // s^(-3/2) = y^3 2^(-3 (26 + p/2)) = m 2^(11 - 62 - lz - 78 - 3p/2)
  const int k = -129 - lz - 3 * (p / 2);
  out = bitsd(((uint64_t)(k + 1074) << 52) + m);
  return true;
}

// s^(-1/2) within about half an ulp; false outside [2^-577, 2^602).
GH_EMU_HD bool rsqrt1(double s, double& out) {
  const uint64_t bits = dbits(s);
  const int E = (int)(bits >> 52);
  if ((unsigned)(E - 446) > 1178u) return false;
  int odd, p;
  uint64_t N, Y2;
  if (!rsqrt_fixed(E, (bits & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull, odd, N, p, Y2)) return false;
#ifdef __CUDA_ARCH__
  const int lz = __clzll((long long)Y2);
#else
  const int lz = __builtin_clzll(Y2);
#endif
  const uint64_t T = Y2 << lz;  // y 2^63 << lz, in [2^63, 2^64)
  const uint64_t m = (T >> 11) + ((T >> 10) & 1);
  // s^(-1/2) = y 2^(-26 - p/2) = m 2^(11 - 63 - lz - 26 - p/2)
  out = bitsd(((uint64_t)(-78 - lz - p / 2 + 1074) << 52) + m);
  return true;
}

// s^(-1) and s^(-3/2), each within about half an ulp (the FP64 adjoint's pair factors);
// false outside [2^-577, 2^602).
GH_EMU_HD bool rsqrt_powers(double s, double& inv1, double& inv3) {
  const uint64_t bits = dbits(s);
  const int E = (int)(bits >> 52);
  if ((unsigned)(E - 446) > 1178u) return false;
  int odd, p;
  uint64_t N, Y2;
  if (!rsqrt_fixed(E, (bits & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull, odd, N, p, Y2)) return false;
  const uint64_t Y2sq = umulhi(Y2, Y2);         // y^2 2^62, y = 1/sqrt(n) in (1/2, 1]
  const uint64_t Y3 = umulhi(Y2sq << 1, Y2);    // y^3 2^62
#ifdef __CUDA_ARCH__
  const int l2 = __clzll((long long)Y2sq), l3 = __clzll((long long)Y3);
#else
  const int l2 = __builtin_clzll(Y2sq), l3 = __builtin_clzll(Y3);
#endif
  const uint64_t T2 = Y2sq << l2, T3 = Y3 << l3;  // in [2^63, 2^64)
  const uint64_t m2 = (T2 >> 11) + ((T2 >> 10) & 1), m3 = (T3 >> 11) + ((T3 >> 10) & 1);
  // s^-1 = y^2 2^(-52 - p) = m2 2^(11 - 62 - l2 - 52 - p),
  // s^(-3/2) = y^3 2^(-3 (26 + p/2)) = m3 2^(11 - 62 - l3 - 78 - 3p/2)
  inv1 = bitsd(((uint64_t)(-103 - l2 - p + 1074) << 52) + m2);
  inv3 = bitsd(((uint64_t)(-129 - l3 - 3 * (p / 2) + 1074) << 52) + m3);
  return true;
}

// ---------------------------------------------------------------------------
// The softened squared distance s = RN(RN(RN(dx^2 + dy^2) + dz^2) + eps^2) with
// every product and sum rounded as the FPU does (round to nearest even).  All terms
// are positive, so a sum needs at most a one-bit renormalisation.  Values are
// (E, M): M in [2^52, 2^53), value M 2^(E - 1075), E the biased exponent.

// RN(d^2) of a normal d = D 2^(Ed - 1075); D^2 is formed exactly from 32-bit halves.
GH_EMU_HD void square_rn(int Ed, uint64_t D, int& E, uint64_t& M) {
  const uint32_t h = (uint32_t)(D >> 32), l = (uint32_t)D;  // h < 2^21
  const uint64_t ll = (uint64_t)l * l;
  const uint64_t x = (uint64_t)(2 * h) * l;  // < 2^54
  const uint64_t lo = ll + (x << 32);
  const uint64_t hi = (uint64_t)h * h + (x >> 32) + (lo < ll);  // D^2 = hi 2^64 + lo, hi in [2^40, 2^42)
  const int big = (int)(hi >> 41);  // D^2 >= 2^105
  uint64_t m;
  uint64_t rest;  // the bits below m, left-aligned
  if (big) {
    m = (hi << 11) | (lo >> 53);
    rest = lo << 11;
  } else {
    m = (hi << 12) | (lo >> 52);
    rest = lo << 12;
  }
  m += (rest >> 63) & (uint64_t)(((rest << 1) != 0) | (m & 1));
  E = 2 * Ed - 1023 + big;  // D^2 2^(2 Ed - 2150) = m 2^(52 + big + 2 Ed - 2150)
  const int carry = (int)(m >> 53);
  M = m >> carry;
  E += carry;
}

// RN(a + b) of two positive normals.
GH_EMU_HD void add_pos_rn(int Ea, uint64_t Ma, int Eb, uint64_t Mb, int& E, uint64_t& M) {
  if (Ea < Eb) {
    const int te = Ea;
    Ea = Eb;
    Eb = te;
    const uint64_t tm = Ma;
    Ma = Mb;
    Mb = tm;
  }
  const int d = Ea - Eb;
  if (d >= 54) {  // b < ulp(a) / 2
    E = Ea;
    M = Ma;
    return;
  }
  const uint64_t bs = Mb << 10;
  const uint64_t S = (Ma << 10) + (bs >> d);  // < 2^64
  const bool lost = (bs & ((1ull << d) - 1)) != 0;
  const int big = (int)(S >> 63);
  uint64_t m, rest;
  if (big) {
    m = S >> 11;
    rest = S << 53;
  } else {
    m = S >> 10;
    rest = S << 54;
  }
  m += (rest >> 63) & (uint64_t)(((rest << 1) != 0) | lost | (m & 1));
  const int carry = (int)(m >> 53);
  M = m >> carry;
  E = Ea + big + carry;
}

// Unpacks a double whose magnitude lies in [2^-250, 2^251) (zero excluded) into
// (E, |significand|); false otherwise.
GH_EMU_HD bool unpack_mid(double d, int& E, uint64_t& M) {
  const uint64_t b = dbits(d);
  E = (int)((b >> 52) & 0x7FF);
  M = (b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
  return (unsigned)(E - 773) <= 500u;
}

// Unpacks the squared softening for pair_inv_cube_rn: E = 0 for eps2 = 0; false
// when eps2 lies outside [2^-500, 2^502) (then the caller uses the native path).
GH_EMU_HD bool unpack_eps2(double eps2, int& E, uint64_t& M) {
  const uint64_t b = dbits(eps2);
  E = (int)(b >> 52);
  M = (b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
  if (b == 0) {
    E = 0;
    return true;
  }
  return (unsigned)(E - 523) <= 1001u;
}

// inv = RN(RN(1/s) / RN(sqrt(s))) with s = RN(RN(RN(dx^2 + dy^2) + dz^2) + eps2),
// the pair factor of gravhopper/_jbgrav.c:159-166.  eps2 is given unpacked
// (eps2_E = 0 for eps2 = 0; otherwise 2^-500 <= eps2 < 2^502).  False when a
// component is zero or outside [2^-250, 2^251), or a check fails.
GH_EMU_HD bool pair_inv_cube_rn(double dx, double dy, double dz, int eps2_E, uint64_t eps2_M, double& out) {
  int ex, ey, ez;
  uint64_t mx, my, mz;
  const bool ok = unpack_mid(dx, ex, mx) & unpack_mid(dy, ey, my) & unpack_mid(dz, ez, mz);
  if (!ok) return false;
  int E1, E2, E;
  uint64_t M1, M2, M;
  square_rn(ex, mx, E1, M1);
  square_rn(ey, my, E2, M2);
  add_pos_rn(E1, M1, E2, M2, E, M);
  square_rn(ez, mz, E1, M1);
  add_pos_rn(E, M, E1, M1, E2, M2);
  if (eps2_E) {
    add_pos_rn(E2, M2, eps2_E, eps2_M, E, M);
  } else {
    E = E2;
    M = M2;
  }
  return inv_cube_core(E, M, out);
}

// ---------------------------------------------------------------------------
// Powers of s = dx^2 + dy^2 + dz^2 + eps^2 in 64-bit fixed point, rounded once (the tree
// walk's FP64 interactions, the potential): the differences are aligned at the largest
// exponent e (|d| 2^(62-e) as integers), squared to their top 64 bits and summed, so
// s = S 2^(2e-60) with S to about 2^-58 of s and an exponent that is even as the root
// wants it; then one residual h = 1 - n y0^2 of the FP32 seed, |h| < 2^-20, and a series in h.

GH_EMU_HD int clz64(uint64_t v) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)v);
#else
  return __builtin_clzll(v);
#endif
}

// v >> s, 0 for s > 63.
GH_EMU_HD uint64_t shr_clamp(uint64_t v, int s) {
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
#else
  return s > 63 ? 0 : v >> s;
#endif
}

// a b / 2^64, short by at most 2 (the low halves' product and two carries are left out).
GH_EMU_HD uint64_t umulhi_low(uint64_t a, uint64_t b) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return (uint64_t)ah * bh + (((uint64_t)ah * bl) >> 32) + (((uint64_t)al * bh) >> 32);
}

// The same for signed b, a < 2^63.
GH_EMU_HD int64_t smulhi_low(uint64_t a, int64_t b) {
  const int32_t ah = (int32_t)(a >> 32), bh = (int32_t)(b >> 32);
  const uint32_t al = (uint32_t)a, bl = (uint32_t)b;
  return (int64_t)ah * bh + (int64_t)(((uint64_t)(uint32_t)ah * bl) >> 32) + (((int64_t)al * bh) >> 32);
}

// Top 64 bits of x^2, short by at most 2.
GH_EMU_HD uint64_t square_hi(uint64_t x) {
  const uint32_t h = (uint32_t)(x >> 32), l = (uint32_t)x;
  return (uint64_t)h * h + 2 * (((uint64_t)h * l) >> 32);
}

// eps^2 for the aligned sum: eps^2 = W 2^(2(Ee-1023)-60), W in [2^60, 2^62); W = 0 for
// eps^2 = 0.  False (the caller keeps to FP64) outside [2^-300, 2^300].
GH_EMU_HD bool align_eps2(double eps2, int& Ee, uint64_t& W) {
  const uint64_t b = dbits(eps2);
  const int E = (int)(b >> 52);
  Ee = 0;
  W = 0;
  if (b == 0) return true;
  if ((unsigned)(E - 723) > 600u) return false;
  const int e = E - 1023, half = e >> 1;  // floor(e / 2)
  Ee = half + 1023;
  W = ((b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull) << (8 + (e & 1));
  return true;
}

// s = n 4^e, n = N10 2^-62 in [1, 4); false unless the largest of |dx|, |dy|, |dz|, eps
// lies in [2^-150, 2^151).
GH_EMU_HD bool aligned_norm2(double dx, double dy, double dz, int Ee, uint64_t W, uint64_t& N10, int& e) {
  const uint64_t M52 = 0x000FFFFFFFFFFFFFull, ONE = 0x0010000000000000ull;
  const uint64_t bx = dbits(dx), by = dbits(dy), bz = dbits(dz);
  const int Ex = (int)(bx >> 52) & 0x7FF, Ey = (int)(by >> 52) & 0x7FF, Ez = (int)(bz >> 52) & 0x7FF;
  int E = Ex > Ey ? Ex : Ey;
  E = Ez > E ? Ez : E;
  E = Ee > E ? Ee : E;
  // a zero or subnormal difference has its implicit bit set here, 2^-800 below the rest
  const uint64_t X = shr_clamp(((bx & M52) | ONE) << 10, E - Ex);
  const uint64_t Y = shr_clamp(((by & M52) | ONE) << 10, E - Ey);
  const uint64_t Z = shr_clamp(((bz & M52) | ONE) << 10, E - Ez);
  const uint64_t S = square_hi(X) + square_hi(Y) + square_hi(Z) + shr_clamp(W, 2 * (E - Ee));  // [2^60, 2^64)
  const int big = (S >> 62) != 0;
  N10 = big ? S : S << 2;
  e = E - 1023 + big;
  return (unsigned)(E - 873) <= 300u;
}

// Seed of 1/sqrt(n), n = N10 2^-62, as Y0 = y0 2^30 in (2^29, 2^30], and the residual
// h = 1 - n y0^2 as H = h 2^60.  The approximation (relative error at most 2^-22.9), the
// conversion of n and the seed's 23 bits leave |h| < 2^-20.  The device does not check that,
// so n has to lie in [1, 4); host builds, whose seed may be any, do, unless GH_EMU_DEVICE_SEED
// is defined (tests).
GH_EMU_HD bool rsqrt_seed_residual(uint64_t N10, uint32_t& Y0, uint64_t& Y0sq, int64_t& H) {
  const uint32_t hi = (uint32_t)(N10 >> 32);
#ifdef __CUDA_ARCH__
  const float r = rsqrt_seed(__uint2float_rn(hi));  // y0 2^-15
  Y0 = (fbits(__fmaf_rn(r, 0x1p15f, 1.0f)) - 0x3F800000u) << 7;
#else
  const float r = rsqrt_seed((float)hi);
  Y0 = (fbits(fmaf(r, 0x1p15f, 1.0f)) - 0x3F800000u) << 7;
#endif
  Y0sq = (uint64_t)Y0 * Y0;  // y0^2 2^60, at most a little above 2^60
  H = (int64_t)((1ull << 60) - umulhi_low(N10, Y0sq << 2));
#if defined(__CUDA_ARCH__) || defined(GH_EMU_DEVICE_SEED)
  return true;
#else
  return (uint64_t)(H + (1ll << 40)) < (1ull << 41);
#endif
}

// h^2 2^68 of H = h 2^60, |h| < 2^-20.
GH_EMU_HD uint32_t residual_square(int64_t H) {
  const int32_t h = (int32_t)(H >> 10);
#ifdef __CUDA_ARCH__
  return (uint32_t)__mulhi(h, h);
#else
  return (uint32_t)(((int64_t)h * h) >> 32);
#endif
}

// a (1 + c) for a = A 2^32 and c = C 2^-64, |C| < 2^45 (short by at most 1).
GH_EMU_HD uint64_t scale_up(uint32_t A, int64_t C) {
  const int32_t ch = (int32_t)(C >> 32);
  const uint32_t cl = (uint32_t)C;
  return (((uint64_t)A << 32) | (uint32_t)(((uint64_t)A * cl) >> 32)) + (uint64_t)((int64_t)(int32_t)A * ch);
}

// 1/sqrt(s), s = n 4^e, n = N10 2^-62 in [1, 4), rounded once; false when the seed check of
// host builds fails (rsqrt_seed_residual).
GH_EMU_HD bool inv_root_rn(uint64_t N10, int e, double& out) {
  uint64_t Y0sq;
  uint32_t Y0;
  int64_t H;
  if (!rsqrt_seed_residual(N10, Y0, Y0sq, H)) return false;
  // y = y0 (1 + c), c = h (1/2 + 3/8 h) as C = c 2^64; the next term is below 2^-61
  const int64_t C = (H << 3) + (int64_t)((3 * residual_square(H)) >> 7);
  const uint64_t Y = scale_up(Y0, C);        // y 2^62, in [2^61, 2^62] to rounding
  const uint64_t mant = (Y + 256) >> 9;      // in [2^52, 2^53]; 2^53 carries into the exponent
  out = bitsd(((uint64_t)(1021 - e) << 52) + mant);  // s^(-1/2) = y 2^-e
  return true;
}

// 1/sqrt(dx^2 + dy^2 + dz^2 + eps^2), rounded once (the potential's pairs); false outside
// the range of aligned_norm2.
GH_EMU_HD bool inv_distance(double dx, double dy, double dz, int Ee, uint64_t W, double& out) {
  uint64_t N10;
  int e;
  const bool ok = aligned_norm2(dx, dy, dz, Ee, W, N10, e);  // before the root reads N10 and e
  return inv_root_rn(N10, e, out) & ok;
}

// Positions in 96-bit two's complement fixed point, unit 2^(E - 94) for |x| < 2^E: exact for
// |x| >= 2^(E - 42), truncated below, so a difference is off by less than two units.
struct Fix96 {
  uint32_t w[3];
};
GH_EMU_HD Fix96 to_fix96(double x, int E) {
  const uint64_t b = dbits(x);
  const int ex = (int)(b >> 52) & 0x7FF;
  const uint64_t M = ex ? (b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull : 0;
  const int sh = (ex - 1075) - (E - 94);  // <= 41
  const uint64_t lo = sh >= 0 ? M << sh : shr_clamp(M, -sh);
  const uint32_t hi = sh > 0 ? (uint32_t)(M >> (64 - sh)) : 0u;
  const uint64_t neg = (uint64_t)0 - (b >> 63);  // all ones when negative: ~v + 1
  const uint64_t l2 = (lo ^ neg) + (b >> 63);
  Fix96 r;
  r.w[0] = (uint32_t)l2;
  r.w[1] = (uint32_t)(l2 >> 32);
  r.w[2] = (hi ^ (uint32_t)neg) + (uint32_t)((b >> 63) & (l2 == 0));
  return r;
}

// |a - b| in 96 bits (one unit short of it when negative).
GH_EMU_HD void fix96_distance(const Fix96& a, const Fix96& b, uint32_t& d0, uint32_t& d1, uint32_t& d2) {
#ifdef __CUDA_ARCH__
  asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
      : "=r"(d0), "=r"(d1), "=r"(d2)
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]));
#else
  const uint64_t al = ((uint64_t)a.w[1] << 32) | a.w[0], bl = ((uint64_t)b.w[1] << 32) | b.w[0], dl = al - bl;
  d0 = (uint32_t)dl;
  d1 = (uint32_t)(dl >> 32);
  d2 = a.w[2] - b.w[2] - (al < bl);
#endif
  const uint32_t s = (uint32_t)((int32_t)d2 >> 31);
  d0 ^= s;
  d1 ^= s;
  d2 ^= s;
}

GH_EMU_HD uint32_t shl_funnel(uint32_t lo, uint32_t hi, int s) {  // 0 <= s <= 31
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}

GH_EMU_HD int clz32(uint32_t v) {
#ifdef __CUDA_ARCH__
  return __clz((int)v);
#else
  return v ? __builtin_clz(v) : 32;
#endif
}

// inv_distance of two fixed-point positions, without a floating-point difference.  e_eps
// and W as align_eps2 gives them (e_eps = Ee - 1023), room = E - e_eps >= 0 (a large number
// for eps = 0): the squares are aligned at the largest difference's leading bit, or at the
// softening's.  False below sqrt(d^2 + eps^2) = 2^(E - 31), where n would leave [1, 4).
GH_EMU_HD bool inv_distance_fix96(const Fix96* a, const Fix96* b, int E, int room, uint64_t W, double& out) {
  uint32_t x0, x1, x2, y0, y1, y2, z0, z1, z2;
  fix96_distance(a[0], b[0], x0, x1, x2);
  fix96_distance(a[1], b[1], y0, y1, y2);
  fix96_distance(a[2], b[2], z0, z1, z2);
  int sh = clz32(x2 | y2 | z2) - 1;  // in [0, 31]
  sh = room < sh ? room : sh;
  const uint64_t X = ((uint64_t)shl_funnel(x1, x2, sh) << 32) | shl_funnel(x0, x1, sh);
  const uint64_t Y = ((uint64_t)shl_funnel(y1, y2, sh) << 32) | shl_funnel(y0, y1, sh);
  const uint64_t Z = ((uint64_t)shl_funnel(z1, z2, sh) << 32) | shl_funnel(z0, z1, sh);
  const uint64_t S = square_hi(X) + square_hi(Y) + square_hi(Z) + shr_clamp(W, 2 * (room - sh));
  const int big = (S >> 62) != 0;
  return ((S >> 60) != 0) & inv_root_rn(big ? S : S << 2, E - sh + big, out);
}

// m s^(-3/2), rounded once: s^(-3/2) = y0^3 (1 + 3/2 h + 15/8 h^2), whose first omitted term is
// below 2^-58.  False outside the range of aligned_norm2 and for |m| outside [2^-500, 2^501).
GH_EMU_HD bool mass_inv_cube(double m, double dx, double dy, double dz, int Ee, uint64_t W, double& out) {
  uint64_t N10, Y0sq;
  uint32_t Y0;
  int64_t H;
  int e;
  const uint64_t bm = dbits(m);
  const int Em = (int)(bm >> 52) & 0x7FF;
  bool ok = aligned_norm2(dx, dy, dz, Ee, W, N10, e);
  ok &= (unsigned)(Em - 523) <= 1000u;  // |m| in [2^-500, 2^501)
  ok &= rsqrt_seed_residual(N10, Y0, Y0sq, H);
  if (!ok) return false;
  // y0^3 2^61, then times 1 + c, c = h (3/2 + 15/8 h) as C = c 2^64, |C| < 2^45
  const uint64_t Y3 = umulhi_low(Y0sq << 2, (uint64_t)Y0 << 33);
  const int64_t C = H * 24 + (int64_t)((15 * (uint64_t)residual_square(H)) >> 7);
  const uint64_t F = Y3 + (uint64_t)(smulhi_low(Y3, C));
  // times the mass's significand mm in [1, 2): T0 = mm y^3 2^62 in [2^59, 2^63]
  const uint64_t T0 = umulhi_low(F << 2, ((bm & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull) << 11);
  const int lz = clz64(T0);
  const uint64_t T = T0 << lz;
  const uint64_t mant = (T >> 11) + ((T >> 10) & 1);  // in [2^52, 2^53]
  // s^(-3/2) = y^3 2^(-3e): out = mant 2^k
  const int k = (Em - 1023) - 51 - lz - 3 * e;
  out = bitsd((((uint64_t)(k + 1074) << 52) + mant) | (bm & 0x8000000000000000ull));
  return true;
}

// m s^(-3/2) = m of a zero mass, where mass_inv_cube refuses nothing but that: false for
// another mass or outside the range of aligned_norm2 (there the power may overflow).
GH_EMU_HD bool zero_mass_inv_cube(double m, double dx, double dy, double dz, int Ee, double& out) {
  const int Ex = (int)(dbits(dx) >> 52) & 0x7FF, Ey = (int)(dbits(dy) >> 52) & 0x7FF, Ez = (int)(dbits(dz) >> 52) & 0x7FF;
  int E = Ex > Ey ? Ex : Ey;
  E = Ez > E ? Ez : E;
  E = Ee > E ? Ee : E;
  if ((dbits(m) << 1) != 0 || (unsigned)(E - 873) > 300u) return false;
  out = m;
  return true;
}

}  // namespace emu
}  // namespace gh
