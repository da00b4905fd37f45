// Vector-Jacobian product of the direct-sum acceleration, and the softened
// potential, as all-pairs kernels.  Neither has a counterpart in the reference.
//
// With a_k = sum_j m_j d_kj / s_kj^{3/2}, d_kj = x_j - x_k, s_kj = |d_kj|^2 + eps^2, and
// an incoming cotangent lambda (N,3) on the code-unit accelerations:
//   dL/dx_k = sum_{j != k} [ q u - p (d.u) d ],   u = m_k lambda_j - m_j lambda_k,
//             q = s^{-3/2}, p = 3 s^{-5/2}   (the softened tidal tensor applied to u)
//   dL/dm_k = - sum_{j != k} q (lambda_j . d)
// Potential: phi_k = - sum_{j != k} m_j s^{-1/2}, each unordered pair once.
//
// Work split (mixed VJP): a 2-D grid of (target tile, source split); each CTA writes
// per-target partial sums for its split to scratch and a reduction kernel adds the splits
// in split order, so results do not depend on scheduling.  FP64 VJP and potential: each
// unordered pair of blocks in one CTA, its sums likewise reduced in a fixed order.  Mixed: FP32
// pair arithmetic on coordinates relative to the mass-weighted centre, per-chunk FP32
// partials folded into two-sum (hi, lo) accumulators, FP64 reduction.
#include <mutex>

#include "direct.cuh"
#include "engine.h"

namespace gh {

constexpr int AJ_THREADS = 128;

__device__ __forceinline__ double rsqrt_nr(double s) {
  double y;
  asm("rsqrt.approx.f64 %0, %1;" : "=d"(y) : "d"(s));
#pragma unroll
  for (int it = 0; it < 2; it++) {
    double e = fma(-s * y, y, 1.0);
    y = fma(0.5 * y, e, y);
  }
  return y;
}

// ---------------------------------------------------------------------------
// FP64 VJP.  A pair's term of dL/dx changes sign with the order of its particles, so each
// unordered pair is taken once: row I of AJ_THREADS targets meets blocks I .. I + nblocks/2
// (cyclic; of two opposite blocks only the lower row takes the pairs), a warp's lanes at
// different sources of a block, whose sums wait in shared memory, one set per warp.  Where that is few
// CTAs, `parts` of them share a pair of blocks.
// FP64-pipe bound (93 % busy at N = 16,384): 38 operations per unordered pair against 2 x 28 with ordered ones (per
// VJP, N = 500 160 -> 39 us, 2000 253 -> 184, 4096 877 -> 625, 16,384 13.08 -> 8.97 ms).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(AJ_THREADS)
    vjp_pairs_f64_kernel(const double* __restrict__ pos, const double* __restrict__ mass,
                         const double* __restrict__ lam, int64_t n, double eps2, int nblocks, int row0, int parts, int len,
                         double* __restrict__ part_i, double* __restrict__ part_j) {
  constexpr int NW = AJ_THREADS / 32;
  __shared__ double src[7][AJ_THREADS];  // x, y, z, mass, lambda
  __shared__ double col[NW][4][AJ_THREADS];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int I = row0 + blockIdx.y;
  const int dmax = nblocks / 2;
  const int end = (dmax + 1) * parts, e0 = blockIdx.x * len, e1 = e0 + len < end ? e0 + len : end;
  const int64_t i = (int64_t)I * AJ_THREADS + tid, ii = i < n ? i : 0;
  const double xi = pos[3 * ii], yi = pos[3 * ii + 1], zi = pos[3 * ii + 2], mi = mass[ii];
  const double lxi = lam[3 * ii], lyi = lam[3 * ii + 1], lzi = lam[3 * ii + 2];
  double gx = 0.0, gy = 0.0, gz = 0.0, gm = 0.0;
  for (int e = e0; e < e1; e++) {
    const int d = e / parts, k0 = (e - d * parts) * (AJ_THREADS / parts), k1 = k0 + AJ_THREADS / parts;
    if (2 * d == nblocks && d > 0 && I >= nblocks / 2) break;  // the lower rows' pairs
    const int J = I + d < nblocks ? I + d : I + d - nblocks;
    const int64_t j0 = (int64_t)J * AJ_THREADS, j = j0 + tid;
    __syncthreads();
    if (j < n) {
#pragma unroll
      for (int k = 0; k < 3; k++) {
        src[k][tid] = pos[3 * j + k];
        src[4 + k][tid] = lam[3 * j + k];
      }
      src[3][tid] = mass[j];
    }
#pragma unroll
    for (int w = 0; w < NW; w++)
#pragma unroll
      for (int c = 0; c < 4; c++) col[w][c][tid] = 0.0;
    __syncthreads();
    const int jn = i < n ? (int)(n - j0 < AJ_THREADS ? n - j0 : AJ_THREADS) : 0;  // sources to take
    for (int k = d | k0 ? k0 : 1; k < k1; k++) {  // k = 0 of the block with itself: the particle itself
      const int q = (tid + k) & (AJ_THREADS - 1);
      if (q < jn) {
        const double dx = src[0][q] - xi, dy = src[1][q] - yi, dz = src[2][q] - zi;
        const double s = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
        double r2, r3;  // s^-1 and s^(-3/2) on the integer pipes; FP64 Newton steps outside its range
        if (!emu::rsqrt_powers(s, r2, r3)) {
          const double r = rsqrt_nr(s);
          r2 = r * r;
          r3 = r2 * r;
        }
        const double p = 3.0 * r3 * r2, mj = src[3][q];
        const double lx = src[4][q], ly = src[5][q], lz = src[6][q];
        const double ux = mi * lx - mj * lxi, uy = mi * ly - mj * lyi, uz = mi * lz - mj * lzi;
        const double du = fma(dx, ux, fma(dy, uy, dz * uz));
        const double pd = p * du;
        gx = fma(r3, ux, fma(-pd, dx, gx));
        gy = fma(r3, uy, fma(-pd, dy, gy));
        gz = fma(r3, uz, fma(-pd, dz, gz));
        gm = fma(-r3, fma(lx, dx, fma(ly, dy, lz * dz)), gm);
        if (d) {
          double* c = &col[warp][0][q];
          c[0] = fma(-r3, ux, fma(pd, dx, c[0]));
          c[AJ_THREADS] = fma(-r3, uy, fma(pd, dy, c[AJ_THREADS]));
          c[2 * AJ_THREADS] = fma(-r3, uz, fma(pd, dz, c[2 * AJ_THREADS]));
          c[3 * AJ_THREADS] = fma(r3, fma(lxi, dx, fma(lyi, dy, lzi * dz)), c[3 * AJ_THREADS]);
        }
      }
      __syncwarp();  // the neighbouring lane takes this source next
    }
    __syncthreads();
    if (d) {
      double* o = part_j + ((int64_t)blockIdx.y * dmax * parts + e - parts) * 4 * AJ_THREADS + tid;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        double a = col[0][c][tid];
#pragma unroll
        for (int w = 1; w < NW; w++) a += col[w][c][tid];
        o[c * AJ_THREADS] = a;
      }
    }
  }
  double* o = part_i + ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * 4 * AJ_THREADS + tid;
  o[0] = gx;
  o[AJ_THREADS] = gy;
  o[2 * AJ_THREADS] = gz;
  o[3 * AJ_THREADS] = gm;
}

// ---------------------------------------------------------------------------
// Mixed VJP: FP32 pair arithmetic on packed f32x2 lanes (two targets per thread
// register pair, VJ_P packs per thread), sources duplicated per lane pair in shared
// memory, per-chunk partials folded into two-sum (hi, lo) accumulators; 8 floats of
// partials per (split, target): hi/lo of gx, gy, gz, gm.  Per pair: 30 FP32 lane-ops
// (3 sub, 3 fma for s, 4 for q and -3q/s, 6 for u (3 with equal masses), 3 for d.u,
// 1, 6 for g, 4 for gm) and one MUFU rsqrt.
// ---------------------------------------------------------------------------
constexpr int VJ_THREADS = 128;
constexpr int VJ_P = 2;
constexpr int VJ_TILE = VJ_THREADS * 2 * VJ_P;
constexpr int VJ_JT = VJ_THREADS;

// EQ (all masses equal): u = m (lambda_j - lambda_k) with the mass taken out, one
// subtraction instead of a product and an FMA per component; the caller scales the
// position gradient by m once (the mass gradient's terms hold no mass).
template <bool SELFCHK, bool EQ = false>
__device__ __forceinline__ void vjp_chunk(const float4* __restrict__ tile, int64_t jbase, const int64_t* ka,
                                          const f2* tx, const f2* ty, const f2* tz, const f2* tm, const f2* tlx,
                                          const f2* tly, const f2* tlz, f2 E2, f2* gx, f2* gy, f2* gz, f2* gm) {
  const f2 M3 = f2make(-3.f, -3.f);
#pragma unroll 2
  for (int k = 0; k < VJ_JT; k++) {
    const float4 A = tile[4 * k], B = tile[4 * k + 1], C = tile[4 * k + 2], D = tile[4 * k + 3];
    const f2 X = f2make(A.x, A.y), Y = f2make(A.z, A.w), Z = f2make(B.x, B.y), NM = f2make(B.z, B.w);
    const f2 LX = f2make(C.x, C.y), LY = f2make(C.z, C.w), LZ = f2make(D.x, D.y);
#pragma unroll
    for (int p = 0; p < VJ_P; p++) {
      const f2 dx = f2sub(X, tx[p]), dy = f2sub(Y, ty[p]), dz = f2sub(Z, tz[p]);
      f2 s = f2fma(dx, dx, E2);
      s = f2fma(dy, dy, s);
      s = f2fma(dz, dz, s);
      float sa, sb;
      f2split(s, sa, sb);
      float ra = rsqrt_approx(sa), rb = rsqrt_approx(sb);
      if (SELFCHK) {
        ra = (jbase + k == ka[2 * p]) ? 0.f : ra;
        rb = (jbase + k == ka[2 * p + 1]) ? 0.f : rb;
      }
      const f2 r = f2make(ra, rb);
      const f2 r2 = f2mul(r, r);
      const f2 q = f2mul(r2, r);
      const f2 np = f2mul(f2mul(q, M3), r2);
      const f2 ux = EQ ? f2sub(LX, tlx[p]) : f2fma(NM, tlx[p], f2mul(tm[p], LX));
      const f2 uy = EQ ? f2sub(LY, tly[p]) : f2fma(NM, tly[p], f2mul(tm[p], LY));
      const f2 uz = EQ ? f2sub(LZ, tlz[p]) : f2fma(NM, tlz[p], f2mul(tm[p], LZ));
      f2 du = f2mul(dx, ux);
      du = f2fma(dy, uy, du);
      du = f2fma(dz, uz, du);
      const f2 npd = f2mul(np, du);
      gx[p] = f2fma(npd, dx, f2fma(q, ux, gx[p]));
      gy[p] = f2fma(npd, dy, f2fma(q, uy, gy[p]));
      gz[p] = f2fma(npd, dz, f2fma(q, uz, gz[p]));
      f2 ld = f2mul(dx, LX);
      ld = f2fma(dy, LY, ld);
      ld = f2fma(dz, LZ, ld);
      gm[p] = f2fma(q, ld, gm[p]);
    }
  }
}

__global__ void __launch_bounds__(VJ_THREADS, 4)
    vjp_mixed_kernel(const float4* __restrict__ src, const float4* __restrict__ lsrc, int64_t n, float eps2,
                     int64_t jlen, float* __restrict__ part, const double* __restrict__ meqp) {
  __shared__ __align__(16) float4 tile[4 * VJ_JT];
  const int tid = threadIdx.x;
  const int64_t tbase = (int64_t)blockIdx.x * VJ_TILE;
  const int64_t split = blockIdx.y;
  const int64_t j0 = split * jlen, j1 = (j0 + jlen) < n ? j0 + jlen : n;
  // equal masses: the sums are taken with unit masses (staged as such for the general
  // loop of a partial chunk: -1 for a source, 0 for padding, 1 for every target) and the
  // position gradient is scaled by the mass in the reduction
  const bool eq = __ldg(meqp) != 0.0;
  f2 tx[VJ_P], ty[VJ_P], tz[VJ_P], tm[VJ_P], tlx[VJ_P], tly[VJ_P], tlz[VJ_P];
  f2 hx[VJ_P], hy[VJ_P], hz[VJ_P], hm[VJ_P], lx[VJ_P], ly[VJ_P], lz[VJ_P], lm[VJ_P];
  int64_t ka[2 * VJ_P];
#pragma unroll
  for (int p = 0; p < VJ_P; p++) {
    float4 P0[2], L0[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int64_t k = tbase + (2 * p + h) * VJ_THREADS + tid;
      ka[2 * p + h] = k;
      P0[h] = k < n ? src[k] : make_float4(0.f, 0.f, 0.f, 0.f);
      L0[h] = k < n ? lsrc[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    tx[p] = f2make(P0[0].x, P0[1].x);
    ty[p] = f2make(P0[0].y, P0[1].y);
    tz[p] = f2make(P0[0].z, P0[1].z);
    tm[p] = eq ? f2make(1.f, 1.f) : f2make(P0[0].w, P0[1].w);
    tlx[p] = f2make(L0[0].x, L0[1].x);
    tly[p] = f2make(L0[0].y, L0[1].y);
    tlz[p] = f2make(L0[0].z, L0[1].z);
    hx[p] = hy[p] = hz[p] = hm[p] = lx[p] = ly[p] = lz[p] = lm[p] = 0ull;
  }
  const f2 E2 = f2make(eps2, eps2);
  for (int64_t c = j0; c < j1; c += VJ_JT) {
    __syncthreads();
    {
      const int64_t j = c + tid;
      const float4 P = j < j1 ? src[j] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 L = j < j1 ? lsrc[j] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float w = eq ? (j < j1 ? 1.f : 0.f) : P.w;
      tile[4 * tid + 0] = make_float4(P.x, P.x, P.y, P.y);
      tile[4 * tid + 1] = make_float4(P.z, P.z, -w, -w);
      tile[4 * tid + 2] = make_float4(L.x, L.x, L.y, L.y);
      tile[4 * tid + 3] = make_float4(L.z, L.z, 0.f, 0.f);
    }
    __syncthreads();
    f2 gx[VJ_P], gy[VJ_P], gz[VJ_P], gm[VJ_P];
#pragma unroll
    for (int p = 0; p < VJ_P; p++) gx[p] = gy[p] = gz[p] = gm[p] = 0ull;
    // only a chunk that overlaps this tile's targets can pair a target with itself
    const bool self = c < tbase + VJ_TILE && c + VJ_JT > tbase;
    if (eq && c + VJ_JT <= j1) {  // a full chunk of equal masses
      if (self)
        vjp_chunk<true, true>(tile, c, ka, tx, ty, tz, tm, tlx, tly, tlz, E2, gx, gy, gz, gm);
      else
        vjp_chunk<false, true>(tile, c, ka, tx, ty, tz, tm, tlx, tly, tlz, E2, gx, gy, gz, gm);
    } else {
      if (self)
        vjp_chunk<true>(tile, c, ka, tx, ty, tz, tm, tlx, tly, tlz, E2, gx, gy, gz, gm);
      else
        vjp_chunk<false>(tile, c, ka, tx, ty, tz, tm, tlx, tly, tlz, E2, gx, gy, gz, gm);
    }
#pragma unroll
    for (int p = 0; p < VJ_P; p++) {
      f2 sm, e;
      f2two_sum(hx[p], gx[p], sm, e);
      hx[p] = sm;
      lx[p] = f2add(lx[p], e);
      f2two_sum(hy[p], gy[p], sm, e);
      hy[p] = sm;
      ly[p] = f2add(ly[p], e);
      f2two_sum(hz[p], gz[p], sm, e);
      hz[p] = sm;
      lz[p] = f2add(lz[p], e);
      f2two_sum(hm[p], gm[p], sm, e);
      hm[p] = sm;
      lm[p] = f2add(lm[p], e);
    }
  }
#pragma unroll
  for (int p = 0; p < VJ_P; p++) {
    float a[8], b[8];
    f2split(hx[p], a[0], b[0]);
    f2split(lx[p], a[1], b[1]);
    f2split(hy[p], a[2], b[2]);
    f2split(ly[p], a[3], b[3]);
    f2split(hz[p], a[4], b[4]);
    f2split(lz[p], a[5], b[5]);
    f2split(hm[p], a[6], b[6]);
    f2split(lm[p], a[7], b[7]);
    // dL/dm_k = -sum q (lambda_j . d): the mass terms were accumulated with + sign
    a[6] = -a[6];
    a[7] = -a[7];
    b[6] = -b[6];
    b[7] = -b[7];
    const int64_t k0 = ka[2 * p], k1 = ka[2 * p + 1];
    if (k0 < n) {
      float* o = part + (split * n + k0) * 8;
#pragma unroll
      for (int q = 0; q < 8; q++) o[q] = a[q];
    }
    if (k1 < n) {
      float* o = part + (split * n + k1) * 8;
#pragma unroll
      for (int q = 0; q < 8; q++) o[q] = b[q];
    }
  }
}

// One thread per target and component: (hi, lo) pairs are 8 bytes of consecutive threads,
// and the splits' sums are added in split order (one thread per target with 4-byte loads 32
// bytes apart took 41 us at N = 16,384, 32 splits).
__global__ void vjp_reduce_mixed_kernel(const float2* __restrict__ part, int splits, int64_t n,
                                        const double* __restrict__ meqp, double* __restrict__ gpos,
                                        double* __restrict__ gmass) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 4 * n) return;
  double a = 0.0;
#pragma unroll 8
  for (int s = 0; s < splits; s++) {
    const float2 o = part[(int64_t)s * n * 4 + i];
    a += (double)o.x + (double)o.y;
  }
  const int64_t k = i >> 2;
  const int q = (int)(i & 3);
  if (q == 3) {
    if (gmass) gmass[k] = a;
    return;
  }
  const double meq = *meqp;
  gpos[3 * k + q] = (meq != 0.0 ? meq : 1.0) * a;  // equal masses: the sums were taken with unit masses
}

// ---------------------------------------------------------------------------
// Potential, FP64: each unordered pair once.  Blocks of AJ_THREADS particles; CTA (split,
// row I) takes row block I, one target per thread, against blocks I + d (mod T) for a range
// of d in 0 .. T/2, so every pair of blocks is met by exactly one row (d = 0: the block with
// itself, one-sided; with T even, d = T/2 by the lower half of the rows).  Lane t of a warp
// takes source (t + k) mod AJ_THREADS at step k and adds the pair's other half to that
// source's sum in shared memory, a private copy per warp.  The partial sums of rows (part_i)
// and columns (part_j) are added in a fixed order.
// The differences come from 96-bit fixed-point positions and the inverse distance from
// 64-bit fixed point (f64emu.cuh), about 155 instructions per unordered pair and warp (54
// cycles of an SM as measured, ALU 71 % busy) with two DFMAs on the FP64 pipe (32 of the
// cycles).  With FP64 differences it took 94 cycles, and the one-sided sum in FP64 296 (three
// differences, three DFMAs of the squared distance, a comparison, a DFMA, each twice).
// N = 65,536: 62.9 -> 20.0 -> 11.7 ms; 8192: 996 -> 364 -> 225 us; 1000: 74 -> 70 -> 56 -> 28
// in shares.
// Two or four targets per thread: the same from N = 30,000 on, slower below (fewer CTAs).
// ---------------------------------------------------------------------------
struct PairEps {
  double eps2;
  uint64_t W;
  int E;
  bool ok;
};

// y = s^(-1/2) of a pair; false (no contribution) where s is not positive.
__device__ __forceinline__ bool pair_inv_distance(double dx, double dy, double dz, const PairEps& pe, double& y) {
  if (pe.ok && emu::inv_distance(dx, dy, dz, pe.E, pe.W, y)) return true;
  const double s = fma(dx, dx, fma(dy, dy, fma(dz, dz, pe.eps2)));
  y = rsqrt_nr(s);
  return s > 0.0;
}

// Largest |coordinate| of pos[i], i = first, first + step, ... below n3, over a warp, as the
// bits of a double (they order like the values).
__device__ __forceinline__ unsigned long long largest_of_warp(const double* __restrict__ pos, int64_t first, int64_t step,
                                                              int64_t n3) {
  unsigned long long m = 0;
  for (int64_t k = first; k < n3; k += step) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(pos[k]) & 0x7FFFFFFFFFFFFFFFull;
    m = b > m ? b : m;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long q = __shfl_xor_sync(0xffffffffu, m, o);
    m = q > m ? q : m;
  }
  return m;
}

__global__ void __launch_bounds__(256)
    largest_coordinate_kernel(const double* __restrict__ pos, int64_t n3, unsigned long long* __restrict__ out) {
  const unsigned long long m =
      largest_of_warp(pos, (int64_t)blockIdx.x * 256 + threadIdx.x, (int64_t)gridDim.x * 256, n3);
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// WHOLE: each pair of blocks by one CTA (the loop over its 128 steps has fixed bounds: 4 %
// faster at every large N); else in `parts` shares.
template <bool WHOLE>
__global__ void __launch_bounds__(AJ_THREADS)
    potential_pairs_kernel(const double* __restrict__ pos, const double* __restrict__ mass, int64_t n, double eps2,
                           const unsigned long long* __restrict__ largest, int nblocks, int row0, int shares, int len,
                           double* __restrict__ part_i, double* __restrict__ part_j) {
  constexpr int NW = AJ_THREADS / 32;
  __shared__ uint4 src[3][AJ_THREADS];  // (x, y0), (y1, y2, z0, z1), (z2, -, mass): words of the positions
  __shared__ double col[NW][AJ_THREADS];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int I = row0 + blockIdx.y;
  const int dmax = nblocks / 2, parts = WHOLE ? 1 : shares;
  const int end = (dmax + 1) * parts, e0 = blockIdx.x * len, e1 = e0 + len < end ? e0 + len : end;
  unsigned long long top_bits;
  if (largest) {
    top_bits = *largest;
  } else {  // one block of particles: no launches for it
    __shared__ unsigned long long warp_top[NW];
    const unsigned long long m = largest_of_warp(pos, tid, AJ_THREADS, 3 * n);
    if ((tid & 31) == 0) warp_top[warp] = m;
    __syncthreads();
    top_bits = warp_top[0];
#pragma unroll
    for (int w = 1; w < NW; w++) top_bits = warp_top[w] > top_bits ? warp_top[w] : top_bits;
  }
  PairEps pe;
  pe.eps2 = eps2;
  pe.ok = emu::align_eps2(eps2, pe.E, pe.W);
  // |x| < 2^E; room: how far the softening's leading bit lies below 2^E
  const int top = (int)(top_bits >> 52), E = top - 1022;
  const int room = pe.W ? E - (pe.E - 1023) : 1 << 20;
  const bool fix = pe.ok && (unsigned)(top - 873) <= 300u && room >= 0;
  const int64_t i = (int64_t)I * AJ_THREADS + tid;
  const double mass_i = i < n ? mass[i] : 0.0;
  emu::Fix96 me[3];
#pragma unroll
  for (int k = 0; k < 3; k++) me[k] = emu::to_fix96(i < n ? pos[3 * i + k] : 0.0, E);
  double phi = 0.0;
  for (int e = e0; e < e1; e++) {
    const int d = e / parts, k0 = (e - d * parts) * (AJ_THREADS / parts), k1 = k0 + AJ_THREADS / parts;
    if (2 * d == nblocks && d > 0 && I >= nblocks / 2) break;  // the lower rows' pairs
    const int J = I + d < nblocks ? I + d : I + d - nblocks;
    const int64_t j0 = (int64_t)J * AJ_THREADS, j = j0 + tid;
    __syncthreads();
    if (j < n) {
      emu::Fix96 p[3];
#pragma unroll
      for (int k = 0; k < 3; k++) p[k] = emu::to_fix96(pos[3 * j + k], E);
      const uint64_t m = (uint64_t)__double_as_longlong(mass[j]);
      src[0][tid] = make_uint4(p[0].w[0], p[0].w[1], p[0].w[2], p[1].w[0]);
      src[1][tid] = make_uint4(p[1].w[1], p[1].w[2], p[2].w[0], p[2].w[1]);
      src[2][tid] = make_uint4(p[2].w[2], 0u, (uint32_t)m, (uint32_t)(m >> 32));
    }
    const int jn = i < n ? (int)(n - j0 < AJ_THREADS ? n - j0 : AJ_THREADS) : 0;  // sources to take
#pragma unroll
    for (int w = 0; w < NW; w++) col[w][tid] = 0.0;
    __syncthreads();
    for (int k = d | k0 ? k0 : 1; k < (WHOLE ? AJ_THREADS : k1); k++) {  // k = 0 of the block with itself: the particle itself
      const int q = (tid + k) & (AJ_THREADS - 1);
      if (q < jn) {
        const uint4 A = src[0][q], B = src[1][q], C = src[2][q];
        const emu::Fix96 p[3] = {{A.x, A.y, A.z}, {A.w, B.x, B.y}, {B.z, B.w, C.x}};
        const double mass_j = __hiloint2double((int)C.w, (int)C.z);
        double v;
        bool add = fix && emu::inv_distance_fix96(p, me, E, room, pe.W, v);
        if (!add) {
          const double* x = pos + 3 * (j0 + q);
          add = pair_inv_distance(x[0] - pos[3 * i], x[1] - pos[3 * i + 1], x[2] - pos[3 * i + 2], pe, v);
        }
        if (add) {
          phi = fma(-mass_j, v, phi);
          if (d) col[warp][q] = fma(-mass_i, v, col[warp][q]);
        }
      }
      __syncwarp();  // the neighbouring lane takes this source next
    }
    __syncthreads();
    if (d) {
      double a = col[0][tid];
#pragma unroll
      for (int w = 1; w < NW; w++) a += col[w][tid];
      part_j[((int64_t)blockIdx.y * dmax * parts + e - parts) * AJ_THREADS + tid] = a;
    }
  }
  part_i[((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * AJ_THREADS + tid] = phi;
}

// Adds the sums of rows row0 .. row0 + rows - 1: a particle's own row, split by split, then
// the rows that met its block as a column, in row order; the shares of a pair of blocks among
// themselves first (added one by one to the whole sum they doubled its error: 3e-16 against
// 1.4e-16 in the potential of 1500 particles).  C sums per particle, one per blockIdx.y: the
// first of them to out (stride C < 4 ? C : 3), a fourth to out4.
template <int C, int PARTS>
__global__ void pairs_reduce_kernel(const double* __restrict__ part_i, const double* __restrict__ part_j, int64_t n,
                                    int nblocks, int row0, int rows, int splits, double* __restrict__ out,
                                    double* __restrict__ out4) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int c = blockIdx.y;
  double* to = c == 3 ? out4 + k : out + k * (C < 4 ? C : 3) + c;
  const int J = (int)(k / AJ_THREADS), o = (int)(k - (int64_t)J * AJ_THREADS) + c * AJ_THREADS, dmax = nblocks / 2;
  double a = row0 ? *to : 0.0;
  if (J >= row0 && J < row0 + rows) {
    const double* own = part_i + (int64_t)(J - row0) * splits * C * AJ_THREADS + o;
    int s = 0;
    for (; s + PARTS <= splits; s += PARTS) {
      double t = own[(int64_t)s * C * AJ_THREADS];
#pragma unroll
      for (int q = 1; q < PARTS; q++) t += own[(int64_t)(s + q) * C * AJ_THREADS];
      a += t;
    }
    for (; s < splits; s++) a += own[(int64_t)s * C * AJ_THREADS];
  }
  for (int r = 0; r < rows; r++) {
    const int I = row0 + r;
    const int d = J >= I ? J - I : J - I + nblocks;
    if (d < 1 || d > dmax || (2 * d == nblocks && I >= nblocks / 2)) continue;
    const double* col = part_j + ((int64_t)r * dmax + d - 1) * PARTS * C * AJ_THREADS + o;
    double t = *col;
#pragma unroll
    for (int q = 1; q < PARTS; q++) t += col[(int64_t)q * C * AJ_THREADS];
    a += t;
  }
  *to = a;
}

template <int C>
static int launch_pairs_reduce(const double* part_i, const double* part_j, int64_t n, int nblocks, int row0, int rows,
                               int parts, int splits, double* out, double* out4, int sums, cudaStream_t st) {
  const auto kernel = parts == 1   ? pairs_reduce_kernel<C, 1>
                      : parts == 8 ? pairs_reduce_kernel<C, 8>
                                   : pairs_reduce_kernel<C, 32>;
  kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)sums), 256, 0, st>>>(part_i, part_j, n, nblocks, row0, rows, splits,
                                                                           out, out4);
  GH_LAUNCH_CHECK();
  return GH_OK;
}

// Mass-weighted centre for the FP32 sources, in 256 chains (particles t, t + 256, ...) of
// FP64 sums and a fixed tree over the chains, and whether every mass equals the first
// (finite, nonzero; a NaN never does).  One warp of chains per block: a block of all 256
// ran its FP64 sums on one SM, one dependent load after another (37 us at N = 16,384).
constexpr int MO_CHAINS = 256;

__global__ void __launch_bounds__(32)
    origin_chains_kernel(const double* __restrict__ pos, const double* __restrict__ mass, int64_t n,
                         dvec4* __restrict__ chain, int* __restrict__ differ) {
  const double m0 = n > 0 ? mass[0] : 0.0;
  dvec4 a = make_dvec4(0.0, 0.0, 0.0, 0.0);
  bool ne = false;
  constexpr int U = 8;  // loads in flight
  for (int64_t i = blockIdx.x * 32 + threadIdx.x; i < n; i += U * MO_CHAINS) {
    double m[U], x[U], y[U], z[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int64_t j = i + u * MO_CHAINS < n ? i + u * MO_CHAINS : i;
      m[u] = mass[j];
      x[u] = pos[3 * j];
      y[u] = pos[3 * j + 1];
      z[u] = pos[3 * j + 2];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      ne |= !(m[u] == m0);
      if (i + u * MO_CHAINS < n) {
        a.x += m[u] * x[u];
        a.y += m[u] * y[u];
        a.z += m[u] * z[u];
        a.w += m[u];
      }
    }
  }
  chain[blockIdx.x * 32 + threadIdx.x] = a;
  ne = __any_sync(0xffffffffu, ne);
  if (threadIdx.x == 0) differ[blockIdx.x] = ne;
}

// FP32 relative sources (x, y, z, m) and cotangents (lx, ly, lz, 0).  Every block adds the
// chains up for itself; block 0 leaves the centre in origin[0..2] and the common mass (0
// when the masses differ) in origin[3].
__global__ void __launch_bounds__(MO_CHAINS)
    vjp_prepare_mixed_kernel(const double* __restrict__ pos, const double* __restrict__ mass,
                             const double* __restrict__ lam, int64_t n, const dvec4* __restrict__ chain,
                             const int* __restrict__ differ, double* __restrict__ origin, float4* __restrict__ src,
                             float4* __restrict__ lsrc) {
  __shared__ dvec4 red[MO_CHAINS];
  red[threadIdx.x] = chain[threadIdx.x];
  __syncthreads();
  for (int s = MO_CHAINS / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      red[threadIdx.x].x += red[threadIdx.x + s].x;
      red[threadIdx.x].y += red[threadIdx.x + s].y;
      red[threadIdx.x].z += red[threadIdx.x + s].z;
      red[threadIdx.x].w += red[threadIdx.x + s].w;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const dvec4 r = red[0];
    const double o0 = r.x / r.w, o1 = r.y / r.w, o2 = r.z / r.w;
    const bool ok = r.w != 0.0 && isfinite(o0) && isfinite(o1) && isfinite(o2);
    red[0] = make_dvec4(ok ? o0 : 0.0, ok ? o1 : 0.0, ok ? o2 : 0.0, 0.0);
    if (blockIdx.x == 0) {
      bool ne = false;
      for (int k = 0; k < MO_CHAINS / 32; k++) ne |= differ[k] != 0;
      const double m0 = mass[0];
      origin[0] = red[0].x;
      origin[1] = red[0].y;
      origin[2] = red[0].z;
      origin[3] = (!ne && m0 != 0.0 && isfinite(m0)) ? m0 : 0.0;
    }
  }
  __syncthreads();
  const dvec4 o = red[0];
  const int64_t i = (int64_t)blockIdx.x * MO_CHAINS + threadIdx.x;
  if (i >= n) return;
  src[i] = make_float4((float)(pos[3 * i] - o.x), (float)(pos[3 * i + 1] - o.y), (float)(pos[3 * i + 2] - o.z),
                       (float)mass[i]);
  lsrc[i] = make_float4((float)lam[3 * i], (float)lam[3 * i + 1], (float)lam[3 * i + 2], 0.f);
}

// ---------------------------------------------------------------------------
struct AdjWS {
  Buffer part, part_j, src, lsrc, origin;
};
static AdjWS g_adj[64];
static std::mutex g_adj_mu;

// Bytes of column sums held at once, at most; kept for the life of the process, as every
// workspace (with the rows' sums, some 40 MB, from 92,673 particles on for the potential, 46,337
// for the FP64 VJP).
constexpr size_t PAIR_SCRATCH = 256u << 20;

// How an unordered-pair sum of `comps` values per particle is laid out.
struct PairPlan {
  int nblocks, parts, len;  // CTAs' shares of a pair of blocks, and how many of them one CTA takes
  int64_t rows, splits;     // rows of one launch, CTAs per row
};

static int plan_pairs(AdjWS& ws, int64_t n, int comps, int parts, int num_sms, PairPlan* out) {
  const int nblocks = (int)((n + AJ_THREADS - 1) / AJ_THREADS), dmax = nblocks / 2;
  const size_t row_bytes = (size_t)(dmax > 0 ? dmax : 1) * parts * comps * AJ_THREADS * sizeof(double);
  // the rows of one launch: all that the scratch holds, fewer when memory is short
  int64_t rows = (int64_t)(PAIR_SCRATCH / row_bytes);
  if (rows > nblocks) rows = nblocks;
  if (rows < 1) rows = 1;
  for (;;) {
    int64_t splits = (64LL * num_sms + rows - 1) / rows;  // eight waves of about eight CTAs per SM
    const int64_t most = (int64_t)(dmax + 1) * parts;
    if (splits > most) splits = most;
    out->len = (int)((most + splits - 1) / splits);
    splits = (most + out->len - 1) / out->len;
    int rc = ensure(ws.part, (size_t)rows * splits * comps * AJ_THREADS * sizeof(double));
    if (rc == GH_OK) rc = ensure(ws.part_j, (size_t)rows * row_bytes);
    out->nblocks = nblocks;
    out->parts = parts;
    out->rows = rows;
    out->splits = splits;
    if (rc != GH_ERR_OOM || rows == 1) return rc;
    clear_error();
    rows = (rows + 7) / 8;
  }
}

// A pair of blocks is a chain of 128 pairs per lane, some 200 us in the VJP and 45 in the
// potential; shares of it where the pairs of blocks are few.  VJP: N = 100 32 shares 167 -> 15
// us, 1000 8 shares 227 -> 76, 6000 1329 -> 1277; more blocks lose (16,384 8981 -> 9220).
// Potential (device time): N = 30 27 -> 7 us (of one block, which finds its own largest
// coordinate), 130 46 -> 19, 1000 50 -> 23, 3000 69 -> 61; more blocks lose (4000 83 -> 91).
// (pairs_reduce_kernel is made for 1, 8 and 32.)
static int pair_shares(int64_t n, bool vjp) {
  const int64_t nb = (n + AJ_THREADS - 1) / AJ_THREADS, meets = nb * (nb / 2 + 1);
  return meets < 8 ? 32 : (meets < (vjp ? 1200 : 320) ? 8 : 1);
}

int direct_vjp(const double* pos, const double* mass, int64_t n, double eps, const double* lam, int precision,
               double* gpos, double* gmass, cudaStream_t st) {
  if (n < 0) return set_error(GH_ERR_ARG, "negative particle count");
  if (!(eps >= 0.0)) return set_error(GH_ERR_ARG, "eps must be >= 0 (got %g)", eps);
  if (precision != GH_PREC_FP64 && precision != GH_PREC_MIXED)
    return set_error(GH_ERR_ARG, "unknown precision %d", precision);
  if (n == 0) return GH_OK;
  if (!pos || !mass || !lam || !gpos) return set_error(GH_ERR_ARG, "null buffer");
  std::lock_guard<std::mutex> lk(g_adj_mu);
  DeviceInfo di;
  GH_TRY(device_info(&di));
  AdjWS& ws = g_adj[di.device];
  const unsigned rb = (unsigned)((n + 255) / 256);
  if (precision == GH_PREC_FP64) {
    PairPlan pp;
    GH_TRY(plan_pairs(ws, n, 4, pair_shares(n, true), di.num_sms, &pp));
    for (int row0 = 0; row0 < pp.nblocks; row0 += (int)pp.rows) {
      const int here = pp.nblocks - row0 < pp.rows ? pp.nblocks - row0 : (int)pp.rows;
      prof_begin(st);
      vjp_pairs_f64_kernel<<<dim3((unsigned)pp.splits, (unsigned)here), AJ_THREADS, 0, st>>>(
          pos, mass, lam, n, eps * eps, pp.nblocks, row0, pp.parts, pp.len, (double*)ws.part.ptr,
          (double*)ws.part_j.ptr);
      prof_end(st);
      GH_LAUNCH_CHECK();
      GH_TRY(launch_pairs_reduce<4>((const double*)ws.part.ptr, (const double*)ws.part_j.ptr, n, pp.nblocks, row0, here,
                                    pp.parts, (int)pp.splits, gpos, gmass, gmass ? 4 : 3, st));
    }
    return GH_OK;
  }
  GH_TRY(ensure(ws.src, (size_t)n * sizeof(float4)));
  GH_TRY(ensure(ws.lsrc, (size_t)n * sizeof(float4)));
  GH_TRY(ensure(ws.origin, 4 * sizeof(double) + MO_CHAINS * sizeof(dvec4) + MO_CHAINS / 32 * sizeof(int)));
  dvec4* chain = (dvec4*)((double*)ws.origin.ptr + 4);
  int* differ = (int*)(chain + MO_CHAINS);
  origin_chains_kernel<<<MO_CHAINS / 32, 32, 0, st>>>(pos, mass, n, chain, differ);
  GH_LAUNCH_CHECK();
  vjp_prepare_mixed_kernel<<<rb, MO_CHAINS, 0, st>>>(pos, mass, lam, n, chain, differ, (double*)ws.origin.ptr,
                                                     (float4*)ws.src.ptr, (float4*)ws.lsrc.ptr);
  GH_LAUNCH_CHECK();
  // Mixed kernel: tiles of VJ_TILE targets, splits of whole VJ_JT-source chunks, four
  // resident CTAs per SM.  Of the splits that fill 1 to 16 waves of CTAs, the one with the
  // fewest chunks in sequence (half a chunk more per wave for its start): N = 16,384 takes
  // 19 splits of 7 chunks in one wave, not 32 of 4 in two.  Partial sums up to 64 MB.
  const int64_t mtiles = (n + VJ_TILE - 1) / VJ_TILE;
  const int64_t chunks = (n + VJ_JT - 1) / VJ_JT;
  const int64_t slots = 4LL * di.num_sms;
  int64_t best = 0, per = chunks;
  for (int64_t waves = 1; waves <= 16; waves++) {
    const int64_t most = waves * slots / mtiles;  // splits that fit
    if (most < 1 || (most > 1 && most * n * 8 * (int64_t)sizeof(float) > (64 << 20))) continue;
    const int64_t p = (chunks + most - 1) / most, cost = waves * (2 * p + 1);
    if (best == 0 || cost < best) {
      best = cost;
      per = p;
    }
  }
  const int64_t mjlen = per * VJ_JT;
  const int64_t msplits = (n + mjlen - 1) / mjlen;
  GH_TRY(ensure(ws.part, (size_t)msplits * n * 8 * sizeof(float)));
  prof_begin(st);
  vjp_mixed_kernel<<<dim3((unsigned)mtiles, (unsigned)msplits), VJ_THREADS, 0, st>>>(
      (const float4*)ws.src.ptr, (const float4*)ws.lsrc.ptr, n, (float)(eps * eps), mjlen, (float*)ws.part.ptr,
      (const double*)ws.origin.ptr + 3);
  prof_end(st);
  GH_LAUNCH_CHECK();
  vjp_reduce_mixed_kernel<<<(unsigned)((4 * n + 255) / 256), 256, 0, st>>>(
      (const float2*)ws.part.ptr, (int)msplits, n, (const double*)ws.origin.ptr + 3, gpos, gmass);
  GH_LAUNCH_CHECK();
  return GH_OK;
}

// ---------------------------------------------------------------------------
// Backward pass of drift-kick-drift steps.  Forward step (gravhopper.py:405-416):
//   xh = x + c v,  v' = v + dt A F(xh),  x' = xh + c v'      (c = 0.5 dt F_kpc)
// Reverse, given (xbar, vbar) of (x', v'):
//   w = vbar + c xbar;  lam = A dt w;  (gx, gm) = VJP of F at xh with lam;
//   xhbar = xbar + gx;  xbar <- xhbar;  vbar <- w + c xhbar;  mbar += gm
// ---------------------------------------------------------------------------
__global__ void adj_pre_kernel(const double* __restrict__ x, const double* __restrict__ v, int64_t n, double dt,
                               const double* __restrict__ xbar, const double* __restrict__ vbar,
                               double* __restrict__ xh, double* __restrict__ w, double* __restrict__ lam) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * n) return;
  const double c = 0.5 * dt * GH_KMS_MYR_TO_KPC;
  xh[i] = drift_half(x[i], v[i], dt);
  const double wi = vbar[i] + c * xbar[i];
  w[i] = wi;
  lam[i] = (GH_ACCEL_UNIT * dt) * wi;
}

__global__ void adj_post_kernel(int64_t n, double dt, const double* __restrict__ w, const double* __restrict__ gpos,
                                const double* __restrict__ gmass, double* __restrict__ xbar,
                                double* __restrict__ vbar, double* __restrict__ mbar) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 3 * n) {
    const double c = 0.5 * dt * GH_KMS_MYR_TO_KPC;
    const double xhb = xbar[i] + gpos[i];
    xbar[i] = xhb;
    vbar[i] = w[i] + c * xhb;
  }
  if (i < n && mbar) mbar[i] += gmass[i];
}

struct BwdWS {
  Buffer states_x, states_v, work_x, work_v, xh, w, lam, gpos, gmass;
  Buffer chain_x[2], chain_v[2];        // dkd_backward_chain: recomputed segments, two buffers
  cudaStream_t rstream = nullptr;       // dkd_backward_chain: recomputation stream
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
};
static BwdWS g_bwd[64];
static std::mutex g_bwd_mu;

// Back-propagates through `nsteps` recomputed states (sx, sv: state at the start of
// each step) with the VJP kernel: (xbar, vbar) updated in place, mbar incremented.
static int backward_steps(BwdWS& ws, const double* sx, const double* sv, const double* mass, int64_t n,
                          int64_t nsteps, double dt, double eps, int precision, double* xbar, double* vbar,
                          double* mbar, cudaStream_t st) {
  const unsigned b3 = (unsigned)((3 * n + 255) / 256);
  for (int64_t j = nsteps - 1; j >= 0; j--) {
    adj_pre_kernel<<<b3, 256, 0, st>>>(sx + 3 * n * j, sv + 3 * n * j, n, dt, xbar, vbar, (double*)ws.xh.ptr,
                                       (double*)ws.w.ptr, (double*)ws.lam.ptr);
    GH_LAUNCH_CHECK();
    GH_TRY(direct_vjp((const double*)ws.xh.ptr, mass, n, eps, (const double*)ws.lam.ptr, precision,
                      (double*)ws.gpos.ptr, (double*)ws.gmass.ptr, st));
    adj_post_kernel<<<b3, 256, 0, st>>>(n, dt, (const double*)ws.w.ptr, (const double*)ws.gpos.ptr,
                                        (const double*)ws.gmass.ptr, xbar, vbar, mbar);
    GH_LAUNCH_CHECK();
  }
  return GH_OK;
}

int dkd_backward(const double* x0, const double* v0, const double* mass, int64_t n, int64_t nsteps, double dt,
                 double eps, int precision, double* xbar, double* vbar, double* mbar, cudaStream_t st) {
  if (n < 0 || nsteps < 0) return set_error(GH_ERR_ARG, "negative n or nsteps");
  if (n == 0 || nsteps == 0) return GH_OK;
  if (!x0 || !v0 || !mass || !xbar || !vbar) return set_error(GH_ERR_ARG, "null buffer");
  std::lock_guard<std::mutex> lk(g_bwd_mu);
  DeviceInfo di;
  GH_TRY(device_info(&di));
  BwdWS& ws = g_bwd[di.device];
  const size_t vec = (size_t)n * 3 * sizeof(double);
  GH_TRY(ensure(ws.states_x, vec * nsteps));
  GH_TRY(ensure(ws.states_v, vec * nsteps));
  GH_TRY(ensure(ws.work_x, vec));
  GH_TRY(ensure(ws.work_v, vec));
  GH_TRY(ensure(ws.xh, vec));
  GH_TRY(ensure(ws.w, vec));
  GH_TRY(ensure(ws.lam, vec));
  GH_TRY(ensure(ws.gpos, vec));
  GH_TRY(ensure(ws.gmass, (size_t)n * sizeof(double)));
  double* sx = (double*)ws.states_x.ptr;
  double* sv = (double*)ws.states_v.ptr;
  // states[j] = state at the start of step j, j = 0 .. nsteps-1, recomputed from x0, v0
  GH_CUDA_TRY(cudaMemcpyAsync(sx, x0, vec, cudaMemcpyDeviceToDevice, st));
  GH_CUDA_TRY(cudaMemcpyAsync(sv, v0, vec, cudaMemcpyDeviceToDevice, st));
  if (nsteps > 1) {
    GH_CUDA_TRY(cudaMemcpyAsync(ws.work_x.ptr, x0, vec, cudaMemcpyDeviceToDevice, st));
    GH_CUDA_TRY(cudaMemcpyAsync(ws.work_v.ptr, v0, vec, cudaMemcpyDeviceToDevice, st));
    GH_TRY(direct_run((double*)ws.work_x.ptr, (double*)ws.work_v.ptr, mass, n, nsteps - 1, dt, eps, precision,
                      sx + 3 * n, sv + 3 * n, 1, st));
  }
  return backward_steps(ws, sx, sv, mass, n, nsteps, dt, eps, precision, xbar, vbar, mbar, st);
}

// Multi-segment form: the checkpoints of all segments at once; segment s-1 is
// recomputed on a second stream while segment s back-propagates on `st` (two state
// buffers, ordered by events), so the recomputation overlaps the VJP launches.
int dkd_backward_chain(const double* cx, const double* cv, const int64_t* seg, int64_t nseg, const double* mass,
                       int64_t n, double dt, double eps, int precision, double* xbar, double* vbar, double* mbar,
                       cudaStream_t st) {
  if (n < 0 || nseg < 0) return set_error(GH_ERR_ARG, "negative n or segment count");
  if (n == 0 || nseg == 0) return GH_OK;
  if (!cx || !cv || !seg || !mass || !xbar || !vbar) return set_error(GH_ERR_ARG, "null buffer");
  int64_t maxseg = 0;
  for (int64_t s = 0; s < nseg; s++) {
    if (seg[s] < 1) return set_error(GH_ERR_ARG, "segment %lld has %lld steps", (long long)s, (long long)seg[s]);
    if (seg[s] > maxseg) maxseg = seg[s];
  }
  std::lock_guard<std::mutex> lk(g_bwd_mu);
  DeviceInfo di;
  GH_TRY(device_info(&di));
  BwdWS& ws = g_bwd[di.device];
  const size_t vec = (size_t)n * 3 * sizeof(double);
  for (int b = 0; b < 2; b++) {
    GH_TRY(ensure(ws.chain_x[b], vec * maxseg));
    GH_TRY(ensure(ws.chain_v[b], vec * maxseg));
  }
  GH_TRY(ensure(ws.work_x, vec));
  GH_TRY(ensure(ws.work_v, vec));
  GH_TRY(ensure(ws.xh, vec));
  GH_TRY(ensure(ws.w, vec));
  GH_TRY(ensure(ws.lam, vec));
  GH_TRY(ensure(ws.gpos, vec));
  GH_TRY(ensure(ws.gmass, (size_t)n * sizeof(double)));
  if (!ws.rstream) {
    GH_CUDA_TRY(cudaStreamCreateWithFlags(&ws.rstream, cudaStreamNonBlocking));
    for (int b = 0; b < 3; b++) GH_CUDA_TRY(cudaEventCreateWithFlags(&ws.ev[b], cudaEventDisableTiming));
  }
  cudaStream_t rs = ws.rstream;
  cudaEvent_t ev_ready[2] = {ws.ev[0], ws.ev[1]};  // recomputed segment in buffer b
  cudaEvent_t ev_free = ws.ev[2];                  // the backward that last read a buffer
  GH_CUDA_TRY(cudaEventRecord(ev_free, st));        // the caller's work before anything here
  GH_CUDA_TRY(cudaStreamWaitEvent(rs, ev_free, 0));
  auto recompute = [&](int64_t s) -> int {
    const int b = (int)(s & 1);
    double* sx = (double*)ws.chain_x[b].ptr;
    double* sv = (double*)ws.chain_v[b].ptr;
    GH_CUDA_TRY(cudaMemcpyAsync(sx, cx + 3 * n * s, vec, cudaMemcpyDeviceToDevice, rs));
    GH_CUDA_TRY(cudaMemcpyAsync(sv, cv + 3 * n * s, vec, cudaMemcpyDeviceToDevice, rs));
    if (seg[s] > 1) {
      GH_CUDA_TRY(cudaMemcpyAsync(ws.work_x.ptr, cx + 3 * n * s, vec, cudaMemcpyDeviceToDevice, rs));
      GH_CUDA_TRY(cudaMemcpyAsync(ws.work_v.ptr, cv + 3 * n * s, vec, cudaMemcpyDeviceToDevice, rs));
      GH_TRY(direct_run((double*)ws.work_x.ptr, (double*)ws.work_v.ptr, mass, n, seg[s] - 1, dt, eps, precision,
                        sx + 3 * n, sv + 3 * n, 1, rs));
    }
    GH_CUDA_TRY(cudaEventRecord(ev_ready[b], rs));
    return GH_OK;
  };
  GH_TRY(recompute(nseg - 1));
  for (int64_t s = nseg - 1; s >= 0; s--) {
    const int b = (int)(s & 1);
    GH_CUDA_TRY(cudaStreamWaitEvent(st, ev_ready[b], 0));
    if (s >= 1) {
      // buffer (s-1)&1 was last read by the backward of segment s+1
      if (s + 1 < nseg) GH_CUDA_TRY(cudaStreamWaitEvent(rs, ev_free, 0));
      GH_TRY(recompute(s - 1));
    }
    GH_TRY(backward_steps(ws, (const double*)ws.chain_x[b].ptr, (const double*)ws.chain_v[b].ptr, mass, n, seg[s],
                          dt, eps, precision, xbar, vbar, mbar, st));
    GH_CUDA_TRY(cudaEventRecord(ev_free, st));
  }
  return GH_OK;
}

int potential(const double* pos, const double* mass, int64_t n, double eps, double* phi, cudaStream_t st) {
  if (n < 0) return set_error(GH_ERR_ARG, "negative particle count");
  if (!(eps >= 0.0)) return set_error(GH_ERR_ARG, "eps must be >= 0 (got %g)", eps);
  if (n == 0) return GH_OK;
  if (!pos || !mass || !phi) return set_error(GH_ERR_ARG, "null buffer");
  std::lock_guard<std::mutex> lk(g_adj_mu);
  DeviceInfo di;
  GH_TRY(device_info(&di));
  AdjWS& ws = g_adj[di.device];
  PairPlan pp;
  GH_TRY(plan_pairs(ws, n, 1, pair_shares(n, false), di.num_sms, &pp));
  unsigned long long* largest = nullptr;
  if (pp.nblocks > 1) {
    GH_TRY(ensure(ws.origin, sizeof(unsigned long long)));
    largest = (unsigned long long*)ws.origin.ptr;
    GH_CUDA_TRY(cudaMemsetAsync(largest, 0, sizeof(*largest), st));
    const int64_t need = (3 * n + 255) / 256, cap = 2LL * di.num_sms;
    largest_coordinate_kernel<<<(unsigned)(need < cap ? need : cap), 256, 0, st>>>(pos, 3 * n, largest);
    GH_LAUNCH_CHECK();
  }
  for (int row0 = 0; row0 < pp.nblocks; row0 += (int)pp.rows) {
    const int here = pp.nblocks - row0 < pp.rows ? pp.nblocks - row0 : (int)pp.rows;
    const dim3 grid((unsigned)pp.splits, (unsigned)here);
    const auto kernel = pp.parts == 1 ? potential_pairs_kernel<true> : potential_pairs_kernel<false>;
    kernel<<<grid, AJ_THREADS, 0, st>>>(pos, mass, n, eps * eps, largest, pp.nblocks, row0, pp.parts, pp.len,
                                        (double*)ws.part.ptr, (double*)ws.part_j.ptr);
    GH_LAUNCH_CHECK();
    GH_TRY(launch_pairs_reduce<1>((const double*)ws.part.ptr, (const double*)ws.part_j.ptr, n, pp.nblocks, row0, here,
                                  pp.parts, (int)pp.splits, phi, nullptr, 1, st));
  }
  return GH_OK;
}

}  // namespace gh
