// Direct-sum force kernels and the leapfrog epilogues they can run in place of a
// plain store.  Included by direct.cu (force calls, run loop) and by the no-alloc
// variant; everything here is header-only device code plus launch helpers.
#pragma once

#include "gh_common.cuh"
#include "f64emu.cuh"

namespace gh {

// ---------------------------------------------------------------------------
// Packed FP32 pairs (Blackwell f32x2 ALU ops): one instruction, two lanes of work.
// ---------------------------------------------------------------------------
typedef unsigned long long f2;

__device__ __forceinline__ f2 f2make(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2split(f2 v, float& a, float& b) {
  asm("mov.b64 {%0,%1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 f2add(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 f2sub(f2 a, f2 b) {
  f2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 f2mul(f2 a, f2 b) {
  f2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 f2fma(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// Two-sum on both lanes: (s, e) with s + e == a + b exactly, per lane.
__device__ __forceinline__ void f2two_sum(f2 a, f2 b, f2& s, f2& e) {
  s = f2add(a, b);
  f2 bb = f2sub(s, a);
  e = f2add(f2sub(a, f2sub(s, bb)), f2sub(b, bb));
}

// ---------------------------------------------------------------------------
// Leapfrog (drift-kick-drift) arithmetic of Simulation.perform_timestep,
// gravhopper/gravhopper.py:405-416, in kpc, km/s, Myr, with no FMA contraction:
//   xh = x + ((0.5*v)*dt)*F          (F = km*Myr/s -> kpc)
//   v' = v + (a*ACC)*dt              (ACC = G*Msun/kpc^2 in km/s/Myr)
//   x' = xh + ((0.5*v')*dt)*F
// ---------------------------------------------------------------------------
__device__ __forceinline__ double drift_half(double x, double v, double dt) {
  return dadd(x, dmul(dmul(dmul(0.5, v), dt), GH_KMS_MYR_TO_KPC));
}
__device__ __forceinline__ double kick(double v, double a_code, double dt) {
  return dadd(v, dmul(dmul(a_code, GH_ACCEL_UNIT), dt));
}

// ---------------------------------------------------------------------------
// Epilogues.  Each is called once per target with the code-unit acceleration.
// ---------------------------------------------------------------------------

// Store the acceleration (code units) into acc[(N,3)].
struct EpiStore {
  static constexpr bool kFusedStep = false;
  double* acc;
  __device__ __forceinline__ void operator()(int64_t i, double ax, double ay, double az) const {
    acc[3 * i + 0] = ax;
    acc[3 * i + 1] = ay;
    acc[3 * i + 2] = az;
  }
};

// Finish a DKD step for particle i and prepare the next step's sources.
//   x, v     : state at the start of the step (read), state after it (written)
//   src_next : next step's half-drifted sources; float4 relative to `origin` for the
//              mixed form, or FP64 (N,3) in `xh_next` for the FP64 form
//   hist_x/v : optional snapshot slots (N,3) written with the new state
struct EpiDKD {
  static constexpr bool kFusedStep = true;
  double* x;
  double* v;
  const double* mass;
  float4* src_next;      // mixed form (may be null)
  double* xh_next;       // FP64 form (may be null)
  double* hist_x;
  double* hist_v;
  const double* origin;  // device pointer to 3 doubles (mixed form)
  double dt;
  __device__ __forceinline__ void operator()(int64_t i, double ax, double ay, double az) const {
    double a[3] = {ax, ay, az};
    double xn[3], vn[3], xh2[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      double x0 = x[3 * i + k], v0 = v[3 * i + k];
      double xh = drift_half(x0, v0, dt);
      double v1 = kick(v0, a[k], dt);
      double x1 = drift_half(xh, v1, dt);
      xn[k] = x1;
      vn[k] = v1;
      xh2[k] = drift_half(x1, v1, dt);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
      x[3 * i + k] = xn[k];
      v[3 * i + k] = vn[k];
    }
    if (hist_x) {
#pragma unroll
      for (int k = 0; k < 3; k++) {
        hist_x[3 * i + k] = xn[k];
        hist_v[3 * i + k] = vn[k];
      }
    }
    if (src_next) {
      src_next[i] = make_float4((float)dsub(xh2[0], origin[0]), (float)dsub(xh2[1], origin[1]),
                                (float)dsub(xh2[2], origin[2]), (float)mass[i]);
    }
    if (xh_next) {
#pragma unroll
      for (int k = 0; k < 3; k++) xh_next[3 * i + k] = xh2[k];
    }
  }
};

// ---------------------------------------------------------------------------
// FP64 form: bit-exact restatement of directsummation_workhorse
// (gravhopper/_jbgrav.c:140-193) and directsummation_position_workhorse
// (:299-353).  One thread owns F64_R targets and walks every source in ascending
// order, so each component is summed in exactly the reference's order.
// ---------------------------------------------------------------------------
constexpr int F64_THREADS = 128;
constexpr int F64_R = 2;
constexpr int F64_JT = 128;

// The pair terms RN(RN(m d_k) inv) of one (target, source) pair with the reference's
// operations (gravhopper/_jbgrav.c:159-166, 181): d = x_j - x_i, then s and
// inv = 1/s/sqrt(s) on the integer pipes (f64emu.cuh) with the native IEEE operations
// for the inputs that path leaves out.  Without the self-pair exclusion (target
// points) s = 0 gives zero terms (:325-331).
template <bool SELF>
__device__ __forceinline__ void f64_pair_terms(const dvec4& s, double tx, double ty, double tz, double eps2,
                                               bool emu_ok, int e2E, uint64_t e2M, double& vx, double& vy,
                                               double& vz) {
  const double dx = dsub(s.x, tx);
  const double dy = dsub(s.y, ty);
  const double dz = dsub(s.z, tz);
  double inv;
  if (!(emu_ok && emu::pair_inv_cube_rn(dx, dy, dz, e2E, e2M, inv))) {
    double r2 = dmul(dx, dx);
    r2 = dadd(r2, dmul(dy, dy));
    r2 = dadd(r2, dmul(dz, dz));
    const double ss = dadd(r2, eps2);
    if (!emu::inv_cube_rn(ss, inv)) inv = (!SELF && ss == 0.0) ? 0.0 : ddiv(ddiv(1.0, ss), dsqrt(ss));
  }
  vx = dmul(dmul(s.w, dx), inv);
  vy = dmul(dmul(s.w, dy), inv);
  vz = dmul(dmul(s.w, dz), inv);
}

template <bool SELF, class Epi>
__global__ void __launch_bounds__(F64_THREADS)
    direct_f64_kernel(const double* __restrict__ spos, const double* __restrict__ smass, int64_t np,
                      const double* __restrict__ tpos, int64_t nt, double eps2, Epi epi) {
  __shared__ dvec4 tile[F64_JT];
  const int64_t base = (int64_t)blockIdx.x * (F64_THREADS * F64_R) + threadIdx.x;
  double tx[F64_R], ty[F64_R], tz[F64_R], ax[F64_R], ay[F64_R], az[F64_R];
  int64_t ti[F64_R];
  int e2E;
  uint64_t e2M;
  const bool emu_ok = emu::unpack_eps2(eps2, e2E, e2M);  // integer-pipe pair factor usable
#pragma unroll
  for (int r = 0; r < F64_R; r++) {
    ti[r] = base + r * F64_THREADS;
    int64_t t = ti[r] < nt ? ti[r] : 0;
    tx[r] = nt ? tpos[3 * t + 0] : 0.0;
    ty[r] = nt ? tpos[3 * t + 1] : 0.0;
    tz[r] = nt ? tpos[3 * t + 2] : 0.0;
    ax[r] = ay[r] = az[r] = 0.0;
  }
  for (int64_t j0 = 0; j0 < np; j0 += F64_JT) {
    __syncthreads();
    for (int k = threadIdx.x; k < F64_JT; k += F64_THREADS) {
      int64_t j = j0 + k;
      if (j < np) tile[k] = make_dvec4(spos[3 * j], spos[3 * j + 1], spos[3 * j + 2], smass[j]);
    }
    __syncthreads();
    const int jn = (np - j0) < F64_JT ? (int)(np - j0) : F64_JT;
    for (int k = 0; k < jn; k++) {
      const dvec4 s = tile[k];
#pragma unroll
      for (int r = 0; r < F64_R; r++) {
        if (SELF && (j0 + k) == ti[r]) continue;
        double vx, vy, vz;
        f64_pair_terms<SELF>(s, tx[r], ty[r], tz[r], eps2, emu_ok, e2E, e2M, vx, vy, vz);
        ax[r] = dadd(ax[r], vx);
        ay[r] = dadd(ay[r], vy);
        az[r] = dadd(az[r], vz);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < F64_R; r++)
    if (ti[r] < nt) epi(ti[r], ax[r], ay[r], az[r]);
}

// FP64 form for few targets (fewer than eight CTAs of the kernel above per SM): the
// pair terms (m_j d) inv of a chunk of sources are computed by warps 1-7 into shared
// memory while warp 0 adds the previous chunk's terms in ascending j, one lane per
// (target, component), so the sums are the reference's own.  Two term buffers, one
// barrier per chunk.  A self pair contributes +0.0, which leaves every sum unchanged:
// a round-to-nearest sum started at +0.0 is never -0.0.
constexpr int F64O_THREADS = 256;
constexpr int F64O_WORKERS = F64O_THREADS - 32;  // warps 1-7 compute pair terms
constexpr int F64O_TERMS = 2 * F64O_WORKERS;     // pair terms per chunk: two per worker

template <bool SELF, int TB, class Epi>
__global__ void __launch_bounds__(F64O_THREADS)
    direct_f64_ordered_kernel(const double* __restrict__ spos, const double* __restrict__ smass, int64_t np,
                              const double* __restrict__ tpos, int64_t nt, double eps2, Epi epi) {
  static_assert(3 * TB <= 32, "the summing lanes form one warp");
  constexpr int JC = F64O_TERMS / TB;  // sources per chunk
  // Padded rows: odd, so that the summing lanes hit distinct banks, but for TB = 5 (90), where
  // lanes 8 apart share one; 89 is slower there (N = 1520 95.2 us against 93.1).
  constexpr int JP = JC + 1;
  __shared__ dvec4 src[2][JC];
  __shared__ double term[2][3 * TB][JP];
  __shared__ double tp[TB][3];
  __shared__ double res[3 * TB];
  const int tid = threadIdx.x;
  const int64_t t0 = (int64_t)blockIdx.x * TB;
  if (tid < 3 * TB) {
    const int64_t ti = t0 + tid / 3;
    tp[tid / 3][tid % 3] = ti < nt ? tpos[3 * ti + tid % 3] : 0.0;
  }
  const int w = tid - 32;  // worker index (warps 1-7)
  if (w >= 0) {
    for (int k = w; k < JC; k += F64O_WORKERS)
      if (k < np) src[0][k] = make_dvec4(spos[3 * k], spos[3 * k + 1], spos[3 * k + 2], smass[k]);
  }
  __syncthreads();
  double sum = 0.0;  // lanes < 3 TB of warp 0: target tid / 3, component tid % 3
  int e2E;
  uint64_t e2M;
  const bool emu_ok = emu::unpack_eps2(eps2, e2E, e2M);  // integer-pipe pair factor usable
  const int64_t nchunks = (np + JC - 1) / JC;
  for (int64_t c = 0; c <= nchunks; c++) {
    if (w >= 0) {
      if (c + 1 < nchunks) {  // next chunk's sources into the other buffer
        const int64_t j1 = (c + 1) * JC;
        for (int k = w; k < JC; k += F64O_WORKERS) {
          const int64_t j = j1 + k;
          if (j < np) src[(c + 1) & 1][k] = make_dvec4(spos[3 * j], spos[3 * j + 1], spos[3 * j + 2], smass[j]);
        }
      }
      if (c < nchunks) {
        const int64_t j0 = c * JC;
        const int jn = (np - j0) < JC ? (int)(np - j0) : JC;
        const dvec4* sc = src[c & 1];
        double(*tc)[JP] = term[c & 1];
        for (int q = w; q < TB * JC; q += F64O_WORKERS) {
          const int t = q / JC, k = q % JC;
          if (k >= jn) continue;
          double vx = 0.0, vy = 0.0, vz = 0.0;
          if (!(SELF && j0 + k == t0 + t))
            f64_pair_terms<SELF>(sc[k], tp[t][0], tp[t][1], tp[t][2], eps2, emu_ok, e2E, e2M, vx, vy, vz);
          tc[3 * t + 0][k] = vx;
          tc[3 * t + 1][k] = vy;
          tc[3 * t + 2][k] = vz;
        }
      }
    } else if (c >= 1 && tid < 3 * TB) {  // previous chunk's terms, in order
      const int64_t j0 = (c - 1) * JC;
      const int jn = (np - j0) < JC ? (int)(np - j0) : JC;
      const double* row = term[(c - 1) & 1][tid];
      for (int k = 0; k < jn; k++) sum = dadd(sum, row[k]);
    }
    __syncthreads();
  }
  if (tid < 3 * TB) res[tid] = sum;
  __syncthreads();
  if (tid < TB && t0 + tid < nt) epi(t0 + tid, res[3 * tid], res[3 * tid + 1], res[3 * tid + 2]);
}

// ---------------------------------------------------------------------------
// Mixed form: FP32 pair arithmetic on coordinates relative to an origin, f32x2
// packed over pairs of targets, per-chunk FP32 partial sums folded into a
// (hi, lo) two-sum accumulator per target and component, FP64 epilogue.
//
// Work split ("stream-K"): the (target tile, source chunk) grid of
// n_tiles x chunks units is cut into `grid` equal contiguous ranges, one per
// persistent CTA.  A tile split across CTAs leaves per-CTA partials in scratch;
// the CTA that finishes last (per-tile counter) combines them in CTA order, so
// the result does not depend on timing, and runs the epilogue.
// ---------------------------------------------------------------------------
// Tile shapes of the mixed kernel: THREADS per CTA, P f32x2 packs (2P targets) per thread,
// MINB CTAs per SM, JT sources per chunk (a multiple of THREADS).  A chunk is both what
// shared memory holds and what is summed in plain FP32, so JT alone decides a result's
// FP32 rounding: shapes of one JT agree to the two-sums' 2^-48.
struct MixedShape {
  int threads, packs, minb, jt;
};
constexpr MixedShape kMixedShapes[] = {{256, 2, 2, 256}, {256, 4, 1, 256}, {128, 4, 2, 128}, {128, 2, 4, 128},
                                       {512, 2, 1, 512}, {256, 2, 3, 256}, {128, 2, 6, 128}, {256, 1, 4, 256},
                                       {512, 2, 2, 512}, {256, 2, 2, 256}, {512, 2, 1, 512}, {256, 4, 1, 256},
                                       {384, 3, 1, 384}, {64, 1, 8, 256}, {64, 1, 8, 128}, {64, 1, 6, 512}};
// Shapes 9-12 run the scalar FP32 loop (mixed_chunk_scalar); the others the packed f32x2
// loop.
constexpr int kNumMixedShapes = (int)(sizeof(kMixedShapes) / sizeof(kMixedShapes[0]));

struct StreamK {
  int64_t n_tiles;
  int64_t chunks;
  int64_t units;
  int64_t grid;
};

__host__ __device__ __forceinline__ int64_t sk_start(const StreamK& s, int64_t g) {
  return (g * s.units) / s.grid;
}
// CTA whose range contains unit u.
__host__ __device__ __forceinline__ int64_t sk_owner(const StreamK& s, int64_t u) {
  return ((u + 1) * s.grid + s.units - 1) / s.units - 1;
}

// One shared-memory chunk of JT sources against P packed target pairs: FP32 pair
// forces summed into a per-chunk partial, then folded into the (h, l) two-sum
// accumulator.  `tile` holds each source duplicated per lane: (x,x,y,y), (z,z,m,m).
// Per pair: 3 sub, 3 fma (r^2 + eps^2), 1 MUFU rsqrt, 3 mul, 3 fma.  EQ (all sources
// of one mass): the sum of r^-3 d without the mass, which the caller applies once per
// target; 2 multiplies per pair instead of 3.
template <bool GUARD, int P, int JT, bool EQ = false>
__device__ __forceinline__ void mixed_chunk(const float4* __restrict__ tile, const f2* tx, const f2* ty,
                                            const f2* tz, f2 E2, f2* hx, f2* hy, f2* hz, f2* lx, f2* ly,
                                            f2* lz) {
  f2 px[P], py[P], pz[P];
#pragma unroll
  for (int p = 0; p < P; p++) px[p] = py[p] = pz[p] = 0ull;
#pragma unroll 4
  for (int k = 0; k < JT; k++) {
    const float4 a = tile[2 * k + 0];
    const float4 b = tile[2 * k + 1];
    const f2 X = f2make(a.x, a.y), Y = f2make(a.z, a.w);
    const f2 Z = f2make(b.x, b.y), M = f2make(b.z, b.w);
#pragma unroll
    for (int p = 0; p < P; p++) {
      f2 dx = f2sub(X, tx[p]);
      f2 dy = f2sub(Y, ty[p]);
      f2 dz = f2sub(Z, tz[p]);
      f2 r2 = f2fma(dx, dx, E2);
      r2 = f2fma(dy, dy, r2);
      r2 = f2fma(dz, dz, r2);
      float r2a, r2b;
      f2split(r2, r2a, r2b);
      float ia = rsqrt_approx(r2a), ib = rsqrt_approx(r2b);
      if (GUARD) {
        ia = r2a > 0.f ? ia : 0.f;
        ib = r2b > 0.f ? ib : 0.f;
      }
      f2 ri = f2make(ia, ib);
      f2 ri2 = f2mul(ri, ri);
      f2 sc = EQ ? f2mul(ri, ri2) : f2mul(f2mul(M, ri), ri2);
      px[p] = f2fma(sc, dx, px[p]);
      py[p] = f2fma(sc, dy, py[p]);
      pz[p] = f2fma(sc, dz, pz[p]);
    }
  }
#pragma unroll
  for (int p = 0; p < P; p++) {
    f2 s, e;
    f2two_sum(hx[p], px[p], s, e);
    hx[p] = s;
    lx[p] = f2add(lx[p], e);
    f2two_sum(hy[p], py[p], s, e);
    hy[p] = s;
    ly[p] = f2add(ly[p], e);
    f2two_sum(hz[p], pz[p], s, e);
    hz[p] = s;
    lz[p] = f2add(lz[p], e);
  }
}

// The same chunk with scalar FP32 instructions (one target per instruction); its
// sources are stored once each, (x, y, z, m), not duplicated per lane pair.
template <bool GUARD, int P, int JT, bool EQ = false>
__device__ __forceinline__ void mixed_chunk_scalar(const float4* __restrict__ tile, const f2* tx, const f2* ty,
                                                   const f2* tz, f2 E2, f2* hx, f2* hy, f2* hz, f2* lx, f2* ly,
                                                   f2* lz) {
  constexpr int R = 2 * P;
  float sx[R], sy[R], sz[R], ax[R], ay[R], az[R];
#pragma unroll
  for (int p = 0; p < P; p++) {
    f2split(tx[p], sx[2 * p], sx[2 * p + 1]);
    f2split(ty[p], sy[2 * p], sy[2 * p + 1]);
    f2split(tz[p], sz[2 * p], sz[2 * p + 1]);
  }
  float e2, e2b;
  f2split(E2, e2, e2b);
#pragma unroll
  for (int r = 0; r < R; r++) ax[r] = ay[r] = az[r] = 0.f;
#pragma unroll 4
  for (int k = 0; k < JT; k++) {
    const float4 a = tile[k];  // (x, y, z, m): the scalar loop's undoubled layout
#pragma unroll
    for (int r = 0; r < R; r++) {
      const float dx = a.x - sx[r], dy = a.y - sy[r], dz = a.z - sz[r];
      const float r2 = fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, e2)));
      float ri = rsqrt_approx(r2);
      if (GUARD) ri = r2 > 0.f ? ri : 0.f;
      const float sc = EQ ? ri * (ri * ri) : (a.w * ri) * (ri * ri);
      ax[r] = fmaf(sc, dx, ax[r]);
      ay[r] = fmaf(sc, dy, ay[r]);
      az[r] = fmaf(sc, dz, az[r]);
    }
  }
#pragma unroll
  for (int p = 0; p < P; p++) {
    f2 s, e;
    f2two_sum(hx[p], f2make(ax[2 * p], ax[2 * p + 1]), s, e);
    hx[p] = s;
    lx[p] = f2add(lx[p], e);
    f2two_sum(hy[p], f2make(ay[2 * p], ay[2 * p + 1]), s, e);
    hy[p] = s;
    ly[p] = f2add(ly[p], e);
    f2two_sum(hz[p], f2make(az[2 * p], az[2 * p + 1]), s, e);
    hz[p] = s;
    lz[p] = f2add(lz[p], e);
  }
}

// Per-CTA scratch for split tiles: 2 slots (first and last tile of its range),
// each 6 floats (hi/lo for x, y, z) per target of a tile.
__host__ __device__ constexpr int64_t mixed_slot_floats(int threads, int packs) {
  return (int64_t)6 * threads * 2 * packs;
}

template <bool GUARD, int THREADS, int P, int MINB, class Epi, bool PACKED = true, int JT = THREADS>
__global__ void __launch_bounds__(THREADS, MINB)
    direct_mixed_kernel(const float4* __restrict__ src, int64_t np, const float4* __restrict__ tgt,
                        int64_t nt, float eps2, StreamK sk, float* __restrict__ partials,
                        int* __restrict__ counters, Epi epi, const double* __restrict__ eqm) {
  constexpr int R = 2 * P, TILE = THREADS * R;
  constexpr int JS = JT / THREADS;  // sources of a chunk staged by each thread
  static_assert(JT % THREADS == 0, "whole rows of sources");
  constexpr int64_t SLOT = mixed_slot_floats(THREADS, P);
  // Sources duplicated per lane pair: (x,x,y,y) and (z,z,m,m).
  __shared__ __align__(16) float4 tile[2 * 2 * JT];
  __shared__ int s_last;
  const int tid = threadIdx.x;
  int buf = 0;
  const int64_t g = blockIdx.x;
  const int64_t u_begin = sk_start(sk, g), u_end = sk_start(sk, g + 1);
  const f2 E2 = f2make(eps2, eps2);
  // *eqm: the sources' common mass when every source has it (0: masses differ, or no
  // pointer); then the chunks sum r^-3 d and each target's sum is scaled by it once
  const double mq = eqm ? __ldg(eqm) : 0.0;
  const bool eq = mq != 0.0;
  const double msc = eq ? mq : 1.0;  // x * 1.0 == x: the general path's bits are unchanged

  int64_t u = u_begin;
  while (u < u_end) {
    const int64_t t = u / sk.chunks;
    const int64_t c0 = u - t * sk.chunks;
    const int64_t c1 = (sk.chunks - c0) < (u_end - u) ? sk.chunks : c0 + (u_end - u);
    u += c1 - c0;

    // Targets of tile t: target r of this thread is t*TILE + r*THREADS + tid.
    f2 tx[P], ty[P], tz[P];
    f2 hx[P], hy[P], hz[P], lx[P], ly[P], lz[P];
#pragma unroll
    for (int p = 0; p < P; p++) {
      float4 q[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        int64_t i = t * TILE + (2 * p + h) * THREADS + tid;
        q[h] = i < nt ? tgt[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      tx[p] = f2make(q[0].x, q[1].x);
      ty[p] = f2make(q[0].y, q[1].y);
      tz[p] = f2make(q[0].z, q[1].z);
      hx[p] = hy[p] = hz[p] = lx[p] = ly[p] = lz[p] = 0ull;
    }

    // Double-buffered chunks: the next chunk's source is loaded into a register while
    // the current one is computed, and written to the other buffer afterwards, so one
    // barrier per chunk suffices (the barrier of chunk c orders every read of the
    // buffer it reuses, last read in chunk c-1).  Padding sources have zero mass at the
    // origin: their terms are exactly 0.
    // With equal masses (eq) a staged source's w is 1 (0 for padding past the last
    // source) instead of its mass: the equal-mass loop, which ignores w, runs only on
    // full chunks, and the general loop on the partial last chunk then gives r^-3 d
    // for a source and exactly 0 for padding.
    float4 pre[JS];
    auto load = [&](int64_t c) {
#pragma unroll
      for (int q = 0; q < JS; q++) {
        const int64_t j = c * JT + q * THREADS + tid;
        pre[q] = j < np ? src[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (eq) pre[q].w = j < np ? 1.f : 0.f;
      }
    };
    load(c0);
    for (int64_t c = c0; c < c1; c++) {
      float4* tb = tile + buf * (2 * JT);
#pragma unroll
      for (int q = 0; q < JS; q++) {
        const int k = q * THREADS + tid;
        if (PACKED) {
          tb[2 * k + 0] = make_float4(pre[q].x, pre[q].x, pre[q].y, pre[q].y);
          tb[2 * k + 1] = make_float4(pre[q].z, pre[q].z, pre[q].w, pre[q].w);
        } else {
          tb[k] = pre[q];
        }
      }
      __syncthreads();
      if (c + 1 < c1) load(c + 1);
      const bool eq_loop = eq && (c + 1) * JT <= np;  // a full chunk of equal masses
      if (PACKED) {
        if (eq_loop)
          mixed_chunk<GUARD, P, JT, true>(tb, tx, ty, tz, E2, hx, hy, hz, lx, ly, lz);
        else
          mixed_chunk<GUARD, P, JT>(tb, tx, ty, tz, E2, hx, hy, hz, lx, ly, lz);
      } else {
        if (eq_loop)
          mixed_chunk_scalar<GUARD, P, JT, true>(tb, tx, ty, tz, E2, hx, hy, hz, lx, ly, lz);
        else
          mixed_chunk_scalar<GUARD, P, JT>(tb, tx, ty, tz, E2, hx, hy, hz, lx, ly, lz);
      }
      buf ^= 1;
    }

    const bool whole = (c0 == 0 && c1 == sk.chunks);
    if (whole) {
#pragma unroll
      for (int p = 0; p < P; p++) {
        float a[6], b[6];
        f2split(hx[p], a[0], b[0]);
        f2split(lx[p], a[1], b[1]);
        f2split(hy[p], a[2], b[2]);
        f2split(ly[p], a[3], b[3]);
        f2split(hz[p], a[4], b[4]);
        f2split(lz[p], a[5], b[5]);
        int64_t i0 = t * TILE + (2 * p) * THREADS + tid;
        int64_t i1 = i0 + THREADS;
        if (i0 < nt)
          epi(i0, msc * ((double)a[0] + (double)a[1]), msc * ((double)a[2] + (double)a[3]),
              msc * ((double)a[4] + (double)a[5]));
        if (i1 < nt)
          epi(i1, msc * ((double)b[0] + (double)b[1]), msc * ((double)b[2] + (double)b[3]),
              msc * ((double)b[4] + (double)b[5]));
      }
      continue;
    }

    // Split tile: publish this CTA's partial, count in, last one combines.
    const int64_t first_tile = u_begin / sk.chunks;
    float* slot = partials + (2 * g + (t == first_tile ? 0 : 1)) * SLOT;
#pragma unroll
    for (int p = 0; p < P; p++) {
      float a[6], b[6];
      f2split(hx[p], a[0], b[0]);
      f2split(lx[p], a[1], b[1]);
      f2split(hy[p], a[2], b[2]);
      f2split(ly[p], a[3], b[3]);
      f2split(hz[p], a[4], b[4]);
      f2split(lz[p], a[5], b[5]);
      const int r0 = 2 * p, r1 = 2 * p + 1;
#pragma unroll
      for (int q = 0; q < 6; q++) {
        slot[(int64_t)q * TILE + r0 * THREADS + tid] = a[q];
        slot[(int64_t)q * TILE + r1 * THREADS + tid] = b[q];
      }
    }
    __threadfence();
    __syncthreads();
    const int64_t g_first = sk_owner(sk, t * sk.chunks);
    const int64_t g_last = sk_owner(sk, t * sk.chunks + sk.chunks - 1);
    if (tid == 0) {
      int prev = atomicAdd(&counters[t], 1);
      s_last = (prev == (int)(g_last - g_first));
    }
    __syncthreads();
    if (!s_last) continue;
    __threadfence();
    // The partials of CTAs g_first .. g_last in that order, RG of this thread's targets at
    // a time (one target at a time, with the two 64-bit divisions of each CTA's range
    // start in its loop, took 45 of a step's 180 us at N = 16,384).  A CTA's first tile is
    // in its slot 0: this tile is the first of every CTA but possibly g_first, whose range
    // may begin in an earlier tile.
    constexpr int RG = R > 4 ? R / 2 : R;
    const int64_t first_slot = 2 * g_first + (t == sk_start(sk, g_first) / sk.chunks ? 0 : 1);
    const int parts = (int)(g_last - g_first) + 1;
    for (int r0 = 0; r0 < R; r0 += RG) {
      float h[RG][3], l[RG][3];
#pragma unroll
      for (int r = 0; r < RG; r++)
#pragma unroll
        for (int k = 0; k < 3; k++) h[r][k] = l[r][k] = 0.f;
      const float* sl = partials + first_slot * SLOT + r0 * THREADS + tid;
      const float* rest = partials + 2 * (g_first + 1) * SLOT + r0 * THREADS + tid;
#pragma unroll 2
      for (int q = 0; q < parts; q++) {
#pragma unroll
        for (int r = 0; r < RG; r++)
#pragma unroll
          for (int k = 0; k < 3; k++) {
            const float ph = __ldcg(sl + (2 * k) * TILE + r * THREADS);
            const float pl = __ldcg(sl + (2 * k + 1) * TILE + r * THREADS);
            float s, e;
            two_sum(h[r][k], ph, s, e);
            h[r][k] = s;
            l[r][k] = __fadd_rn(l[r][k], __fadd_rn(pl, e));
          }
        sl = rest;
        rest += 2 * SLOT;
      }
#pragma unroll
      for (int r = 0; r < RG; r++) {
        const int64_t i = t * TILE + (r0 + r) * THREADS + tid;
        if (i < nt)
          epi(i, msc * ((double)h[r][0] + (double)l[r][0]), msc * ((double)h[r][1] + (double)l[r][1]),
              msc * ((double)h[r][2] + (double)l[r][2]));
      }
    }
    if (tid == 0) counters[t] = 0;  // ready for the next launch
  }
}

// Launch helper shared by the force call, the run loop and the no-alloc variant.
// `grid_cap` bounds the persistent grid (2 slots of partials per CTA in scratch).
StreamK mixed_plan(int64_t np, int64_t nt, int64_t grid_cap, int tile, int jt);

}  // namespace gh
