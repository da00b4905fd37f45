// Barnes-Hut octree on the GPU with the reference's exact cell geometry and
// opening decisions (gravhopper/_jbgrav.c:360-541, 737-806).
//
// Build (every force evaluation):
//   1. bounding box and root cell with the reference's boxsize rule (_jbgrav.c:747-775);
//   2. per-particle octant keys: at each level the octant is (x>cx, y>cy, z>cz) and the
//      child centre is c + (+-0.5*halfsize), the same FP64 recurrence as
//      gravoct_calc_subnode / gravoct_add_particle (_jbgrav.c:403-428, 453-462); read
//      off the bits of (p - c_0)/size wherever that provably gives the same decisions.
//      21 levels per 64-bit word, MSB first, digit = x | y<<1 | z<<2 (the reference's
//      branch number, _jbgrav.c:441-450), so key order is depth-first order with
//      children in branch order 0..7.  The number of words grows until no two
//      particles share a full key (coincident particles end with GH_ERR_DEPTH);
//   3. sort of the keys: a radix sort of the first word, then runs of equal first
//      words ordered by the other words (a full multi-word radix sort for long runs);
//   4. the node set of the reference's uncompressed octree (every cell that holds a
//      particle and whose parent holds at least two, single-child chains included)
//      laid out in depth-first preorder with skip ("next") indices, from the common
//      prefix lengths of neighbouring keys;
//   5. monopoles: leaves take the particle's position and mass exactly
//      (gravoct_finalize, _jbgrav.c:467-483); a cell holds a contiguous range of the
//      key-ordered particles, so its mass and first moment are differences of exact
//      192-bit fixed-point prefix sums, rounded to FP64 once (the reference rounds
//      after every particle it adds, in insertion order, so the last bits of an
//      internal COM can differ), and the centre of mass is first moment over mass.
// Small systems take the same steps in six launches, the keys ranked by comparison.
// Walk: one warp per 32 consecutive targets in key order.  Each lane applies the
// reference's test "leaf or size/|center - x| < theta" (_jbgrav.c:496-502) to every
// cell its own traversal reaches; the warp visits the union of those cells in
// preorder, a lane skipping the subtrees it accepted.  The test is decided in FP32
// from hi/lo split coordinates with a 1e-4 relative margin; inside the margin it is
// recomputed with the reference's FP64 operations, so every lane takes exactly the
// reference's decisions.  Accepted cells contribute (COM - x) m / (r^2 + eps^2)^1.5 in
// FP64, with the reference's zero for r^2 + eps^2 == 0 (_jbgrav.c:514-520).  An FP64 walk
// of few targets is split over several warps per 32 of them by ranges of the preorder.
#include <cmath>
#include <mutex>

#include "direct.cuh"
#include "engine.h"
#include "fixed192.cuh"
#include "sort.cuh"

namespace gh {

constexpr int KEY_LEVELS = 21;
constexpr int KEY_BITS = 63;
constexpr int TREE_MIN_WORDS = 2;
constexpr int TREE_MAX_WORDS = 6;
constexpr double TREE_MARGIN = 1e-4;

struct TreeRoot {
  double c[3];
  double size;
  double inv;           // RN(1 / size)
  float invf;
  long long margin;     // 0: fast keys allowed; -1: the FP64 recurrence for every particle
  int bad;              // a particle position or mass is NaN or infinite
  int lsb_m, lsb_f;     // fixed-point units (2^lsb) of the mass and first-moment sums
};

// ---------------------------------------------------------------------------
// 1. Bounding box and root cell
// ---------------------------------------------------------------------------
constexpr int BB_THREADS = 256;
constexpr int BB_BLOCKS = 304;

// Doubles ordered as integers (-0.0 below 0.0): comparisons of doubles would be FP64-pipe
// instructions.
__device__ __forceinline__ int64_t ordered_bits(double x) {
  const int64_t b = __double_as_longlong(x);
  return b ^ (int64_t)((uint64_t)(b >> 63) >> 1);
}
__device__ __forceinline__ double from_ordered(int64_t o) {
  return __longlong_as_double(o ^ (int64_t)((uint64_t)(o >> 63) >> 1));
}

struct Box {
  int64_t mn[3], mx[3];  // ordered_bits
  int64_t m;             // bits of the largest |mass|
  bool bad;              // a position or mass is not finite
};

__device__ __forceinline__ Box box_empty() {
  Box b;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    b.mn[k] = 0x7FF0000000000000ll;               // +inf
    b.mx[k] = 0x7FF0000000000000ll ^ -1ll;        // below every finite double
  }
  b.m = 0;
  b.bad = false;
  return b;
}

__device__ __forceinline__ void box_add(Box& b, const double* __restrict__ pos, const double* __restrict__ mass,
                                        int64_t i) {
  const int64_t mb = __double_as_longlong(mass[i]) & 0x7FFFFFFFFFFFFFFFll;
  b.bad = b.bad || mb >= 0x7FF0000000000000ll;
  b.m = mb > b.m ? mb : b.m;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double q = pos[3 * i + k];
    b.bad = b.bad || (__double_as_longlong(q) & 0x7FF0000000000000ll) == 0x7FF0000000000000ll;
    const int64_t o = ordered_bits(q);
    b.mn[k] = o < b.mn[k] ? o : b.mn[k];
    b.mx[k] = o > b.mx[k] ? o : b.mx[k];
  }
}

__device__ __forceinline__ void box_merge(Box& a, const Box& b) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    a.mn[k] = b.mn[k] < a.mn[k] ? b.mn[k] : a.mn[k];
    a.mx[k] = b.mx[k] > a.mx[k] ? b.mx[k] : a.mx[k];
  }
  a.m = b.m > a.m ? b.m : a.m;
  a.bad = a.bad || b.bad;
}

// Merges the lanes' boxes; every lane gets the result.
__device__ __forceinline__ void box_warp(Box& b) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Box c;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      c.mn[k] = __shfl_xor_sync(0xffffffffu, b.mn[k], o);
      c.mx[k] = __shfl_xor_sync(0xffffffffu, b.mx[k], o);
    }
    c.m = __shfl_xor_sync(0xffffffffu, b.m, o);
    c.bad = false;
    box_merge(b, c);
  }
  b.bad = __any_sync(0xffffffffu, b.bad);
}

// Merges a block's boxes (T threads); warp 0 gets the result.
template <int T>
__device__ __forceinline__ void box_block(Box& b) {
  __shared__ Box part[T / 32];
  box_warp(b);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = b;
  __syncthreads();
  if (threadIdx.x < 32) {
    b = threadIdx.x < T / 32 ? part[threadIdx.x] : box_empty();
    box_warp(b);
  }
}

__global__ void __launch_bounds__(BB_THREADS)
    bbox_partial_kernel(const double* __restrict__ pos, const double* __restrict__ mass, int64_t n,
                        Box* __restrict__ part) {
  Box b = box_empty();
  for (int64_t i = (int64_t)blockIdx.x * BB_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * BB_THREADS)
    box_add(b, pos, mass, i);
  box_block<BB_THREADS>(b);
  if (threadIdx.x == 0) part[blockIdx.x] = b;
}

// treeforce_workhorse, _jbgrav.c:764-772: boxsize = extent_x + eps, replaced by
// extent_i + eps when extent_i (without eps) exceeds it; centre = bbox midpoint.
//
// Fast keys.  The reference's cell centres follow c_{l+1} = RN(c_l +- size 2^-(l+2)).
// Along a particle's own path the level-(l+1) centre lies within size 2^-(l+2) of p,
// so that rounding moves it by at most 2^-53 (|p| + size 2^-(l+2)), and after 42
// levels the centre is within E_c = 2^-53 (42 |p| + size/2) of the exact dyadic
// centre (per axis).  With t = (p - c_0) / size + 1/2 computed as
// fma(p - c_0, RN(1/size), 1/2) (error below 2^-52), each of the first 42 octant
// decisions "p > c_l" equals the bit of t at that level unless t lies within
// E_c / size + 2^-52 of a multiple of 2^-42.  keys_kernel keeps that window, doubled,
// in units of 2^-63; particles inside it take the reference's FP64 recurrence, as do
// all particles when the box size is outside [2^-900, 2^900] (margin -1).
__device__ __forceinline__ void root_write(const Box& box, double eps, TreeRoot* __restrict__ root) {
  double mn[3], mx[3];
  for (int k = 0; k < 3; k++) {
    mn[k] = from_ordered(box.mn[k]);
    mx[k] = from_ordered(box.mx[k]);
  }
  const bool bad = box.bad;
  const double mmax = __longlong_as_double(box.m);
  double bs = dadd(dsub(mx[0], mn[0]), eps);
  for (int k = 1; k < 3; k++)
    if (dsub(mx[k], mn[k]) > bs) bs = dadd(dsub(mx[k], mn[k]), eps);
  double amax = 0.0;
  for (int k = 0; k < 3; k++) {
    root->c[k] = dmul(0.5, dadd(mn[k], mx[k]));
    amax = fmax(amax, fabs(root->c[k]));
  }
  root->size = bs;
  root->bad = bad ? 1 : 0;
  // fixed-point units: |m| < 2^Bm and |m x| < 2^(Bm + Bx + 1) (the product's rounding
  // included), headroom for 2^24 particles (fixed192.cuh); floored so that sums of
  // exotic tiny inputs stay normal doubles
  if (!bad) {
    double xmax = 0.0;
    for (int k = 0; k < 3; k++) xmax = fmax(xmax, fmax(fabs(mn[k]), fabs(mx[k])));
    const int bm = fx::bound_exponent(mmax), bx = fx::bound_exponent(xmax);
    root->lsb_m = max(bm - fx::FX_HEADROOM, -1000);
    root->lsb_f = max(bm + bx + 1 - fx::FX_HEADROOM, -1000);
  } else {
    root->lsb_m = root->lsb_f = 0;
  }
  root->inv = ddiv(1.0, bs);
  root->invf = (float)root->inv;
  root->margin = (bs > 0x1p-900 && bs < 0x1p+900 && amax < 0x1p+900) ? 0 : -1;
}

// One warp folds the per-block boxes.
__global__ void root_kernel(const Box* __restrict__ part, int nb, double eps, TreeRoot* __restrict__ root) {
  Box b = box_empty();
  for (int k = threadIdx.x; k < nb; k += 32) box_merge(b, part[k]);
  box_warp(b);
  if (threadIdx.x == 0) root_write(b, eps, root);
}

// Both for a small system, in one block.
constexpr int SB_THREADS = 1024;
__global__ void __launch_bounds__(SB_THREADS)
    box_root_kernel(const double* __restrict__ pos, const double* __restrict__ mass, int64_t n, double eps,
                    TreeRoot* __restrict__ root) {
  Box b = box_empty();
  for (int64_t i = threadIdx.x; i < n; i += SB_THREADS) box_add(b, pos, mass, i);
  box_block<SB_THREADS>(b);
  if (threadIdx.x == 0) root_write(b, eps, root);
}

// ---------------------------------------------------------------------------
// 2. Octant keys
// ---------------------------------------------------------------------------
constexpr int TREE_MAX_LEVELS = KEY_LEVELS * TREE_MAX_WORDS;

// Spreads the low 21 bits of v to every third bit (bit b to bit 3b).
__device__ __forceinline__ uint64_t spread3(uint64_t v) {
  v &= 0x1fffffull;
  v = (v | (v << 32)) & 0x001f00000000ffffull;
  v = (v | (v << 16)) & 0x001f0000ff0000ffull;
  v = (v | (v << 8)) & 0x100f00f00f00f00full;
  v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
  v = (v | (v << 2)) & 0x1249249249249249ull;
  return v;
}

__device__ __forceinline__ unsigned lane_mask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Appends i to list (warp-aggregated) where `need`; every lane of the warp calls it.
__device__ __forceinline__ void warp_append(bool need, int64_t i, int* __restrict__ list, int* __restrict__ count) {
  const unsigned mask = __ballot_sync(0xffffffffu, need);
  if (!mask) return;
  int base = 0;
  if ((threadIdx.x & 31) == 0) base = atomicAdd(count, __popc(mask));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (need) list[base + __popc(mask & lane_mask_lt())] = (int)i;
}

// Fast keys where the decisions are provably the recurrence's (see root_write); the
// block's other particles (about 2 %) then take the reference's recurrence
// (gravoct_calc_subnode, _jbgrav.c:441-462), compacted so that it runs on full warps: it
// is a chain of FP64 additions, each 20 cycles of the SM for a warp however many of its
// lanes take part.  "p > c" is decided on the doubles' bits, in an order-preserving integer
// form, which leaves the additions alone on the FP64 pipe (a DSETP costs as much as one).
// N = 2000 26 -> 11 us, 60,013 39 -> 13, 1M 85 -> 58 against a fast-key kernel and a
// recurrence kernel on a global list (52 us of the 85 were FP64-pipe comparisons, scalings
// and conversions of the fast keys).  Blocks of 1024 from four blocks of 256 per SM on:
// fewer, fuller warps in the chain.

// floor(t 2^63) of t in (0, 1), 2^63 from 1 on, 0 for t <= 0: off the bits of t (its
// comparisons, its scaling and its conversion would all be FP64-pipe instructions).
__device__ __forceinline__ uint64_t unit_bits(double t) {
  const int64_t b = __double_as_longlong(t);
  if (b >= 0x3FF0000000000000ll) return 1ull << 63;
  const uint64_t m = (((uint64_t)b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull) << 10;
  return b <= 0 ? 0ull : emu::shr_clamp(m, 1022 - (int)(b >> 52));
}

// |p| in FP32, short by less than 2^-20 of it (2^-126 for anything smaller, infinity
// beyond the range).
__device__ __forceinline__ float abs_f32(double p) {
  const uint64_t b = (uint64_t)__double_as_longlong(p);
  const int e = ((int)(b >> 52) & 0x7FF) - 896;
  const float f = __uint_as_float(((uint32_t)e << 23) | ((uint32_t)(b >> 29) & 0x7FFFFFu));
  return e <= 0 ? 0x1p-126f : (e >= 255 ? INFINITY : f);
}

template <int T>
__global__ void __launch_bounds__(T)
    keys_kernel(const double* __restrict__ pos, int64_t n, const TreeRoot* __restrict__ root, int words,
                uint64_t* __restrict__ keys, uint32_t* __restrict__ idx) {
  __shared__ int list[T];
  __shared__ int count;
  __shared__ double offs[TREE_MAX_LEVELS];  // child-centre offsets 0.5 * halfsize = size 2^-(l+2), exact
  const double S = root->size;
  for (int l = threadIdx.x; l < words * KEY_LEVELS; l += T)
    offs[l] = dmul(S, __longlong_as_double((long long)(1023 - (l + 2)) << 52));
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * T + threadIdx.x;
  bool need = false;
  if (i < n) {
    idx[i] = (uint32_t)i;
    need = true;
    if (root->margin >= 0 && words == 2) {
      uint64_t K[3];
      bool ok = true;
      const double inv = root->inv;
      const float invf = root->invf;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const double p = pos[3 * i + k];
        K[k] = unit_bits(fma(dsub(p, root->c[k]), inv, 0.5));
        // 2 * 2^63 * (E_c / size + 2^-52) + slack, in FP32 (a bound, not a value)
        const float mf = fmaf(86016.f * 1.01f * abs_f32(p), invf, 5200.f);
        const uint64_t r = K[k] & ((1ull << 21) - 1);
        ok = ok && mf < 1048576.f && r > (uint64_t)mf && r < (1ull << 21) - (uint64_t)mf;
      }
      if (ok) {
        keys[i] = spread3(K[0] >> 42) | (spread3(K[1] >> 42) << 1) | (spread3(K[2] >> 42) << 2);
        keys[n + i] = spread3(K[0] >> 21) | (spread3(K[1] >> 21) << 1) | (spread3(K[2] >> 21) << 2);
        need = false;
      }
    }
  }
  warp_append(need, i, list, &count);
  __syncthreads();
  if (threadIdx.x >= count) return;
  const int64_t j = list[threadIdx.x];
  // adding 0.0 turns -0.0, which ordered_bits puts below 0.0, into 0.0; the sums below
  // are never -0.0
  const int64_t q0 = ordered_bits(dadd(pos[3 * j], 0.0)), q1 = ordered_bits(dadd(pos[3 * j + 1], 0.0)),
                q2 = ordered_bits(dadd(pos[3 * j + 2], 0.0));
  double c0 = dadd(root->c[0], 0.0), c1 = dadd(root->c[1], 0.0), c2 = dadd(root->c[2], 0.0);
  for (int w = 0; w < words; w++) {
    uint64_t k = 0;
#pragma unroll 3
    for (int l = 0; l < KEY_LEVELS; l++) {
      const double off = offs[w * KEY_LEVELS + l];
      const unsigned g0 = q0 > ordered_bits(c0), g1 = q1 > ordered_bits(c1), g2 = q2 > ordered_bits(c2);
      c0 = dadd(c0, g0 ? off : -off);
      c1 = dadd(c1, g1 ? off : -off);
      c2 = dadd(c2, g2 ? off : -off);
      k = (k << 3) | (uint64_t)(g0 | (g1 << 1) | (g2 << 2));
    }
    keys[(int64_t)w * n + j] = k;
  }
}

// Keys of target points (two words, 42 levels of the sources' root cell; points
// outside it clamped to its faces) for the walk's order only: warps that hold
// neighbouring targets visit nearly the same cells.  Any order gives each target the
// same decisions and interactions, so these keys need not be the reference's.
__global__ void target_keys_kernel(const double* __restrict__ tpos, int64_t nt, const TreeRoot* __restrict__ root,
                                   uint64_t* __restrict__ keys, uint32_t* __restrict__ idx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nt) return;
  uint64_t T[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double t = fma(tpos[3 * i + k] - root->c[k], root->inv, 0.5);
    T[k] = t >= 1.0 ? ((1ull << 63) - 1) : (t > 0.0 ? (uint64_t)(t * 0x1p63) : 0ull);  // NaN: 0
  }
  keys[i] = spread3(T[0] >> 42) | (spread3(T[1] >> 42) << 1) | (spread3(T[2] >> 42) << 2);
  keys[nt + i] = spread3(T[0] >> 21) | (spread3(T[1] >> 21) << 1) | (spread3(T[2] >> 21) << 2);
  idx[i] = (uint32_t)i;
}

__device__ __forceinline__ int key_lcp(const uint64_t* __restrict__ keys, int words, int64_t n, int64_t a,
                                       int64_t b) {
  for (int w = 0; w < words; w++) {
    uint64_t x = keys[(int64_t)w * n + a] ^ keys[(int64_t)w * n + b];
    if (x) return w * KEY_LEVELS + (__clzll((long long)x) - 1) / 3;
  }
  return words * KEY_LEVELS;
}

__device__ __forceinline__ unsigned key_digit(const uint64_t* __restrict__ keys, int64_t n, int64_t i, int level) {
  const int w = level / KEY_LEVELS, l = level - w * KEY_LEVELS;
  return (unsigned)((keys[(int64_t)w * n + i] >> (3 * (KEY_LEVELS - 1 - l))) & 7u);
}

// ---------------------------------------------------------------------------
// 3. Sort: the first key word with a radix sort, then the rare runs of equal first
//    words ordered by the remaining words in place.  Equal full keys make the build
//    widen the keys and start again, so the final order is the full-key order.
// ---------------------------------------------------------------------------
constexpr int TIE_MAX_RUN = 256;  // longer runs of equal first words: full radix sort

// Brings key words 1.. into the order of the sorted first word: out[w][i] = in[w][idx[i]].
__global__ void gather_words_kernel(const uint64_t* __restrict__ kin, uint64_t* __restrict__ kout, int words,
                                    int64_t n, const uint32_t* __restrict__ idx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t src = idx[i];
  for (int w = 1; w < words; w++) kout[(int64_t)w * n + i] = kin[(int64_t)w * n + src];
}

__device__ __forceinline__ bool tied_first_word(const uint64_t* __restrict__ k0, int64_t n, int64_t i) {
  const uint64_t k = k0[i];
  return (i > 0 && k0[i - 1] == k) || (i + 1 < n && k0[i + 1] == k);
}

// Each particle in a run of equal first words takes its rank within the run by
// (words 1.., original index) and writes its key and index to that slot of the
// temporaries; flags[2] marks a run longer than TIE_MAX_RUN.
__global__ void tie_rank_kernel(const uint64_t* __restrict__ keys, int words, int64_t n,
                                const uint32_t* __restrict__ idx, uint64_t* __restrict__ kt,
                                uint32_t* __restrict__ it, int* __restrict__ flags) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !tied_first_word(keys, n, i)) return;
  const uint64_t k = keys[i];
  if ((i >= TIE_MAX_RUN && keys[i - TIE_MAX_RUN] == k) || (i + TIE_MAX_RUN < n && keys[i + TIE_MAX_RUN] == k)) {
    atomicOr(&flags[2], 1);  // sorted keys: the run is longer than TIE_MAX_RUN
    return;
  }
  int64_t s = i, e = i + 1;
  while (s > 0 && keys[s - 1] == k) {
    if (i - --s >= TIE_MAX_RUN) {
      atomicOr(&flags[2], 1);
      return;
    }
  }
  while (e < n && keys[e] == k) {
    if (++e - i > TIE_MAX_RUN) {
      atomicOr(&flags[2], 1);
      return;
    }
  }
  const uint32_t me = idx[i];
  int64_t r = 0;
  for (int64_t j = s; j < e; j++) {
    if (j == i) continue;
    int c = 0;  // -1: j before i, +1: j after i
    for (int w = 1; w < words && c == 0; w++) {
      const uint64_t a = keys[(int64_t)w * n + j], b = keys[(int64_t)w * n + i];
      c = a < b ? -1 : (a > b ? 1 : 0);
    }
    if (c < 0 || (c == 0 && idx[j] < me)) r++;
  }
  for (int w = 1; w < words; w++) kt[(int64_t)w * n + s + r] = keys[(int64_t)w * n + i];
  it[s + r] = me;
}

__global__ void tie_copy_kernel(uint64_t* __restrict__ keys, int words, int64_t n, uint32_t* __restrict__ idx,
                                const uint64_t* __restrict__ kt, const uint32_t* __restrict__ it) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !tied_first_word(keys, n, i)) return;
  for (int w = 1; w < words; w++) keys[(int64_t)w * n + i] = kt[(int64_t)w * n + i];
  idx[i] = it[i];
}

// flags[0]: two particles share a full key; flags[1]: deepest leaf level.
__global__ void lcp_kernel(const uint64_t* __restrict__ keys, int words, int64_t n, int* __restrict__ lp,
                           int* __restrict__ flags) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  if (i == 0 || i == n) {
    lp[i] = -1;
    return;
  }
  int l = key_lcp(keys, words, n, i - 1, i);
  lp[i] = l;
  if (l >= words * KEY_LEVELS) atomicOr(&flags[0], 1);
}

// Leaf level d_i = 1 + max(common prefix with either neighbour); particle i opens
// the cells at levels lp[i]+1 .. d_i (count d_i - lp[i]).
__global__ void count_kernel(const int* __restrict__ lp, int64_t n, int* __restrict__ cnt,
                             int* __restrict__ depth, int* __restrict__ flags) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int d = 0;
  if (i < n) {
    const int a = lp[i], b = lp[i + 1];
    d = 1 + (a > b ? a : b);
    depth[i] = d;
    cnt[i] = d - a;
  }
  d = __reduce_max_sync(0xffffffffu, d);
  if ((threadIdx.x & 31) == 0 && d > flags[1]) atomicMax(&flags[1], d);  // flags[1] only grows
}

// ---------------------------------------------------------------------------
// 4. Nodes in preorder
// ---------------------------------------------------------------------------
// The walk's per-node record, 48 bytes (two 32-byte sectors) per visited cell.  A
// leaf's "centre" is its particle's position and its offset is zero, so the offset
// from the target computed for the opening test is, plus O, the offset of the centre
// of mass: accepted cells are at least size/theta away, so O's FP32 rounding is below
// 2^-24 theta of the distance.
struct __align__(16) WalkRec {
  float4 A;   // (cx_hi, cy_hi, cz_hi, size^2)        FP32 opening prefilter
  float4 L;   // (cx_lo, cy_lo, cz_lo, next as bits)   FP32 residuals + skip index
  float4 O;   // (com - c as FP32, mass)              mixed-precision interaction
};

struct NodeArrays {
  WalkRec* R;    // walk records (A, L, O)
  dvec4* C;      // (cx, cy, cz, size)                    exact opening test (internal cells)
  dvec4* M;      // (comx, comy, comz, mass)              interaction
};

// Exact prefix sums over the key-ordered particles: mass and first moment x, y, z.
struct FxMoments {
  fx::I192 c[4];
};
// Two particles per thread: eight left a build of 60,013 particles with 30 blocks in a chain
// of gathers (48 us against 12; whole build 254 -> 221 us, 1,048,576 1059 -> 1011, 4,000,000
// 3640 -> 3365), one costs more scans (1,048,576 1074).
constexpr int MS_THREADS = 256, MS_ITEMS = 2, MS_TILE = MS_THREADS * MS_ITEMS, MS_BITS = 9;
static_assert(MS_TILE == 1 << MS_BITS, "tiles are found by a shift");
constexpr int SB_BITS = 8;  // small builds: tiles of one particle per thread

__device__ __forceinline__ void fxm_add(FxMoments& a, const FxMoments& b) {
#pragma unroll
  for (int k = 0; k < 4; k++) a.c[k] = fx::add(a.c[k], b.c[k]);
}

__device__ __forceinline__ FxMoments fxm_zero() {
  FxMoments r;
#pragma unroll
  for (int k = 0; k < 4; k++) r.c[k] = fx::zero();
  return r;
}

// Prefix over the first j key-ordered particles (j <= n): the tile's prefix plus the
// prefix within the tile.
__device__ __forceinline__ FxMoments fxm_prefix(const FxMoments* __restrict__ local,
                                                const FxMoments* __restrict__ tiles, int tile_bits, int64_t j,
                                                int64_t n) {
  if (j >= n) return tiles[((n - 1) >> tile_bits) + 1];
  FxMoments r = tiles[j >> tile_bits];
  fxm_add(r, local[j]);
  return r;
}

__device__ __forceinline__ float f32_hi(double v) { return (float)v; }
__device__ __forceinline__ float f32_lo(double v, float hi) { return (float)(v - (double)hi); }

// First particle after i that shares fewer than L leading digits with it: a short
// scan of the neighbour prefixes, then a binary search on the keys.
__device__ __forceinline__ int64_t cell_end(const uint64_t* __restrict__ keys, int words, int64_t n,
                                            const int* __restrict__ lp, int64_t i, int L) {
  int64_t j = i + 1;
  for (int s = 0; s < 16; s++, j++)
    if (lp[j] < L) return j;  // lp[n] = -1 ends the scan
  int64_t a = j - 1, b = n - 1;  // a shares >= L digits with i
  // gallop: most cells are small, so bracket the end before bisecting
  for (int64_t step = 32; a + step < b; step *= 2) {
    if (key_lcp(keys, words, n, i, a + step) < L) {
      b = a + step - 1;
      break;
    }
    a += step;
  }
  while (a < b) {
    const int64_t mid = (a + b + 1) >> 1;
    if (key_lcp(keys, words, n, i, mid) >= L)
      a = mid;
    else
      b = mid - 1;
  }
  return a + 1;
}

__device__ __forceinline__ double rcp_f64(double m);

// Leaf k: its particle's position as its centre and centre of mass, and its mass.
__device__ __forceinline__ void write_leaf(const NodeArrays& na, int k, int next, double x, double y, double z, double m) {
  na.M[k] = make_dvec4(x, y, z, m);
  const float hx = (float)x, hy = (float)y, hz = (float)z;
  na.R[k].A = make_float4(hx, hy, hz, 0.f);
  na.R[k].L = make_float4(f32_lo(x, hx), f32_lo(y, hy), f32_lo(z, hz), __int_as_float(next));
  na.R[k].O = make_float4(0.f, 0.f, 0.f, (float)m);
}

// Internal cell k with centre and size C, holding the key-ordered particles [i, end): its
// walk record and its monopole, from exact sums with one rounding each, then firstmoment /
// mass (_jbgrav.c:478) with a Newton-refined reciprocal.
__device__ __forceinline__ void write_cell(const NodeArrays& na, int k, int next, const dvec4& C, int64_t i, int64_t end,
                                           int64_t n, int lsb_m, int lsb_f, const FxMoments* __restrict__ fx_local,
                                           const FxMoments* __restrict__ fx_tiles, int tile_bits) {
  const double c[3] = {C.x, C.y, C.z};
  float4 A, Lo;
  A.x = f32_hi(c[0]);
  A.y = f32_hi(c[1]);
  A.z = f32_hi(c[2]);
  A.w = (float)dmul(C.w, C.w);
  Lo.x = f32_lo(c[0], A.x);
  Lo.y = f32_lo(c[1], A.y);
  Lo.z = f32_lo(c[2], A.z);
  Lo.w = __int_as_float(next);
  na.R[k].A = A;
  na.R[k].L = Lo;
  const FxMoments Pi = fxm_prefix(fx_local, fx_tiles, tile_bits, i, n);
  const FxMoments Pe = fxm_prefix(fx_local, fx_tiles, tile_bits, end, n);
  const double cm = fx::to_double(fx::sub(Pe.c[0], Pi.c[0]), lsb_m);
  const double r = rcp_f64(cm);
  double com[3];
#pragma unroll
  for (int a2 = 0; a2 < 3; a2++) com[a2] = dmul(fx::to_double(fx::sub(Pe.c[a2 + 1], Pi.c[a2 + 1]), lsb_f), r);
  na.M[k] = make_dvec4(com[0], com[1], com[2], cm);
  na.R[k].O = make_float4((float)dsub(com[0], c[0]), (float)dsub(com[1], c[1]), (float)dsub(com[2], c[2]), (float)cm);
}

// Particle i opens the cells at levels lo = lp[i]+1 .. d (its leaf), nodes
// base[i] .. base[i] + d - lo in preorder.  nodes_kernel writes the leaf: the
// particle's position as its centre, its mass, its skip index (gravoct_finalize,
// _jbgrav.c:467-483: a leaf's centre of mass is its particle), and lists the
// particles that open internal cells and the internal cells themselves;
// cell_centres_kernel gives those cells their centre from the reference's FP64
// recurrence along the particle's digits (gravoct_add_particle, _jbgrav.c:403-428),
// cells_kernel their skip index and their monopole.  A leaf is always accepted by the
// walk, so it needs no geometric centre.
__global__ void nodes_kernel(int64_t n, const int* __restrict__ lp, const int* __restrict__ depth,
                             const int* __restrict__ base, const uint32_t* __restrict__ perm,
                             const double* __restrict__ pos, const double* __restrict__ mass, NodeArrays na,
                             int nnodes, int* __restrict__ list, int* __restrict__ count,
                             int2* __restrict__ cells, int* __restrict__ ncells) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool need = false;
  int ncell = 0, k0 = 0;  // this particle's internal cells: nodes k0 .. k0 + ncell - 1
  if (i < n) {
    const int lo = lp[i] + 1, d = depth[i];
    const int k = base[i] + (d - lo);
    const int next = i + 1 < n ? base[i + 1] : nnodes;
    const int64_t p = perm[i];
    write_leaf(na, k, next, pos[3 * p], pos[3 * p + 1], pos[3 * p + 2], mass[p]);
    need = d > lo;
    ncell = d - lo;
    k0 = base[i];
  }
  warp_append(need, i, list, count);
  // the internal cells, one (cell, opener) entry each, for cells_kernel
  const int lane = threadIdx.x & 31;
  int incl = ncell;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  int first = 0;
  if (lane == 31 && incl > 0) first = atomicAdd(ncells, incl);
  first = __shfl_sync(0xffffffffu, first, 31) + incl - ncell;
  for (int j = 0; j < ncell; j++) cells[first + j] = make_int2(k0 + j, (int)i);
}

// Centres of the internal cells from the reference's FP64 recurrence along each
// opener's digits (gravoct_add_particle, _jbgrav.c:403-428): C[k] = (centre, size).
// Only the recurrence runs here, so its FP64 adds keep most lanes of a warp busy; the
// rest of each cell is cells_kernel's, one thread per cell.
__global__ void cell_centres_kernel(const uint64_t* __restrict__ keys, int words, int64_t n,
                                    const int* __restrict__ lp, const int* __restrict__ depth,
                                    const int* __restrict__ base, const TreeRoot* __restrict__ root, NodeArrays na,
                                    const int* __restrict__ list, const int* __restrict__ count) {
  __shared__ double offs[TREE_MAX_LEVELS];  // size 2^-(L+2), exact
  const double S = root->size;
  for (int l = threadIdx.x; l < TREE_MAX_LEVELS; l += blockDim.x)
    offs[l] = dmul(S, __longlong_as_double((long long)(1023 - (l + 2)) << 52));
  __syncthreads();
  const int cnt = *count;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < cnt; q += gridDim.x * blockDim.x) {
    const int64_t i = list[q];
    const int lo = lp[i] + 1, d = depth[i];
    const int k0 = base[i];
    const uint64_t kw0 = keys[i], kw1 = words > 1 ? keys[n + i] : 0ull;  // digits of the first 42 levels
    double c[3] = {root->c[0], root->c[1], root->c[2]};
    for (int L = 0; L < d; L++) {
      if (L >= lo)
        na.C[k0 + (L - lo)] = make_dvec4(c[0], c[1], c[2], dmul(S, __longlong_as_double((long long)(1023 - L) << 52)));
      if (L + 1 < d) {
        const unsigned g = L < KEY_LEVELS       ? (unsigned)(kw0 >> (3 * (KEY_LEVELS - 1 - L))) & 7u
                           : L < 2 * KEY_LEVELS ? (unsigned)(kw1 >> (3 * (2 * KEY_LEVELS - 1 - L))) & 7u
                                                : key_digit(keys, n, i, L);
        const double off = offs[L];
#pragma unroll
        for (int r = 0; r < 3; r++) c[r] = dadd(c[r], ((g >> r) & 1u) ? off : -off);
      }
    }
  }
}

// One internal cell per thread (the (cell, opener) list of nodes_kernel): its skip
// index, its walk record from the centre, and its monopole.  Cell k of opener i is at
// level L = lp[i] + 1 + (k - base[i]) and holds the key-ordered particles [i, end).
__global__ void cells_kernel(const uint64_t* __restrict__ keys, int words, int64_t n, const int* __restrict__ lp,
                             const int* __restrict__ base, const TreeRoot* __restrict__ root, NodeArrays na,
                             int nnodes, const int2* __restrict__ cells, int ncells,
                             const FxMoments* __restrict__ fx_local, const FxMoments* __restrict__ fx_tiles) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= ncells) return;
  const int2 e = cells[q];
  const int k = e.x;
  const int64_t i = e.y;
  const int L = lp[i] + 1 + (k - base[i]);
  const int64_t end = cell_end(keys, words, n, lp, i, L);
  write_cell(na, k, end < n ? base[end] : nnodes, na.C[k], i, end, n, root->lsb_m, root->lsb_f, fx_local, fx_tiles,
             MS_BITS);
}

// ---------------------------------------------------------------------------
// 5. Exact prefix sums of the monopole moments over the key-ordered particles
// ---------------------------------------------------------------------------
// The particles of a cell are a contiguous range [first, end) of the key order, so
// its mass and first moment (m_j x_j, the reference's FP64 products,
// gravoct_add_particle, _jbgrav.c:396-398) are differences of prefix sums.  The sums
// are exact 192-bit fixed-point integers (fixed192.cuh): their values do not depend on
// the order of addition, and each cell's is rounded to FP64 once.

// 1/m from the hardware approximation and two Newton steps y <- y + y (1 - m y).
__device__ __forceinline__ double rcp_f64(double m) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(m));
#pragma unroll
  for (int it = 0; it < 2; it++) y = fma(y, fma(-m, y, 1.0), y);
  return y;
}

__device__ __forceinline__ FxMoments particle_moments(const double* __restrict__ pos,
                                                      const double* __restrict__ mass, int64_t p, int lsb_m,
                                                      int lsb_f) {
  const double m = mass[p];
  FxMoments r;
  r.c[0] = fx::from_double(m, lsb_m);
#pragma unroll
  for (int a = 0; a < 3; a++) r.c[a + 1] = fx::from_double(dmul(m, pos[3 * p + a]), lsb_f);
  return r;
}

// Exclusive scan of the threads' totals within a block of T; returns the thread's
// exclusive prefix.
template <int T>
__device__ __forceinline__ FxMoments fxm_block_exclusive(const FxMoments& tot) {
  __shared__ FxMoments warp_tot[T / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  FxMoments inc = tot;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    FxMoments y;
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int w = 0; w < 3; w++) y.c[k].w[w] = __shfl_up_sync(0xffffffffu, inc.c[k].w[w], d);
    if (lane >= d) fxm_add(inc, y);
  }
  if (lane == 31) warp_tot[warp] = inc;
  __syncthreads();
  FxMoments before = fxm_zero();
  for (int w = 0; w < warp; w++) fxm_add(before, warp_tot[w]);
#pragma unroll
  for (int k = 0; k < 4; k++) before.c[k] = fx::add(before.c[k], fx::sub(inc.c[k], tot.c[k]));
  __syncthreads();  // warp_tot may be reused by the caller's next scan
  return before;
}

// Per tile of MS_THREADS * ITEMS key-ordered particles: the prefix of every particle within its
// tile (fx_local) and the tile's total (fx_tiles[tile]).
template <int ITEMS>
__global__ void __launch_bounds__(MS_THREADS)
    moments_scan_kernel(const double* __restrict__ pos, const double* __restrict__ mass,
                        const uint32_t* __restrict__ perm, int64_t n, const TreeRoot* __restrict__ root,
                        FxMoments* __restrict__ fx_local, FxMoments* __restrict__ fx_tiles) {
  const int lsb_m = root->lsb_m, lsb_f = root->lsb_f;
  const int64_t j0 = ((int64_t)blockIdx.x * MS_THREADS + threadIdx.x) * ITEMS;
  // each item's moments are formed twice (for the thread's total, then for the running
  // prefix): measured cheaper than storing them and reading them back (1.22 against
  // 1.33 ms per build at N = 1M)
  FxMoments tot = fxm_zero();
  for (int r = 0; r < ITEMS; r++)
    if (j0 + r < n) fxm_add(tot, particle_moments(pos, mass, perm[j0 + r], lsb_m, lsb_f));
  FxMoments run = fxm_block_exclusive<MS_THREADS>(tot);
  for (int r = 0; r < ITEMS; r++)
    if (j0 + r < n) {
      fx_local[j0 + r] = run;
      fxm_add(run, particle_moments(pos, mass, perm[j0 + r], lsb_m, lsb_f));
    }
  if (threadIdx.x == MS_THREADS - 1) fx_tiles[blockIdx.x] = run;
}

// Exclusive scan of the tile totals in place; fx_tiles[ntiles] receives the total.
__global__ void __launch_bounds__(MS_THREADS) moments_tiles_kernel(FxMoments* __restrict__ fx_tiles, int64_t ntiles) {
  const int64_t per = (ntiles + MS_THREADS - 1) / MS_THREADS;
  const int64_t a = (int64_t)threadIdx.x * per;
  const int64_t b = a + per < ntiles ? a + per : ntiles;
  FxMoments tot = fxm_zero();
  for (int64_t t = a; t < b; t++) fxm_add(tot, fx_tiles[t]);
  FxMoments run = fxm_block_exclusive<MS_THREADS>(tot);
  for (int64_t t = a; t < b; t++) {
    const FxMoments v = fx_tiles[t];
    fx_tiles[t] = run;
    fxm_add(run, v);
  }
  if (threadIdx.x == MS_THREADS - 1) fx_tiles[ntiles] = run;
}

// ---------------------------------------------------------------------------
// Build of a small system (n <= SB_MAX): a build of a few thousand particles is bound by
// its 27 launches and by latency (250 us at N = 2000, whatever N down to 100), so here it
// is six: box and root, keys, rank, moments, layout (one block) and cells.  The keys are sorted by
// counting smaller ones, n^2 comparisons over all SMs.  Only the two-word keys are
// handled: a tie, a non-finite input or more nodes than the caller's room leaves a status
// and a tree of zero nodes, which the walk takes no step on.  The host reads the status
// after the walk is queued, so the GPU does not wait for it.
// ---------------------------------------------------------------------------
constexpr int SB_MAX = 8192;
constexpr int SB_ITEMS = SB_MAX / SB_THREADS;
enum SmallStatus { SB_OK = 0, SB_BAD = 1, SB_TIE = 2, SB_ROOM = 3 };
// A tie usually recurs in the next step of the same system, and then the small build and the
// walk queued on it were for nothing, so its particle count keeps to the general build until
// as many builds of it in a row had no tie (several systems of one count may take turns).
constexpr int SB_TIE_BUILDS = 4;

// Rank of each key among all (words and index), 16 particles x 16 slices of the others per
// block; writes the keys and indices in order.
constexpr int RK_THREADS = 256, RK_CHUNK = 1024;
__global__ void __launch_bounds__(RK_THREADS)
    small_rank_kernel(const uint64_t* __restrict__ kin, int n, uint64_t* __restrict__ kout, uint32_t* __restrict__ idx) {
  __shared__ uint64_t c0[RK_CHUNK], c1[RK_CHUNK];
  const int slice = threadIdx.x & 15, i = blockIdx.x * 16 + (threadIdx.x >> 4);
  const uint64_t k0 = i < n ? kin[i] : 0ull, k1 = i < n ? kin[n + i] : 0ull;
  int rank = 0;
  for (int b = 0; b < n; b += RK_CHUNK) {
    const int m = n - b < RK_CHUNK ? n - b : RK_CHUNK;
    __syncthreads();
    for (int q = threadIdx.x; q < m; q += RK_THREADS) {
      c0[q] = kin[b + q];
      c1[q] = kin[n + b + q];
    }
    __syncthreads();
#pragma unroll 4
    for (int q = slice; q < m; q += 16) {
      const uint64_t a0 = c0[q], a1 = c1[q];
      rank += a0 < k0 || (a0 == k0 && (a1 < k1 || (a1 == k1 && b + q < i)));
    }
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
  if (slice == 0 && i < n) {
    kout[rank] = k0;
    kout[n + rank] = k1;
    idx[rank] = (uint32_t)i;
  }
}

// Common prefixes, the nodes' places in the preorder (base; base[n] = nodes, or 0 with a
// status) and the prefixes of the moment tiles, in one block; thread t has the contiguous
// key-ordered particles from t * per on.
__global__ void __launch_bounds__(SB_THREADS)
    small_layout_kernel(const uint64_t* __restrict__ keys, int n, int room, const TreeRoot* __restrict__ root,
                        int* __restrict__ lp, int* __restrict__ base, FxMoments* __restrict__ fx_tiles,
                        int* __restrict__ status) {
  __shared__ int warp_sum[SB_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (n + SB_THREADS - 1) / SB_THREADS;
  const int j0 = tid * per < n ? tid * per : n, j1 = j0 + per < n ? j0 + per : n;
  int l[SB_ITEMS + 1], cnt[SB_ITEMS];
  bool tie = false;
#pragma unroll
  for (int r = 0; r <= SB_ITEMS; r++) {
    const int j = j0 + r;
    l[r] = -1;
    if (r <= j1 - j0 && j > 0 && j < n) l[r] = key_lcp(keys, 2, n, j - 1, j);
    tie = tie || l[r] >= 2 * KEY_LEVELS;
  }
  int mine = 0;
#pragma unroll
  for (int r = 0; r < SB_ITEMS; r++) {
    cnt[r] = 1 + (l[r] > l[r + 1] ? l[r] : l[r + 1]) - l[r];
    if (r < j1 - j0) mine += cnt[r];
  }
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_sum[warp] = incl;
  tie = __syncthreads_or(tie);
  int before = incl - mine, total = 0;
  for (int w = 0; w < SB_THREADS / 32; w++) {
    const int s = warp_sum[w];
    if (w < warp) before += s;
    total += s;
  }
#pragma unroll
  for (int r = 0; r < SB_ITEMS; r++)
    if (r < j1 - j0) {
      lp[j0 + r] = l[r];
      base[j0 + r] = before;
      before += cnt[r];
    }
  if (tid == 0) {
    const int st = root->bad ? SB_BAD : (tie ? SB_TIE : (total > room ? SB_ROOM : SB_OK));
    lp[n] = -1;
    base[n] = st == SB_OK ? total : 0;
    status[1] = total;
    status[0] = st;
  }
  if (warp == 1) {  // tile totals -> prefixes: at most 32 tiles
    static_assert(SB_MAX >> SB_BITS <= 32, "one warp scans the tiles");
    const int ntiles = ((n - 1) >> SB_BITS) + 1;
    const FxMoments v = lane < ntiles ? fx_tiles[lane] : fxm_zero();
    FxMoments inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      FxMoments y;
#pragma unroll
      for (int k = 0; k < 4; k++)
#pragma unroll
        for (int w = 0; w < 3; w++) y.c[k].w[w] = __shfl_up_sync(0xffffffffu, inc.c[k].w[w], d);
      if (lane >= d) fxm_add(inc, y);
    }
    if (lane == ntiles - 1) fx_tiles[ntiles] = inc;
#pragma unroll
    for (int k = 0; k < 4; k++) inc.c[k] = fx::sub(inc.c[k], v.c[k]);
    if (lane < ntiles) fx_tiles[lane] = inc;
  }
}

// A block of key-ordered particles: their leaves and the centres of the internal cells
// that they open, by the reference's FP64 recurrence along their digits (see nodes_kernel,
// cell_centres_kernel), then the rest of those cells, one thread each: the block's nodes
// are contiguous in the preorder.
constexpr int SC_CELL_THREADS = 64;
__global__ void __launch_bounds__(SC_CELL_THREADS)
    small_cells_kernel(const double* __restrict__ pos, const double* __restrict__ mass,
                       const uint64_t* __restrict__ keys, const uint32_t* __restrict__ perm, int n,
                       const TreeRoot* __restrict__ root, const int* __restrict__ lp, const int* __restrict__ base,
                       NodeArrays na, const FxMoments* __restrict__ fx_local, const FxMoments* __restrict__ fx_tiles) {
  __shared__ double offs[2 * KEY_LEVELS], sizes[2 * KEY_LEVELS];
  __shared__ int s_lp[SC_CELL_THREADS], s_base[SC_CELL_THREADS + 1];
  const int tid = threadIdx.x, i0 = blockIdx.x * SC_CELL_THREADS, i = i0 + tid;
  const int nnodes = base[n];
  if (nnodes == 0) return;
  const int m = n - i0 < SC_CELL_THREADS ? n - i0 : SC_CELL_THREADS;
  if (tid < 2 * KEY_LEVELS) {
    sizes[tid] = dmul(root->size, __longlong_as_double((long long)(1023 - tid) << 52));
    offs[tid] = dmul(root->size, __longlong_as_double((long long)(1023 - (tid + 2)) << 52));
  }
  if (tid == 0) s_base[m] = base[i0 + m];
  if (tid < m) {
    s_lp[tid] = lp[i];
    s_base[tid] = base[i];
  }
  __syncthreads();
  if (tid < m) {
    const int lo = s_lp[tid] + 1, k0 = s_base[tid], d = lo + s_base[tid + 1] - k0 - 1;
    const int64_t p = perm[i];
    write_leaf(na, k0 + (d - lo), k0 + (d - lo) + 1, pos[3 * p], pos[3 * p + 1], pos[3 * p + 2], mass[p]);
    if (d > lo) {
      const uint64_t kw0 = keys[i], kw1 = keys[n + i];
      double c[3] = {root->c[0], root->c[1], root->c[2]};
      for (int L = 0; L < d; L++) {
        if (L >= lo) na.C[k0 + (L - lo)] = make_dvec4(c[0], c[1], c[2], sizes[L]);
        if (L + 1 < d) {
          const unsigned g = L < KEY_LEVELS ? (unsigned)(kw0 >> (3 * (KEY_LEVELS - 1 - L))) & 7u
                                            : (unsigned)(kw1 >> (3 * (2 * KEY_LEVELS - 1 - L))) & 7u;
          const double off = offs[L];
#pragma unroll
          for (int r = 0; r < 3; r++) c[r] = dadd(c[r], ((g >> r) & 1u) ? off : -off);
        }
      }
    }
  }
  __syncthreads();
  const int lsb_m = root->lsb_m, lsb_f = root->lsb_f;
  for (int k = s_base[0] + tid; k < s_base[m]; k += SC_CELL_THREADS) {
    int a = 0, b = m - 1;  // the particle that opens node k: the last with base <= k
    while (a < b) {
      const int mid = (a + b + 1) >> 1;
      if (s_base[mid] <= k)
        a = mid;
      else
        b = mid - 1;
    }
    if (k == s_base[a + 1] - 1) continue;  // its leaf
    const int64_t end = cell_end(keys, 2, n, lp, i0 + a, s_lp[a] + 1 + k - s_base[a]);
    write_cell(na, k, end < n ? base[end] : nnodes, na.C[k], i0 + a, end, n, lsb_m, lsb_f, fx_local, fx_tiles, SB_BITS);
  }
}

// ---------------------------------------------------------------------------
// Walk
// ---------------------------------------------------------------------------
constexpr int TW_THREADS = 128;
constexpr int TW_MINB = 9;  // 56 registers: 36 warps per SM (10: 48 registers, spills, slower)

__device__ __forceinline__ double rsqrt_f64(double s) {
  double y;
  asm("rsqrt.approx.f64 %0, %1;" : "=d"(y) : "d"(s));
  // two Newton steps: y <- y + 0.5 y (1 - s y^2)
#pragma unroll
  for (int it = 0; it < 2; it++) {
    double e = fma(-s * y, y, 1.0);
    y = fma(0.5 * y, e, y);
  }
  return y;
}

// Mixed: accepted cells interact in FP32: the hi/lo split offset of the cell's
// centre (keeps ~2^-48 of |x|) plus the FP32 offset of its centre of mass; partial
// sums folded into a two-sum (hi, lo) accumulator every TW_FOLD warp steps.  Otherwise
// FP64 with the factor from fixed point (f64emu.cuh).
// The opening decisions are the same exact ones in both forms.
constexpr int TW_FOLD = 32;
// FP64: a lane's accepted cells wait in a FIFO of TW_FQ entries and are evaluated in
// rounds that run when at least TW_FQ_ROUND lanes have one waiting (or a FIFO is
// full), so the FP64 pipe (1/74 of the FP32 rate on GB300) issues fewer partly empty
// instructions; each lane still adds its interactions in visiting order.
constexpr int TW_FQ = 32;
constexpr int TW_FQ_ROUND = 28;
static_assert((TW_FQ & (TW_FQ - 1)) == 0, "the FIFO index wraps with a mask");

// Softening as the fixed-point interaction wants it (f64emu.cuh); ok = false keeps every
// interaction on the FP64 operations.
struct WalkEps {
  double eps2;
  uint64_t W;
  int E;
  bool ok;
};

// m s^(-3/2) where the fixed-point factor does not take the pair: FP64 operations, 0 for
// s = 0; but a zero mass, which has no place in that factor either, is its own (as FP64 it
// cost its whole round: 300,000 particles, a fifth massless, 6.30 -> 4.42 ms, none 3.82).  A
// call: inline, it cost the rounds that do not take it up to 0.5 % (60,013 1377 -> 1365 us).
template <bool GUARD>
__device__ __noinline__ double walk_factor_rare(double m, double dx, double dy, double dz, double eps2, int Ee, bool ok) {
  double f;
  if (ok && emu::zero_mass_inv_cube(m, dx, dy, dz, Ee, f)) return f;
  const double s = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
  if (GUARD && s == 0.0) return 0.0;
  const double y = rsqrt_f64(s);
  return m * (y * (y * y));
}

// One FP64 interaction: the cell's monopole (nM) times s^(-3/2), from the differences to
// the rounded factor in 64-bit fixed point; FP64 operations outside that form's range.
// Bound by the FP64 pipe, which a warp's DFMA holds for 17 cycles of the SM and a DADD
// or DMUL for 20 (measured): three differences and three sums are left on it, busy for 96 of
// the 109 cycles that a round takes at N = 1M (29 of 32 lanes hold an interaction), where s
// and its factor took four more.  With the walk's steps and the fixed-point factor a round is
// 273 instructions (issue 63 % busy).
// Force at N = 1M Hernquist + disk: theta 0.7 29.0 -> 18.5 ms, theta 0.5 71.6 -> 44.9;
// the differences as FMAs by an opaque 1.0 (17 cycles instead of 20): 18.8.
template <bool GUARD>
__device__ __forceinline__ void walk_interact_f64(const dvec4* __restrict__ nM, int node, double p0, double p1,
                                                  double p2, const WalkEps& E, double& ax, double& ay, double& az) {
  const dvec4 M = nM[node];
  const double dx = M.x - p0, dy = M.y - p1, dz = M.z - p2;
  double f;
  if (!(E.ok && emu::mass_inv_cube(M.w, dx, dy, dz, E.E, E.W, f)))
    f = walk_factor_rare<GUARD>(M.w, dx, dy, dz, E.eps2, E.E, E.ok);
  ax = fma(f, dx, ax);
  ay = fma(f, dy, ay);
  az = fma(f, dz, az);
}

// A target's position as the opening test wants it: FP32 hi and residual, and the
// squared distance below which the exact test is needed (FP32 differences lose too much
// relative to |x|, and FP32 stays in its normal range: with theta >= 1e-3 a cell whose
// size^2 is below that range is then accepted, as the exact test would).
struct WalkTarget {
  f2 h01, l01;
  float h2, l2, near2;
};
__device__ __forceinline__ WalkTarget walk_target(double p0, double p1, double p2) {
  WalkTarget T;
  const float h0 = (float)p0, h1 = (float)p1;
  T.h2 = (float)p2;
  T.l2 = f32_lo(p2, T.h2);
  T.h01 = f2make(h0, h1);
  T.l01 = f2make(f32_lo(p0, h0), f32_lo(p1, h1));
  T.near2 = fmaxf(1e-18f * (h0 * h0 + h1 * h1 + T.h2 * T.h2), 1e-30f);
  return T;
}

// Offset of a cell's centre (A, Lo: its record) from the target.
__device__ __forceinline__ void walk_offset(const WalkTarget& T, const float4& A, const float4& Lo, f2& dxy, float& dz) {
  dxy = f2add(f2sub(f2make(A.x, A.y), T.h01), f2sub(f2make(Lo.x, Lo.y), T.l01));
  dz = (A.z - T.h2) + (Lo.z - T.l2);
}

// gravoct_calc_accel's opening test with the reference's FP64 operations, on the target's
// position, which pos(p0, p1, p2) gives.  Rare, and a call: inline, its division and square
// root took the registers and the branches of every step.
template <class Pos>
__device__ __noinline__ bool walk_exact(const dvec4* __restrict__ nC, int node, Pos pos, double theta) {
  double p0, p1, p2;
  pos(p0, p1, p2);
  const dvec4 C = nC[node];
  const double e0 = dsub(C.x, p0), e1 = dsub(C.y, p1), e2 = dsub(C.z, p2);
  double nd = dmul(e0, e0);
  nd = dadd(nd, dmul(e1, e1));
  nd = dadd(nd, dmul(e2, e2));
  return ddiv(C.w, dsqrt(nd)) < theta;
}

// Whether a visited cell is accepted: a leaf always, another when size / distance < theta,
// decided in FP32 outside the margins, else exactly (exact counts those).  One branch, the
// rare one: the rest is predicates.
template <class Pos>
__device__ __forceinline__ bool walk_accept(const WalkTarget& T, f2 dxy, float dz, float s2, bool leaf, bool visit,
                                            float th2_lo, float th2_hi, const dvec4* __restrict__ nC, int node,
                                            const Pos& pos, double theta, unsigned& exact) {
  float dx, dy;
  f2split(dxy, dx, dy);
  const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
  // d2 = inf (overflow) accepts, as the exact test does for so distant a cell
  const bool usable = d2 > T.near2;
  bool accept = leaf | (usable & (s2 < th2_lo * d2));
  if (visit & !accept & !(usable & (s2 > th2_hi * d2))) {
    exact++;
    accept = walk_exact(nC, node, pos, theta);
  }
  return accept & visit;
}

// Walk counters of a warp into stats.
__device__ __forceinline__ void walk_count(unsigned long long* stats, unsigned n_step, unsigned n_visit, unsigned n_inter,
                                           unsigned n_exact, unsigned n_leaf, unsigned n_chain) {
  // one cell record read per warp step; the other counts summed over lanes
  n_visit = __reduce_add_sync(0xffffffffu, n_visit);
  n_inter = __reduce_add_sync(0xffffffffu, n_inter);
  n_exact = __reduce_add_sync(0xffffffffu, n_exact);
  n_leaf = __reduce_add_sync(0xffffffffu, n_leaf);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&stats[0], (unsigned long long)n_step);
    atomicAdd(&stats[1], (unsigned long long)n_visit);
    atomicAdd(&stats[2], (unsigned long long)n_inter);
    atomicAdd(&stats[3], (unsigned long long)n_exact);
    atomicAdd(&stats[4], (unsigned long long)n_leaf);
    atomicAdd(&stats[5], (unsigned long long)n_chain);
  }
}

// A cell with one child cell: the child's subtree ends where the cell's does.
__device__ __forceinline__ bool walk_is_chain(const WalkRec* __restrict__ nR, int node, int nnodes) {
  const int nxt = __float_as_int(nR[node].L.w);
  return nxt != node + 1 && node + 1 < nnodes && __float_as_int(nR[node + 1].L.w) == nxt;
}

// Mixed walk.  A step is a chain (record, opening test, the lanes' next node) of some 50
// instructions, most of them waiting for the one before.  So a step has one branch, for the
// rare exact test, its interaction is formed by every lane, the fold is a loop of its own
// around the steps, and the position for the exact test is read again instead of held.
// (N = 262,144: 50 -> 48 instructions a step, but 62 -> 70 % of the issue slots, waits on
// the pipes 3.2 -> 2.2 warps per issue.)  N = 16,384 theta 0.7 408 -> 318 us, 60,013 505 ->
// 399, 1,048,576 theta 0.5 9.62 -> 8.49 ms (the FP64 walk, whose steps also end in rounds of
// interactions: 344 -> 322 us, 1141 -> 1085, 17.34 -> 17.20 ms at theta 0.7).  More warps
// with fewer registers (spills), the next record's load ahead of the interaction, and votes
// in place of the minimum were all slower.
template <bool GUARD, bool STATS, class Epi>
__global__ void __launch_bounds__(TW_THREADS, TW_MINB)
    tree_walk_kernel(const WalkRec* __restrict__ nR, const dvec4* __restrict__ nC, const int* __restrict__ nodes,
                     const double* __restrict__ tpos, const uint32_t* __restrict__ order, int64_t nt,
                     double eps2, double theta, float th2_lo, float th2_hi, Epi epi,
                     unsigned long long* __restrict__ stats) {
  const int nnodes = *nodes;
  if (nnodes == 0) return;  // a build that did not succeed
  const int64_t slot = (int64_t)blockIdx.x * TW_THREADS + threadIdx.x;
  const bool valid = slot < nt;
  const auto pos = [=](double& p0, double& p1, double& p2) {  // read again by the exact test
    const int64_t t = order ? (int64_t)order[slot] : slot;
    p0 = tpos[3 * t];
    p1 = tpos[3 * t + 1];
    p2 = tpos[3 * t + 2];
  };
  double p0 = 0.0, p1 = 0.0, p2 = 0.0;
  if (valid) pos(p0, p1, p2);
  const WalkTarget T = walk_target(p0, p1, p2);
  const float eps2f = (float)eps2;
  float px = 0.f, py = 0.f, pz = 0.f;                                // FP32 partial
  float hx = 0.f, hy = 0.f, hz = 0.f, qx = 0.f, qy = 0.f, qz = 0.f;  // two-sum hi, lo
  unsigned n_step = 0, n_visit = 0, n_inter = 0, n_exact = 0, n_leaf = 0, n_chain = 0;  // walk counters (STATS)
  int skip = valid ? 0 : 0x7fffffff;
  int node = __reduce_min_sync(0xffffffffu, skip);
  while (node < nnodes) {
    int left = TW_FOLD;
    do {
      if (STATS) {
        n_step++;
        n_chain += walk_is_chain(nR, node, nnodes);
      }
      const float4 A = nR[node].A;
      const float4 Lo = nR[node].L;
      const float4 O = nR[node].O;
      const int nx = __float_as_int(Lo.w);
      const bool visit = node >= skip, leaf = nx == node + 1;
      f2 dxy;
      float dz;
      walk_offset(T, A, Lo, dxy, dz);
      const bool accept = walk_accept(T, dxy, dz, A.w, leaf, visit, th2_lo, th2_hi, nC, node, pos, theta, n_exact);
      if (STATS) {
        n_visit += visit;
        n_inter += accept;
        n_leaf += accept && leaf;
      }
      // formed by every lane, added where accepted: no branch
      float ex, ey;
      f2split(f2add(dxy, f2make(O.x, O.y)), ex, ey);
      const float ez = dz + O.z;
      const float s = fmaf(ex, ex, fmaf(ey, ey, fmaf(ez, ez, eps2f)));
      float r = rsqrt_approx(s);
      if (GUARD) r = s > 0.f ? r : 0.f;
      const float f = O.w * (r * (r * r));
      if (accept) {
        px = fmaf(f, ex, px);
        py = fmaf(f, ey, py);
        pz = fmaf(f, ez, pz);
        skip = nx;
      }
      node = __reduce_min_sync(0xffffffffu, visit & !accept ? node + 1 : skip);
    } while (--left && node < nnodes);
    // fold the FP32 partials every TW_FOLD warp steps (at most one interaction per
    // target per step); what is left of them at the end is added as it is
    if (left == 0) {
      float sx, ex;
      two_sum(hx, px, sx, ex);
      hx = sx;
      qx += ex;
      two_sum(hy, py, sx, ex);
      hy = sx;
      qy += ex;
      two_sum(hz, pz, sx, ex);
      hz = sx;
      qz += ex;
      px = py = pz = 0.f;
    }
  }
  if (STATS) walk_count(stats, n_step, n_visit, n_inter, n_exact, n_leaf, n_chain);
  if (valid)
    epi(order ? (int64_t)order[slot] : slot, (double)hx + (double)qx + (double)px, (double)hy + (double)qy + (double)py,
        (double)hz + (double)qz + (double)pz);
}

// How a walk is split over warps: `segs` warps per 32 targets, each walking one range of
// the preorder.  Targets that have a place of their own in it (particles, sorted points)
// open cells that are near them in space: those of d nodes around that place and, beyond,
// the ones that lie along the faces of larger cells, whose number grows like the faces'
// area, d^(2/3).  So the ranges are equal in the 2/3 power of the distance from that place
// (equal in its logarithm, the far ranges held up to 17 times the average's steps: force
// 664 us at N = 16,384 against 575, and equal ranges 630).  Just two meet next to the
// place, where they are equal in the logarithm (262,144: 4.66 -> 4.59 ms).  32 unsorted
// points are anywhere, so theirs are equal.
struct WalkSplit {
  int segs;
  double* part;           // [group][seg][component][lane] partial sums
  int* count;             // per group: segments finished (zero between launches)
  const int* base;        // first node of each key-ordered particle (null: equal ranges)
  const uint64_t* keys;   // the particles' first two key words, n each,
  const uint64_t* tkeys;  // and the sorted points' (null: the targets are the particles)
  int64_t n;
};
constexpr float TW_SEG_NEAR = 128.f;  // nodes around its own place that a group visits densely
constexpr float TW_SEG_POWER = 2.f / 3.f;

// Place in the preorder of target slot q.
__device__ __forceinline__ int walk_own(const WalkSplit& sp, int64_t q, int64_t nt, int nnodes) {
  if (!sp.tkeys) return sp.base[q];
  const uint64_t k0 = sp.tkeys[q], k1 = sp.tkeys[nt + q];
  int64_t a = 0, b = sp.n;  // first particle whose key is not below the point's
  while (a < b) {
    const int64_t m = (a + b) >> 1;
    const uint64_t w = sp.keys[m];
    if (w < k0 || (w == k0 && sp.keys[sp.n + m] < k1))
      a = m + 1;
    else
      b = m;
  }
  return a < sp.n ? sp.base[a] : nnodes;
}

// First node of segment s (of K) for a group whose own place is node `own` (-1: none).
// Never falls with s: steps of u are 2e-5 and more, __powf is good to 1e-6 there.
__device__ __forceinline__ int walk_bound(int s, int K, int own, int nnodes) {
  if (s <= 0) return 0;
  if (s >= K) return nnodes;
  if (own < 0) return (int)((int64_t)nnodes * s / K);
  const float l = 1.f + (float)own / TW_SEG_NEAR, r = 1.f + (float)(nnodes - own) / TW_SEG_NEAR;
  float d;
  bool before;
  if (K == 2) {
    before = l > r;
    d = sqrtf(before ? l / r : r / l) - 1.f;
  } else {
    const float left = __powf(l, TW_SEG_POWER) - 1.f, right = __powf(r, TW_SEG_POWER) - 1.f;
    const float u = (left + right) * (float)s / (float)K - left;
    before = u < 0.f;
    d = __powf(1.f + fabsf(u), 1.f / TW_SEG_POWER) - 1.f;
  }
  const int b = before ? own - (int)(TW_SEG_NEAR * d) : own + (int)(TW_SEG_NEAR * d);
  return b < 0 ? 0 : (b > nnodes ? nnodes : b);
}

// FP64 walk.  SPLIT: warp w of the grid takes segment w % segs of target group w / segs.
// The segment's first node a lies inside a chain of ancestor cells; the warp first takes
// each lane's decisions on that chain (their interactions belong to the segments that hold
// those cells), so that every cell and interaction is met exactly once, in the segment that
// holds it.  The group's last segment to finish adds the partial sums in segment order: the
// result does not depend on timing.
template <bool GUARD, bool STATS, bool SPLIT, class Epi>
__global__ void __launch_bounds__(TW_THREADS, TW_MINB)
    tree_walk_f64_kernel(const WalkRec* __restrict__ nR, const dvec4* __restrict__ nC, const dvec4* __restrict__ nM,
                         const int* __restrict__ nodes, const double* __restrict__ tpos,
                         const uint32_t* __restrict__ order, int64_t nt, double eps2, double theta, float th2_lo,
                         float th2_hi, Epi epi, WalkSplit sp, unsigned long long* __restrict__ stats) {
  const int nnodes = *nodes;
  if (nnodes == 0) return;  // a build that did not succeed
  const int lane = threadIdx.x & 31;
  const unsigned set = SPLIT ? blockIdx.x / sp.segs : blockIdx.x;  // of neighbouring target groups
  const int seg = SPLIT ? (int)(blockIdx.x - set * sp.segs) : 0;
  const int64_t group = (int64_t)set * (TW_THREADS / 32) + (threadIdx.x >> 5);
  if (group * 32 >= nt) return;  // whole warps
  const int64_t slot = group * 32 + lane;
  const bool valid = slot < nt;
  const int64_t t = valid ? (order ? (int64_t)order[slot] : slot) : 0;
  double p0 = 0.0, p1 = 0.0, p2 = 0.0;
  if (valid) {
    p0 = tpos[3 * t];
    p1 = tpos[3 * t + 1];
    p2 = tpos[3 * t + 2];
  }
  const auto pos = [=](double& a0, double& a1, double& a2) {
    a0 = p0;
    a1 = p1;
    a2 = p2;
  };
  WalkTarget T = walk_target(p0, p1, p2);
  // keeps the compiler from forming the residuals again inside the loop to save registers,
  // where each is three FP64-pipe instructions (one residual per interaction was: 29.0
  // against 18.5 ms per force at N = 1M, theta 0.7)
  asm volatile("" : "+f"(T.h2), "+f"(T.l2), "+l"(T.l01));
  double ax = 0.0, ay = 0.0, az = 0.0;
  __shared__ int fq[TW_FQ][TW_THREADS];  // this lane's accepted cells, FIFO
  int fq_head = 0, fq_n = 0;
  WalkEps we;
  we.eps2 = eps2;
  we.ok = emu::align_eps2(eps2, we.E, we.W);
  unsigned n_step = 0, n_visit = 0, n_inter = 0, n_exact = 0, n_leaf = 0, n_chain = 0;  // walk counters (STATS)
  int skip = valid ? 0 : 0x7fffffff;
  int end = nnodes;
  if (SPLIT) {
    const int64_t mid = group * 32 + 16 < nt ? group * 32 + 16 : nt - 1;
    const int own = sp.base ? walk_own(sp, mid, nt, nnodes) : -1;
    const int first = walk_bound(seg, sp.segs, own, nnodes);
    end = walk_bound(seg + 1, sp.segs, own, nnodes);
    int c = 0;
    while (c < first) {  // the cells that hold `first`
      const float4 Lo = nR[c].L;
      const int nx = __float_as_int(Lo.w);
      if (nx <= first) {
        c = nx;
        continue;
      }
      if (c >= skip) {
        f2 dxy;
        float dz;
        const float4 A = nR[c].A;
        walk_offset(T, A, Lo, dxy, dz);
        if (walk_accept(T, dxy, dz, A.w, false, true, th2_lo, th2_hi, nC, c, pos, theta, n_exact)) skip = nx;
      }
      c++;
    }
    if (skip < first) skip = first;
  }
  int node = __reduce_min_sync(0xffffffffu, skip);
  while (node < end) {
    if (STATS) {
      n_step++;
      n_chain += walk_is_chain(nR, node, nnodes);
    }
    const float4 A = nR[node].A;
    const float4 Lo = nR[node].L;
    const int nx = __float_as_int(Lo.w);
    const bool visit = node >= skip, leaf = nx == node + 1;
    f2 dxy;
    float dz;
    walk_offset(T, A, Lo, dxy, dz);
    const bool accept = walk_accept(T, dxy, dz, A.w, leaf, visit, th2_lo, th2_hi, nC, node, pos, theta, n_exact);
    if (STATS) {
      n_visit += visit;
      n_inter += accept;
      n_leaf += accept && leaf;
    }
    if (accept) {
      fq[(fq_head + fq_n) & (TW_FQ - 1)][threadIdx.x] = node;  // evaluated in a later round
      fq_n++;
      skip = nx;
    }
    const int lane_next = visit & !accept ? node + 1 : skip;
    // a round of FP64 interactions when enough lanes have one waiting; a FIFO that
    // just became full forces one, so a FIFO never holds more than TW_FQ
    const unsigned waiting = __ballot_sync(0xffffffffu, fq_n > 0);
    if (__popc(waiting) >= TW_FQ_ROUND || __any_sync(0xffffffffu, fq_n == TW_FQ)) {
      if (fq_n > 0) {
        const int c = fq[fq_head][threadIdx.x];
        fq_head = (fq_head + 1) & (TW_FQ - 1);
        fq_n--;
        walk_interact_f64<GUARD>(nM, c, p0, p1, p2, we, ax, ay, az);
      }
    }
    node = __reduce_min_sync(0xffffffffu, lane_next);
  }
  while (fq_n > 0) {  // the cells still waiting, in order
    const int c = fq[fq_head][threadIdx.x];
    fq_head = (fq_head + 1) & (TW_FQ - 1);
    fq_n--;
    walk_interact_f64<GUARD>(nM, c, p0, p1, p2, we, ax, ay, az);
  }
  if (STATS) walk_count(stats, n_step, n_visit, n_inter, n_exact, n_leaf, n_chain);
  if (SPLIT) {
    __syncwarp();
    double* mine = sp.part + (group * sp.segs + seg) * 96 + lane;
    mine[0] = ax;
    mine[32] = ay;
    mine[64] = az;
    __threadfence();
    __syncwarp();
    int last = 0;
    if (lane == 0) last = atomicAdd(&sp.count[group], 1) == sp.segs - 1;
    last = __shfl_sync(0xffffffffu, last, 0);
    if (!last) return;
    __threadfence();
    const double* all = sp.part + group * sp.segs * 96 + lane;
    ax = ay = az = 0.0;
    for (int k = 0; k < sp.segs; k++) {
      ax += __ldcg(all + 96 * k);
      ay += __ldcg(all + 96 * k + 32);
      az += __ldcg(all + 96 * k + 64);
    }
    if (lane == 0) sp.count[group] = 0;  // ready for the next launch
  }
  if (valid) epi(t, ax, ay, az);
}

// ---------------------------------------------------------------------------
// Workspace and host driver
// ---------------------------------------------------------------------------
struct TreeWS {
  int num_sms = 0;  // of its device
  Buffer part, root, keys, keys_tmp, idx, idx_tmp, rs, lp, cnt, depth, base, scan, flags;
  Buffer nA, nC, nM, fxl, fxt, xh[2];
  Buffer wpart, wcount;       // split walks: partial sums, finished segments per group
  size_t wcount_zeroed = 0;
  Buffer tkeys, tkeys_tmp, tidx, tidx_tmp, trs;  // target points' walk order
  Buffer list;                // particles that open internal cells
  Buffer cells;               // (internal cell, opener) pairs
  int* host_flags = nullptr;  // pinned: the 8 device flags, nnodes, the root's non-finite flag; [10..11] small build
  cudaEvent_t small_built = nullptr;
  // Per particle count: how many more general builds, from the last whose two-word keys tied
  // on, before the small build is tried again.
  uint8_t small_tied[SB_MAX + 1] = {};
  int64_t small_room = 0;     // nodes that a small build may write
  int words = TREE_MIN_WORDS;
  int64_t full_sort_n = -1;  // particle count whose last build needed the full multi-word sort
};
static TreeWS g_tree[64];
static std::recursive_mutex g_tree_mu;

// The current device's workspace (under g_tree_mu).
static int tree_workspace(TreeWS** ws) {
  DeviceInfo di;
  GH_TRY(device_info(&di));
  *ws = &g_tree[di.device];
  (*ws)->num_sms = di.num_sms;
  return GH_OK;
}

static NodeArrays node_arrays(TreeWS& ws) {
  NodeArrays na;
  na.R = (WalkRec*)ws.nA.ptr;
  na.C = (dvec4*)ws.nC.ptr;
  na.M = (dvec4*)ws.nM.ptr;
  return na;
}

struct BuiltTree {
  int64_t n = 0;  // particles
  int nnodes = 0;              // (unknown while pending)
  int maxdepth = 0;
  const int* nodes = nullptr;  // the same on the device; 0 when the build did not succeed
  bool pending = false;        // a small build whose status has not been read
  const uint32_t* torder = nullptr;  // target points in key order (when sorted)
};

// Target points are walked in key order from this many on (below, the sort's fixed
// cost exceeds what the coherent warps save).
constexpr int64_t TGT_SORT_MIN = 8192;

static int bad_input() {
  return set_error(GH_ERR_ARG,
                   "tree: particle positions and masses must be finite (the reference's octree insert "
                   "does not terminate on NaN or infinite coordinates)");
}

// Queues the build of a small system; small_finish reads its status.
static int small_build(TreeWS& ws, const double* pos, const double* mass, int64_t n, double eps, cudaStream_t st,
                       BuiltTree* out) {
  if (!ws.small_built) GH_CUDA_TRY(cudaEventCreateWithFlags(&ws.small_built, cudaEventDisableTiming));
  if (ws.small_room < 4 * n + 1024) ws.small_room = 4 * n + 1024;
  const size_t room = (size_t)ws.small_room;
  GH_TRY(ensure(ws.root, sizeof(TreeRoot)));
  GH_TRY(ensure(ws.lp, (n + 1) * sizeof(int)));
  GH_TRY(ensure(ws.base, (n + 1) * sizeof(int)));
  GH_TRY(ensure(ws.idx, n * sizeof(uint32_t)));
  GH_TRY(ensure(ws.idx_tmp, n * sizeof(uint32_t)));
  GH_TRY(ensure(ws.keys, (size_t)2 * n * sizeof(uint64_t)));
  GH_TRY(ensure(ws.keys_tmp, (size_t)2 * n * sizeof(uint64_t)));
  GH_TRY(ensure(ws.nA, room * sizeof(WalkRec)));
  GH_TRY(ensure(ws.nC, room * sizeof(dvec4)));
  GH_TRY(ensure(ws.nM, room * sizeof(dvec4)));
  GH_TRY(ensure(ws.fxl, (size_t)n * sizeof(FxMoments)));
  GH_TRY(ensure(ws.fxt, (size_t)(((n - 1) >> SB_BITS) + 2) * sizeof(FxMoments)));
  TreeRoot* root = (TreeRoot*)ws.root.ptr;
  uint64_t *keys = (uint64_t*)ws.keys.ptr, *ktmp = (uint64_t*)ws.keys_tmp.ptr;
  uint32_t* idx = (uint32_t*)ws.idx.ptr;
  int *lp = (int*)ws.lp.ptr, *base = (int*)ws.base.ptr;
  FxMoments *fxl = (FxMoments*)ws.fxl.ptr, *fxt = (FxMoments*)ws.fxt.ptr;
  box_root_kernel<<<1, SB_THREADS, 0, st>>>(pos, mass, n, eps, root);
  GH_LAUNCH_CHECK();
  keys_kernel<256><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(pos, n, root, 2, ktmp, (uint32_t*)ws.idx_tmp.ptr);
  GH_LAUNCH_CHECK();
  small_rank_kernel<<<(unsigned)((n + 15) / 16), RK_THREADS, 0, st>>>(ktmp, (int)n, keys, idx);
  GH_LAUNCH_CHECK();
  moments_scan_kernel<1><<<(unsigned)((n + MS_THREADS - 1) / MS_THREADS), MS_THREADS, 0, st>>>(pos, mass, idx, n, root,
                                                                                               fxl, fxt);
  GH_LAUNCH_CHECK();
  small_layout_kernel<<<1, SB_THREADS, 0, st>>>(keys, (int)n, (int)ws.small_room, root, lp, base, fxt,
                                                ws.host_flags + 10);
  GH_LAUNCH_CHECK();
  GH_CUDA_TRY(cudaEventRecord(ws.small_built, st));
  small_cells_kernel<<<(unsigned)((n + SC_CELL_THREADS - 1) / SC_CELL_THREADS), SC_CELL_THREADS, 0, st>>>(
      pos, mass, keys, idx, (int)n, root, lp, base, node_arrays(ws), fxl, fxt);
  GH_LAUNCH_CHECK();
  out->n = n;
  out->nodes = base + n;
  out->pending = true;
  return GH_OK;
}

// Waits for a small build's status.  *again: it did not succeed for a reason that the next
// tree_build of the same particles takes care of (a walk queued on it has done nothing).
static int small_finish(TreeWS& ws, BuiltTree* bt, bool* again) {
  *again = false;
  if (!bt->pending) return GH_OK;
  bt->pending = false;
  GH_CUDA_TRY(cudaEventSynchronize(ws.small_built));
  const volatile int* status = ws.host_flags + 10;
  bt->nnodes = status[1];
  switch (status[0]) {
    case SB_OK: return GH_OK;
    case SB_BAD: return bad_input();
    case SB_TIE: ws.small_tied[bt->n] = SB_TIE_BUILDS; break;
    default: ws.small_room = (int64_t)status[1] + status[1] / 4;
  }
  *again = true;
  return GH_OK;
}


// `defer`: a small system's build may be left pending (small_finish after the walk).
static int tree_build(TreeWS& ws, const double* pos, const double* mass, int64_t n, double eps,
                      cudaStream_t st, BuiltTree* out, bool defer = false, const double* tpos = nullptr,
                      int64_t nt = 0) {
  Trace tr("tree build");
  *out = BuiltTree();
  const bool sort_targets = tpos != nullptr && nt >= TGT_SORT_MIN;
  if (sort_targets && nt > (1LL << 31))
    return set_error(GH_ERR_ARG, "tree: at most 2^31 target points (got %lld)", (long long)nt);
  // int32 node indices: at most 127 cells per particle
  if (n > (1LL << 24)) return set_error(GH_ERR_ARG, "tree: at most 16777216 particles (got %lld)", (long long)n);
  if (!ws.host_flags) GH_CUDA_TRY(cudaMallocHost((void**)&ws.host_flags, 16 * sizeof(int)));
  const bool wait_fault = inject_take(GH_INJECT_TREE_WAIT);  // test hook: as if a look-back wait had run out
  if (n <= SB_MAX && !ws.small_tied[n] && !sort_targets && !wait_fault) {
    GH_TRY(small_build(ws, pos, mass, n, eps, st, out));
    if (defer) return GH_OK;
    bool again;
    GH_TRY(small_finish(ws, out, &again));
    if (!again) return GH_OK;
    return tree_build(ws, pos, mass, n, eps, st, out, false, tpos, nt);
  }
  const int T = 256;
  // 1. root cell
  GH_TRY(ensure(ws.part, BB_BLOCKS * sizeof(Box)));
  GH_TRY(ensure(ws.root, sizeof(TreeRoot)));
  int nb = (int)((n + BB_THREADS - 1) / BB_THREADS);
  if (nb > BB_BLOCKS) nb = BB_BLOCKS;
  bbox_partial_kernel<<<nb, BB_THREADS, 0, st>>>(pos, mass, n, (Box*)ws.part.ptr);
  GH_LAUNCH_CHECK();
  root_kernel<<<1, 32, 0, st>>>((const Box*)ws.part.ptr, nb, eps, (TreeRoot*)ws.root.ptr);
  GH_LAUNCH_CHECK();
  const TreeRoot* root = (const TreeRoot*)ws.root.ptr;
  const unsigned gn = (unsigned)((n + T - 1) / T), gn1 = (unsigned)((n + 1 + T - 1) / T);
  GH_TRY(ensure(ws.lp, (n + 1) * sizeof(int)));
  GH_TRY(ensure(ws.cnt, n * sizeof(int)));
  GH_TRY(ensure(ws.depth, n * sizeof(int)));
  GH_TRY(ensure(ws.base, (n + 1) * sizeof(int)));
  GH_TRY(ensure(ws.scan, scan_scratch_ints(n) * sizeof(int)));
  // flags: [0] full-key tie, [1] deepest level, [2] long run, [4] cell openers,
  // [5] a bounded wait in the sort gave up, [6] internal cells listed
  GH_TRY(ensure(ws.flags, 8 * sizeof(int)));
  GH_TRY(ensure(ws.list, n * sizeof(int)));
  GH_TRY(ensure(ws.idx, n * sizeof(uint32_t)));
  GH_TRY(ensure(ws.idx_tmp, n * sizeof(uint32_t)));
  GH_TRY(ensure(ws.rs, radix_scratch_words(n) * sizeof(uint32_t)));
  // 2-3. keys, sort, prefix structure; widen the keys while particles tie
  // A long run of equal first words usually recurs in the next build of the same
  // system (a stepping loop), so the full sort is kept for that particle count.
  bool full_sort = ws.full_sort_n == n;
  for (;;) {
    const int words = ws.words;
    GH_TRY(ensure(ws.keys, (size_t)words * n * sizeof(uint64_t)));
    GH_TRY(ensure(ws.keys_tmp, (size_t)words * n * sizeof(uint64_t)));
    uint64_t* keys = (uint64_t*)ws.keys.ptr;
    uint64_t* ktmp = (uint64_t*)ws.keys_tmp.ptr;
    uint32_t* idx = (uint32_t*)ws.idx.ptr;
    uint32_t* itmp = (uint32_t*)ws.idx_tmp.ptr;
    int* flags = (int*)ws.flags.ptr;
    GH_CUDA_TRY(cudaMemsetAsync(flags, 0, 8 * sizeof(int), st));
    if (n >= 4LL * 256 * ws.num_sms)  // four blocks of 256 per SM (see keys_kernel)
      keys_kernel<1024><<<(unsigned)((n + 1023) / 1024), 1024, 0, st>>>(pos, n, root, words, keys, idx);
    else
      keys_kernel<256><<<gn, 256, 0, st>>>(pos, n, root, words, keys, idx);
    GH_LAUNCH_CHECK();
    if (full_sort) {
      GH_TRY(radix_sort_keys(keys, idx, ktmp, itmp, words, KEY_BITS, n, (uint32_t*)ws.rs.ptr, st, flags + 5));
    } else {
      GH_TRY(radix_sort_keys(keys, idx, ktmp, itmp, 1, KEY_BITS, n, (uint32_t*)ws.rs.ptr, st, flags + 5));
      gather_words_kernel<<<gn, T, 0, st>>>(keys, ktmp, words, n, idx);
      GH_LAUNCH_CHECK();
      GH_CUDA_TRY(cudaMemcpyAsync(keys + n, ktmp + n, (size_t)(words - 1) * n * sizeof(uint64_t),
                                  cudaMemcpyDeviceToDevice, st));
      tie_rank_kernel<<<gn, T, 0, st>>>(keys, words, n, idx, ktmp, itmp, (int*)ws.flags.ptr);
      GH_LAUNCH_CHECK();
      tie_copy_kernel<<<gn, T, 0, st>>>(keys, words, n, idx, ktmp, itmp);
      GH_LAUNCH_CHECK();
    }
    if (wait_fault)
      GH_CUDA_TRY(cudaMemsetAsync(flags + 5, 1, 1, st));
    lcp_kernel<<<gn1, T, 0, st>>>(keys, words, n, (int*)ws.lp.ptr, (int*)ws.flags.ptr);
    GH_LAUNCH_CHECK();
    count_kernel<<<gn, T, 0, st>>>((const int*)ws.lp.ptr, n, (int*)ws.cnt.ptr, (int*)ws.depth.ptr,
                                   (int*)ws.flags.ptr);
    GH_LAUNCH_CHECK();
    GH_TRY(exclusive_scan_i32((const int*)ws.cnt.ptr, (int*)ws.base.ptr, n, (int*)ws.scan.ptr, st));
    if (sort_targets) {  // the targets' walk order; its sort reports a given-up wait in flags[5] too
      GH_TRY(ensure(ws.tkeys, (size_t)2 * nt * sizeof(uint64_t)));
      GH_TRY(ensure(ws.tkeys_tmp, (size_t)2 * nt * sizeof(uint64_t)));
      GH_TRY(ensure(ws.tidx, (size_t)nt * sizeof(uint32_t)));
      GH_TRY(ensure(ws.tidx_tmp, (size_t)nt * sizeof(uint32_t)));
      GH_TRY(ensure(ws.trs, radix_scratch_words(nt) * sizeof(uint32_t)));
      target_keys_kernel<<<(unsigned)((nt + T - 1) / T), T, 0, st>>>(tpos, nt, root, (uint64_t*)ws.tkeys.ptr,
                                                                     (uint32_t*)ws.tidx.ptr);
      GH_LAUNCH_CHECK();
      GH_TRY(radix_sort_keys((uint64_t*)ws.tkeys.ptr, (uint32_t*)ws.tidx.ptr, (uint64_t*)ws.tkeys_tmp.ptr,
                             (uint32_t*)ws.tidx_tmp.ptr, 2, KEY_BITS, nt, (uint32_t*)ws.trs.ptr, st, flags + 5));
      out->torder = (const uint32_t*)ws.tidx.ptr;
    }
    GH_CUDA_TRY(cudaMemcpyAsync(ws.host_flags, ws.flags.ptr, 8 * sizeof(int), cudaMemcpyDeviceToHost, st));
    GH_CUDA_TRY(cudaMemcpyAsync(ws.host_flags + 8, (int*)ws.base.ptr + n, sizeof(int), cudaMemcpyDeviceToHost,
                                st));
    GH_CUDA_TRY(cudaMemcpyAsync(ws.host_flags + 9, &root->bad, sizeof(int), cudaMemcpyDeviceToHost, st));
    GH_CUDA_TRY(cudaStreamSynchronize(st));
    // The kernels so far index only by particle and sort slot, whatever the keys hold,
    // so non-finite input is refused here, before any cell is built from it.
    if (ws.host_flags[9]) return bad_input();
    if (ws.host_flags[5]) return set_error(GH_ERR_TIMEOUT, "tree: radix sort look-back gave up");
    if (ws.host_flags[2] && !full_sort) {  // a long run of equal first words
      full_sort = true;
      ws.full_sort_n = n;
      continue;
    }
    if (!ws.host_flags[0]) break;
    if (ws.words >= TREE_MAX_WORDS)
      return set_error(GH_ERR_DEPTH,
                       "tree: particles share their first %d octree levels (coincident positions?)",
                       TREE_MAX_WORDS * KEY_LEVELS);
    ws.words++;
  }
  const int words = ws.words;
  const int maxdepth = ws.host_flags[1];
  const int nnodes = ws.host_flags[8];
  if (n <= SB_MAX) {
    uint8_t& tied = ws.small_tied[n];
    if (maxdepth > 2 * KEY_LEVELS)  // a leaf below both words' levels: they tied
      tied = SB_TIE_BUILDS;
    else if (tied)
      tied--;
  }
  // 4. nodes
  GH_TRY(ensure(ws.nA, (size_t)nnodes * sizeof(WalkRec)));
  GH_TRY(ensure(ws.nC, (size_t)nnodes * sizeof(dvec4)));
  GH_TRY(ensure(ws.nM, (size_t)nnodes * sizeof(dvec4)));
  const int64_t ntiles = (n + MS_TILE - 1) / MS_TILE;
  GH_TRY(ensure(ws.fxl, (size_t)n * sizeof(FxMoments)));
  GH_TRY(ensure(ws.fxt, (size_t)(ntiles + 1) * sizeof(FxMoments)));
  // every node that is not a particle's leaf is an internal cell
  const int64_t ncells = (int64_t)nnodes - n;
  GH_TRY(ensure(ws.cells, (size_t)(ncells > 0 ? ncells : 1) * sizeof(int2)));
  NodeArrays na = node_arrays(ws);
  {
    const uint64_t* keys = (const uint64_t*)ws.keys.ptr;
    const int* lp = (const int*)ws.lp.ptr;
    const int* dep = (const int*)ws.depth.ptr;
    const int* bs = (const int*)ws.base.ptr;
    const uint32_t* perm = (const uint32_t*)ws.idx.ptr;
    int* openers = (int*)ws.flags.ptr + 4;
    FxMoments* fxl = (FxMoments*)ws.fxl.ptr;
    FxMoments* fxt = (FxMoments*)ws.fxt.ptr;
    // 5. exact prefix sums of the moments (the cells' monopoles come from them below)
    moments_scan_kernel<MS_ITEMS><<<(unsigned)ntiles, MS_THREADS, 0, st>>>(pos, mass, perm, n, root, fxl, fxt);
    GH_LAUNCH_CHECK();
    moments_tiles_kernel<<<1, MS_THREADS, 0, st>>>(fxt, ntiles);
    GH_LAUNCH_CHECK();
    // 4. leaves, then the internal cells' centres, then the rest of each internal cell
    int2* cells = (int2*)ws.cells.ptr;
    nodes_kernel<<<gn, T, 0, st>>>(n, lp, dep, bs, perm, pos, mass, na, nnodes, (int*)ws.list.ptr, openers, cells,
                                   (int*)ws.flags.ptr + 6);
    GH_LAUNCH_CHECK();
    const unsigned resident = 4u * (unsigned)ws.num_sms;
    cell_centres_kernel<<<gn < resident ? gn : resident, T, 0, st>>>(keys, words, n, lp, dep, bs, root, na,
                                                                    (const int*)ws.list.ptr, openers);
    GH_LAUNCH_CHECK();
    if (ncells > 0) {
      cells_kernel<<<(unsigned)((ncells + T - 1) / T), T, 0, st>>>(keys, words, n, lp, bs, root, na, nnodes, cells,
                                                                   (int)ncells, fxl, fxt);
      GH_LAUNCH_CHECK();
    }
  }
  out->n = n;
  out->nnodes = nnodes;
  out->nodes = (const int*)ws.base.ptr + n;
  out->maxdepth = maxdepth;
  return GH_OK;
}

// Walk counters, off unless gh_tree_stats(1): [0] warp cell steps (one 48-byte
// record read each), [1] cells visited summed over targets, [2] target-cell
// interactions, [3] exact FP64 opening tests, [4] interactions with leaves.
static bool g_stats_on = false;
static int64_t g_stats_walks = 0;
static Buffer g_stats[64];

// Warps per target group of an FP64 walk.  A warp walks hundreds to thousands of cells in
// a chain of dependent steps, so a walk with fewer groups than the GPU holds warps
// (36 per SM) takes as long as its longest chain; splitting the chains fills the GPU, at
// about 2 % more steps per doubling (the ancestors of each segment's first cell).
// All in all 14,000 warps and n / 5 more were fastest (a larger tree has more steps to
// share), at most 64 per group of particles, 128 of sorted points and 256 of unsorted ones.
// Where that is less than 12 for each of many groups, two, whose ranges meet at the group's
// own place: with Hernquist + disk, 11 / two (us), theta 0.7 and 0.5: N = 75,000 1651 / 1532
// and 3103 / 3119, 90,113 1916 / 1920 and 3795 / 4026, 110,000 2158 / 2222 and 4330 / 4981,
// 131,072 2563 / 2361 and 5145 / 5095, 200,000 3669 / 3513 and 7932 / 8092; 3 to 8 are worse
// than the better of the two.  So neither wins throughout, and the line is where theta 0.7
// changes sides for good.  3/8 of a million targets fill the GPU unsplit (393,217: 6833 us, two
// 6704; 1,048,576 18.7 ms, two 19.1).  Force, unsplit -> split, theta 0.7: N = 500 Plummer 302 -> 96 us,
// 2000 577 -> 131, 8000 840 -> 303; Hernquist + disk 16,384 1304 -> 575, 30,000 1541 ->
// 842, 60,013 1726 -> 1372, 131,072 2392 -> 2359, 262,144 4638 -> 4477.  Points in a 250,000-particle system, theta 0.5: 100
// unsorted 17.6 -> 0.85 ms, 8100 16.9 -> 2.9, 10,000 sorted 7.0 -> 1.8, 30,011 6.0 -> 2.8,
// 100,000 6.3 -> 5.5.
static int walk_segments(int64_t groups, int64_t n, int cap) {
  if (groups > 12288) return 1;
  const int64_t warps = 14000 + (n < 262144 ? n : 262144) / 5, k = warps / groups;
  if (k < 12 && groups > 2816) return 2;
  return (int)(k < cap ? k : cap);
}

template <bool G, class Epi>
static int launch_walk_f64(TreeWS& ws, const NodeArrays& na, const BuiltTree& bt, const double* tpos,
                           const uint32_t* order, int64_t nt, bool self, double eps2, double theta, float lo, float hi,
                           const Epi& epi, unsigned long long* stats, cudaStream_t st) {
  const int64_t groups = (nt + 31) / 32;
  WalkSplit sp = {};
  sp.segs = stats ? 1 : walk_segments(groups, bt.n, self ? 64 : (order ? 128 : 256));  // the counters are those of whole walks
  const size_t cb = (size_t)groups * sizeof(int);
  if (sp.segs > 1) {  // at most 51 MB of scratch; without it the walk is not split
    int rc = ensure(ws.wpart, (size_t)groups * sp.segs * 96 * sizeof(double));
    if (rc == GH_OK && ws.wcount.bytes < cb) ws.wcount_zeroed = 0;
    if (rc == GH_OK) rc = ensure(ws.wcount, cb);
    if (rc == GH_ERR_OOM) {
      clear_error();
      sp.segs = 1;
    } else if (rc != GH_OK) {
      return rc;
    }
  }
  const unsigned blocks = (unsigned)((groups + TW_THREADS / 32 - 1) / (TW_THREADS / 32)) * (unsigned)sp.segs;
  if (sp.segs > 1) {
    if (ws.wcount_zeroed < cb) {
      GH_CUDA_TRY(cudaMemsetAsync(ws.wcount.ptr, 0, ws.wcount.bytes, st));
      ws.wcount_zeroed = ws.wcount.bytes;
    }
    sp.part = (double*)ws.wpart.ptr;
    sp.count = (int*)ws.wcount.ptr;
    if (self || order) sp.base = (const int*)ws.base.ptr;
    if (!self && order) {
      sp.keys = (const uint64_t*)ws.keys.ptr;
      sp.tkeys = (const uint64_t*)ws.tkeys.ptr;
      sp.n = bt.n;
    }
  }
  prof_begin(st);
  if (stats)
    tree_walk_f64_kernel<G, true, false, Epi><<<blocks, TW_THREADS, 0, st>>>(na.R, na.C, na.M, bt.nodes, tpos, order,
                                                                             nt, eps2, theta, lo, hi, epi, sp, stats);
  else if (sp.segs > 1)
    tree_walk_f64_kernel<G, false, true, Epi><<<blocks, TW_THREADS, 0, st>>>(na.R, na.C, na.M, bt.nodes, tpos, order,
                                                                             nt, eps2, theta, lo, hi, epi, sp, nullptr);
  else
    tree_walk_f64_kernel<G, false, false, Epi><<<blocks, TW_THREADS, 0, st>>>(
        na.R, na.C, na.M, bt.nodes, tpos, order, nt, eps2, theta, lo, hi, epi, sp, nullptr);
  prof_end(st);
  return GH_OK;
}

template <bool G, class Epi>
static void launch_walk_mixed(const NodeArrays& na, const BuiltTree& bt, const double* tpos, const uint32_t* order,
                              int64_t nt, double eps2, double theta, float lo, float hi, const Epi& epi,
                              unsigned long long* stats, cudaStream_t st) {
  const unsigned blocks = (unsigned)((nt + TW_THREADS - 1) / TW_THREADS);
  prof_begin(st);
  if (stats)
    tree_walk_kernel<G, true, Epi><<<blocks, TW_THREADS, 0, st>>>(na.R, na.C, bt.nodes, tpos, order, nt, eps2, theta,
                                                                  lo, hi, epi, stats);
  else
    tree_walk_kernel<G, false, Epi><<<blocks, TW_THREADS, 0, st>>>(na.R, na.C, bt.nodes, tpos, order, nt, eps2, theta,
                                                                   lo, hi, epi, nullptr);
  prof_end(st);
}

template <class Epi>
static int tree_walk(TreeWS& ws, const BuiltTree& bt, const double* tpos, const uint32_t* order, int64_t nt, bool self,
                     double eps, double theta, int precision, const Epi& epi, cudaStream_t st) {
  if (nt == 0) return GH_OK;
  Trace tr("tree walk");
  const double eps2 = eps * eps;
  // theta <= 0 or NaN: the prefilter opens every cell and accepts none; below 1e-3
  // it decides nothing (every internal cell takes the exact test)
  float lo = -1.f, hi = -1.f;
  if (theta >= 1e-3) {
    lo = (float)(theta * theta * (1.0 - TREE_MARGIN));
    hi = (float)(theta * theta * (1.0 + TREE_MARGIN));
  } else if (theta > 0.0) {
    hi = INFINITY;
  }
  NodeArrays na = node_arrays(ws);
  const bool mixed = precision == GH_PREC_MIXED;
  const bool guard = mixed ? !((float)eps2 > 0.f) : eps2 == 0.0;
  unsigned long long* stats = nullptr;
  if (g_stats_on) {
    DeviceInfo di;
    GH_TRY(device_info(&di));
    Buffer& b = g_stats[di.device];
    if (!b.ptr) {
      GH_TRY(ensure(b, 8 * sizeof(unsigned long long)));
      GH_CUDA_TRY(cudaMemsetAsync(b.ptr, 0, 8 * sizeof(unsigned long long), st));
    }
    stats = (unsigned long long*)b.ptr;
    g_stats_walks++;
  }
  if (mixed) {
    if (guard)
      launch_walk_mixed<true>(na, bt, tpos, order, nt, eps2, theta, lo, hi, epi, stats, st);
    else
      launch_walk_mixed<false>(na, bt, tpos, order, nt, eps2, theta, lo, hi, epi, stats, st);
  } else {
    if (guard)
      GH_TRY(launch_walk_f64<true>(ws, na, bt, tpos, order, nt, self, eps2, theta, lo, hi, epi, stats, st));
    else
      GH_TRY(launch_walk_f64<false>(ws, na, bt, tpos, order, nt, self, eps2, theta, lo, hi, epi, stats, st));
  }
  GH_LAUNCH_CHECK();
  return GH_OK;
}

static int check_tree_args(int64_t np, int64_t nt, double eps, int precision) {
  if (np < 0 || nt < 0) return set_error(GH_ERR_ARG, "negative particle count");
  if (precision != GH_PREC_FP64 && precision != GH_PREC_MIXED)
    return set_error(GH_ERR_ARG, "unknown precision %d", precision);
  if (!(eps >= 0.0)) return set_error(GH_ERR_ARG, "eps must be >= 0 (got %g)", eps);
  return GH_OK;
}

int tree_force(const double* pos, const double* mass, int64_t np, const double* tpos, int64_t nt, double eps,
               double theta, int precision, double* acc, cudaStream_t st) {
  GH_TRY(check_tree_args(np, nt, eps, precision));
  const bool self = (tpos == nullptr);
  if (self) nt = np;
  if (nt == 0) return GH_OK;
  if (!acc || (np > 0 && (!pos || !mass))) return set_error(GH_ERR_ARG, "null buffer passed to tree force");
  if (np == 0) {
    GH_CUDA_TRY(cudaMemsetAsync(acc, 0, (size_t)nt * 3 * sizeof(double), st));
    return GH_OK;
  }
  std::lock_guard<std::recursive_mutex> lk(g_tree_mu);
  TreeWS* w = nullptr;
  GH_TRY(tree_workspace(&w));
  TreeWS& ws = *w;
  EpiStore epi{acc};
  for (bool again = true; again;) {
    BuiltTree bt;
    GH_TRY(tree_build(ws, pos, mass, np, eps, st, &bt, !g_stats_on, self ? nullptr : tpos, self ? 0 : nt));
    if (self)
      GH_TRY(tree_walk(ws, bt, pos, (const uint32_t*)ws.idx.ptr, np, true, eps, theta, precision, epi, st));
    else
      GH_TRY(tree_walk(ws, bt, tpos, bt.torder, nt, false, eps, theta, precision, epi, st));
    GH_TRY(small_finish(ws, &bt, &again));
  }
  return GH_OK;
}

int tree_run(double* x, double* v, const double* mass, int64_t np, int64_t nsteps, double dt, double eps,
             double theta, int precision, double* hist_x, double* hist_v, int64_t stride, cudaStream_t st) {
  GH_TRY(check_tree_args(np, 0, eps, precision));
  std::lock_guard<std::recursive_mutex> lk(g_tree_mu);
  TreeWS* w = nullptr;
  GH_TRY(tree_workspace(&w));
  TreeWS& ws = *w;
  GH_TRY(ensure(ws.xh[0], (size_t)np * 3 * sizeof(double)));
  GH_TRY(ensure(ws.xh[1], (size_t)np * 3 * sizeof(double)));
  GH_TRY(drift_prepare_f64(x, v, np, dt, (double*)ws.xh[0].ptr, st));
  for (int64_t s = 0; s < nsteps; s++) {
    Trace step("tree dkd step");
    const int cur = (int)(s & 1), nxt = cur ^ 1;
    const double* xh = (const double*)ws.xh[cur].ptr;
    EpiDKD epi;
    epi.x = x;
    epi.v = v;
    epi.mass = mass;
    epi.dt = dt;
    epi.src_next = nullptr;
    epi.origin = nullptr;
    epi.xh_next = (double*)ws.xh[nxt].ptr;
    epi.hist_x = epi.hist_v = nullptr;
    if (hist_x && stride > 0 && (s + 1) % stride == 0) {
      const int64_t slot = (s + 1) / stride - 1;
      epi.hist_x = hist_x + slot * np * 3;
      epi.hist_v = hist_v + slot * np * 3;
    }
    for (bool again = true; again;) {
      BuiltTree bt;
      GH_TRY(tree_build(ws, xh, mass, np, eps, st, &bt, !g_stats_on));
      GH_TRY(tree_walk(ws, bt, xh, (const uint32_t*)ws.idx.ptr, np, true, eps, theta, precision, epi, st));
      GH_TRY(small_finish(ws, &bt, &again));
    }
  }
  return GH_OK;
}

}  // namespace gh

// ---------------------------------------------------------------------------
// Invariant check of a built tree (gh_tree_validate)
// ---------------------------------------------------------------------------
// out: [0] leaves, [1] skip index out of range, [2] children that do not tile their
// cell's subtree, [3] cells with more than 8 child cells, [4] cell mass not the sum of
// its children's, [5] a child's centre of mass outside its cell, [6] walk record not
// matching the FP64 cell, [7] root subtree not the whole preorder.
namespace gh {
__global__ void tree_validate_kernel(const WalkRec* __restrict__ R, const dvec4* __restrict__ C,
                                     const dvec4* __restrict__ M, int nnodes, unsigned long long* __restrict__ out) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnodes; k += gridDim.x * blockDim.x) {
    const int nx = __float_as_int(R[k].L.w);
    if (k == 0 && nx != nnodes) atomicAdd(&out[7], 1ull);
    if (nx <= k || nx > nnodes) {
      atomicAdd(&out[1], 1ull);
      continue;
    }
    const dvec4 Mk = M[k];
    if (nx == k + 1) {  // leaf: its record is its particle
      atomicAdd(&out[0], 1ull);
      const float4 A = R[k].A;
      if (A.x != (float)Mk.x || A.y != (float)Mk.y || A.z != (float)Mk.z || R[k].O.w != (float)Mk.w)
        atomicAdd(&out[6], 1ull);
      continue;
    }
    const dvec4 Ck = C[k];
    const float4 A = R[k].A;
    if (A.x != (float)Ck.x || A.y != (float)Ck.y || A.z != (float)Ck.z || A.w != (float)(Ck.w * Ck.w) ||
        R[k].O.w != (float)Mk.w)
      atomicAdd(&out[6], 1ull);
    // children: k + 1, then each one's skip index, up to this cell's skip index (at most 8
    // steps are taken; a ninth child counts as a violation)
    const double half = 0.5 * Ck.w * (1.0 + 1e-12);
    double msum = 0.0;
    int c = k + 1, kids = 0;
    while (c < nx && kids <= 8) {
      const dvec4 Mc = M[c];
      msum += Mc.w;
      if (fabs(Mc.x - Ck.x) > half || fabs(Mc.y - Ck.y) > half || fabs(Mc.z - Ck.z) > half)
        atomicAdd(&out[5], 1ull);
      const int cn = __float_as_int(R[c].L.w);
      if (cn <= c || cn > nx) break;
      c = cn;
      kids++;
    }
    if (kids > 8) atomicAdd(&out[3], 1ull);
    else if (c != nx) atomicAdd(&out[2], 1ull);
    if (!(fabs(msum - Mk.w) <= 1e-12 * fabs(Mk.w))) atomicAdd(&out[4], 1ull);
  }
}
}  // namespace gh

extern "C" int gh_tree_validate(const double* pos, const double* mass, int64_t np, double eps, int64_t* out,
                                void* stream) {
  using namespace gh;
  clear_error();
  if (!out) return set_error(GH_ERR_ARG, "tree validate: null output");
  if (np <= 0) return set_error(GH_ERR_ARG, "tree validate: no particles");
  if (!pos || !mass) return set_error(GH_ERR_ARG, "null buffer");
  cudaStream_t st = (cudaStream_t)stream;
  std::lock_guard<std::recursive_mutex> lk(g_tree_mu);
  DeviceInfo di;
  GH_TRY(device_info(&di));
  TreeWS* w = nullptr;
  GH_TRY(tree_workspace(&w));
  TreeWS& ws = *w;
  BuiltTree bt;
  GH_TRY(tree_build(ws, pos, mass, np, eps, st, &bt));
  static Buffer counts[64];
  GH_TRY(ensure(counts[di.device], 8 * sizeof(unsigned long long)));
  unsigned long long* dc = (unsigned long long*)counts[di.device].ptr;
  GH_CUDA_TRY(cudaMemsetAsync(dc, 0, 8 * sizeof(unsigned long long), st));
  NodeArrays na = node_arrays(ws);
  tree_validate_kernel<<<2 * di.num_sms, 256, 0, st>>>(na.R, na.C, na.M, bt.nnodes, dc);
  GH_LAUNCH_CHECK();
  unsigned long long h[8];
  GH_CUDA_TRY(cudaMemcpyAsync(h, dc, sizeof(h), cudaMemcpyDeviceToHost, st));
  GH_CUDA_TRY(cudaStreamSynchronize(st));
  out[0] = bt.nnodes;
  for (int k = 0; k < 8; k++) out[k + 1] = (int64_t)h[k];
  return GH_OK;
}

extern "C" int gh_tree_stats(int enable) {
  using namespace gh;
  clear_error();
  std::lock_guard<std::recursive_mutex> lk(g_tree_mu);
  g_stats_on = enable != 0;
  return GH_OK;
}

extern "C" int gh_tree_stats_read(int64_t* out) {
  using namespace gh;
  clear_error();
  if (!out) return set_error(GH_ERR_ARG, "tree stats: null output");
  std::lock_guard<std::recursive_mutex> lk(g_tree_mu);
  DeviceInfo di;
  GH_TRY(device_info(&di));
  Buffer& b = g_stats[di.device];
  unsigned long long h[6] = {0, 0, 0, 0, 0, 0};
  if (b.ptr) {
    GH_CUDA_TRY(cudaDeviceSynchronize());
    GH_CUDA_TRY(cudaMemcpy(h, b.ptr, sizeof(h), cudaMemcpyDeviceToHost));
    GH_CUDA_TRY(cudaMemset(b.ptr, 0, sizeof(h)));
    GH_CUDA_TRY(cudaDeviceSynchronize());
  }
  out[0] = g_stats_walks;
  for (int k = 0; k < 6; k++) out[k + 1] = (int64_t)h[k];
  g_stats_walks = 0;
  return GH_OK;
}
