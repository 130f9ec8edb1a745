// Bounds, Morton keys, tree keys, gathers, leapfrog halves, node discovery, upsweep and the
// node hash table.
//
// FP64 arithmetic that must reproduce the reference bit for bit uses the explicitly rounded
// intrinsics (__dadd_rn, __dmul_rn, ...), so the compiler cannot contract it into FMAs.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>

#include "bh_internal.cuh"
#include "bh_tilesort.cuh"

namespace bh {
namespace {

constexpr int kThreads = 256;

// ---------------------------------------------------------------------------------------
// exact-arithmetic helpers
// ---------------------------------------------------------------------------------------

// Magic-bit spread of src/MortonKeys.hpp:100-104 with the masks of :51-58, on the full 64-bit
// word (high garbage bits of wrapped coordinates behave as in the reference).
__device__ __forceinline__ uint64_t spread_bits(uint64_t v) {
  v = (v | v << 32) & 0x1f00000000ffffull;
  v = (v | v << 16) & 0x1f0000ff0000ffull;
  v = (v | v << 8) & 0x100f00f00f00f00full;
  v = (v | v << 4) & 0x10c30c30c30c30c3ull;
  v = (v | v << 2) & 0x1249249249249249ull;
  return v;
}

// Float-float arithmetic (a value is hi + lo): TwoSum (Knuth), FMA-based TwoProduct and a
// Newton-corrected quotient (Dekker 1971). About 44 significant bits from FP32 operations.
struct FF {
  float hi, lo;
};
__device__ __forceinline__ FF ff_norm(float s, float e) {
  const float hi = s + e;
  return {hi, e - (hi - s)};
}
__device__ __forceinline__ FF ff_add(FF a, FF b) {
  const float s = a.hi + b.hi;
  const float bb = s - a.hi;
  float e = (a.hi - (s - bb)) + (b.hi - bb);
  e += a.lo + b.lo;
  return ff_norm(s, e);
}
__device__ __forceinline__ FF ff_prod(float a, float b) {
  const float p = a * b;
  return {p, fmaf(a, b, -p)};
}
__device__ __forceinline__ FF ff_mul(FF a, FF b) {
  const float p = a.hi * b.hi;
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  return ff_norm(p, e);
}
__device__ __forceinline__ FF ff_div(FF n, FF d) {
  const float q = n.hi / d.hi;
  const float p = q * d.hi;
  const float pe = fmaf(q, d.hi, -p);
  const float r = (((n.hi - p) - pe) + fmaf(-q, d.lo, n.lo)) / d.hi;
  return ff_norm(q, r);
}
// Splits a double into a float-float pair (hi = nearest float, lo = nearest float of the rest):
// the pair matches the double to about 2^-48 relative.
__device__ __forceinline__ void ff_split(double x, float& hi, float& lo) {
  hi = __double2float_rn(x);
  lo = __double2float_rn(__dsub_rn(x, (double)hi));
}

// x ~ n + f from a float-float value: n = nearest integer of hi (exactly representable), f the
// signed remainder (|f| <= 0.5 + |lo|), accurate to the pair's own error.
__device__ __forceinline__ void ff_int_frac(FF x, float& n, float& f) {
  n = rintf(x.hi);
  f = (x.hi - n) + x.lo;
}

// The reference's (spatialKey)(double) cast (src/MortonKeys.hpp:162-164) as x86-64 code
// generated by gcc evaluates it: below 2^63 (or NaN) a signed truncation, 0x8000000000000000
// when that is out of range; otherwise a truncation of x - 2^63 with bit 63 flipped.
__device__ __forceinline__ uint64_t x86_trunc_u64(double x) {
  if (!(x >= 0x1p63)) {
    if (x >= -0x1p63) return (uint64_t)__double2ll_rz(x);
    return 0x8000000000000000ull;
  }
  double y = __dsub_rn(x, 0x1p63);
  if (y < 0x1p63) return (uint64_t)__double2ll_rz(y) ^ 0x8000000000000000ull;
  return 0ull;
}

// One axis of computeMortonKey (src/MortonKeys.hpp:137-181) in the reference's own FP64
// arithmetic: (p + S) * frac, then the cast.
__device__ __noinline__ uint64_t morton_coord_exact(float x, double S, double frac) {
  return x86_trunc_u64(__dmul_rn(__dadd_rn((double)x, S), frac));
}

// The same axis with an FP32 fast path. v = (p + S) * frac is formed in float-float: for
// |v| < 2^22 the pair is within 2^-23 of the exact v, and the reference's two FP64 roundings put
// its value within |v| 2^-52 <= 2^-30 of it. When the pair lies farther than 2^-21 from every
// integer, both therefore truncate to the same integer, which the fast path returns (as the
// 64-bit two's-complement word the cast produces for |v| < 2^63). Otherwise (near an integer,
// |v| >= 2^22, or not finite) the FP64 path decides.
__device__ __forceinline__ uint64_t morton_coord(float x, const Geom& g) {
  const FF v = ff_mul(ff_add({x, 0.f}, {g.size_hi, g.size_lo}), {g.frac_hi, g.frac_lo});
  float n, f;
  ff_int_frac(v, n, f);
  if (fabsf(v.hi) < 0x1p22f && fabsf(f) > 0x1p-21f) {
    const bool pos = n > 0.f || (n == 0.f && f > 0.f);
    // truncation toward zero: floor for positive v, ceiling for negative v
    const float q = pos ? (f < 0.f ? n - 1.f : n) : (f > 0.f ? n + 1.f : n);
    return (uint64_t)(long long)q;
  }
  return morton_coord_exact(x, g.size, g.frac);
}

// computeMortonKey: the three axes interleaved x<<2 | y<<1 | z with bit 63 set
// (interleaveBits, src/MortonKeys.hpp:95-124).
__device__ __forceinline__ uint64_t morton_key(float4 p, const Geom& g) {
  const uint64_t wx = morton_coord(p.x, g), wy = morton_coord(p.y, g), wz = morton_coord(p.z, g);
  return (1ull << 63) | (spread_bits(wx) << 2) | (spread_bits(wy) << 1) | spread_bits(wz);
}

// 21-bit octant path of one coordinate below a root of centre c0 and edge E, exactly as the
// reference's descent computes it: at each depth compare p > c (DetermineOctant,
// src/OctantUtils.hpp:64-70), halve the size and move the centre by (+-0.5) * size
// (HOTNode child constructor, src/HashedNode.cpp:52-56), one FP64 rounding per level.
__device__ __noinline__ uint32_t tree_path_exact(double p, double c0, double E) {
  double c = c0, s = E;
  uint32_t k = 0;
  for (int d = 0; d < kMaxDepth; ++d) {
    uint32_t b = p > c ? 1u : 0u;
    k = (k << 1) | b;
    s = __dmul_rn(s, 0.5);
    c = __dadd_rn(c, __dmul_rn(b ? 0.5 : -0.5, s));
  }
  return k;
}

// Same path from one scaled coordinate. In exact arithmetic the level-d comparison points
// are the integers of [1, 2^21 - 1] in the units u = (p - c0) * 2^21 / E + 2^20, and the
// strict '>' makes the path ceil(u) - 1 clamped to [0, 2^21 - 1]. The reference's rounded
// centres differ from the exact ones by at most 21 half-ulps: below 2^-26 * (1 + |c0| / E) key
// units. u is formed in float-float (the splits of c0 and 2^21 / E and the pair arithmetic add
// below 2^-24 * (1 + |c0| / E)). Whenever u lies closer than the margin
// (2^-20 * (1 + |c0| / E)) to a comparison point, or is not finite, the exact recurrence
// decides instead.
__device__ __forceinline__ uint32_t tree_path(float p, int a, const Geom& g) {
  const FF d = ff_add({p, 0.f}, {-g.tc_hi[a], -g.tc_lo[a]});
  const FF u = ff_add(ff_mul(d, {g.tscale_hi, g.tscale_lo}), {1048576.f, 0.f});
  float n, f;
  ff_int_frac(u, n, f);
  float dist;
  uint32_t path;
  if (n < 1.f || (n == 1.f && f < 0.f)) {  // u < 1
    dist = (1.f - n) - f;
    path = 0u;
  } else if (n > 2097151.f || (n == 2097151.f && f > 0.f)) {  // u > 2^21 - 1
    dist = (n - 2097151.f) + f;
    path = 2097151u;
  } else {
    dist = fabsf(f);
    path = (uint32_t)(f < 0.f ? n - 1.f : n);
  }
  if (dist > g.tmargin_f) return path;  // false for NaN
  return tree_path_exact((double)p, g.tc[a], g.tedge);
}

__device__ __forceinline__ uint64_t tree_key(float4 p, const Geom& g) {
  const uint32_t kx = tree_path(p.x, 0, g), ky = tree_path(p.y, 1, g), kz = tree_path(p.z, 2, g);
  return (1ull << 63) | (spread_bits(kx) << 2) | (spread_bits(ky) << 1) | spread_bits(kz);
}

__device__ __forceinline__ void fill_tree_geom(Geom& g, const double tc[3], double tedge) {
  g.tc[0] = tc[0];
  g.tc[1] = tc[1];
  g.tc[2] = tc[2];
  g.tedge = tedge;
  g.tscale = __ddiv_rn(2097152.0, tedge);
  double cm = fmax(fabs(tc[0]), fmax(fabs(tc[1]), fabs(tc[2])));
  g.tmargin = 0x1p-20 * (1.0 + cm / tedge);
  // float-float copies for the key fast paths (size and frac are set by every caller first)
  ff_split(g.size, g.size_hi, g.size_lo);
  ff_split(g.frac, g.frac_hi, g.frac_lo);
  for (int a = 0; a < 3; ++a) ff_split(tc[a], g.tc_hi[a], g.tc_lo[a]);
  ff_split(g.tscale, g.tscale_hi, g.tscale_lo);
  g.tedge2 = __double2float_rn(__dmul_rn(tedge, tedge));
  g.tmargin_f = __double2float_rn(g.tmargin);
}

// ---------------------------------------------------------------------------------------
// bounds (OctantBounds(Body*, N), src/OctantUtils.cpp:27-59)
// ---------------------------------------------------------------------------------------

// Partial of one block: FP64 sums and FP32 maxima of the absolute coordinates.
struct BoundsPartial {
  double sum[3];
  float mx[3];
  float pad;
};
constexpr int kBoundsPerLane = 10;  // partials per lane of the finishing warp (at most 320 blocks)

// The step's geometry, from the sums and maxima in every lane of one warp: centre = sum * (1 / N)
// (Vec3D::operator/=, src/MathUtils.cpp:81-90), size = max(0, max_a (max_i |p_ia| - c_a)). fl(|p| - c)
// is monotone in |p|, so the maximum over bodies of the rounded differences equals the rounded
// difference of the maximum. The three FP64 quotients run on three lanes at once, and each lane
// splits one value for the key fast paths (the values are fill_tree_geom's, bit for bit).
__device__ __forceinline__ void finish_geom(const double (&s)[3], const float (&mx)[3], int n, double inv_n,
                                            double edge_factor, Geom* __restrict__ g) {
  const int lane = threadIdx.x & 31;
  double c[3];
  double S = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    c[a] = n != 0 ? __dmul_rn(s[a], inv_n) : s[a];
    const double v = __dsub_rn((double)mx[a], c[a]);
    if (v > S) S = v;
  }
  const double tedge = __dmul_rn(S, edge_factor);
  const double cm = fmax(fabs(c[0]), fmax(fabs(c[1]), fabs(c[2])));
  // lane 0: 2^21 / (2 S), lane 1: 2^21 / tedge, lane 2: cm / tedge
  const double q = __ddiv_rn(lane == 2 ? cm : 2097152.0, lane == 0 ? __dmul_rn(2.0, S) : tedge);
  // lanes 0-5 hold frac, tscale, margin, size and the centre (6 and 7 its last axes)
  const double v = lane == 2 ? 0x1p-20 * (1.0 + q) : lane == 3 ? S : lane == 4 ? c[0] : lane == 5 ? c[1] : lane == 6 ? c[2] : q;
  float hi, lo;
  ff_split(v, hi, lo);
  switch (lane) {
    case 0:
      g->frac = v;
      g->frac_hi = hi;
      g->frac_lo = lo;
      break;
    case 1:
      g->tscale = v;
      g->tscale_hi = hi;
      g->tscale_lo = lo;
      break;
    case 2:
      g->tmargin = v;
      g->tmargin_f = hi;
      break;
    case 3:
      g->size = v;
      g->size_hi = hi;
      g->size_lo = lo;
      break;
    case 4:
    case 5:
    case 6:
      g->center[lane - 4] = v;
      g->tc[lane - 4] = v;
      g->tc_hi[lane - 4] = hi;
      g->tc_lo[lane - 4] = lo;
      break;
    case 7:
      g->tedge = tedge;
      g->tedge2 = __double2float_rn(__dmul_rn(tedge, tedge));
      break;
    default: break;
  }
}

// Bounds in one launch. Per block: FP64 sums of x, y, z (each thread strides through the bodies in a
// fixed order, then a fixed-shape tree) and FP32 maxima of |x|, |y|, |z|. The last block to finish
// combines the partials in one warp (lane l sums partials l, l + 32, ... in order, then a fixed
// shuffle tree): the result does not depend on which block that is. Blocks beyond the bodies
// would add zeros and are not launched. Bound by FP64 latency (chains of dependent additions on a
// pipe 64 times slower than FP32): with a second kernel whose finish ran on one lane, a loop of
// dependent loads and 304 blocks whatever the bodies, the app's frame of 4 444 took 147 us, now 126.
__global__ __launch_bounds__(kThreads) void k_bounds(const float4* __restrict__ pos, int n, double inv_n,
                                                     double edge_factor, BoundsPartial* __restrict__ partial,
                                                     unsigned* __restrict__ done, Geom* __restrict__ g) {
  double sx = 0, sy = 0, sz = 0;
  float mx = 0.f, my = 0.f, mz = 0.f;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
    float4 p = pos[i];
    sx = __dadd_rn(sx, (double)p.x);
    sy = __dadd_rn(sy, (double)p.y);
    sz = __dadd_rn(sz, (double)p.z);
    mx = fmaxf(mx, fabsf(p.x));
    my = fmaxf(my, fabsf(p.y));
    mz = fmaxf(mz, fabsf(p.z));
  }
  __shared__ double sh[3][kThreads / 32];
  __shared__ float shm[3][kThreads / 32];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sx = __dadd_rn(sx, __shfl_down_sync(0xffffffffu, sx, o));
    sy = __dadd_rn(sy, __shfl_down_sync(0xffffffffu, sy, o));
    sz = __dadd_rn(sz, __shfl_down_sync(0xffffffffu, sz, o));
    mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
    my = fmaxf(my, __shfl_down_sync(0xffffffffu, my, o));
    mz = fmaxf(mz, __shfl_down_sync(0xffffffffu, mz, o));
  }
  if (lane == 0) {
    sh[0][w] = sx;
    sh[1][w] = sy;
    sh[2][w] = sz;
    shm[0][w] = mx;
    shm[1][w] = my;
    shm[2][w] = mz;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double acc = sh[threadIdx.x][0];
    float m = shm[threadIdx.x][0];
#pragma unroll
    for (int i = 1; i < kThreads / 32; ++i) {
      acc = __dadd_rn(acc, sh[threadIdx.x][i]);
      m = fmaxf(m, shm[threadIdx.x][i]);
    }
    partial[blockIdx.x].sum[threadIdx.x] = acc;
    partial[blockIdx.x].mx[threadIdx.x] = m;
    __threadfence();
  }
  if (w != 0) return;
  __syncwarp();
  if (lane == 0) s_last = atomicInc(done, gridDim.x - 1) == gridDim.x - 1;  // wraps to 0 for the next launch
  __syncwarp();
  if (!s_last) return;
  __threadfence();
  double s[3] = {0, 0, 0};
  float m[3] = {0.f, 0.f, 0.f};
  double v[kBoundsPerLane][3];
  float vm[kBoundsPerLane][3];
#pragma unroll
  for (int k = 0; k < kBoundsPerLane; ++k) {  // all loads together, then the dependent sums
    const int b = lane + 32 * k;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      v[k][a] = b < (int)gridDim.x ? __ldcg(&partial[b].sum[a]) : 0.0;
      vm[k][a] = b < (int)gridDim.x ? __ldcg(&partial[b].mx[a]) : 0.f;
    }
  }
#pragma unroll
  for (int k = 0; k < kBoundsPerLane; ++k) {
    if (32 * k >= (int)gridDim.x) break;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      s[a] = __dadd_rn(s[a], v[k][a]);
      m[a] = fmaxf(m[a], vm[k][a]);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      s[a] = __dadd_rn(s[a], __shfl_down_sync(0xffffffffu, s[a], o));
      m[a] = fmaxf(m[a], __shfl_down_sync(0xffffffffu, m[a], o));
    }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    s[a] = __shfl_sync(0xffffffffu, s[a], 0);
    m[a] = __shfl_sync(0xffffffffu, m[a], 0);
  }
  finish_geom(s, m, n, inv_n, edge_factor, g);
}

__global__ void k_set_geom(Geom* __restrict__ g, double c0, double c1, double c2, double S, double t0, double t1,
                           double t2, double tedge) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  g->center[0] = c0;
  g->center[1] = c1;
  g->center[2] = c2;
  g->size = S;
  g->frac = __ddiv_rn(2097152.0, __dmul_rn(2.0, S));
  double tc[3] = {t0, t1, t2};
  fill_tree_geom(*g, tc, tedge);
}

// ---------------------------------------------------------------------------------------
// keys, gathers, leapfrog
// ---------------------------------------------------------------------------------------

// body_sys (optional): system of each body; each system then uses its own geometry
// sys_geom[body_sys[i]] (batched ensembles), otherwise the single geometry *g.
__global__ __launch_bounds__(kThreads) void k_morton(const float4* __restrict__ pos, int n,
                                                     const Geom* __restrict__ g, const uint16_t* __restrict__ body_sys,
                                                     uint64_t* __restrict__ keys, uint32_t* __restrict__ idx) {
  int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const Geom& gg = body_sys ? g[body_sys[i]] : *g;
  keys[i] = morton_key(pos[i], gg);
  idx[i] = (uint32_t)i;
}

// decodeMortonKey (src/MortonKeys.hpp:204-228): each axis's 21 bits de-interleaved, then
// x_int / 2^21 * 2 * S - S (the division and doubling are exact; one rounding each for the
// product and the difference, as in the reference's FP64 expression).
__global__ __launch_bounds__(kThreads) void k_decode_morton(const uint64_t* __restrict__ keys, int n, double S,
                                                            double* __restrict__ pos3) {
  const int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const uint64_t k = keys[i];
  uint32_t q[3] = {0u, 0u, 0u};
#pragma unroll
  for (int b = 0; b < kMaxDepth; ++b)
#pragma unroll
    for (int a = 0; a < 3; ++a) q[a] |= (uint32_t)((k >> (3 * b + 2 - a)) & 1ull) << b;
#pragma unroll
  for (int a = 0; a < 3; ++a) pos3[3 * i + a] = __dsub_rn(__dmul_rn((double)q[a] * 0x1p-20, S), S);
}

__global__ __launch_bounds__(kThreads) void k_treekey(const float4* __restrict__ pos, int n,
                                                      const Geom* __restrict__ g, uint64_t* __restrict__ tkeys,
                                                      uint32_t* __restrict__ tidx) {
  int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  tkeys[i] = tree_key(pos[i], *g);
  tidx[i] = (uint32_t)i;
}

__global__ __launch_bounds__(kThreads) void k_gather(const uint32_t* __restrict__ perm, int n,
                                                     const float4* __restrict__ pin, const float4* __restrict__ vin,
                                                     float4* __restrict__ pout, float4* __restrict__ vout) {
  int j = blockIdx.x * kThreads + threadIdx.x;
  if (j >= n) return;
  uint32_t i = perm[j];
  pout[j] = pin[i];
  vout[j] = vin[i];
}

// First half-kick and drift of one body (ComputePositionAtHalfTimeStep, src/Body.hpp:306-313).
__device__ __forceinline__ void kick_drift(float4& p, float4& v, float4 a, float dt, float half_dt) {
  v.x += a.x * half_dt;
  v.y += a.y * half_dt;
  v.z += a.z * half_dt;
  p.x += v.x * dt;
  p.y += v.y * dt;
  p.z += v.z * dt;
}

// Gather into the new (Morton) order fused with the first half-kick and the drift and with the tree
// key of the drifted position.
__global__ __launch_bounds__(kThreads) void k_gather_kd_treekey(
    const uint32_t* __restrict__ perm, int n, const float4* __restrict__ pin, const float4* __restrict__ vin,
    const float4* __restrict__ acc, int acc_follows_body, float dt, float half_dt, const Geom* __restrict__ g,
    const uint16_t* __restrict__ body_sys, float4* __restrict__ pout, float4* __restrict__ vout,
    uint64_t* __restrict__ tkeys, uint32_t* __restrict__ tidx) {
  int j = blockIdx.x * kThreads + threadIdx.x;
  if (j >= n) return;
  const uint32_t i = perm ? perm[j] : (uint32_t)j;  // no permutation: bodies keep their order
  float4 p = pin[i], v = vin[i];
  kick_drift(p, v, acc[acc_follows_body ? i : (uint32_t)j], dt, half_dt);
  pout[j] = p;
  vout[j] = v;
  // the sort keeps every system in its body range, so slot j's system is body_sys[j]
  tkeys[j] = tree_key(p, body_sys ? g[body_sys[j]] : *g);
  tidx[j] = (uint32_t)j;
}

// ---- systems small enough to sort by tiles (tile_sort_max): the stages around the sort in its kernels

// Morton keys, tile-sorted with their slots (kSeg: by the slots' systems first).
template <int kTile, bool kSeg>
__global__ __launch_bounds__(kTile) void k_morton_tiles(const float4* __restrict__ pos, int n,
                                                            const Geom* __restrict__ g,
                                                            const uint16_t* __restrict__ body_sys,
                                                            uint64_t* __restrict__ kout, uint32_t* __restrict__ vout) {
  const int base = blockIdx.x * kTile, i = base + threadIdx.x;
  const uint32_t sys = kSeg ? (i < n ? (uint32_t)body_sys[i] : 0xffffffffu) : 0u;
  const uint64_t key = i < n ? morton_key(pos[i], kSeg ? g[sys] : *g) : ~0ull;
  tile_sort_store<kTile, kSeg>(key, (uint32_t)i, sys, base, n, kout, vout);
}

// The Morton merge, with k_gather_kd_treekey's work at each body's place in the sorted order: kout
// (optional) receives the sorted keys, ktree the tree keys by slot.
template <int kTile, bool kSeg>
__global__ __launch_bounds__(32 * kMergeParts) void k_merge_kd(
    const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin, int n, const float4* __restrict__ pin,
    const float4* __restrict__ velin, const float4* __restrict__ acc, int acc_follows_body, float dt, float half_dt,
    const Geom* __restrict__ g, const uint16_t* __restrict__ body_sys, const uint32_t* __restrict__ off,
    float4* __restrict__ pout, float4* __restrict__ vout, uint64_t* __restrict__ kout, uint64_t* __restrict__ ktree) {
  int j;
  uint64_t key;
  uint32_t i;
  if (!merge_rank<kTile, kSeg>(kin, vin, body_sys, off, n, j, key, i)) return;
  float4 p = pin[i], v = velin[i];
  kick_drift(p, v, acc[acc_follows_body ? i : (uint32_t)j], dt, half_dt);
  pout[j] = p;
  vout[j] = v;
  if (kout) kout[j] = key;
  ktree[j] = tree_key(p, kSeg ? g[body_sys[j]] : *g);
}

// Tree keys (given, or of the positions), tile-sorted with their slots.
template <int kTile, bool kSeg>
__global__ __launch_bounds__(kTile) void k_tree_tiles(const uint64_t* __restrict__ ktree,
                                                          const float4* __restrict__ pos, int n,
                                                          const Geom* __restrict__ g,
                                                          const uint16_t* __restrict__ body_sys,
                                                          uint64_t* __restrict__ kout, uint32_t* __restrict__ vout) {
  const int base = blockIdx.x * kTile, i = base + threadIdx.x;
  const uint32_t sys = kSeg ? (i < n ? (uint32_t)body_sys[i] : 0xffffffffu) : 0u;
  const uint64_t key = i < n ? (ktree ? ktree[i] : tree_key(pos[i], *g)) : ~0ull;
  tile_sort_store<kTile, kSeg>(key, (uint32_t)i, sys, base, n, kout, vout);
}

// The half-kick and drift of bodies that keep their slots (the differentiable path), with the tree keys
// of the drifted positions tile-sorted. The bodies are taken in the previous tree order, in which
// the new keys are nearly sorted and the merge has little to search (65 536 bodies: 75 -> 34 us
// against slot order); bodies of one key keep that order.
template <int kTile, bool kSeg>
__global__ __launch_bounds__(kTile) void k_kd_tiles(const float4* __restrict__ pin,
                                                        const float4* __restrict__ velin,
                                                        const float4* __restrict__ acc,
                                                        const uint32_t* __restrict__ order, int n, float dt,
                                                        float half_dt, const Geom* __restrict__ g,
                                                        float4* __restrict__ pout, float4* __restrict__ velout,
                                                        uint64_t* __restrict__ kout, uint32_t* __restrict__ vout) {
  const int base = blockIdx.x * kTile, k = base + threadIdx.x;
  uint64_t key = ~0ull;
  uint32_t i = 0;
  if (k < n) {
    i = min(order[k], (uint32_t)n - 1u);
    float4 p = pin[i], v = velin[i];
    kick_drift(p, v, acc[i], dt, half_dt);
    pout[i] = p;
    velout[i] = v;
    key = tree_key(p, *g);
  }
  tile_sort_store<kTile, kSeg>(key, i, 0u, base, n, kout, vout);
}

// The tree-key merge, with the positions gathered into tree order.
template <int kTile, bool kSeg>
__global__ __launch_bounds__(32 * kMergeParts) void k_merge_tree(const uint64_t* __restrict__ kin,
                                                              const uint32_t* __restrict__ vin, int n,
                                                              const float4* __restrict__ pos,
                                                              const uint16_t* __restrict__ body_sys,
                                                              const uint32_t* __restrict__ off,
                                                              uint64_t* __restrict__ tkey,
                                                              uint32_t* __restrict__ tslot,
                                                              float4* __restrict__ tpos) {
  int r;
  uint64_t key;
  uint32_t slot;
  if (!merge_rank<kTile, kSeg>(kin, vin, body_sys, off, n, r, key, slot)) return;
  tkey[r] = key;
  tslot[r] = slot;
  tpos[r] = pos[slot];
}

__global__ __launch_bounds__(kThreads) void k_kick_drift(float4* __restrict__ pos, float4* __restrict__ vel,
                                                         const float4* __restrict__ acc, int n, float dt,
                                                         float half_dt, int drift) {
  int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  float4 v = vel[i], a = acc[i];
  v.x += a.x * half_dt;
  v.y += a.y * half_dt;
  v.z += a.z * half_dt;
  vel[i] = v;
  if (drift) {
    float4 p = pos[i];
    p.x += v.x * dt;
    p.y += v.y * dt;
    p.z += v.z * dt;
    pos[i] = p;
  }
}

__global__ __launch_bounds__(kThreads) void k_gather_tree(const uint32_t* __restrict__ tslot, int n,
                                                          const float4* __restrict__ pos,
                                                          float4* __restrict__ tpos) {
  int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  tpos[i] = pos[tslot[i]];
}

// ---------------------------------------------------------------------------------------
// node discovery
// ---------------------------------------------------------------------------------------
// The node set equals the reference's insertion result: the root, plus every prefix K of a
// body's depth-21 path whose parent holds more than leaf_cap bodies (for leaf capacity 1:
// count(parent) >= 2). Bodies are sorted by path, so every node is a contiguous body range.
// Two builds produce the same records: the all-depths build further down (leaf capacities up to
// 64), and this level build (larger ones).
// One launch per depth turns the internal nodes of depth d into the node records of depth
// d+1, appended in key order: children get contiguous indices, depths are stored level by
// level (breadth-first), and a decoupled look-back over 256-node tiles assigns the indices.

__global__ void k_tree_init(int n, uint64_t* __restrict__ nkey, int2* __restrict__ nrange,
                            int* __restrict__ level_bounds, uint32_t* __restrict__ level_tile_ctr) {
  int t = threadIdx.x;
  if (t < kLevels) level_tile_ctr[t] = 0;
  if (t <= kLevels + 1) level_bounds[t] = (t == 0) ? 0 : (t == 1 ? (n > 0 ? 1 : 0) : -1);
  if (t == 0 && n > 0) {
    nkey[0] = 1ull;
    nrange[0] = make_int2(0, n);
  }
}

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
constexpr uint32_t kLbAgg = 1u << 30, kLbPrefix = 2u << 30, kLbMask = (1u << 30) - 1;
constexpr int kLbSpin = 1 << 22;

// K independent binary searches in the sorted child digits of one node: search j finds, inside
// [bnd[2Hj], bnd[2H(j+1)]), the first index whose digit is >= 2Hj + H, and stores it there.
template <int K, int H>
__device__ __forceinline__ void split_search(const uint64_t* __restrict__ tkey, int shift, int (&bnd)[9]) {
  int a[K], b[K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    a[j] = bnd[2 * H * j];
    b[j] = bnd[2 * H * (j + 1)];
  }
  for (;;) {
    bool any = false;
#pragma unroll
    for (int j = 0; j < K; ++j) any |= a[j] < b[j];
    if (!any) break;
    int dig[K];
#pragma unroll
    for (int j = 0; j < K; ++j)  // loads first, so the K searches wait on the memory together
      dig[j] = a[j] < b[j] ? (int)((tkey[(a[j] + b[j]) >> 1] >> shift) & 7ull) : 0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if (a[j] >= b[j]) continue;
      const int m = (a[j] + b[j]) >> 1;
      if (dig[j] < 2 * H * j + H)
        a[j] = m + 1;
      else
        b[j] = m;
    }
  }
#pragma unroll
  for (int j = 0; j < K; ++j) bnd[2 * H * j + H] = a[j];
}

// Decoupled look-back over the tiles of one level (one thread): publishes the tile's child
// count, sums the predecessors' counts back to the first inclusive prefix (eight predecessor
// words per round trip, independent loads in flight together), publishes its own inclusive
// prefix and returns the exclusive one. Waits are bounded; on expiry the timeout bit is set.
__device__ uint32_t tile_lookback(uint32_t* __restrict__ lb, int tile, uint32_t btotal, uint32_t* __restrict__ err) {
  uint32_t* mine = lb + tile;
  st_relaxed(mine, (tile == 0 ? kLbPrefix : kLbAgg) | btotal);
  uint32_t excl = 0;
  if (tile == 0) return 0;
  constexpr int kWin = 8;
  int k = tile - 1, spins = 0;
  while (k >= 0) {
    uint32_t v[kWin];
#pragma unroll
    for (int q = 0; q < kWin; ++q)  // tile 0 always holds a prefix, so k - q < 0 is never consumed
      v[q] = (k - q >= 0) ? ld_relaxed(lb + (k - q)) : kLbPrefix;
    int used = 0;
    bool done = false;
#pragma unroll
    for (int q = 0; q < kWin; ++q) {
      if (done || used < q) continue;  // stop at a prefix or at the first unpublished tile
      const uint32_t f = v[q] & ~kLbMask;
      if (f == 0) continue;
      excl += v[q] & kLbMask;
      used = q + 1;
      done = f == kLbPrefix;
    }
    if (done) break;
    k -= used;
    if (used == 0) {
      if (++spins > kLbSpin) {
        atomicOr(err, kErrTimeout);
        break;
      }
      __nanosleep(32);
    }
  }
  st_relaxed(mine, kLbPrefix | ((excl + btotal) & kLbMask));
  return excl;
}

// The eight child ranges of one node by the whole warp: lanes 4(v-1) .. 4(v-1)+3 search for the
// first index of [lo, hi) whose child digit is >= v (v = 1..7) with four probes per round, so
// each round shrinks the interval about fivefold and the seven searches run together (about
// log5 of the range in dependent loads instead of seven binary searches). Invariant per
// search: every index below a has a smaller digit, and b is the answer or hi.
__device__ __forceinline__ void warp_child_bounds(const uint64_t* __restrict__ tkey, int shift, int lo, int hi,
                                                  int lane, int (&bnd)[9]) {
  const int g = lane >> 2, k = lane & 3, v = g + 1;
  const bool searcher = g < 7;
  int a = lo, b = hi;
  for (int it = 0; it < 40; ++it) {  // 40 rounds cover any 31-bit range
    const bool big = searcher && (b - a > 4);
    if (!__any_sync(0xffffffffu, big)) break;
    const int step = (b - a) / 5;
    bool ge = false;
    if (big) ge = (int)((tkey[a + (k + 1) * step] >> shift) & 7ull) >= v;
    const uint32_t grp = (__ballot_sync(0xffffffffu, ge) >> (4 * g)) & 0xFu;
    if (big) {
      if (grp) {
        const int f = __ffs(grp) - 1;
        b = a + (f + 1) * step;
        if (f > 0) a = a + f * step + 1;
      } else {
        a = a + 4 * step + 1;
      }
    }
  }
  const bool probe = searcher && (a + k < b);
  const bool ge = probe && (int)((tkey[a + k] >> shift) & 7ull) >= v;
  const uint32_t grp = (__ballot_sync(0xffffffffu, ge) >> (4 * g)) & 0xFu;
  const int ans = grp ? a + __ffs(grp) - 1 : b;
  bnd[0] = lo;
  bnd[8] = hi;
#pragma unroll
  for (int u = 1; u < 8; ++u) bnd[u] = __shfl_sync(0xffffffffu, ans, 4 * (u - 1));
}

__global__ __launch_bounds__(kThreads) void k_level(int d, const uint64_t* __restrict__ tkey, int leaf_cap,
                                                    uint64_t* __restrict__ nkey, int2* __restrict__ nrange,
                                                    WalkNode* __restrict__ wn, uint8_t* __restrict__ childbyte,
                                                    int* __restrict__ level_bounds,
                                                    uint32_t* __restrict__ tile_ctr, uint32_t* __restrict__ lb,
                                                    long long node_cap, uint32_t* __restrict__ err) {
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_warp[kThreads / 32];
  __shared__ uint32_t s_excl;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int lo = level_bounds[d], hi = level_bounds[d + 1];
  const int count = hi - lo;
  if (count <= 0) {
    if (blockIdx.x == 0 && t == 0) level_bounds[d + 2] = hi < 0 ? -1 : hi;
    return;
  }
  if (*((volatile uint32_t*)err) & kErrNodes) {
    if (blockIdx.x == 0 && t == 0) level_bounds[d + 2] = hi;
    return;
  }
  const int shift = 3 * (kMaxDepth - 1 - d);
  if (count <= kLevelWarpNodes) {
    // few nodes with long body ranges (the top levels): one warp per node, tiles of one node
    // per warp, the child ranges found by the warp-cooperative search
    constexpr int kW = kThreads / 32;
    const int ntiles_w = (count + kW - 1) / kW;
    for (;;) {
      if (t == 0) s_tile = atomicAdd(&tile_ctr[d], 1u);
      __syncthreads();
      const int tile = (int)s_tile;
      __syncthreads();
      if (tile >= ntiles_w) break;
      const int node = lo + tile * kW + w;
      const bool valid = node < hi;  // warp-uniform
      int2 r = make_int2(0, 0);
      bool internal = false;
      int bnd[9];
      int nc = 0;
      uint32_t mask = 0;
      if (valid) {
        r = nrange[node];
        internal = r.y > leaf_cap && d < kMaxDepth;
        if (internal) {
          warp_child_bounds(tkey, shift, r.x, r.x + r.y, lane, bnd);
          for (int v = 0; v < 8; ++v)
            if (bnd[v + 1] > bnd[v]) {
              ++nc;
              mask |= 1u << v;
            }
        }
      }
      if (lane == 0) s_warp[w] = (uint32_t)nc;
      __syncthreads();
      uint32_t wadd = 0, btotal = 0;
      for (int i = 0; i < kW; ++i) {
        if (i < w) wadd += s_warp[i];
        btotal += s_warp[i];
      }
      if (t == 0) {
        const uint32_t excl = tile_lookback(lb, tile, btotal, err);
        s_excl = excl;
        if (tile == ntiles_w - 1) level_bounds[d + 2] = hi + (int)(excl + btotal);
      }
      __syncthreads();
      const long long child_base = (long long)hi + s_excl + wadd;
      if (valid) {
        const bool fits = child_base + nc <= node_cap;
        if (!fits && lane == 0) atomicOr(err, kErrNodes);
        const bool make = internal && fits;
        if (make && lane < 8 && ((mask >> lane) & 1u)) {  // lane v writes child v
          const int ci = (int)child_base + __popc(mask & ((1u << lane) - 1u));
          nkey[ci] = (nkey[node] << 3) | (uint64_t)lane;
          nrange[ci] = make_int2(bnd[lane], bnd[lane + 1] - bnd[lane]);
        }
        if (lane == 0) {
          wn[node].link = make_int4(make ? (int)child_base : -1, make ? nc : 0, r.x, r.y);
          childbyte[node] = (uint8_t)(make ? mask : 0u);
        }
      }
      __syncthreads();
    }
    return;
  }
  const int ntiles = (count + kThreads - 1) / kThreads;
  for (;;) {
    if (t == 0) s_tile = atomicAdd(&tile_ctr[d], 1u);
    __syncthreads();
    const int tile = (int)s_tile;
    __syncthreads();
    if (tile >= ntiles) break;
    const int node = lo + tile * kThreads + t;
    const bool valid = node < hi;
    int2 r = make_int2(0, 0);
    int bnd[9];
    int nc = 0;
    uint32_t mask = 0;
    bool internal = false;
    if (valid) {
      r = nrange[node];
      internal = r.y > leaf_cap && d < kMaxDepth;
      if (internal) {
        // the first index with child digit >= v, for v = 4, then 2 and 6, then 1, 3, 5, 7: each
        // round searches inside the intervals the previous round split off, and its searches are
        // independent, so their loads overlap (three dependent search depths instead of seven)
        bnd[0] = r.x;
        bnd[8] = r.x + r.y;
        split_search<1, 4>(tkey, shift, bnd);
        split_search<2, 2>(tkey, shift, bnd);
        split_search<4, 1>(tkey, shift, bnd);
        for (int v = 0; v < 8; ++v)
          if (bnd[v + 1] > bnd[v]) {
            ++nc;
            mask |= 1u << v;
          }
      }
    }
    // block exclusive scan of child counts
    uint32_t x = (uint32_t)nc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    uint32_t wadd = 0, btotal = 0;
    for (int i = 0; i < kThreads / 32; ++i) {
      if (i < w) wadd += s_warp[i];
      btotal += s_warp[i];
    }
    const uint32_t my_excl = x - (uint32_t)nc + wadd;
    // tile look-back (thread 0)
    if (t == 0) {
      const uint32_t excl = tile_lookback(lb, tile, btotal, err);
      s_excl = excl;
      if (tile == ntiles - 1) level_bounds[d + 2] = hi + (int)(excl + btotal);
    }
    __syncthreads();
    const long long child_base = (long long)hi + s_excl + my_excl;
    if (valid) {
      bool fits = child_base + nc <= node_cap;
      if (!fits) atomicOr(err, kErrNodes);
      int first = -1;
      if (internal && fits) {
        first = (int)child_base;
        int k = 0;
        const uint64_t pk = nkey[node];
        for (int v = 0; v < 8; ++v) {
          if (!(mask & (1u << v))) continue;
          int ci = first + k++;
          nkey[ci] = (pk << 3) | (uint64_t)v;
          nrange[ci] = make_int2(bnd[v], bnd[v + 1] - bnd[v]);
        }
      }
      wn[node].link = make_int4(first, (internal && fits) ? nc : 0, r.x, r.y);
      childbyte[node] = (uint8_t)((internal && fits) ? mask : 0u);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------
// Parallel build: every depth at once
// ---------------------------------------------------------------------------------------
// The same node set, order and records as k_tree_init + k_level, without a chain of levels.
// With the tree keys sorted, a depth-e cell is a contiguous run of bodies, and:
//   * the depth-e cell of body i holds more than L bodies exactly when some run of L + 1
//     consecutive bodies containing i shares its first e digits; the keys being sorted, a run
//     [j, j + L] shares as many digits as its end keys do. So with w(j) = digits shared by keys j
//     and j + L, E(i) = max of w(j) over j in [i - L, i] is the deepest such depth;
//   * a node of depth d >= 1 is a non-empty cell whose parent cell holds more than L bodies
//     (the parent's parent then does too), so a depth-d node starts at body i exactly when keys
//     i - 1 and i differ in the first d digits and d <= E(i) + 1 (and d <= 21): every depth
//     from (digits shared with key i - 1) + 1 to min(E(i) + 1, 21).
// The build counts node starts per depth for each tile of bodies (k_nodes_count), scans the
// counts of each depth over the tiles (k_nodes_scan), writes every node from the thread of its
// first body (k_nodes_write: index = level start + starts of its depth before it; its cell's
// end by a galloping search; its first child is node (d + 1, i); its parent is the last
// depth-(d - 1) node starting at or before i), and lets each parent's last child set the
// parent's child count and child byte (k_nodes_link).
constexpr int kPBThreads = 512;
constexpr int kPBWarps = kPBThreads / 32;
constexpr int kPBMaxLeaf = 64;  // halo of the window maxima; larger leaf capacities use k_level

// Octal digits (from the top) that two tree keys share; 21 when they are equal (the marker bit
// 63 is set in both).
__device__ __forceinline__ int common_digits(uint64_t a, uint64_t b) {
  const uint64_t x = a ^ b;
  return x ? (__clzll((long long)x) - 1) / 3 : kMaxDepth;
}

// Per-warp counts of node starts for each depth 1..21 (ballots only over the depths the warp's
// bodies start nodes at; a warp of 32 neighbouring bodies spans a few depths of the 21).
__device__ __forceinline__ void warp_start_counts(int lo, int hi, uint32_t (*s_wc)[kPBWarps]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int wlo = __reduce_min_sync(0xffffffffu, lo), whi = __reduce_max_sync(0xffffffffu, hi);
  for (int d = 1 + lane; d <= kMaxDepth; d += 32)
    if (d < wlo || d > whi) s_wc[d - 1][w] = 0u;
  for (int d = wlo; d <= whi; ++d) {
    const unsigned b = __ballot_sync(0xffffffffu, lo <= d && d <= hi);
    if (lane == 0) s_wc[d - 1][w] = (uint32_t)__popc(b);
  }
}

// Start depths of the tile's bodies: lo | hi << 8 (none when lo > hi), and per-warp counts of
// starts for each depth 1..21 in s_wc. In an ensemble (kSeg) bodies of different systems share no
// digit, not even the root.
template <bool kSeg>
__device__ void node_start_depths(const uint64_t* __restrict__ tkey, const uint16_t* __restrict__ body_sys, int n,
                                  int leaf_cap, int t0, uint32_t (*s_wc)[kPBWarps], uint32_t* span_out) {
  __shared__ uint64_t s_k[kPBThreads + 2 * kPBMaxLeaf];
  __shared__ uint16_t s_sys[kSeg ? kPBThreads + 2 * kPBMaxLeaf : 1];
  __shared__ int8_t s_w[kPBThreads + kPBMaxLeaf];
  const int t = threadIdx.x, L = leaf_cap;
  const int base = t0 - L;  // s_k[x - base] is key x, for x in [t0 - L, t0 + T + L)
  for (int x = t; x < kPBThreads + 2 * L; x += kPBThreads) {
    const int g = base + x;
    const bool in = g >= 0 && g < n;
    s_k[x] = in ? tkey[g] : 0ull;
    if (kSeg) s_sys[x] = in ? body_sys[g] : 0;
  }
  __syncthreads();
  auto shared_digits = [&](int x, int y) {
    return kSeg && s_sys[x] != s_sys[y] ? -1 : common_digits(s_k[x], s_k[y]);
  };
  for (int x = t; x < kPBThreads + L; x += kPBThreads) {  // w(j) for j in [t0 - L, t0 + T)
    const int j = base + x;
    s_w[x] = (int8_t)((j >= 0 && j + L < n) ? shared_digits(x, x + L) : -1);
  }
  __syncthreads();
  const int i = t0 + t;
  int lo = 1, hi = 0;
  if (i < n) {
    const int lcp = i == 0 ? -1 : shared_digits(i - 1 - base, i - base);
    int e = -1;
    for (int q = 0; q <= L; ++q) e = max(e, (int)s_w[t + q]);  // j = i - L + q
    lo = max(lcp + 1, 1);
    hi = min(e + 1, kMaxDepth);
  }
  if (i < n) span_out[i] = (uint32_t)lo | ((uint32_t)hi << 8);
  warp_start_counts(lo, hi, s_wc);
  __syncthreads();
}

template <bool kSeg>
__global__ __launch_bounds__(kPBThreads) void k_nodes_count(const uint64_t* __restrict__ tkey,
                                                            const uint16_t* __restrict__ body_sys, int n, int leaf_cap,
                                                            uint32_t* __restrict__ span,
                                                            uint32_t* __restrict__ tile_cnt, int ntiles) {
  __shared__ uint32_t s_wc[kMaxDepth][kPBWarps];
  node_start_depths<kSeg>(tkey, body_sys, n, leaf_cap, blockIdx.x * kPBThreads, s_wc, span);
  if (threadIdx.x < kMaxDepth) {
    uint32_t c = 0;
    for (int q = 0; q < kPBWarps; ++q) c += s_wc[threadIdx.x][q];
    tile_cnt[(size_t)threadIdx.x * ntiles + blockIdx.x] = c;
  }
}

// Block d - 1 scans depth d's tile counts (exclusive, in place) and stores the depth's total.
__global__ __launch_bounds__(1024) void k_nodes_scan(uint32_t* __restrict__ tile_cnt, int ntiles,
                                                     uint32_t* __restrict__ totals) {
  __shared__ uint32_t s_warp[32];
  uint32_t* c = tile_cnt + (size_t)blockIdx.x * ntiles;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int per = (ntiles + 1023) / 1024, a = min(ntiles, t * per), b = min(ntiles, a + per);
  uint32_t sum = 0;
  for (int q = a; q < b; ++q) sum += c[q];
  uint32_t x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[w] = x;
  __syncthreads();
  if (w == 0) {
    const uint32_t v = s_warp[lane];
    uint32_t z = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, z, o);
      if (lane >= o) z += y;
    }
    s_warp[lane] = z - v;
    if (lane == 31) totals[blockIdx.x] = z;
  }
  __syncthreads();
  uint32_t run = x - sum + s_warp[w];
  for (int q = a; q < b; ++q) {
    const uint32_t v = c[q];
    c[q] = run;
    run += v;
  }
}

// Level starts (s_lb, from the depth totals) and, per depth and warp of this tile, the index of
// the warp's first node start (s_first); returns the node count.
__device__ long long node_first_indices(int roots, uint32_t lo, uint32_t hi, const uint32_t* __restrict__ tile_excl,
                                        int ntiles, const uint32_t* __restrict__ totals, long long* s_lb,
                                        uint32_t (*s_first)[kPBWarps]) {
  const int t = threadIdx.x;
  if (t == 0) {
    s_lb[0] = 0;
    s_lb[1] = roots;
    for (int d = 1; d <= kMaxDepth; ++d) s_lb[d + 1] = s_lb[d] + totals[d - 1];
  }
  warp_start_counts((int)lo, (int)hi, s_first);
  __syncthreads();
  if (t < kMaxDepth) {
    uint32_t run = (uint32_t)s_lb[t + 1] + tile_excl[(size_t)t * ntiles + blockIdx.x];
    for (int q = 0; q < kPBWarps; ++q) {
      const uint32_t v = s_first[t][q];
      s_first[t][q] = run;
      run += v;
    }
  }
  __syncthreads();
  return s_lb[kLevels];
}

// Node records from the thread of each node's first body: key, first body, parent, first
// child (node (d + 1, i); a node is internal exactly when d < the body's deepest start depth).
// The body counts, child counts and child bytes follow in k_nodes_link. The roots come first, one
// per system of an ensemble (kSeg), from the thread of the system's first body.
template <bool kSeg>
__global__ __launch_bounds__(kPBThreads) void k_nodes_write(const uint64_t* __restrict__ tkey,
                                                            const uint16_t* __restrict__ body_sys,
                                                            const uint32_t* __restrict__ off, int roots, int n,
                                                            const uint32_t* __restrict__ span,
                                                            const uint32_t* __restrict__ tile_excl, int ntiles,
                                                            const uint32_t* __restrict__ totals,
                                                            uint64_t* __restrict__ nkey, int2* __restrict__ nrange,
                                                            WalkNode* __restrict__ wn, uint8_t* __restrict__ childbyte,
                                                            int* __restrict__ nparent, int* __restrict__ level_bounds,
                                                            long long node_cap, uint32_t* __restrict__ err) {
  __shared__ long long s_lb[kLevels + 1];
  __shared__ uint32_t s_first[kMaxDepth][kPBWarps];
  const int t = threadIdx.x, lane = t & 31;
  const int i = blockIdx.x * kPBThreads + t;
  const uint32_t sp = i < n ? span[i] : 1u;
  const int lo = (int)(sp & 0xFFu), hi = (int)(sp >> 8);
  const long long m = node_first_indices(roots, (uint32_t)lo, (uint32_t)hi, tile_excl, ntiles, totals, s_lb, s_first);
  if (blockIdx.x == 0) {
    if (t <= kLevels + 1) level_bounds[t] = (int)min(s_lb[min(t, kLevels)], 0x7fffffffll);
    if (t == 0 && m > node_cap) atomicOr(err, kErrNodes);
  }
  if (m > node_cap) return;  // the host grows the arena and builds again
  const uint32_t lt = (1u << lane) - 1u;
  const uint64_t ki = i < n ? tkey[i] : 0ull;
  int child = -1;  // index of node (d + 1, i), when it exists
  // the warp's depths, and one above them for the parents of its shallowest nodes
  const int wlo = __reduce_min_sync(0xffffffffu, lo), whi = __reduce_max_sync(0xffffffffu, hi);
  for (int d = whi; d >= max(1, wlo - 1); --d) {
    const bool f = lo <= d && d <= hi;
    const unsigned b = __ballot_sync(0xffffffffu, f);
    const int idx = (int)s_first[d - 1][t >> 5] + __popc(b & lt);  // node (d, i) if f, else the next start
    if (child >= 0) nparent[child] = idx + (f ? 1 : 0) - 1;  // the last depth-d node starting at or before i
    if (f) {
      nkey[idx] = ki >> (3 * (kMaxDepth - d));
      nrange[idx] = make_int2(i, 0);
      wn[idx].link = make_int4(d < hi ? child : -1, 0, i, 0);
      childbyte[idx] = 0;
      child = idx;
    } else {
      child = -1;
    }
  }
  if (i >= n) return;
  const int root = kSeg ? body_sys[i] : 0, first = kSeg ? (int)off[root] : 0;
  if (child >= 0) nparent[child] = root;  // depth-1 nodes hang from the root
  if (i == first) {
    const int count = kSeg ? (int)off[root + 1] - first : n;
    nkey[root] = 1ull;
    nrange[root] = make_int2(first, count);
    wn[root].link = make_int4(child, 0, first, count);  // child: the first depth-1 node, or -1
    childbyte[root] = 0;
    nparent[root] = -1;
  }
}

// Body counts, child counts and child bytes, one thread per node. Siblings are contiguous and
// their cells adjacent, so a node's cell ends where its next sibling's starts, and a last
// child's where its parent's ends (the climb passes only through last children: about 1.3
// nodes on average). The last child of each parent (the next node has another parent) also
// counts its siblings from the parent's first child and ORs their digits.
__global__ __launch_bounds__(kThreads) void k_nodes_link(const int* __restrict__ level_bounds,
                                                         const uint64_t* __restrict__ nkey,
                                                         const int* __restrict__ nparent, int2* __restrict__ nrange,
                                                         WalkNode* __restrict__ wn, uint8_t* __restrict__ childbyte,
                                                         const uint32_t* __restrict__ err) {
  if (*err & kErrNodes) return;
  const int m = level_bounds[kLevels], roots = level_bounds[1];
  auto last_child = [&](int j) { return j + 1 >= m || nparent[j + 1] != nparent[j]; };
  for (int j = roots + blockIdx.x * kThreads + threadIdx.x; j < m; j += gridDim.x * kThreads) {
    const bool last = last_child(j);
    int a = j;
    bool up = last;
    while (up) {
      a = nparent[a];
      if (a < roots) break;
      up = last_child(a);
    }
    const int first = nrange[j].x;
    const int cnt = (up ? nrange[a].x + nrange[a].y : nrange[a + 1].x) - first;  // up: the climb reached a root
    nrange[j].y = cnt;
    wn[j].link.w = cnt;
    if (!last) continue;
    const int p = nparent[j];
    const int fc = wn[p].link.x;
    uint32_t mask = 0;
    for (int c = fc; c <= j; ++c) mask |= 1u << (uint32_t)(nkey[c] & 7ull);
    wn[p].link.y = j - fc + 1;
    childbyte[p] = (uint8_t)mask;
  }
}

// ---------------------------------------------------------------------------------------
// upsweep
// ---------------------------------------------------------------------------------------

// Parallel-axis quadrupole contribution of one child (or member body) of mass m at offset x
// from the node's centre of mass, the reference's formulas (src/HashedOctree.cpp:778-808).
__device__ __forceinline__ void quad_add(float q[6], float m, float x, float y, float z) {
  const float m3 = 3.f * m;
  q[1] = fmaf(m3 * x, y, q[1]);
  q[2] = fmaf(m3 * x, z, q[2]);
  q[4] = fmaf(m3 * y, z, q[4]);
  const float r2m = m * fmaf(x, x, fmaf(y, y, z * z));
  q[0] += fmaf(m3 * x, x, -r2m);
  q[3] += fmaf(m3 * y, y, -r2m);
  q[5] += fmaf(m3 * z, z, -r2m);
}

// Upsweep without a climb: every node's multipole straight from its bodies. A node is the range
// [first, first + count) of the tree order, so its mass and centre of mass are range sums and its
// quadrupole a second range sum about that centre; no node waits for another, where a bottom-up
// climb is one L2 round trip and one atomic per level and child. Bound by the dependent float-float
// sums of each node. Device time of the upsweep, climb -> this (chunk launches included): 4 444
// bodies (literal) 45 -> 12 us, 16 384 (leaf 1) 41 -> 20, 100 003 (leaf 1) 97 -> 41, 2^22 (leaf 16)
// 250 -> 204, the ensemble of 4.7e7 bodies 4.5 -> 2.35 ms. Chunk records (k_chunk_moments: the moments of every
// aligned 64 and 4096 bodies) keep a large node's range to at most 126 bodies, 126 chunks and its
// supers, which bounds the work at 2^22 bodies, where the visits of a body per level would not.
//   count <= 16     one thread in systems of more than 65 536 bodies (32 nodes per warp: the
//                   fewest instructions); below that a team, whose chain of sums is shorter
//   count <= 1024   a team of 8 lanes (64 without chunk records)
//   count <= 16384  a warp (256 without)
//   larger          the block
// The block collects the larger nodes of its tile and takes them after the small ones. Nodes are
// numbered level by level, so the largest come first: the head of the list is dealt node by node to
// all blocks, the rest in tiles of neighbouring nodes from a queue.
constexpr int kThreadNode = 16;  // largest node of a thread
constexpr int kTeam = 8;
constexpr int kTeamDirect = 64, kTeamNode = 1024;  // largest node of a team without / with chunks
constexpr int kWarpDirect = 256, kWarpNode = 16384;
constexpr int kChunk = 64;    // bodies per chunk record
constexpr int kSuper = 64;    // chunks per super record

// First moments of a range: mass and sum of mass * position, in float-float.
struct Moments {
  FF m, x, y, z;
  __device__ __forceinline__ void body(float4 p) {
    m = ff_add(m, {p.w, 0.f});
    x = ff_add(x, ff_prod(p.x, p.w));
    y = ff_add(y, ff_prod(p.y, p.w));
    z = ff_add(z, ff_prod(p.z, p.w));
  }
  __device__ __forceinline__ void record(const NodeUp& r) {
    const FF rm = {r.mass_hi, r.mass_lo};
    m = ff_add(m, rm);
    x = ff_add(x, ff_mul({r.com_hi[0], r.com_lo[0]}, rm));
    y = ff_add(y, ff_mul({r.com_hi[1], r.com_lo[1]}, rm));
    z = ff_add(z, ff_mul({r.com_hi[2], r.com_lo[2]}, rm));
  }
  // sums over lanes that differ in the bits below W; the order of the two operands does not
  // change an ff_add, so every lane ends with the same pair
  template <int W>
  __device__ __forceinline__ void reduce() {
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) {
      m = ff_add(m, {__shfl_xor_sync(0xffffffffu, m.hi, o), __shfl_xor_sync(0xffffffffu, m.lo, o)});
      x = ff_add(x, {__shfl_xor_sync(0xffffffffu, x.hi, o), __shfl_xor_sync(0xffffffffu, x.lo, o)});
      y = ff_add(y, {__shfl_xor_sync(0xffffffffu, y.hi, o), __shfl_xor_sync(0xffffffffu, y.lo, o)});
      z = ff_add(z, {__shfl_xor_sync(0xffffffffu, z.hi, o), __shfl_xor_sync(0xffffffffu, z.lo, o)});
    }
  }
  __device__ __forceinline__ void centre() {  // sums -> centre of mass
    if (m.hi == 0.f) return;
    x = ff_div(x, m);
    y = ff_div(y, m);
    z = ff_div(z, m);
  }
};

// Quadrupole of a range about a centre, FP32 partial sums.
struct Quad {
  float q[6];
  __device__ __forceinline__ void body(float4 p, const Moments& c) {
    quad_add(q, p.w, (p.x - c.x.hi) - c.x.lo, (p.y - c.y.hi) - c.y.lo, (p.z - c.z.hi) - c.z.lo);
  }
  __device__ __forceinline__ void record(const NodeUp& r, const Moments& c) {
    quad_add(q, r.mass_hi, (r.com_hi[0] - c.x.hi) + (r.com_lo[0] - c.x.lo),
             (r.com_hi[1] - c.y.hi) + (r.com_lo[1] - c.y.lo), (r.com_hi[2] - c.z.hi) + (r.com_lo[2] - c.z.lo));
#pragma unroll
    for (int k = 0; k < 6; ++k) q[k] += r.q[k];
  }
  template <int W>
  __device__ __forceinline__ void reduce() {
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < 6; ++k) q[k] += __shfl_xor_sync(0xffffffffu, q[k], o);
  }
};

// Literal barycentre: the member with the smallest Morton slot, as (slot << 32 | tree position).
template <int W>
__device__ __forceinline__ unsigned long long min_reduce(unsigned long long v) {
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ unsigned long long first_member(const uint32_t* __restrict__ tslot, int b) {
  return ((unsigned long long)tslot[b] << 32) | (unsigned)b;
}

// One node's records from its sums, 16 bytes for each `part` 0..6.
__device__ __forceinline__ void write_multipole(int node, int part, const Moments& c, const Quad& q, bool single,
                                                float s2, WalkNode* __restrict__ wn, NodeUp* __restrict__ nf) {
  float4 v;
  switch (part) {
    case 0: v = make_float4(c.x.hi, c.y.hi, c.z.hi, c.m.hi); break;
    case 1: v = make_float4(c.x.lo, c.y.lo, c.z.lo, c.m.lo); break;
    case 2: v = make_float4(q.q[0], q.q[1], q.q[2], q.q[3]); break;
    case 3: v = make_float4(q.q[4], q.q[5], 0.f, 0.f); break;
    case 4: v = make_float4(c.x.hi, c.y.hi, c.z.hi, single ? -s2 : s2); break;
    case 5: v = make_float4(c.m.hi, q.q[0], q.q[1], q.q[2]); break;
    default: v = make_float4(q.q[3], q.q[4], q.q[5], 0.f); break;
  }
  float4* dst = part < 4 ? reinterpret_cast<float4*>(nf + node) + part
                         : (part == 4 ? &wn[node].mac : (part == 5 ? &wn[node].mq : &wn[node].q2));
  *dst = v;
}

__device__ __noinline__ float node_edge2_exact(double root_edge, int d) {
  const double edge = ldexp(root_edge, -d);
  return __double2float_rn(__dmul_rn(edge, edge));
}

// Edge^2 of a node, the FP64 square rounded to float. Where the root's square and the node's are both
// normal floats, that is the rounded root's square times 4^-depth (exact); otherwise (the square of an edge
// above 2^64 is no float, although those of the nodes below may be) it is formed in FP64.
__device__ __forceinline__ float node_edge2(uint64_t key, int first, const Geom* __restrict__ g,
                                            const uint16_t* __restrict__ body_sys) {
  const int d = (63 - __clzll((long long)key)) / 3;
  const Geom& root = body_sys ? g[body_sys[first]] : *g;
  const float s2 = ldexpf(root.tedge2, -2 * d);
  return s2 >= FLT_MIN && s2 <= FLT_MAX ? s2 : node_edge2_exact(root.tedge, d);
}

// A node's range as bodies, chunks and supers: bodies [first, b0) and [b1, end), chunks [c0, d0)
// and [d1, c1), supers [s0, s1). Without chunks (or supers) their ranges are empty.
struct Split {
  int first, b0, b1, end, c0, d0, d1, c1, s0, s1;
  __device__ __forceinline__ Split(int2 r, const NodeUp* chunks, const NodeUp* supers) {
    first = r.x;
    end = r.x + r.y;
    b0 = b1 = end;
    c0 = d0 = d1 = c1 = s0 = s1 = 0;
    if (!chunks) return;
    const int lo = (first + kChunk - 1) / kChunk, hi = end / kChunk;
    if (lo >= hi) return;
    b0 = lo * kChunk;
    b1 = hi * kChunk;
    c0 = lo;
    d0 = d1 = c1 = hi;
    const int slo = (lo + kSuper - 1) / kSuper, shi = hi / kSuper;
    if (!supers || slo >= shi) return;
    d0 = slo * kSuper;
    d1 = shi * kSuper;
    s0 = slo;
    s1 = shi;
  }
  // body(p, b) for every body and record(r) for every record, thread l of W
  template <class Body, class Record>
  __device__ __forceinline__ void each(int l, int W, const float4* __restrict__ tpos,
                                       const NodeUp* __restrict__ chunks, const NodeUp* __restrict__ supers,
                                       Body body, Record record) const {
    const int nhead = b0 - first, nbody = nhead + (end - b1);
#pragma unroll 2
    for (int i = l; i < nbody; i += W) {
      const int b = i < nhead ? first + i : b1 + (i - nhead);
      body(tpos[b], b);
    }
    if (c0 >= c1) return;
    const int chead = d0 - c0, nchunk = chead + (c1 - d1);
#pragma unroll 2
    for (int i = l; i < nchunk; i += W) record(chunks[i < chead ? c0 + i : d1 + (i - chead)]);
#pragma unroll 2
    for (int i = s0 + l; i < s1; i += W) record(supers[i]);
  }
};

// Moments of every aligned kChunk bodies (a team each) or, with records, of every kSuper chunk
// records (a warp each): mass, centre of mass and quadrupole, or, in literal mode, the mass and the
// member with the smallest Morton slot.
template <bool kQuad, int W>
__global__ __launch_bounds__(kThreads) void k_chunk_moments(const float4* __restrict__ tpos,
                                                            const uint32_t* __restrict__ tslot,
                                                            const NodeUp* __restrict__ recs, int n, int per,
                                                            NodeUp* __restrict__ out) {
  const int l = threadIdx.x % W, chunk = blockIdx.x * (kThreads / W) + threadIdx.x / W;
  const long long b0 = (long long)chunk * per, b1 = min((long long)n, b0 + per);
  Moments c = {};
  Quad q = {};
  unsigned long long who = ~0ull;
  for (long long b = b0 + l; b < b1; b += W) {
    if (recs) {
      const NodeUp r = recs[b];
      if (kQuad)
        c.record(r);
      else {
        c.m = ff_add(c.m, {r.mass_hi, r.mass_lo});
        who = min(who, ((unsigned long long)r.min_slot << 32) | r.min_body);
      }
    } else {
      const float4 p = tpos[b];
      if (kQuad)
        c.body(p);
      else {
        c.m = ff_add(c.m, {p.w, 0.f});
        who = min(who, first_member(tslot, (int)b));
      }
    }
  }
  c.reduce<W>();
  if (kQuad) {
    c.centre();
    for (long long b = b0 + l; b < b1; b += W) {
      if (recs)
        q.record(recs[b], c);
      else
        q.body(tpos[b], c);
    }
    q.reduce<W>();
  } else {
    who = min_reduce<W>(who);
  }
  if (b0 >= n || l != 0) return;
  NodeUp r;
  r.com_hi[0] = c.x.hi;
  r.com_hi[1] = c.y.hi;
  r.com_hi[2] = c.z.hi;
  r.com_lo[0] = c.x.lo;
  r.com_lo[1] = c.y.lo;
  r.com_lo[2] = c.z.lo;
  r.mass_hi = c.m.hi;
  r.mass_lo = c.m.lo;
#pragma unroll
  for (int k = 0; k < 6; ++k) r.q[k] = q.q[k];
  r.min_slot = (uint32_t)(who >> 32);
  r.min_body = (uint32_t)who;
  out[chunk] = r;
}

// A node of one thread, team or warp (W lanes, lane l of it).
template <bool kQuad, int W>
__device__ __forceinline__ void node_direct(int node, int2 r, int l, const uint64_t* __restrict__ nkey,
                                            const float4* __restrict__ tpos, const uint32_t* __restrict__ tslot,
                                            const NodeUp* __restrict__ chunks, WalkNode* __restrict__ wn,
                                            NodeUp* __restrict__ nf, const Geom* __restrict__ g,
                                            const uint16_t* __restrict__ body_sys) {
  const int end = r.x + r.y;
  Moments c = {};
  Quad q = {};
  if (r.y == 1) {
    const float4 p = tpos[r.x];
    c.m = {p.w, 0.f};
    c.x = {p.x, 0.f};
    c.y = {p.y, 0.f};
    c.z = {p.z, 0.f};
  }
  const bool many = r.y > 1;
  if (__any_sync(0xffffffffu, many)) {
    Moments s = {};
    unsigned long long who = ~0ull;
    auto add = [&](float4 p, int b) {
      if (kQuad)
        s.body(p);
      else {
        s.m = ff_add(s.m, {p.w, 0.f});
        who = min(who, first_member(tslot, b));
      }
    };
    auto quad = [&](float4 p, int) { q.body(p, s); };
    // one thread: four bodies' loads together, then the dependent sums
    auto batches = [&](auto f) {
      for (int b0 = r.x; b0 < end; b0 += 4) {
        float4 p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = tpos[min(b0 + j, end - 1)];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (b0 + j < end) f(p[j], b0 + j);
      }
    };
    const Split sp(many ? r : make_int2(0, 0), W > 1 ? chunks : nullptr, nullptr);
    if (W == 1) {
      if (many) batches(add);
    } else {
      sp.each(l, W, tpos, chunks, nullptr, add, [&](const NodeUp& rec) {
        if (kQuad)
          s.record(rec);
        else {
          s.m = ff_add(s.m, {rec.mass_hi, rec.mass_lo});
          who = min(who, ((unsigned long long)rec.min_slot << 32) | rec.min_body);
        }
      });
    }
    s.reduce<W>();
    if (kQuad) {
      s.centre();
      if (W == 1) {
        if (many) batches(quad);
      } else {
        sp.each(l, W, tpos, chunks, nullptr, quad, [&](const NodeUp& rec) { q.record(rec, s); });
      }
      q.reduce<W>();
    } else {
      who = min_reduce<W>(who);
      if (many) {
        const float4 p = tpos[(uint32_t)who];
        s.x = {p.x, 0.f};
        s.y = {p.y, 0.f};
        s.z = {p.z, 0.f};
      }
    }
    if (many) c = s;
  }
  if (r.y <= 0) return;
  const float s2 = node_edge2(nkey[node], r.x, g, body_sys);
  if (W > 1) {
    if (l < 7) write_multipole(node, l, c, q, r.y == 1, s2, wn, nf);
  } else {
#pragma unroll
    for (int part = 0; part < 7; ++part) write_multipole(node, part, c, q, r.y == 1, s2, wn, nf);
  }
}

// The multipole of every node (computeTreeBaryCenters / computeNodeBaryCenters,
// src/HashedOctree.cpp:721-855, as intended; or the literal pseudo-barycentres).
// kFirst lanes (1 or kTeam) take each node of up to kFirstNode bodies in the first place.
template <bool kQuad, int kFirst>
__global__ __launch_bounds__(kThreads) void k_multipoles(const int* __restrict__ level_bounds,
                                                         const uint64_t* __restrict__ nkey,
                                                         const int2* __restrict__ nrange,
                                                         const float4* __restrict__ tpos,
                                                         const uint32_t* __restrict__ tslot,
                                                         const NodeUp* __restrict__ chunks,
                                                         const NodeUp* __restrict__ supers,
                                                         WalkNode* __restrict__ wn, NodeUp* __restrict__ nf,
                                                         const Geom* __restrict__ g,
                                                         const uint16_t* __restrict__ body_sys,
                                                         const uint32_t* __restrict__ err, Counters* __restrict__ ctr) {
  constexpr int kWarps = kThreads / 32, kTeams = kThreads / kTeam;
  constexpr int kNodes = kThreads / kFirst;  // nodes per block and pass
  __shared__ int s_team[kNodes], s_warp[kNodes], s_big[kNodes];
  __shared__ int s_count[3], s_next;
  __shared__ Moments s_mom[kWarps];
  __shared__ Quad s_quad[kWarps];
  __shared__ unsigned long long s_who[kWarps];
  if (*err & kErrNodes) return;
  const int m = level_bounds[kLevels];
  const int team_node = chunks ? kTeamNode : kTeamDirect, warp_node = chunks ? kWarpNode : kWarpDirect;
  const int first_node = kFirst == 1 ? kThreadNode : team_node;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (blockIdx.x == 0 && t == 0) {
    int d = 0;
    while (d < kMaxDepth && level_bounds[d + 2] > level_bounds[d + 1]) ++d;
    ctr->max_depth = d;
  }
  if (t < 3) s_count[t] = 0;
  __syncthreads();
  // the head: the first nodes of the tree, among them the largest, dealt one by one to the blocks
  // (a node per warp, or per team in small systems); then tiles of neighbouring nodes from a queue
  const int head = kFirst == 1 ? kWarps * (int)gridDim.x : kTeams * (int)gridDim.x;
  for (int tile = -1;;) {
    int node, l;
    if (tile < 0 && kFirst == 1) {
      l = lane;
      node = lane == 0 ? w * (int)gridDim.x + (int)blockIdx.x : m;
    } else {
      l = t % kFirst;
      node = tile < 0 ? (t / kFirst) * (int)gridDim.x + (int)blockIdx.x : head + tile * kNodes + t / kFirst;
    }
    int2 r = node < m ? nrange[node] : make_int2(0, 0);
    if (r.y > first_node) {
      if (l == 0) {
        const int kind = r.y > warp_node ? 2 : (r.y > team_node ? 1 : 0);
        (kind == 2 ? s_big : (kind == 1 ? s_warp : s_team))[atomicAdd(&s_count[kind], 1)] = node;
      }
      r.y = 0;
    }
    node_direct<kQuad, kFirst>(node, r, l, nkey, tpos, tslot, chunks, wn, nf, g, body_sys);
    if (t == 0) s_next = tile < 0 ? (int)blockIdx.x : (int)gridDim.x + (int)atomicAdd(&ctr->node_next, 1u);
    __syncthreads();
    tile = s_next;
    const int nteam = s_count[0], nwarp = s_count[1], nbig = s_count[2];
    if (kFirst == 1)
      for (int k = (w * 32) / kTeam; k < nteam; k += kTeams) {  // warp-uniform: a warp takes four nodes
        const int at = k + lane / kTeam;
        const int tn = at < nteam ? s_team[at] : 0;
        node_direct<kQuad, kTeam>(tn, at < nteam ? nrange[tn] : make_int2(0, 0), t % kTeam, nkey, tpos, tslot, chunks, wn,
                                  nf, g, body_sys);
      }
    for (int k = w; k < nwarp; k += kWarps)
      node_direct<kQuad, 32>(s_warp[k], nrange[s_warp[k]], lane, nkey, tpos, tslot, chunks, wn, nf, g, body_sys);
    for (int k = 0; k < nbig; ++k) {
      const int big = s_big[k];
      const int2 rb = nrange[big];
      const Split sp(rb, chunks, supers);
      Moments c = {};
      Quad q = {};
      unsigned long long who = ~0ull;
      sp.each(
          t, kThreads, tpos, chunks, supers,
          [&](float4 p, int b) {
            if (kQuad)
              c.body(p);
            else {
              c.m = ff_add(c.m, {p.w, 0.f});
              who = min(who, first_member(tslot, b));
            }
          },
          [&](const NodeUp& rec) {
            if (kQuad)
              c.record(rec);
            else {
              c.m = ff_add(c.m, {rec.mass_hi, rec.mass_lo});
              who = min(who, ((unsigned long long)rec.min_slot << 32) | rec.min_body);
            }
          });
      c.reduce<32>();
      if (!kQuad) who = min_reduce<32>(who);
      if (lane == 0) {
        s_mom[w] = c;
        s_who[w] = who;
      }
      __syncthreads();
      c = s_mom[lane % kWarps];
      c.reduce<kWarps>();
      if (kQuad) {
        c.centre();
        sp.each(
            t, kThreads, tpos, chunks, supers, [&](float4 p, int) { q.body(p, c); },
            [&](const NodeUp& rec) { q.record(rec, c); });
        q.reduce<32>();
        if (lane == 0) s_quad[w] = q;
        __syncthreads();
        q = s_quad[lane % kWarps];
        q.reduce<kWarps>();
      } else {
        who = min_reduce<kWarps>(s_who[lane % kWarps]);
        const float4 p = tpos[(uint32_t)who];
        c.x = {p.x, 0.f};
        c.y = {p.y, 0.f};
        c.z = {p.z, 0.f};
      }
      if (t < 7) write_multipole(big, t, c, q, false, node_edge2(nkey[big], rb.x, g, body_sys), wn, nf);
      __syncthreads();  // the sums' shared memory serves the next node
    }
    __syncthreads();
    if (t < 3) s_count[t] = 0;
    __syncthreads();
    if (head + (long long)tile * kNodes >= m) break;
  }
}

// ---------------------------------------------------------------------------------------
// node hash table (replaces the std::unordered_map of LinearHashedOctree,
// src/HashedOctree.hpp:134; lookups as in lookUpNode, src/HashedOctree.cpp:111-115)
// ---------------------------------------------------------------------------------------

__device__ __forceinline__ size_t hash_slot(uint64_t key, size_t mask) {
  return (size_t)((key * 0x9E3779B97F4A7C15ull) >> 17) & mask;
}

constexpr int kHashProbeLimit = 4096;

__global__ __launch_bounds__(kThreads) void k_hash_insert(const uint64_t* __restrict__ nkey,
                                                          const int* __restrict__ level_bounds,
                                                          unsigned long long* __restrict__ hk,
                                                          int* __restrict__ hv, size_t cap,
                                                          long long node_cap, uint32_t* __restrict__ err) {
  const int m = (int)min((long long)level_bounds[kLevels], node_cap);
  const size_t mask = cap - 1;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < m; i += gridDim.x * kThreads) {
    unsigned long long key = nkey[i];
    size_t h = hash_slot(key, mask);
    int probe = 0;
    for (;;) {
      unsigned long long prev = atomicCAS(&hk[h], 0ull, key);
      if (prev == 0ull || prev == key) {
        hv[h] = i;
        break;
      }
      if (++probe >= kHashProbeLimit) {
        atomicOr(err, kErrHash);
        break;
      }
      h = (h + 1) & mask;
    }
  }
}

__global__ void k_hash_lookup(const unsigned long long* __restrict__ hk, const int* __restrict__ hv, size_t cap,
                              uint64_t key, int* __restrict__ out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const size_t mask = cap - 1;
  size_t h = hash_slot(key, mask);
  int res = -1;
  for (int probe = 0; probe < kHashProbeLimit; ++probe) {
    unsigned long long k = hk[h];
    if (k == key) {
      res = hv[h];
      break;
    }
    if (k == 0ull) break;
    h = (h + 1) & mask;
  }
  *out = res;
}

// Register-only FMA loop for the measured FP32 roofline (8 independent chains per thread).
__global__ __launch_bounds__(kThreads) void k_fp32_peak(float* sink, int iters) {
  float a0 = threadIdx.x * 1e-7f, a1 = a0 + 1e-7f, a2 = a0 + 2e-7f, a3 = a0 + 3e-7f;
  float a4 = a0 + 4e-7f, a5 = a0 + 5e-7f, a6 = a0 + 6e-7f, a7 = a0 + 7e-7f;
  const float b = 0.999999f, c = 1e-7f;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      a0 = fmaf(a0, b, c);
      a1 = fmaf(a1, b, c);
      a2 = fmaf(a2, b, c);
      a3 = fmaf(a3, b, c);
      a4 = fmaf(a4, b, c);
      a5 = fmaf(a5, b, c);
      a6 = fmaf(a6, b, c);
      a7 = fmaf(a7, b, c);
    }
  }
  float r = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (r == 12345.678f) sink[0] = r;  // keeps the loop alive; never true for these inputs
}

// ---------------------------------------------------------------------------------------
// batched ensembles: system s owns the fixed body range [off[s], off[s + 1])
// ---------------------------------------------------------------------------------------

// OctantBounds of every system, one block per system: FP64 sums in a fixed order (thread
// stride, then a fixed tree), FP32 maxima of |p|, then the same finish as k_bounds.
__global__ __launch_bounds__(kThreads) void k_batch_bounds(const float4* __restrict__ pos,
                                                           const uint32_t* __restrict__ off, double edge_factor,
                                                           Geom* __restrict__ sys_geom) {
  const int s = blockIdx.x;
  const int b0 = (int)off[s], b1 = (int)off[s + 1];
  double sx = 0, sy = 0, sz = 0;
  float mx = 0.f, my = 0.f, mz = 0.f;
  for (int i = b0 + threadIdx.x; i < b1; i += kThreads) {
    const float4 p = pos[i];
    sx = __dadd_rn(sx, (double)p.x);
    sy = __dadd_rn(sy, (double)p.y);
    sz = __dadd_rn(sz, (double)p.z);
    mx = fmaxf(mx, fabsf(p.x));
    my = fmaxf(my, fabsf(p.y));
    mz = fmaxf(mz, fabsf(p.z));
  }
  __shared__ double sh[3][kThreads / 32];
  __shared__ float shm[3][kThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sx = __dadd_rn(sx, __shfl_down_sync(0xffffffffu, sx, o));
    sy = __dadd_rn(sy, __shfl_down_sync(0xffffffffu, sy, o));
    sz = __dadd_rn(sz, __shfl_down_sync(0xffffffffu, sz, o));
    mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
    my = fmaxf(my, __shfl_down_sync(0xffffffffu, my, o));
    mz = fmaxf(mz, __shfl_down_sync(0xffffffffu, mz, o));
  }
  if (lane == 0) {
    sh[0][w] = sx;
    sh[1][w] = sy;
    sh[2][w] = sz;
    shm[0][w] = mx;
    shm[1][w] = my;
    shm[2][w] = mz;
  }
  __syncthreads();
  if (w != 0) return;
  double s3[3];
  float m3[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    s3[a] = sh[a][0];
    m3[a] = shm[a][0];
#pragma unroll
    for (int k = 1; k < kThreads / 32; ++k) {
      s3[a] = __dadd_rn(s3[a], sh[a][k]);
      m3[a] = fmaxf(m3[a], shm[a][k]);
    }
  }
  finish_geom(s3, m3, b1 - b0, __ddiv_rn(1.0, (double)(b1 - b0)), edge_factor, sys_geom + s);
}

// Secondary sort key: the system of the body each sorted element came from. A stable sort of
// the key-sorted elements by it groups them back into their systems, in key order.
__global__ __launch_bounds__(kThreads) void k_sys_keys(const uint32_t* __restrict__ vals, int n,
                                                       const uint16_t* __restrict__ body_sys,
                                                       uint64_t* __restrict__ k2) {
  const int j = blockIdx.x * kThreads + threadIdx.x;
  if (j < n) k2[j] = (uint64_t)body_sys[vals[j]];
}

// Tree-order positions and tree keys of a batched ensemble: the (system, key) sort leaves the
// permutation in tslot, the keys themselves are gathered from their per-slot copy.
__global__ __launch_bounds__(kThreads) void k_gather_tree_keys(const uint32_t* __restrict__ tslot, int n,
                                                               const float4* __restrict__ pos,
                                                               const uint64_t* __restrict__ key_by_slot,
                                                               float4* __restrict__ tpos,
                                                               uint64_t* __restrict__ tkey) {
  const int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = tslot[i];
  tpos[i] = pos[s];
  tkey[i] = key_by_slot[s];
}

// One root per system at depth 0, in system order.
__global__ void k_tree_init_batch(int nsys, const uint32_t* __restrict__ off, uint64_t* __restrict__ nkey,
                                  int2* __restrict__ nrange, int* __restrict__ level_bounds,
                                  uint32_t* __restrict__ level_tile_ctr) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nsys) {
    nkey[t] = 1ull;
    nrange[t] = make_int2((int)off[t], (int)(off[t + 1] - off[t]));
  }
  if (t < kLevels) level_tile_ctr[t] = 0;
  if (t <= kLevels + 1) level_bounds[t] = (t == 0) ? 0 : (t == 1 ? nsys : -1);
}

inline int grid_for(long long n) { return (int)((n + kThreads - 1) / kThreads); }

}  // namespace

// ---------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------

int bounds_blocks(int sms) { return std::min(2 * sms, 32 * kBoundsPerLane); }
size_t bounds_bytes(int blocks) { return sizeof(BoundsPartial) * (size_t)blocks; }

void launch_bounds(bh_ctx* c, const float4* pos, int n, double edge_factor) {
  c->launches += 1;
  const int blocks = std::max(1, std::min(c->bounds_blocks, grid_for(n)));
  k_bounds<<<blocks, kThreads, 0, c->stream>>>(pos, n, n > 0 ? 1.0 / (double)n : 0.0, edge_factor,
                                               static_cast<BoundsPartial*>(c->bounds_partial),
                                               &c->counters->bounds_done, c->geom);
}

void launch_set_geom(bh_ctx* c, const double center[3], double size, const double tcenter[3], double tedge) {
  c->launches += 1;
  k_set_geom<<<1, 32, 0, c->stream>>>(c->geom, center[0], center[1], center[2], size, tcenter[0], tcenter[1],
                                      tcenter[2], tedge);
}

void launch_morton(bh_ctx* c, const float4* pos, int n, uint64_t* keys, uint32_t* idx, bool batch) {
  if (n > 0) c->launches += 1;
  if (n > 0)
    k_morton<<<grid_for(n), kThreads, 0, c->stream>>>(pos, n, batch ? c->sys_geom : c->geom,
                                                       batch ? c->body_sys : nullptr, keys, idx);
}

void launch_decode_morton(bh_ctx* c, const uint64_t* keys, int n, double size, double* pos3) {
  if (n <= 0) return;
  c->launches += 1;
  k_decode_morton<<<grid_for(n), kThreads, 0, c->stream>>>(keys, n, size, pos3);
}

void launch_treekey(bh_ctx* c, const float4* pos, int n, uint64_t* tkeys, uint32_t* tidx) {
  if (n > 0) c->launches += 1;
  if (n > 0) k_treekey<<<grid_for(n), kThreads, 0, c->stream>>>(pos, n, c->geom, tkeys, tidx);
}

void launch_gather(bh_ctx* c, const uint32_t* perm, int n, const float4* pin, const float4* vin, float4* pout,
                   float4* vout) {
  if (n > 0) c->launches += 1;
  if (n > 0) k_gather<<<grid_for(n), kThreads, 0, c->stream>>>(perm, n, pin, vin, pout, vout);
}

void launch_gather_kd_treekey(bh_ctx* c, const uint32_t* perm, int n, const float4* pin, const float4* vin,
                              const float4* acc, int acc_follows_body, float dt, float4* pout, float4* vout,
                              uint64_t* tkeys, uint32_t* tidx, bool batch) {
  if (n > 0) c->launches += 1;
  if (n > 0)
    k_gather_kd_treekey<<<grid_for(n), kThreads, 0, c->stream>>>(
        perm, n, pin, vin, acc, acc_follows_body, dt, 0.5f * dt, batch ? c->sys_geom : c->geom,
        batch ? c->body_sys : nullptr, pout, vout, tkeys, tidx);
}

// The stages of a step up to the tree order, for systems that sort by tiles. The tile-sorted pairs pass
// through keys[1] / vals[1]; merged spans, where the sort has them, through arrays that are free until
// the tree order (tkey / tslot) and the build (nkey, vals[0]).
void launch_morton_tiles(bh_ctx* c, const float4* pos, int n, bool batch) {
  c->launches += 1;
  const TileShape sh = step_shape(n, batch);
  (batch ? BH_TILE_KERNEL_SEG(k_morton_tiles, sh)
         : BH_TILE_KERNEL(k_morton_tiles, sh))<<<sh.tile_blocks(), sh.tile, 0, c->stream>>>(
      pos, n, batch ? c->sys_geom : c->geom, c->body_sys, c->keys[1], c->vals[1]);
  if (sh.span) launch_merge_spans(c, n, c->tkey, c->tslot);
}

void launch_merge_kd(bh_ctx* c, int n, const float4* pin, const float4* vin, const float4* acc, int acc_follows_body,
                     float dt, float4* pout, float4* vout, uint64_t* kout, uint64_t* ktree, bool batch) {
  c->launches += 1;
  const TileShape sh = step_shape(n, batch);
  (batch ? BH_TILE_KERNEL_SEG(k_merge_kd, sh)
         : BH_MERGE_KERNEL(k_merge_kd, sh))<<<sh.merge_blocks(), sh.merge_threads(), 0, c->stream>>>(
      sh.span ? c->tkey : c->keys[1], sh.span ? c->tslot : c->vals[1], n, pin, vin, acc, acc_follows_body, dt,
      0.5f * dt, batch ? c->sys_geom : c->geom,
      c->body_sys, c->sys_off, pout, vout, kout, ktree);
}

void launch_kd_tiles(bh_ctx* c, int n, const float4* pin, const float4* vin, const float4* acc, float dt, float4* pout,
                     float4* vout) {
  c->launches += 1;
  const TileShape sh = step_shape(n);
  BH_TILE_KERNEL(k_kd_tiles, sh)<<<sh.tile_blocks(), sh.tile, 0, c->stream>>>(
      pin, vin, acc, c->tslot, n, dt, 0.5f * dt, c->geom, pout, vout, c->keys[1], c->vals[1]);
  if (sh.span) launch_merge_spans(c, n, c->nkey, c->vals[0]);
}

void launch_tree_tiles(bh_ctx* c, const uint64_t* ktree, const float4* pos, int n, bool batch) {
  c->launches += 1;
  const TileShape sh = step_shape(n, batch);
  (batch ? BH_TILE_KERNEL_SEG(k_tree_tiles, sh)
         : BH_TILE_KERNEL(k_tree_tiles, sh))<<<sh.tile_blocks(), sh.tile, 0, c->stream>>>(
      ktree, pos, n, c->geom, c->body_sys, c->keys[1], c->vals[1]);
  if (sh.span) launch_merge_spans(c, n, c->nkey, c->vals[0]);
}

void launch_merge_tree(bh_ctx* c, const float4* pos, int n, bool batch) {
  c->launches += 1;
  const TileShape sh = step_shape(n, batch);
  (batch ? BH_TILE_KERNEL_SEG(k_merge_tree, sh)
         : BH_MERGE_KERNEL(k_merge_tree, sh))<<<sh.merge_blocks(), sh.merge_threads(), 0, c->stream>>>(
      sh.span ? c->nkey : c->keys[1], sh.span ? c->vals[0] : c->vals[1], n, pos, c->body_sys, c->sys_off, c->tkey, c->tslot, c->tpos);
}

void launch_kick_drift(bh_ctx* c, float4* pos, float4* vel, const float4* acc, int n, float dt, int drift) {
  if (n > 0) c->launches += 1;
  if (n > 0) k_kick_drift<<<grid_for(n), kThreads, 0, c->stream>>>(pos, vel, acc, n, dt, 0.5f * dt, drift);
}

void launch_gather_tree(bh_ctx* c, const uint32_t* tslot, int n, const float4* pos, float4* tpos) {
  if (n > 0) c->launches += 1;
  if (n > 0) k_gather_tree<<<grid_for(n), kThreads, 0, c->stream>>>(tslot, n, pos, tpos);
}

// Function attributes set once per process, before any stream capture (none at present).
void tree_init() {}

void launch_build(bh_ctx* c, int n, int leaf_cap, bool batch) {
  if (n >= 1 && leaf_cap <= kPBMaxLeaf) {
    // every depth at once: counts per tile and depth (in lb_level), their scans (totals in
    // level_tile_ctr), the node records (start depths of each body in vals[1], free after the
    // sorts), then child counts and bytes
    const int ntiles = (n + kPBThreads - 1) / kPBThreads;
    uint32_t* span = c->vals[1];
    uint32_t* tile = c->lb_level;
    uint32_t* totals = c->level_tile_ctr;
    c->launches += 4;
    (batch ? k_nodes_count<true> : k_nodes_count<false>)<<<ntiles, kPBThreads, 0, c->stream>>>(
        c->tkey, c->body_sys, n, leaf_cap, span, tile, ntiles);
    k_nodes_scan<<<kMaxDepth, 1024, 0, c->stream>>>(tile, ntiles, totals);
    (batch ? k_nodes_write<true> : k_nodes_write<false>)<<<ntiles, kPBThreads, 0, c->stream>>>(
        c->tkey, c->body_sys, c->sys_off, batch ? c->nsys : 1, n, span, tile, ntiles, totals, c->nkey, c->nrange,
        c->wnode, c->nchildbyte, c->nparent, c->level_bounds, (long long)c->node_cap, c->err);
    const int lgrid = (int)std::min<size_t>((size_t)c->sms * 8, (c->node_cap + kThreads - 1) / kThreads);
    k_nodes_link<<<lgrid, kThreads, 0, c->stream>>>(c->level_bounds, c->nkey, c->nparent, c->nrange, c->wnode,
                                                    c->nchildbyte, c->err);
    return;
  }
  c->launches += 1 + kLevels;
  if (batch)
    k_tree_init_batch<<<(max(c->nsys, kLevels + 2) + 255) / 256, 256, 0, c->stream>>>(
        c->nsys, c->sys_off, c->nkey, c->nrange, c->level_bounds, c->level_tile_ctr);
  else
    k_tree_init<<<1, 64, 0, c->stream>>>(n, c->nkey, c->nrange, c->level_bounds, c->level_tile_ctr);
  const int max_tiles = c->lb_level_tiles;
  cudaMemsetAsync(c->lb_level, 0, sizeof(uint32_t) * (size_t)kLevels * max_tiles, c->stream);
  const int grid = c->sms * 4;
  for (int d = 0; d < kLevels; ++d)
    k_level<<<grid, kThreads, 0, c->stream>>>(d, c->tkey, leaf_cap, c->nkey, c->nrange, c->wnode, c->nchildbyte,
                                              c->level_bounds, c->level_tile_ctr,
                                              c->lb_level + (size_t)d * max_tiles, (long long)c->node_cap, c->err);
}

// Systems above this many bodies sum their larger nodes from chunk records (one more launch, about
// 6 us: as much as the root's 32 rounds of a block without them),
constexpr int kChunkMinBodies = 8192;
// and above this many from super records (another one).
constexpr int kSuperMinBodies = 262144;
// Above this many bodies a thread takes each small node, below it a team of kTeam lanes (100 003
// bodies at leaf capacity 1: 44 us by teams, 35 by threads; 2^22: 415 by teams).
constexpr int kThreadMinBodies = 65536;

void launch_upsweep(bh_ctx* c, int n, int mode, bool batch) {
  if (n <= 0) return;
  const bool quad = mode == BH_MULTIPOLE_QUADRUPOLE;
  // the records (about one byte per body) in the sorts' key scratch, free until the next sort
  NodeUp* chunks = n > kChunkMinBodies ? reinterpret_cast<NodeUp*>(c->keys[1]) : nullptr;
  NodeUp* supers = nullptr;
  if (chunks) {
    const int nchunks = (n + kChunk - 1) / kChunk, teams = kThreads / kTeam;
    c->launches += 1;
    (quad ? k_chunk_moments<true, kTeam> : k_chunk_moments<false, kTeam>)<<<(nchunks + teams - 1) / teams, kThreads, 0,
                                                                            c->stream>>>(c->tpos, c->tslot, nullptr, n,
                                                                                         kChunk, chunks);
    if (n > kSuperMinBodies) {
      const int nsupers = (nchunks + kSuper - 1) / kSuper, warps = kThreads / 32;
      supers = chunks + nchunks;
      c->launches += 1;
      (quad ? k_chunk_moments<true, 32> : k_chunk_moments<false, 32>)<<<(nsupers + warps - 1) / warps, kThreads, 0,
                                                                        c->stream>>>(c->tpos, c->tslot, chunks, nchunks,
                                                                                     kSuper, supers);
    }
  }
  c->launches += 1;
  // up to two nodes per body
  const bool threads = n > kThreadMinBodies;
  const int per_pass = kThreads / (threads ? 1 : kTeam);
  const int grid = (int)std::min<long long>((long long)c->sms * 8, (2ll * n + per_pass - 1) / per_pass);
  auto kernel = quad ? (threads ? k_multipoles<true, 1> : k_multipoles<true, kTeam>)
                     : (threads ? k_multipoles<false, 1> : k_multipoles<false, kTeam>);
  kernel<<<grid, kThreads, 0, c->stream>>>(
      c->level_bounds, c->nkey, c->nrange, c->tpos, c->tslot, chunks, supers, c->wnode, c->nup,
      batch ? c->sys_geom : c->geom, batch ? c->body_sys : nullptr, c->err, c->counters);
}

void launch_batch_bounds(bh_ctx* c, const float4* pos, double edge_factor) {
  c->launches += 1;
  k_batch_bounds<<<c->nsys, kThreads, 0, c->stream>>>(pos, c->sys_off, edge_factor, c->sys_geom);
}

void launch_gather_tree_keys(bh_ctx* c, const uint32_t* tslot, int n, const float4* pos,
                             const uint64_t* key_by_slot, float4* tpos, uint64_t* tkey) {
  if (n <= 0) return;
  c->launches += 1;
  k_gather_tree_keys<<<grid_for(n), kThreads, 0, c->stream>>>(tslot, n, pos, key_by_slot, tpos, tkey);
}

void launch_sys_keys(bh_ctx* c, const uint32_t* vals, int n, uint64_t* k2) {
  if (n <= 0) return;
  c->launches += 1;
  k_sys_keys<<<grid_for(n), kThreads, 0, c->stream>>>(vals, n, c->body_sys, k2);
}

void launch_hash(bh_ctx* c) {
  cudaMemsetAsync(c->hash_keys, 0, sizeof(uint64_t) * c->hash_cap, c->stream);
  c->launches += 1;
  k_hash_insert<<<c->sms * 8, kThreads, 0, c->stream>>>(c->nkey, c->level_bounds, (unsigned long long*)c->hash_keys,
                                                     c->hash_vals, c->hash_cap, (long long)c->node_cap, c->err);
}

void launch_lookup(bh_ctx* c, uint64_t key, int* out_index) {
  c->launches += 1;
  k_hash_lookup<<<1, 32, 0, c->stream>>>((const unsigned long long*)c->hash_keys, c->hash_vals, c->hash_cap, key,
                                         out_index);
}

void launch_fp32_peak(cudaStream_t st, float* sink, int blocks) {
  k_fp32_peak<<<blocks, kThreads, 0, st>>>(sink, 4096);
}

}  // namespace bh
