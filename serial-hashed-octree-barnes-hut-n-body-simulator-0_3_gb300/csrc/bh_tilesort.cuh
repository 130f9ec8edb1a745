// Stable sort of up to tile_sort_max() (u64 key, u32 value) pairs in two launches, or three, as building
// blocks that the stage kernels fuse with what makes the keys and with what consumes the sorted order.
//
//   tile:  a block sorts 128, 256 or 512 pairs. Each warp ranks its 32 keys by comparing them all (a
//          broadcast read per comparison), which gives 4 or 16 sorted runs in shared memory; a
//          key's place in the tile is its place in its run plus, by binary search, its place in
//          the other runs.
//   spans: (larger sorts) the same as the merge within every 32 tiles, a warp for 32 keys.
//   merge: a key's final place is its place in its tile or span plus, by binary search, its place in
//          every other one. A block takes 32 keys and its warps share the tiles.
//
// Equal keys count when they stand in an earlier run or tile, so the sort is stable. The radix sort's
// eight digit passes are a chain of 10 dependent launches, this is two or three; its work grows with
// n^2 over the tile or span, which sets the limits.
//
// Segments (ensembles): every system keeps its slot range, and pairs are ordered by (system, key).
// Slots are grouped by system, so system s fills the same places of a tile before and after the
// tile sort, and its keys need only be searched inside their system's part of each tile.
#pragma once
#include "bh_internal.cuh"

namespace bh {

// Keys per tile: small tiles are sorted sooner, large ones leave the merge fewer tiles.
constexpr int kTileSmall = 128, kTileLarge = 512;
// Keys of a sort with small tiles, at most. Keys to tree order of a step with tiles of 512 / 128 (us):
// 1 000 bodies 36 / 27, 4 444 38 / 31, 16 384 47 / 46, 32 768 61 / 63, 65 536 86 / 137.
constexpr int kTileSmallMax = 16384;
constexpr int kMergeParts = 8;  // warps of a merge block, at most
// Larger sorts take a middle launch that merges spans of 32 tiles (a warp for every 32 keys), and the
// final merge takes the spans: a key is searched in 32 + n / span runs instead of n / tile.
constexpr int kTileSpan = 256;
constexpr int kSpanThreads = 128;
// A step's sorts up to here stay at two launches. Whole steps with two / three launches (us, theta 1.2,
// leaf capacity 8): 32 768 bodies 183 / 195, 49 152 218 / 225, 65 536 242 / 242, 80 000 289 / 272, 98 304
// 326 / 293, 163 840 495 / 380.
constexpr int kTwoLaunchMax = 65536;
// Pairs in random order gain sooner, as fewer tiles agree. Two launches / tiles of 128 / tiles of 256 (us):
// 24 000 35 / 41 / 45, 40 001 57 / 47 / 53, 65 536 89 / 53 / 51, 98 304 156 / 70 / 64.
constexpr int kTwoLaunchPairsMax = 32768;
constexpr int kSpanSmallMax = 65536;

// Sorted order of (system, key); without segments the systems are all 0 and the compiler drops them.
template <bool kSeg>
__device__ __forceinline__ bool tile_less(uint32_t sa, uint64_t a, uint32_t sb, uint64_t b, bool or_equal) {
  const bool key = or_equal ? a <= b : a < b;
  return kSeg ? (sa < sb || (sa == sb && key)) : key;
}

// Sorts the block's kTileKeys pairs (thread t holds pair t of the tile; pairs at or beyond n hold key
// ~0 and the largest system, so they stay last) and stores those below n. All threads call it.
template <int kTileKeys, bool kSeg>
__device__ __forceinline__ void tile_sort_store(uint64_t key, uint32_t val, uint32_t sys, int base, int n,
                                                uint64_t* __restrict__ kout, uint32_t* __restrict__ vout) {
  constexpr int kTileRuns = kTileKeys / 32;
  __shared__ uint64_t s_in[kTileKeys], s_run[kTileKeys];
  __shared__ uint32_t s_sin[kSeg ? kTileKeys : 1], s_srun[kSeg ? kTileKeys : 1];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  s_in[t] = key;
  if (kSeg) s_sin[t] = sys;
  __syncwarp();
  int r = 0;
#pragma unroll 8
  for (int j = 0; j < 32; ++j)
    r += tile_less<kSeg>(kSeg ? s_sin[w * 32 + j] : 0u, s_in[w * 32 + j], sys, key, j < lane) ? 1 : 0;
  s_run[w * 32 + r] = key;
  if (kSeg) s_srun[w * 32 + r] = sys;
  __syncthreads();
#pragma unroll(kTileRuns > 4 ? 5 : 3)
  for (int q = 1; q < kTileRuns; ++q) {
    const int run = (w + q) % kTileRuns;
    const uint64_t* k = s_run + run * 32;
    const uint32_t* s = s_srun + (kSeg ? run * 32 : 0);
    const bool before = run < w;
    int p = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (tile_less<kSeg>(kSeg ? s[p + step - 1] : 0u, k[p + step - 1], sys, key, before)) p += step;
    if (tile_less<kSeg>(kSeg ? s[p] : 0u, k[p], sys, key, before)) p += 1;
    r += p;
  }
  if (base + r < n) {
    kout[base + r] = key;
    vout[base + r] = val;
  }
}

// Number of keys of the sorted range kin[lo, lo + len), at most kTileKeys, that sort before `key` (equal
// ones included for an earlier tile).
template <int kTileKeys>
__device__ __forceinline__ int tile_count(const uint64_t* __restrict__ kin, int lo, int len, uint64_t key,
                                          bool earlier) {
  int p = 0;
  for (int step = kTileKeys; step > 0; step >>= 1) {
    const bool fits = p + step <= len;
    const uint64_t k = kin[lo + (fits ? p + step - 1 : 0)];
    if (fits && (earlier ? k <= key : k < key)) p += step;
  }
  return p;
}

// How many of the keys of [o0, o1) outside tile `own` sort before each lane's key: this warp's share of
// the tiles (32 at a time, from tile t0 on, `step` tiles further each time), to be added up over the
// warps. The warp's 32 keys stand in order, kfirst to klast.
// A lane takes a tile and finds how many of its keys come before the first and before the last of the
// 32. Where the two agree (most tiles, once the bodies are in the previous step's order) that is the
// count for all 32 keys; the others are searched between the two, a key per lane.
template <int kTileKeys>
__device__ __forceinline__ int tile_counts(const uint64_t* __restrict__ kin, int o0, int o1, int own, int t0, int step32,
                                           uint64_t key, uint64_t kfirst, uint64_t klast) {
  const int lane = threadIdx.x & 31, tlast = (o1 - 1) / kTileKeys;
  int cnt = 0, shared_cnt = 0;  // shared_cnt: this lane's tiles, keys before all 32
  for (; t0 <= tlast; t0 += step32) {
    const int tile = t0 + lane;
    int lo = max(o0, tile * kTileKeys), len = min(o1, (tile + 1) * kTileKeys) - lo, c0 = 0, c1 = 0;
    if (tile <= tlast && tile != own) {
      for (int step = kTileKeys; step > 0; step >>= 1) {  // the two searches side by side
        const bool f0 = c0 + step <= len, f1 = c1 + step <= len;
        const uint64_t k0 = kin[lo + (f0 ? c0 + step - 1 : 0)], k1 = kin[lo + (f1 ? c1 + step - 1 : 0)];
        if (f0 && (tile < own ? k0 <= kfirst : k0 < kfirst)) c0 += step;
        if (f1 && (tile < own ? k1 <= klast : k1 < klast)) c1 += step;
      }
      shared_cnt += c0;
    }
    uint32_t open = __ballot_sync(0xffffffffu, c1 > c0);
    lo += c0;
    len = c1 - c0;
    while (open) {  // four tiles' searches in flight
      constexpr int kFlight = 4;
      int clo[kFlight], clen[kFlight], p[kFlight], longest = 0;
      bool earlier[kFlight];
#pragma unroll
      for (int q = 0; q < kFlight; ++q) {
        const int src = open ? __ffs(open) - 1 : 0;
        clo[q] = __shfl_sync(0xffffffffu, lo, src);
        if (!open) clo[q] = 0;  // an empty search reads key 0
        clen[q] = open ? __shfl_sync(0xffffffffu, len, src) : 0;
        earlier[q] = t0 + src < own;
        open &= open - 1;
        p[q] = 0;
        longest = max(longest, clen[q]);
      }
      for (int step = 1 << (31 - __clz(longest)); step > 0; step >>= 1) {
#pragma unroll
        for (int q = 0; q < kFlight; ++q) {
          const bool fits = p[q] + step <= clen[q];
          const uint64_t k = kin[clo[q] + (fits ? p[q] + step - 1 : 0)];
          if (fits && (earlier[q] ? k <= key : k < key)) p[q] += step;
        }
      }
#pragma unroll
      for (int q = 0; q < kFlight; ++q) cnt += p[q];
    }
  }
  return cnt + __reduce_add_sync(0xffffffffu, shared_cnt);
}

// Final places of the block's 32 keys (tile-sorted slots 32 blockIdx.x ..): true in the lanes of the
// first warp that hold a key, with its place, key and value. All threads call it; the block's warps
// share the tiles.
// kSeg: pairs ordered by (system, key), off the systems' slot ranges, body_sys each slot's system. A
// slot's system is that of every pair the tile sort may put there.
template <int kTileKeys, bool kSeg>
__device__ __forceinline__ bool tile_merge_rank(const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                const uint16_t* __restrict__ body_sys,
                                                const uint32_t* __restrict__ off, int n, int& place, uint64_t& key,
                                                uint32_t& val) {
  __shared__ int s_cnt[kMergeParts][32];
  const int lane = threadIdx.x & 31, part = threadIdx.x >> 5, parts = blockDim.x >> 5;
  const int b0 = blockIdx.x * 32, i = b0 + lane, own = b0 / kTileKeys;
  const int last = min(31, n - 1 - b0);  // the block's last key
  const bool valid = lane <= last;
  key = kin[min(i, n - 1)];
  const uint64_t kfirst = __shfl_sync(0xffffffffu, key, 0), klast = __shfl_sync(0xffffffffu, key, last);
  int o0 = 0, o1 = n;
  bool same = true;
  if (kSeg) {
    const int sys = body_sys[min(i, n - 1)];
    o0 = (int)off[sys];
    o1 = (int)off[sys + 1];
    same = __all_sync(0xffffffffu, sys == __shfl_sync(0xffffffffu, sys, 0));
  }
  int cnt = 0;
  if (same) {
    cnt = tile_counts<kTileKeys>(kin, o0, o1, own, o0 / kTileKeys + part * 32, parts * 32, key, kfirst, klast);
  } else {  // several systems among the block's keys: each lane searches its own system's tiles
    const int tfirst = __reduce_min_sync(0xffffffffu, o0 / kTileKeys);
    const int tlast = __reduce_max_sync(0xffffffffu, (o1 - 1) / kTileKeys);
    for (int tile = tfirst + part; tile <= tlast; tile += parts) {
      const int lo = max(o0, tile * kTileKeys), len = min(o1, (tile + 1) * kTileKeys) - lo;
      if (tile != own && len > 0) cnt += tile_count<kTileKeys>(kin, lo, len, key, tile < own);
    }
  }
  s_cnt[part][lane] = cnt;
  __syncthreads();
  if (part != 0 || !valid) return false;
  place = o0 + (i - max(o0, own * kTileKeys));
  for (int q = 0; q < parts; ++q) place += s_cnt[q][lane];
  val = vin[i];
  return true;
}

// The same with a warp for every 32 keys, for merges of about 32 tiles: within spans of kSpanKeys keys
// (0: over all n). No barrier; whole warps return early.
template <int kTileKeys, int kSpanKeys>
__device__ __forceinline__ bool span_merge_rank(const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                int n, int& place, uint64_t& key, uint32_t& val) {
  const int lane = threadIdx.x & 31;
  const int b0 = (int)(blockIdx.x * blockDim.x + threadIdx.x - lane), i = b0 + lane, own = b0 / kTileKeys;
  if (b0 >= n) return false;
  const int last = min(31, n - 1 - b0);
  key = kin[min(i, n - 1)];
  const uint64_t kfirst = __shfl_sync(0xffffffffu, key, 0), klast = __shfl_sync(0xffffffffu, key, last);
  const int o0 = kSpanKeys ? b0 / kSpanKeys * kSpanKeys : 0, o1 = kSpanKeys ? min(n, o0 + kSpanKeys) : n;
  const int cnt = tile_counts<kTileKeys>(kin, o0, o1, own, o0 / kTileKeys, 32, key, kfirst, klast);
  if (lane > last) return false;
  place = o0 + (i - own * kTileKeys) + cnt;
  val = vin[i];
  return true;
}

// The final merge's places: of tiles, by blocks that share them, or of merged spans, a warp per 32 keys.
template <int kTileKeys, bool kSeg>
__device__ __forceinline__ bool merge_rank(const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                           const uint16_t* __restrict__ body_sys, const uint32_t* __restrict__ off,
                                           int n, int& place, uint64_t& key, uint32_t& val) {
  if (kTileKeys > kTileLarge) return span_merge_rank<kTileKeys, 0>(kin, vin, n, place, key, val);
  return tile_merge_rank<kTileKeys, kSeg>(kin, vin, body_sys, off, n, place, key, val);
}

// The launches of a sort of n keys: tiles of `tile` keys, merged in spans of `span` keys (0: not), then
// runs of `run()` keys into the result.
struct TileShape {
  int n, tile, span;
  int run() const { return span ? span : tile; }
  int tile_blocks() const { return (n + tile - 1) / tile; }
  // without spans a warp for every 32 tiles, up to eight, share 32 keys
  int merge_threads() const {
    const int parts = (tile_blocks() + 31) / 32;
    return span ? kSpanThreads : 32 * (parts < kMergeParts ? parts : kMergeParts);
  }
  int merge_blocks() const { return span ? (n + kSpanThreads - 1) / kSpanThreads : (n + 31) / 32; }
};

// In a step the keys are nearly in order. Ensembles (seg) never merge spans: their systems are short.
inline TileShape step_shape(int n, bool seg = false) {
  if (!seg && n > kTwoLaunchMax) return {n, kTileSpan, 32 * kTileSpan};
  return {n, n <= kTileSmallMax ? kTileSmall : kTileLarge, 0};
}
// Pairs in any order.
inline TileShape pairs_shape(int n) {
  if (n > kSpanSmallMax) return {n, kTileSpan, 32 * kTileSpan};
  if (n > kTwoLaunchPairsMax) return {n, kTileSmall, 32 * kTileSmall};
  return {n, n <= kTileSmallMax ? kTileSmall : kTileLarge, 0};
}

// The kernel instance of a shape's tiles and of its final merge.
#define BH_TILE_KERNEL(kernel, shape)                      \
  ((shape).tile == kTileSmall  ? kernel<kTileSmall, false> \
   : (shape).tile == kTileSpan ? kernel<kTileSpan, false>  \
                               : kernel<kTileLarge, false>)
#define BH_TILE_KERNEL_SEG(kernel, shape) \
  ((shape).tile == kTileSmall ? kernel<kTileSmall, true> : kernel<kTileLarge, true>)
#define BH_MERGE_KERNEL(kernel, shape)                      \
  ((shape).run() == kTileSmall   ? kernel<kTileSmall, false> \
   : (shape).run() == kTileLarge ? kernel<kTileLarge, false> \
                                 : kernel<32 * kTileSpan, false>)

}  // namespace bh
