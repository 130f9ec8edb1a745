// Two-launch stable sort of up to kTileSortMax (u64 key, u32 value) pairs, as building blocks that
// the stage kernels fuse with what makes the keys and with what consumes the sorted order.
//
//   tile:  a block sorts 128 or 512 pairs. Each warp ranks its 32 keys by comparing them all (a
//          broadcast read per comparison), which gives 4 or 16 sorted runs in shared memory; a
//          key's place in the tile is its place in its run plus, by binary search, its place in
//          the other runs.
//   merge: a key's final place is its place in its tile plus, by binary search, its place in every
//          other tile. A block takes 32 keys and its eight warps share the tiles.
//
// Equal keys count when they stand in an earlier run or tile, so the sort is stable. The radix sort's
// eight digit passes are a chain of 10 dependent launches, this is two; its work grows with n^2 over
// the tile, which sets the limit.
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

// Final places of the block's 32 keys (tile-sorted slots 32 blockIdx.x ..): true in the lanes of the
// first warp that hold a key, with its place, key and value. All threads call it.
// A warp takes 32 tiles at once, a tile per lane, and finds how many of its keys come before the
// block's first and before its last key. Where the two agree (most tiles, once the bodies are
// in the previous step's order) that is the count for all 32 keys; the others are searched between
// the two, a key per lane.
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
    const int tfirst = o0 / kTileKeys, tlast = (o1 - 1) / kTileKeys;
    int shared_cnt = 0;  // this lane's tiles: keys before all of the block's
    for (int t0 = tfirst + part * 32; t0 <= tlast; t0 += parts * 32) {
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
    cnt += __reduce_add_sync(0xffffffffu, shared_cnt);
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

// Tile size for n keys (both launches of a sort), and the launches' shapes.
inline int tile_keys(int n) { return n <= kTileSmallMax ? kTileSmall : kTileLarge; }
inline int tile_blocks(int n) { return (n + tile_keys(n) - 1) / tile_keys(n); }
inline int merge_blocks(int n) { return (n + 31) / 32; }
// a warp for every 32 tiles, up to eight
inline int merge_threads(int n) {
  const int parts = (tile_blocks(n) + 31) / 32;
  return 32 * (parts < kMergeParts ? parts : kMergeParts);
}

// Launches kernel<tile size, segments> with the tile of n keys.
#define BH_TILE_KERNEL(kernel, n, seg)                                                      \
  (tile_keys(n) == kTileSmall ? ((seg) ? kernel<kTileSmall, true> : kernel<kTileSmall, false>) \
                              : ((seg) ? kernel<kTileLarge, true> : kernel<kTileLarge, false>))

}  // namespace bh
