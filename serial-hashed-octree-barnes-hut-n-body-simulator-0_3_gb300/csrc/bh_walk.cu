// Launches of the force walk (bh_walk_kernel.cuh): launch shapes by the number of bodies, the shapes the
// autotuner chooses from, ensembles, and the recording walk of the differentiable path. Compiled to flush
// FP32 denormals (build.py).
#include <algorithm>
#include <type_traits>

#include "bh_walk_kernel.cuh"

namespace bh {
namespace {

struct WalkArgs {
  float theta2, eps2, half_dt;
  float4 *acc_slot, *vel_kick, *vel_copy;
  bool batch;
};

template <bool kQuad, bool kSelf, class Cfg = CfgDefault, int kGroup = 32>
void launch_walk_t(bh_ctx* c, int n, const WalkArgs& a) {
  const bool own = kGroup == c->batch_group;  // else a shape of groups of 32 on a smaller ensemble
  const int4* table = !a.batch ? nullptr : own ? c->groups : c->groups32;
  const int ngroups = !a.batch ? (n + kGroup - 1) / kGroup : own ? c->ngroups : c->ngroups32;
  const int grid = min(walk_grid<kQuad, kSelf, false, Cfg, kGroup>(), walk_blocks<Cfg, kGroup>(ngroups));
  k_walk<kQuad, kSelf, false, Cfg, kGroup><<<grid, Cfg::kThreads, 0, c->stream>>>(
      c->wnode, c->tpos, c->tslot, n, a.theta2, a.eps2, a.acc_slot, a.vel_kick, a.half_dt, a.vel_copy,
      table, ngroups, c->counters, c->err);
}

// The walk with groups of `group` bodies (32, 16, 8 or 4; an ensemble's table is built for it).
template <bool kQuad, bool kSelf>
void launch_walk_group(bh_ctx* c, int n, const WalkArgs& a, int group) {
  switch (group) {
    case 4: launch_walk_t<kQuad, kSelf, CfgDefault, 4>(c, n, a); break;
    case 8: launch_walk_t<kQuad, kSelf, CfgDefault, 8>(c, n, a); break;
    case 16: launch_walk_t<kQuad, kSelf, CfgDefault, 16>(c, n, a); break;
    default: launch_walk_t<kQuad, kSelf, CfgDefault, 32>(c, n, a); break;
  }
}

// Launch shapes the autotuner chooses from for the quadrupole walk with positive softening
// (the benchmarked path): block size, register budget (resident blocks per SM) and stack depth.
// Static shared memory caps a block at 48 KB, which bounds warps x stack depth.
using Cfg1 = WalkCfg<8, 3, 384>;
using Cfg2 = WalkCfg<8, 2, 384>;
using Cfg3 = WalkCfg<4, 8, 384>;
using Cfg4 = WalkCfg<4, 6, 384>;
using Cfg5 = WalkCfg<4, 8, 512>;
using Cfg6 = WalkCfg<8, 4, 384, 1>;
using Cfg7 = WalkCfg<4, 8, 384, 1>;
// Variant 0, the default, takes its group size from the number of bodies (walk_group_size), 1 to 7 walk
// groups of 32; variants 8 and 9 take 16 and 8, and 10 and 11 do so at 104 registers (two 8-warp blocks
// per SM): small single systems, where a few warps per SM walk and the walk's time is one warp's chain
// of dependent latencies. Ensembles have tables of the default's groups and of groups of 32, so for them
// 8 to 11 are variant 0.
constexpr int kVariants = 12;

// The 104-register shape of the small groups, while about one wave of its blocks (16 warps per SM)
// holds them all: a warp then walks one group, and its latency is the walk's. Quadrupole walk, us at 64
// (groups of 16: 80) / 104 registers: 1 000 bodies in groups of 4 46.7 / 42.7; 10 000 (2 500 groups) 114.5 /
// 104.0; 16 384 in groups of 8 160.0 / 145.4, of 4 (4 096 groups) 171.8 / 178.7; 32 768 in groups of 16
// (2 048 groups) 223 / 237, 65 536 (4 096 groups) 360 / 403: for groups of 16 the line could lie lower.
constexpr int kWideMaxGroups = 3072;
bool walk_wide(int ngroups, int group) { return group < 32 && ngroups <= kWideMaxGroups; }

template <class Cfg, int kGroup = 32>
WalkVariant variant_info() {
  cudaFuncAttributes fa{};
  cudaFuncGetAttributes(&fa, k_walk<true, false, false, Cfg, kGroup>);
  return {Cfg::kWarps, Cfg::kMinBlocks, Cfg::kStack, Cfg::kForm, fa.numRegs, kGroup};
}

// f(shape, group size) with the default shape for that many groups of `group` bodies: 104 registers while
// the groups are few (see walk_wide), 80 for groups of 16 (65 536 bodies 417 us at 64, 360 at 80), else 64.
template <class F>
auto with_default_shape(int ngroups, int group, F f) {
  using std::integral_constant;
  const bool wide = walk_wide(ngroups, group);
  switch (group) {
    case 4: return wide ? f(Cfg2{}, integral_constant<int, 4>{}) : f(CfgDefault{}, integral_constant<int, 4>{});
    case 8: return wide ? f(Cfg2{}, integral_constant<int, 8>{}) : f(CfgDefault{}, integral_constant<int, 8>{});
    case 16: return wide ? f(Cfg2{}, integral_constant<int, 16>{}) : f(Cfg1{}, integral_constant<int, 16>{});
    default: return f(CfgDefault{}, integral_constant<int, 32>{});
  }
}

void launch_quad_default(bh_ctx* c, int n, const WalkArgs& a, int group) {
  with_default_shape(a.batch ? c->ngroups : (n + group - 1) / group, group, [&](auto cfg, auto g) {
    launch_walk_t<true, false, decltype(cfg), decltype(g)::value>(c, n, a);
  });
}

void launch_quad_variant(bh_ctx* c, int v, int n, const WalkArgs& a) {
  if (a.batch && v >= 8) v = 0;
  switch (v) {
    case 1: launch_walk_t<true, false, Cfg1>(c, n, a); break;
    case 2: launch_walk_t<true, false, Cfg2>(c, n, a); break;
    case 3: launch_walk_t<true, false, Cfg3>(c, n, a); break;
    case 4: launch_walk_t<true, false, Cfg4>(c, n, a); break;
    case 5: launch_walk_t<true, false, Cfg5>(c, n, a); break;
    case 6: launch_walk_t<true, false, Cfg6>(c, n, a); break;
    case 7: launch_walk_t<true, false, Cfg7>(c, n, a); break;
    case 8: launch_walk_t<true, false, CfgDefault, 16>(c, n, a); break;
    case 9: launch_walk_t<true, false, CfgDefault, 8>(c, n, a); break;
    case 10: launch_walk_t<true, false, Cfg2, 16>(c, n, a); break;
    case 11: launch_walk_t<true, false, Cfg2, 8>(c, n, a); break;
    default: launch_quad_default(c, n, a, a.batch ? c->batch_group : walk_group_size(n)); break;
  }
}

}  // namespace

int walk_variants() { return kVariants; }

// Small groups give more warps and, with their boxes, fewer entries a body (at 16 384 bodies, leaf
// capacity 1, a group of 32 / 16 / 8 evaluates 2200 / 1835 / 1569 entries), but each group traverses
// the tree. Quadrupole walk, us with groups of 4 / 8 / 16 / 32, each in its default shape (theta 0.5; leaf
// capacity 1 up to 16 384 bodies, 8 above): 1 000 bodies 43 / 51 / 66 / 142; 10 000 104 / 116 / 152 / 309;
// 16 384 172 / 145 / 166 / 352; 32 768 274 / 240 / 237 / 357; 65 536 525 / 401 / 360 / 455; 131 072 1036 /
// 754 / 668 / 755; 262 144 2125 / 1474 / 1237 / 1200. The literal walk crosses at the same sizes.
int walk_group_size(size_t n) {
  if (n < 12288) return 4;
  if (n < 24576) return 8;
  return n < 196608 ? 16 : 32;
}

WalkVariant walk_variant_info(const bh_ctx* c, int v) {
  if (c->batch && v >= 8) v = 0;  // as in launch_quad_variant
  switch (v) {
    case 1: return variant_info<Cfg1>();
    case 2: return variant_info<Cfg2>();
    case 3: return variant_info<Cfg3>();
    case 4: return variant_info<Cfg4>();
    case 5: return variant_info<Cfg5>();
    case 6: return variant_info<Cfg6>();
    case 7: return variant_info<Cfg7>();
    case 8: return variant_info<CfgDefault, 16>();
    case 9: return variant_info<CfgDefault, 8>();
    case 10: return variant_info<Cfg2, 16>();
    case 11: return variant_info<Cfg2, 8>();
    default: break;
  }
  const int group = c->batch ? c->batch_group : walk_group_size(c->n);
  const int ngroups = c->batch ? c->ngroups : (int)((c->n + group - 1) / group);
  return with_default_shape(ngroups, group,
                            [](auto cfg, auto g) { return variant_info<decltype(cfg), decltype(g)::value>(); });
}

// One force-only walk with the given variant (the autotuner's trial); acc_out by slot.
void launch_walk_variant(bh_ctx* c, int v, int n, float theta, float eps, float4* acc_out, bool batch) {
  if (n <= 0) return;
  c->launches += 1;
  launch_quad_variant(c, v, n, WalkArgs{theta * theta, eps * eps, 0.f, acc_out, nullptr, nullptr, batch});
}

namespace {
template <bool kQuad, bool kSelf>
void walk_grids_all_groups() {
  walk_grid<kQuad, kSelf, false, CfgDefault, 32>();
  walk_grid<kQuad, kSelf, false, CfgDefault, 16>();
  walk_grid<kQuad, kSelf, false, CfgDefault, 8>();
  walk_grid<kQuad, kSelf, false, CfgDefault, 4>();
}
}  // namespace

// Occupancy queries done once per process, before any stream capture.
void walk_init() {
  walk_grids_all_groups<true, true>();
  walk_grids_all_groups<true, false>();
  walk_grids_all_groups<false, true>();
  walk_grids_all_groups<false, false>();
  walk_grid<true, false, true, CfgDefault>();
  walk_grid<true, false, true, Cfg1, 16>();
  walk_grid<true, false, true, Cfg2, 16>();
  walk_grid<true, false, false, Cfg1, 16>();
  walk_grid<true, false, false, Cfg1>();
  walk_grid<true, false, false, Cfg2>();
  walk_grid<true, false, false, Cfg2, 16>();
  walk_grid<true, false, false, Cfg2, 8>();
  walk_grid<true, false, false, Cfg2, 4>();
  walk_grid<true, false, false, Cfg3>();
  walk_grid<true, false, false, Cfg4>();
  walk_grid<true, false, false, Cfg5>();
  walk_grid<true, false, false, Cfg6>();
  walk_grid<true, false, false, Cfg7>();
}

void launch_walk(bh_ctx* c, int n, float theta, float eps, int mode, float4* acc_slot, float4* vel_kick,
                 float half_dt, bool batch, float4* vel_copy) {
  if (n <= 0) return;
  c->launches += 1;
  const WalkArgs a{theta * theta, eps * eps, half_dt, acc_slot, vel_kick, vel_copy, batch};
  const bool quad = mode == BH_MULTIPOLE_QUADRUPOLE;
  const bool self = !(a.eps2 > 0.f);
  const int group = batch ? c->batch_group : walk_group_size(n);
  if (quad && !self)
    launch_quad_variant(c, batch ? c->batch_variant : c->walk_variant, n, a);
  else if (quad)
    launch_walk_group<true, true>(c, n, a, group);
  else if (self)
    launch_walk_group<false, true>(c, n, a, group);
  else
    launch_walk_group<false, false>(c, n, a, group);
}

}  // namespace bh

namespace bh {

template <class Cfg, int kGroup>
static void launch_walk_record_t(bh_ctx* c, int n, float theta, float eps, float4* acc_slot, float4* vel_kick,
                                 float half_dt, Chunk* tape, unsigned* tape_count, int tape_cap) {
  const int grid = min(walk_grid<true, false, true, Cfg, kGroup>(), walk_blocks<Cfg, kGroup>((n + kGroup - 1) / kGroup));
  k_walk<true, false, true, Cfg, kGroup><<<grid, Cfg::kThreads, 0, c->stream>>>(
      c->wnode, c->tpos, c->tslot, n, theta * theta, eps * eps, acc_slot, vel_kick, half_dt, nullptr, nullptr, 0,
      c->counters, c->err, tape, tape_count, tape_cap);
}

// Bodies per group of the differentiable path: 16 where the force walk's groups are at most 16.
int record_group_size(size_t n) { return std::min(32, std::max(16, walk_group_size(n))); }

// The recording walk without its tape, for the forward pass: the same groups whatever the context's variant,
// so that a recomputed step repeats the forward step's sums bit for bit. (Forward steps in groups of 4 or
// 8 would walk faster below 24 576 bodies, 1 000 in 43 us instead of 66, 16 384 in 145 instead of 166, but
// recomputed trajectories would drift away from them.)
void launch_walk_unrecorded(bh_ctx* c, int n, float theta, float eps, float4* acc_slot, float4* vel_kick,
                            float half_dt) {
  if (n <= 0) return;
  c->launches += 1;
  launch_quad_default(c, n, WalkArgs{theta * theta, eps * eps, half_dt, acc_slot, vel_kick, nullptr, false},
                      record_group_size(n));
}

// The walk of the differentiable path: quadrupole multipoles, positive softening, and every
// flushed interaction buffer appended to `tape` (tape_count counts chunks; overflow of tape_cap
// sets the tape error bit).
void launch_walk_record(bh_ctx* c, int n, float theta, float eps, float4* acc_slot, float4* vel_kick, float half_dt,
                        Chunk* tape, unsigned* tape_count, int tape_cap) {
  if (n <= 0) return;
  c->launches += 1;
  auto launch = record_group_size(n) == 32  ? launch_walk_record_t<CfgDefault, 32>
                : walk_wide((n + 15) / 16, 16) ? launch_walk_record_t<Cfg2, 16>
                                               : launch_walk_record_t<Cfg1, 16>;
  launch(c, n, theta, eps, acc_slot, vel_kick, half_dt, tape, tape_count, tape_cap);
}

}  // namespace bh
