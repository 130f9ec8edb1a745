// The potential of every body over the current tree, for the conservation diagnostics: the force walk's kernel
// with the potential's terms, in the force walk's groups. Compiled without the flush of denormals that the
// force walk has: d.Q.d / D^5 of a cell has a factor 1 / D^5 that is denormal from D = 4e7 on (a solar
// system in km), and bodies closer than 1.1e-19 have denormal squared distances.
#include "bh_walk_kernel.cuh"

namespace bh {
namespace {

template <bool kQuad, int kGroup>
void launch_potential_t(bh_ctx* c, int n, float theta2, float eps2, float* pot_slot) {
  const int ngroups = (n + kGroup - 1) / kGroup;
  const int grid = min(walk_grid<kQuad, true, false, CfgDefault, kGroup, true>(), walk_blocks<CfgDefault, kGroup>(ngroups));
  k_walk<kQuad, true, false, CfgDefault, kGroup, true><<<grid, CfgDefault::kThreads, 0, c->stream>>>(
      c->wnode, c->tpos, c->tslot, n, theta2, eps2, reinterpret_cast<float4*>(pot_slot), nullptr, 0.f, nullptr, nullptr,
      0, c->counters, c->err);
}

template <bool kQuad>
void launch_potential_group(bh_ctx* c, int n, float theta2, float eps2, float* pot_slot) {
  switch (walk_group_size(n)) {
    case 4: launch_potential_t<kQuad, 4>(c, n, theta2, eps2, pot_slot); break;
    case 8: launch_potential_t<kQuad, 8>(c, n, theta2, eps2, pot_slot); break;
    case 16: launch_potential_t<kQuad, 16>(c, n, theta2, eps2, pot_slot); break;
    default: launch_potential_t<kQuad, 32>(c, n, theta2, eps2, pot_slot); break;
  }
}

}  // namespace

void launch_potential(bh_ctx* c, int n, float theta, float eps, int mode, float* pot_slot) {
  if (n <= 0) return;
  c->launches += 1;
  if (mode == BH_MULTIPOLE_QUADRUPOLE)
    launch_potential_group<true>(c, n, theta * theta, eps * eps, pot_slot);
  else
    launch_potential_group<false>(c, n, theta * theta, eps * eps, pot_slot);
}

}  // namespace bh
