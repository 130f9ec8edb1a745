// Conservation diagnostics (bh_energy_diag): kinetic and potential energy, linear and angular
// momentum of the current state. The reference has none; these measure the drift of the
// integrator and the tree force over a run.
//
// The potential of body i is taken over the current tree with the reference's opening test
// (s^2 / d^2 < theta^2 with s the node edge and d the distance to the node's barycentre,
// src/HashedOctree.cpp:872-885) and the multipoles the tree was built with:
//   accepted node  phi -= M / D + (d.Q.d) / (2 D^5),   D^2 = |d|^2 + eps^2,  d = C - x
//   opened leaf    phi -= m_j / D for every member j at a position other than x
// (the potential whose gradient is the monopole + quadrupole force of the walk). The force walk's kernel
// computes it, a warp per group of bodies (with one thread per body on its own stack, and buffers
// allocated by each call, the diagnostics of 131 071 bodies took 1.89 ms, now 0.74). Energy sums are
// accumulated in FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "bh_internal.cuh"

namespace bh {
namespace {

constexpr int kThreads = 128;
constexpr int kSums = kDiagSums;  // kinetic, potential, momentum (3), angular momentum (3), mass, mass-weighted x (3)

__device__ __forceinline__ void block_add(double (&v)[kSums], double* __restrict__ out) {
  __shared__ double sh[kThreads / 32][kSums];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < kSums; ++k) {
    double x = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sh[w][k] = x;
  }
  __syncthreads();
  if (threadIdx.x < kSums) {
    double x = 0;
    for (int i = 0; i < kThreads / 32; ++i) x += sh[i][threadIdx.x];
    if (x != 0.0) atomicAdd(out + threadIdx.x, x);
  }
}

// Kinetic and potential energy, momentum, angular momentum, mass and centre of mass over the slots.
__global__ __launch_bounds__(kThreads) void k_moments(const float4* __restrict__ pos, const float4* __restrict__ vel,
                                                      const float* __restrict__ pot, int n,
                                                      double* __restrict__ sums) {
  double v[kSums] = {};
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
    const float4 p = pos[i], u = vel[i];
    const double m = p.w, x = p.x, y = p.y, z = p.z, vx = u.x, vy = u.y, vz = u.z;
    v[0] += 0.5 * m * (vx * vx + vy * vy + vz * vz);
    v[1] += 0.5 * m * (double)pot[i];
    v[2] += m * vx;
    v[3] += m * vy;
    v[4] += m * vz;
    v[5] += m * (y * vz - z * vy);
    v[6] += m * (z * vx - x * vz);
    v[7] += m * (x * vy - y * vx);
    v[8] += m;
    v[9] += m * x;
    v[10] += m * y;
    v[11] += m * z;
  }
  block_add(v, sums);
}

}  // namespace
}  // namespace bh

using namespace bh;

extern "C" {

bh_status bh_energy_diag(bh_ctx* c, double theta, double eps, bh_energy* out, float* pot_out) {
  bh::Range range_("bh_energy_diag");
  if (!c || !out || !(theta >= 0) || !(eps >= 0)) return BH_ERR_INVALID_ARG;
  if (!c->tree_valid) return BH_ERR_NO_TREE;
  cudaSetDevice(c->device);
  const int n = (int)c->n;
  std::memset(out, 0, sizeof(*out));
  if (n == 0) return BH_OK;
  // phi by slot in the sorts' value scratch, the sums in the status block
  float* pot = reinterpret_cast<float*>(c->vals[1]);
  clear_device_flags(c);
  cudaMemsetAsync(c->status->sums, 0, sizeof(double) * kSums, c->stream);
  bh::launch_potential(c, n, (float)theta, (float)eps, c->tree_mode, pot);
  const int grid = std::min((n + kThreads - 1) / kThreads, c->sms * 2);
  c->launches += 1;
  k_moments<<<grid, kThreads, 0, c->stream>>>(c->pos[c->cur], c->vel[c->cur], pot, n, c->status->sums);
  if (pot_out) cudaMemcpyAsync(pot_out, pot, sizeof(float) * n, cudaMemcpyDeviceToHost, c->stream);
  uint32_t e = 0;
  BH_TRY(last_launch());
  BH_TRY(sync_and_check(c, &e));
  if (e) return err_to_status(e);
  const double* h = c->h_status->sums;
  out->kinetic = h[0];
  out->potential = h[1];
  out->total = h[0] + h[1];
  for (int a = 0; a < 3; ++a) {
    out->momentum[a] = h[2 + a];
    out->angular_momentum[a] = h[5 + a];
    out->com[a] = h[8] != 0 ? h[9 + a] / h[8] : 0.0;
  }
  out->mass = h[8];
  return BH_OK;
}

}  // extern "C"
