// The PSO's two paths for quadratic forms of other dimensions than the
// library's: the per-iteration kernel serves up to 512, the one-launch kernel
// only where eight particles and the matrix fit a block.
#include <cstdint>

#include "zb_pso_swarm.cuh"

using zeus::Gaussian;

static_assert(zb::swarm_built<Gaussian<150>, 150>());
static_assert(!zb::swarm_built<Gaussian<168>, 168>()); // more than an SM's shared memory
static_assert(!zb::swarm_built<Gaussian<264>, 264>());
static_assert(!zb::swarm_built<Gaussian<520>, 520>());

template <int D>
void
launch(const double* C, double* out)
{
  Gaussian<D> f;
  f.C = C;
  zb::PsoWork w{};
  if constexpr (zb::swarm_built<Gaussian<D>, D>())
    zb::pso_swarm_kernel<Gaussian<D>, D><<<1, 32>>>(f, zb::SwarmArgs{});
  else if constexpr (D <= zb::kPsoDmmaMaxDim)
    zb::pso_init_dmma_kernel<D><<<1, zb::kPsoBlock>>>(f, 8, -1.0, 1.0, 1, w, out, out);
}

template void launch<40>(const double*, double*);
template void launch<150>(const double*, double*);
template void launch<160>(const double*, double*);
template void launch<168>(const double*, double*);
template void launch<264>(const double*, double*);
template void launch<512>(const double*, double*);
