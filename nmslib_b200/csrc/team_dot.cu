// The team search kernels for cosine and negative-dot-product indices.
#include "team_kernel.cuh"

namespace nmsg {
namespace {
template <int D>
void* select(const DevIndex& ix, int warps, bool with_old) {
  if (with_old) return (void*)search_team_kernel<D, 0, 8, true>;
  // as in team_l2.cu; cosine 1M x 100, M 24, efSearch 200, 600 / 2,000 queries: 1,090 / 2,026 -> 963 / 1,734 us
  switch (ix.n16 >> 5) {
    case 3:
      return warps == 4 ? (void*)search_team_kernel<D, 3, 4, false> : (void*)search_team_kernel<D, 3, 8, false>;
    case 4:
      return warps == 4 ? (void*)search_team_kernel<D, 4, 4, false> : (void*)search_team_kernel<D, 4, 8, false>;
  }
  return warps == 4 ? (void*)search_team_kernel<D, 0, 4, false> : (void*)search_team_kernel<D, 0, 8, false>;
}
}  // namespace
void* team_kernel_dot(const DevIndex& ix, int warps, bool with_old) {
  return ix.dist_type == kNormCosine ? select<kTeamCos>(ix, warps, with_old) : select<kTeamNeg>(ix, warps, with_old);
}
}  // namespace nmsg
