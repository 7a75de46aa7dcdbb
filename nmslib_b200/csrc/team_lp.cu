// The team search kernels for L1 and LInf indices.
#include "team_kernel.cuh"

namespace nmsg {
namespace {
template <int D>
void* select(int warps, bool with_old) {
  if (with_old) return (void*)search_team_kernel<D, 0, 8, true>;
  return warps == 4 ? (void*)search_team_kernel<D, 0, 4, false> : (void*)search_team_kernel<D, 0, 8, false>;
}
}  // namespace
void* team_kernel_lp(const DevIndex& ix, int warps, bool with_old) {
  return ix.dist_type == kL1 ? select<kTeamL1>(warps, with_old) : select<kTeamLInf>(warps, with_old);
}
}  // namespace nmsg
