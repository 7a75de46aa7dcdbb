// The team search kernels for l2sqr_sift indices.
#include "team_kernel.cuh"

namespace nmsg {
// Eight warps only: their limit ends where four would start.
void* team_kernel_sift(bool with_old) {
  return with_old ? (void*)search_team_kernel<kTeamSift, 0, 8, true>
                  : (void*)search_team_kernel<kTeamSift, 0, 8, false>;
}
}  // namespace nmsg
