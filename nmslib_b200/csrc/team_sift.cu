// The team search kernels for l2sqr_sift indices.
#include "team_kernel.cuh"

namespace nmsg {
void* team_kernel_sift(int warps, bool with_old) {
  if (with_old)
    return warps == 4 ? (void*)search_team_kernel<kTeamSift, 0, 4, true>
                      : (void*)search_team_kernel<kTeamSift, 0, 8, true>;
  return warps == 4 ? (void*)search_team_kernel<kTeamSift, 0, 4, false>
                    : (void*)search_team_kernel<kTeamSift, 0, 8, false>;
}
}  // namespace nmsg
