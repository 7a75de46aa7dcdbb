// The team search kernels for squared L2 indices.
#include "team_kernel.cuh"

namespace nmsg {
void* team_kernel_l2(const DevIndex& ix, int warps, bool with_old) {
  if (with_old) return (void*)search_team_kernel<kTeamL2, 0, 8, true>;
  // rows of 96 to 159 floats (the lengths of the common data sets): loops of known length, all of a row in
  // flight, instead of the loop that tests every block. 1M x 128, efSearch 100, 16 / 600 / 1,500 queries:
  // 345 / 853 / 1,339 -> 318 / 798 / 1,284 us
  switch (ix.n16 >> 5) {
    case 3:
      return warps == 4 ? (void*)search_team_kernel<kTeamL2, 3, 4, false>
                        : (void*)search_team_kernel<kTeamL2, 3, 8, false>;
    case 4:
      return warps == 4 ? (void*)search_team_kernel<kTeamL2, 4, 4, false>
                        : (void*)search_team_kernel<kTeamL2, 4, 8, false>;
  }
  return warps == 4 ? (void*)search_team_kernel<kTeamL2, 0, 4, false>
                    : (void*)search_team_kernel<kTeamL2, 0, 8, false>;
}
}  // namespace nmsg
