// The Chord round on compressed dDI problems, four and six copies, integer fields: the kernels of anneal_group.cuh.
#include "anneal_group.cuh"

namespace arp {
cudaError_t int_chord46(const DDParams& a, int P, int warps, cudaStream_t st) {
  return P == 4 ? grp::dispatch<4, grp::kChord>(a, warps, st) : grp::dispatch<6, grp::kChord>(a, warps, st);
}
}  // namespace arp
