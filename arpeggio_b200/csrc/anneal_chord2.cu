// The Chord round on compressed dDI problems, two copies, integer fields: the kernels of anneal_group.cuh.
#include "anneal_group.cuh"

namespace arp {
cudaError_t int_chord2(const DDParams& a, int warps, cudaStream_t st) { return grp::dispatch<2, grp::kChord>(a, warps, st); }
}  // namespace arp
