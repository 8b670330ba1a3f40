// Warm-started first accept on compressed dDI problems (two copies, integer fields): the kernels of anneal_group.cuh.
#include "anneal_group.cuh"

namespace arp {
cudaError_t int_warm(const DDParams& a, int warps, cudaStream_t st) { return grp::dispatch<2, grp::kWarm>(a, warps, st); }
}  // namespace arp
