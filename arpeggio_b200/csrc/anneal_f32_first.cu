// First accept on compressed dDI problems with FP32 fields: the kernels of anneal_group_f32.cuh.
#include "anneal_group_f32.cuh"

namespace arp {
cudaError_t f32_first(const DDParams& a, int P, int warps, cudaStream_t st) {
  return P == 2   ? grpf::dispatch<2, false>(a, warps, st)
         : P == 4 ? grpf::dispatch<4, false>(a, warps, st)
                  : grpf::dispatch<6, false>(a, warps, st);
}
}  // namespace arp
