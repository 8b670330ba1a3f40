// The Chord round on compressed dDI problems with FP32 fields: the kernels of anneal_group_f32.cuh.
#include "anneal_group_f32.cuh"

namespace arp {
cudaError_t f32_chord(const DDParams& a, int P, int warps, cudaStream_t st) {
  return P == 2   ? grpf::dispatch<2, true>(a, warps, st)
         : P == 4 ? grpf::dispatch<4, true>(a, warps, st)
                  : grpf::dispatch<6, true>(a, warps, st);
}
}  // namespace arp
