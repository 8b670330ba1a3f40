// The Chord round with the engine model's own numbers, integer fields: the kernels of anneal_group.cuh.
#include "anneal_group.cuh"

namespace arp {
cudaError_t int_engine(const DDParams& a, int P, cudaStream_t st) {
  return P == 2   ? grp::dispatch<2, grp::kEngine>(a, 0, st)
         : P == 4 ? grp::dispatch<4, grp::kEngine>(a, 0, st)
                  : grp::dispatch<6, grp::kEngine>(a, 0, st);
}
}  // namespace arp
