// Persistent mixed-size first accept.
// Every problem of every size class of a mixed batch in one grid per coordinate-slot count NS (at most four
// launches): the grid is sized to the SMs' resident blocks, and each block takes problems from a work counter in
// global memory (one atomicAdd per problem, no waiting on other blocks) until the batch is done, running the
// per-size body compiled for its NS.  Problems are numbered class by class, the classes in decreasing cost per
// problem (L R D), so the costly problems start first and the short ones fill the tail.  Each problem's anneals are
// exactly those of the per-class launch (same body, same counters), so the outputs do not depend on the schedule.
#include <cstring>

#include "anneal_group.cuh"

namespace arp {

constexpr int kMaxMixed = 64;

struct MixedArgs {
  PhiloxKeys K;  // one key for the whole batch (kernel parameter: the rounds read it as constant operands)
  int total;
  int* counter;
  int first[kMaxMixed + 1];  // problems of class c: first[c] .. first[c + 1] - 1
  DDParams cls[kMaxMixed];
};

// The mapping of each slot count's group: one that holds its largest coordinate count (the per-class dispatch picks
// narrower ones for large batches up to 16 coordinates and from 33 to 48).
template <int NS>
struct MixedMap {
  static constexpr int LN = NS <= 2 ? 8 : 16, C = NS == 1 ? 4 : NS == 3 ? 6 : 8;
};

template <int NS>
__global__ void __launch_bounds__(grp::max_threads<MixedMap<NS>::LN, MixedMap<NS>::C>(), NS <= 2 ? 3 : 1)
    k_anneal_mixed(const __grid_constant__ MixedArgs g) {
  __shared__ int s_item;
  for (;;) {
    __syncthreads();  // the previous problem's shared memory is no longer read
    if (threadIdx.x == 0) s_item = atomicAdd(g.counter, 1);
    __syncthreads();
    const int i = s_item;
    if (i >= g.total) break;
    int c = 0;
    while (c + 1 < kMaxMixed && g.first[c + 1] <= i) ++c;
    grp::problem<MixedMap<NS>::LN, MixedMap<NS>::C, 2, grp::kFirst>(g.cls[c], g.K, i - g.first[c], 0);
  }
}

template <int NS>
static cudaError_t launch_mixed(MixedArgs& g, int Lmax, int warps, int* counter, cudaStream_t st) {
  constexpr int LN = MixedMap<NS>::LN, C = MixedMap<NS>::C, WMAX = grp::max_threads<LN, C>() / 32;
  const auto kern = k_anneal_mixed<NS>;
  static DeviceAttr attr;
  cudaError_t e = smem_attr(attr, kern, 226 * 1024);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if (warps <= 0) warps = tuned_warps(NS, 2, 0, 0);
  int W = 0, nb = 0;  // the width with the most resident warps per SM, or the caller's
  for (int w = 1; w <= WMAX; w *= 2) {
    const size_t s = grp::smem_bytes<LN, C, 2>(Lmax, w);
    int n = 0;
    if (s > 226 * 1024) break;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, 32 * w, s)) != cudaSuccess) return e;
    if (n > 0 && (warps > 0 ? w <= warps : n * w >= nb * W)) {
      W = w;
      nb = n;
    }
  }
  if (nb < 1) return cudaErrorInvalidConfiguration;
  long long grid = (long long)nb * sms;
  if (grid > g.total) grid = g.total;
  g.counter = counter;
  e = cudaMemsetAsync(counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)grid, 32 * W, grp::smem_bytes<LN, C, 2>(Lmax, W), st>>>(g);
  return cudaGetLastError();
}

}  // namespace arp

using namespace arp;

/* Persistent mixed-size first accept: see the header.  Classes are grouped by slot count and ordered by cost. */
extern "C" int arp_anneal_first_accept_mixed(const arp_mixed_class* cls, int ncls, int P, uint32_t k0, uint32_t k1,
                                             int warps, int* counters, int32_t* status, void* stream) {
  if (ncls < 0 || ncls > kMaxMixed || P != 2) return ARP_ERR_SHAPE;
  if (ncls == 0) return ARP_OK;
  if (!cls || !counters) return ARP_ERR_ARG;
  if (!(warps == 0 || warps == 1 || warps == 2 || warps == 4 || warps == 8)) return ARP_ERR_ARG;
  for (int c = 0; c < ncls; ++c) {
    const arp_mixed_class& m = cls[c];
    const int rc = check_dd(m.Gt, m.h, m.T, m.L, 2, m.R, m.D, m.B, m.inst, m.start, m.out_s, m.out_de, m.out_st);
    if (rc != ARP_OK) return rc;
  }
  const PhiloxKeys K = philox_keys(k0, k1);
  cudaStream_t st = (cudaStream_t)stream;
  for (int ns = 4; ns >= 1; --ns) {
    // this group's classes, in decreasing cost per problem
    int idx[kMaxMixed], n = 0, Lmax = 1;
    for (int c = 0; c < ncls; ++c)
      if ((cls[c].D + 31) / 32 == ns && cls[c].B > 0) idx[n++] = c;
    if (n == 0) continue;
    auto cost = [&](int c) { return (double)cls[c].L * cls[c].R * cls[c].D; };
    for (int i = 1; i < n; ++i)
      for (int j = i; j > 0 && cost(idx[j]) > cost(idx[j - 1]); --j) {
        const int t = idx[j];
        idx[j] = idx[j - 1];
        idx[j - 1] = t;
      }
    MixedArgs g;
    memset(&g, 0, sizeof(g));
    g.K = K;
    int total = 0;
    for (int i = 0; i < n; ++i) {
      const arp_mixed_class& m = cls[idx[i]];
      DDParams& a = g.cls[i];
      a.Gt = m.Gt;
      a.h = m.h;
      a.T = m.T;
      a.c = nullptr;
      a.L = m.L;
      a.qi = m.q;
      a.R = m.R;
      a.D = m.D;
      a.B = m.B;
      a.inst = m.inst;
      a.start = m.start;
      a.out_s = m.out_s;
      a.out_de = m.out_de;
      a.out_st = m.out_st;
      a.status = status;
      a.split = 1;
      a.m0 = nullptr;
      a.perm = nullptr;
      a.warm_r = 1 << 30;
      a.cdf = nullptr;
      a.ra = nullptr;
      g.first[i] = total;
      total += m.B;
      if (m.L > Lmax && m.L <= grp::kMaxSched) Lmax = m.L;
    }
    for (int i = n; i <= kMaxMixed; ++i) g.first[i] = total;
    g.total = total;
    cudaError_t e;
    switch (ns) {
      case 1: e = launch_mixed<1>(g, Lmax, warps, counters + 0, st); break;
      case 2: e = launch_mixed<2>(g, Lmax, warps, counters + 1, st); break;
      case 3: e = launch_mixed<3>(g, Lmax, warps, counters + 2, st); break;
      default: e = launch_mixed<4>(g, Lmax, warps, counters + 3, st); break;
    }
    if (e != cudaSuccess) return ARP_ERR_LAUNCH;
  }
  return ARP_OK;
}
