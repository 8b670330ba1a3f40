// Entry points of the anneals on compressed dDI problems: argument checks and the dispatch to the kernels of
// anneal_group.cuh (integer fields) and anneal_group_f32.cuh (FP32 fields), compiled one file per rule.
#include "arp_common.cuh"
#include "arp_internal.h"

namespace arp {

// Warps per block chosen by a caller's autotuner per (slots NS, copies P, policy: first accept, Chord round, warm
// first accept, FP32 fields); 0 = occupancy heuristic.  Process-wide, set through arp_anneal_tune.
static int g_tuned_warps[5][7][3][2];

int tuned_warps(int NS, int P, int policy, int precision) { return g_tuned_warps[NS][P][policy][precision]; }

int check_dd(const void* Gt, const void* h, const void* T, int L, int P, int R, int D, int B, const uint32_t* inst,
             int start, const int8_t* out_s, const void* out_de, const int64_t* out_st) {
  if (B < 0 || R < 1 || D < 1 || D > 128 || L < 1 || !(P == 2 || P == 4 || P == 6)) return ARP_ERR_SHAPE;
  if (start != 0 && start != 1) return ARP_ERR_ARG;
  if (B > 0 && (!Gt || !h || !T || !inst || !out_s || !out_de || !out_st)) return ARP_ERR_ARG;
  return ARP_OK;
}

int default_warps(int R) { return 0; }  // 0: chosen per kernel by occupancy

// The Philox round keys of (k0, k1), once per launch: the rounds read them as constant operands.
static DDParams with_keys(const DDParams& a0) {
  DDParams a = a0;
  const PhiloxKeys K = philox_keys(a.k0, a.k1);
  for (int i = 0; i < 10; ++i) {
    a.rk0[i] = K.k0[i];
    a.rk1[i] = K.k1[i];
  }
  return a;
}

cudaError_t anneal_dispatch(int policy, bool flt, const DDParams& a0, int P, int warps, cudaStream_t st) {
  const DDParams a = with_keys(a0);
  if (warps <= 0) warps = tuned_warps((a.D + 31) / 32, P, policy, flt ? 1 : 0);
  if (flt) return policy == 0 ? f32_first(a, P, warps, st) : f32_chord(a, P, warps, st);
  if (policy == 0) return P == 2 ? int_first2(a, warps, st) : int_first46(a, P, warps, st);
  return P == 2 ? int_chord2(a, warps, st) : int_chord46(a, P, warps, st);
}

// Warm-started first accept (integer fields, P = 2).
static cudaError_t launch_warm(const DDParams& a, cudaStream_t st) {
  return int_warm(with_keys(a), tuned_warps((a.D + 31) / 32, 2, 2, 0), st);
}

}  // namespace arp

using namespace arp;

extern "C" int arp_anneal_chord_engine(const int32_t* Gt, const int32_t* h, const int32_t* T, const int32_t* c,
                                       int L, int q, int P, int R, int D, int B, const uint32_t* inst, uint32_t k0,
                                       uint32_t k1, int8_t* out_s, int64_t* out_de, int64_t* out_st,
                                       int32_t* status, void* stream) {
  int rc = check_dd(Gt, h, T, L, P, R, D, B, inst, 0, out_s, out_de, out_st);
  if (rc || B == 0) return rc;
  DDParams a{Gt, h, T, c, L, q, 0.0f, R, D, B, inst, 0u, k0, k1, 0, out_s, out_de, out_st, status};
  return int_engine(a, P, (cudaStream_t)stream) == cudaSuccess ? ARP_OK : ARP_ERR_LAUNCH;
}

extern "C" int arp_anneal_first_accept(const int32_t* Gt, const int32_t* h, const int32_t* T, int L, int q, int P,
                                       int R, int D, int B, const uint32_t* inst, uint32_t k0, uint32_t k1,
                                       int start, int8_t* out_s, int64_t* out_de, int64_t* out_st,
                                       int32_t* status, void* stream) {
  int rc = check_dd(Gt, h, T, L, P, R, D, B, inst, start, out_s, out_de, out_st);
  if (rc || B == 0) return rc;
  DDParams a{Gt, h, T, nullptr, L, q, 0.0f, R, D, B, inst, 0u, k0, k1, start, out_s, out_de, out_st, status};
  return anneal_dispatch(0, false, a, P, default_warps(R), (cudaStream_t)stream) == cudaSuccess ? ARP_OK
                                                                                                : ARP_ERR_LAUNCH;
}

extern "C" int arp_anneal_chord_dd(const int32_t* Gt, const int32_t* h, const int32_t* T, const int32_t* c, int L,
                                   int q, int P, int R, int D, int B, const uint32_t* inst, uint32_t k0, uint32_t k1,
                                   int start, int8_t* out_s, int64_t* out_de, int64_t* out_st, int32_t* status,
                                   void* stream) {
  int rc = check_dd(Gt, h, T, L, P, R, D, B, inst, start, out_s, out_de, out_st);
  if (rc || B == 0) return rc;
  DDParams a{Gt, h, T, c, L, q, 0.0f, R, D, B, inst, 0u, k0, k1, start, out_s, out_de, out_st, status};
  return anneal_dispatch(1, false, a, P, default_warps(R), (cudaStream_t)stream) == cudaSuccess ? ARP_OK
                                                                                                : ARP_ERR_LAUNCH;
}

extern "C" int arp_anneal_chord_dd_n1(const int32_t* Gt, const int32_t* h, const int32_t* T, const int32_t* c, int L,
                                      int q, int P, int R, int D, int B, const uint32_t* inst, uint32_t k0,
                                      uint32_t k1, int start, int8_t* out_s, int64_t* out_de, int64_t* out_st,
                                      int64_t* out_n1, int32_t* status, void* stream) {
  int rc = check_dd(Gt, h, T, L, P, R, D, B, inst, start, out_s, out_de, out_st);
  if (rc || B == 0) return rc;
  if (!out_n1) return ARP_ERR_ARG;
  DDParams a{Gt, h, T, c, L, q, 0.0f, R, D, B, inst, 0u, k0, k1, start, out_s, out_de, out_st, status};
  a.out_n1 = out_n1;
  return anneal_dispatch(1, false, a, P, default_warps(R), (cudaStream_t)stream) == cudaSuccess ? ARP_OK
                                                                                                : ARP_ERR_LAUNCH;
}

extern "C" int arp_anneal_dd_f32(int policy, const float* Gt, const float* h, const float* T, const float* c, int L,
                                 float q, int P, int R, int D, int B, const uint32_t* inst, uint32_t k0, uint32_t k1,
                                 int start, int8_t* out_s, float* out_de, int64_t* out_st, int32_t* status,
                                 void* stream) {
  if (policy != 0 && policy != 1) return ARP_ERR_ARG;
  int rc = check_dd(Gt, h, T, L, P, R, D, B, inst, start, out_s, out_de, out_st);
  if (rc || B == 0) return rc;
  DDParams a{Gt, h, T, c, L, 0, q, R, D, B, inst, 0u, k0, k1, start, out_s, out_de, out_st, status};
  cudaError_t e = anneal_dispatch(policy, true, a, P, default_warps(R), (cudaStream_t)stream);
  return e == cudaSuccess ? ARP_OK : ARP_ERR_LAUNCH;
}

extern "C" int arp_anneal_first_accept_warm_sampled(const int32_t* Gt, const int32_t* h, const int32_t* T, int L,
                                                    int q, int P, int R, int D, int B, const uint32_t* inst,
                                                    uint32_t k0, uint32_t k1, const int8_t* m0, const uint32_t* cdf,
                                                    const uint8_t* perm, int warm_r, const int32_t* ra,
                                                    int8_t* out_s, int64_t* out_de, int64_t* out_st,
                                                    int32_t* status, void* stream) {
  int rc = check_dd(Gt, h, T, L, P, R, D, B, inst, 1, out_s, out_de, out_st);
  if (rc || B == 0) return rc;
  if (P != 2) return ARP_ERR_SHAPE;
  if (!m0 || !perm || !cdf || warm_r < 0) return ARP_ERR_ARG;
  DDParams a{Gt, h, T, nullptr, L, q, 0.0f, R, D, B, inst, 0u, k0, k1, 1, out_s, out_de, out_st, status};
  a.m0 = m0;
  a.perm = perm;
  a.warm_r = warm_r;
  a.cdf = cdf;
  a.ra = ra;
  return launch_warm(a, (cudaStream_t)stream) == cudaSuccess ? ARP_OK : ARP_ERR_LAUNCH;
}

extern "C" int arp_anneal_first_accept_warm_mix(const int32_t* Gt, const int32_t* h, const int32_t* T, int L, int q,
                                                int P, int R, int D, int B, const uint32_t* inst, uint32_t k0,
                                                uint32_t k1, const int8_t* m0, const uint8_t* perm, int warm_r,
                                                int8_t* out_s, int64_t* out_de, int64_t* out_st, int32_t* status,
                                                void* stream) {
  int rc = check_dd(Gt, h, T, L, P, R, D, B, inst, 1, out_s, out_de, out_st);
  if (rc || B == 0) return rc;
  if (P != 2) return ARP_ERR_SHAPE;
  if (!m0 || !perm || warm_r < 0) return ARP_ERR_ARG;
  DDParams a{Gt, h, T, nullptr, L, q, 0.0f, R, D, B, inst, 0u, k0, k1, 1, out_s, out_de, out_st, status};
  a.m0 = m0;
  a.perm = perm;
  a.warm_r = warm_r;
  return launch_warm(a, (cudaStream_t)stream) == cudaSuccess ? ARP_OK : ARP_ERR_LAUNCH;
}

extern "C" int arp_anneal_first_accept_warm(const int32_t* Gt, const int32_t* h, const int32_t* T, int L, int q, int P,
                                            int R, int D, int B, const uint32_t* inst, uint32_t k0, uint32_t k1,
                                            const int8_t* m0, const uint8_t* perm, int8_t* out_s, int64_t* out_de,
                                            int64_t* out_st, int32_t* status, void* stream) {
  int rc = check_dd(Gt, h, T, L, P, R, D, B, inst, 1, out_s, out_de, out_st);
  if (rc || B == 0) return rc;
  if (P != 2) return ARP_ERR_SHAPE;
  if (!m0 || !perm) return ARP_ERR_ARG;
  DDParams a{Gt, h, T, nullptr, L, q, 0.0f, R, D, B, inst, 0u, k0, k1, 1, out_s, out_de, out_st, status};
  a.m0 = m0;
  a.perm = perm;
  return launch_warm(a, (cudaStream_t)stream) == cudaSuccess ? ARP_OK : ARP_ERR_LAUNCH;
}

extern "C" int arp_anneal_tune(int D, int P, int policy, int precision, int warps) {
  if (D < 1 || D > 128 || !(P == 2 || P == 4 || P == 6) || policy < 0 || policy > 2 ||
      (precision != 0 && precision != 1) || (policy == 2 && (P != 2 || precision != 0)))
    return ARP_ERR_SHAPE;
  if (!(warps == 0 || warps == 1 || warps == 2 || warps == 4 || warps == 8)) return ARP_ERR_ARG;
  g_tuned_warps[(D + 31) / 32][P][policy][precision] = warps;
  return ARP_OK;
}

