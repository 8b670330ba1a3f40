// Anneals on compressed dDI problems with FP32 fields, and the entry points of the integer anneals (anneal_group.cuh).
//
// Problem (arpeggio_ref59.py:41-85, chord_ref.py:72-123): the dDI coupling over N = P D spins is
// J = -offdiag(G (x) 1 1^T), so one lane field per coordinate, w_j = h_j - 2 (G m)_j with m = sum of the P
// copies, serves every copy: the field of spin (p, j) is w_j + 2 G_jj s_pj.
//
// Mapping (one warp = one anneal, lanes across threads): thread `lane` owns coordinates j = t*32 + lane for
// t < NS = ceil(D/32); its fields w[t] live in registers; spins are warp-uniform bit masks Sm[p][t]; G sits
// in shared memory transposed and zero-padded to NS*32 columns (Gs[j][i] = G[i][j]) so a flip of lane j
// streams one contiguous row.  A block holds one problem and W warps that take anneals r = w, w + W, ...
//
// First accept, exactly the reference's index-order scan: every remaining lane of the active copy tests
// against the current fields at once, a ballot + ffs picks the first accepted lane j, the flip commits
// (rank-1 update of every field from row j), and lanes after j re-test with the same draws.  Lanes that
// rejected before j stay rejected, as in the sequential scan, because their decision came before the flip.
// Chord: one snapshot test of the active copy, then the accepted lanes commit in index order.
//
// RNG: Philox4x32-10 with the reference's counters -- start (2^32-1, p*D+j, r, inst) word 0 ('rand') or
// (2^32-1, j, r, inst) ('bal'); pass k = n*P + p uses word n&3 of block (n>>2, p*D+j, r, inst).  One block
// serves four sweeps, so each quad of sweeps computes P*NS blocks per thread once (registers) instead of
// one block per test (the reference's arpeggio_fx.cu:75).
#include <climits>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "arp_common.cuh"
#include "arp_internal.h"

namespace arp {


constexpr int32_t kMaxG = 1 << 18, kMaxH = 1 << 28, kMaxT = 1 << 26;
constexpr int kMaxDevices = 64;

template <int NS, int P, bool CHORD, bool FLT, bool CACHE>
__global__ void __launch_bounds__(256) k_anneal_dd(const DDParams a) {
  using FT = typename std::conditional<FLT, float, int32_t>::type;
  using ET = typename std::conditional<FLT, float, long long>::type;
  constexpr int DP = NS * 32;
  extern __shared__ __align__(16) unsigned char smem[];
  FT* Gs = reinterpret_cast<FT*>(smem);
  __shared__ int s_bad;
  const int D = a.D, L = a.L, R = a.R;
  const int split = a.split, b = blockIdx.x / split, bs = blockIdx.x - b * split;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, W = blockDim.x >> 5;
  pdl_trigger();
  pdl_wait();
  if (threadIdx.x == 0) s_bad = 0;
  __syncthreads();
  {
    const FT* Gg = reinterpret_cast<const FT*>(a.Gt) + (size_t)b * D * D;
    bool bad = false;
    for (int x = threadIdx.x; x < D * DP; x += blockDim.x) {
      const int j = x / DP, i = x - j * DP;
      const FT v = i < D ? Gg[(size_t)j * D + i] : FT(0);
      if constexpr (!FLT) bad |= (v > kMaxG || v < -kMaxG);
      Gs[x] = v;
    }
    if constexpr (!FLT) {
      const int32_t* hg = reinterpret_cast<const int32_t*>(a.h) + (size_t)b * D;
      for (int x = threadIdx.x; x < D; x += blockDim.x) bad |= (hg[x] > kMaxH || hg[x] < -kMaxH);
      const int32_t* Tg = reinterpret_cast<const int32_t*>(a.T);
      const int32_t* cg = reinterpret_cast<const int32_t*>(a.c);
      for (int x = threadIdx.x; x < L; x += blockDim.x) {
        bad |= (Tg[x] > kMaxT || Tg[x] < -kMaxT);
        if (cg) bad |= (cg[x] > kMaxT || cg[x] < -kMaxT);
      }
      bad |= (a.qi > kMaxT || a.qi < -kMaxT);
    }
    if (bad) s_bad = 1;
  }
  __syncthreads();
  if (s_bad) {
    if (threadIdx.x == 0) set_status(a.status, ARP_ERR_RANGE);
    return;
  }
  const uint32_t inst = a.inst ? a.inst[b] : a.inst0 + (uint32_t)b;
  FT dg[NS], hv[NS];
  uint32_t vmask[NS];
#pragma unroll
  for (int t = 0; t < NS; ++t) {
    const int j = t * 32 + lane;
    const int nv = D - t * 32;
    vmask[t] = nv >= 32 ? ARP_FULL : (nv > 0 ? (1u << nv) - 1u : 0u);
    dg[t] = j < D ? Gs[j * DP + j] : FT(0);
    hv[t] = j < D ? reinterpret_cast<const FT*>(a.h)[(size_t)b * D + j] : FT(0);
  }
  const FT* Tg = reinterpret_cast<const FT*>(a.T);
  const FT* cg = reinterpret_cast<const FT*>(a.c);

  for (int r = bs + split * wid; r < R; r += split * W) {
    uint32_t Sm[P][NS], Bm[P][NS];
    // ---- start state (arpeggio_fx.cu:48-57)
    if (a.start == 0) {
#pragma unroll
      for (int p = 0; p < P; ++p)
#pragma unroll
        for (int t = 0; t < NS; ++t) {
          uint32_t c0 = 0xFFFFFFFFu, c1 = (uint32_t)(p * D + t * 32 + lane), c2 = (uint32_t)r, c3 = inst;
          philox10(c0, c1, c2, c3, a.k0, a.k1);
          Sm[p][t] = __ballot_sync(ARP_FULL, c0 >= 0x80000000u) & vmask[t];
        }
    } else {
#pragma unroll
      for (int t = 0; t < NS; ++t) {
        uint32_t c0 = 0xFFFFFFFFu, c1 = (uint32_t)(t * 32 + lane), c2 = (uint32_t)r, c3 = inst;
        philox10(c0, c1, c2, c3, a.k0, a.k1);
        const int pat = bal_pattern(P, (uint32_t)(((uint64_t)c0 * (uint64_t)bal_choose(P)) >> 32));
#pragma unroll
        for (int p = 0; p < P; ++p) Sm[p][t] = __ballot_sync(ARP_FULL, (pat >> p) & 1) & vmask[t];
      }
    }
    // ---- lane fields w = h - 2 G m (arpeggio_fx.cu:58-66); float: sum in j order, one rounding per op
    FT w[NS];
    FT acc[NS];
#pragma unroll
    for (int t = 0; t < NS; ++t) acc[t] = FT(0);
#pragma unroll
    for (int tj = 0; tj < NS; ++tj) {
      for (int l = 0; l < 32; ++l) {
        const int j = tj * 32 + l;
        if (j >= D) break;
        int m = 0;
#pragma unroll
        for (int p = 0; p < P; ++p) m += ((Sm[p][tj] >> l) & 1u) ? 1 : -1;
        if (m == 0) continue;
        const FT* gr = Gs + j * DP + lane;
#pragma unroll
        for (int t = 0; t < NS; ++t) {
          if constexpr (FLT)
            acc[t] = __fadd_rn(acc[t], __fmul_rn(gr[t * 32], (float)m));
          else
            acc[t] += gr[t * 32] * m;
        }
      }
    }
#pragma unroll
    for (int t = 0; t < NS; ++t) {
      if constexpr (FLT)
        w[t] = __fsub_rn(hv[t], __fmul_rn(2.0f, acc[t]));
      else
        w[t] = hv[t] - 2 * acc[t];
    }
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int t = 0; t < NS; ++t) Bm[p][t] = Sm[p][t];

    ET de = ET(0), best;
    if constexpr (FLT)
      best = __int_as_float(0x7f800000);
    else
      best = 1LL << 62;
    long long flips = 0, tests = 0;
    const int nquad = (L + 4 * P - 1) / (4 * P);
    for (int q4 = 0; q4 < nquad; ++q4) {
      uint32_t cw[CACHE ? P : 1][CACHE ? NS : 1][4];
      if constexpr (CACHE) {
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
          for (int t = 0; t < NS; ++t) {
            uint32_t c0 = (uint32_t)q4, c1 = (uint32_t)(p * D + t * 32 + lane), c2 = (uint32_t)r, c3 = inst;
            philox10(c0, c1, c2, c3, a.k0, a.k1);
            cw[p][t][0] = c0;
            cw[p][t][1] = c1;
            cw[p][t][2] = c2;
            cw[p][t][3] = c3;
          }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const int k = (q4 * 4 + i) * P + p;
          if (k >= L) break;
          // ---- per-lane thresholds for this pass
          FT th[NS];
          FT qk;
          if constexpr (FLT) {
            const float A = __fmul_rn(4.0f, Tg[k]);
            qk = (CHORD && cg) ? __fsub_rn(a.qf, cg[k]) : a.qf;
#pragma unroll
            for (int t = 0; t < NS; ++t) {
              uint32_t u;
              if constexpr (CACHE) {
                u = cw[p][t][i];
              } else {
                uint32_t c0 = (uint32_t)q4, c1 = (uint32_t)(p * D + t * 32 + lane), c2 = (uint32_t)r, c3 = inst;
                philox10(c0, c1, c2, c3, a.k0, a.k1);
                u = i == 0 ? c0 : (i == 1 ? c1 : (i == 2 ? c2 : c3));
              }
              th[t] = __fmul_rn(__fsub_rn(unit24(u), 0.5f), A);
            }
          } else {
            const int32_t Tk = Tg[k];
            const long long A = 4LL * Tk;
            const int32_t Bk = a.qi + 2 * Tk - ((CHORD && cg) ? cg[k] : 0);
#pragma unroll
            for (int t = 0; t < NS; ++t) {
              uint32_t u;
              if constexpr (CACHE) {
                u = cw[p][t][i];
              } else {
                uint32_t c0 = (uint32_t)q4, c1 = (uint32_t)(p * D + t * 32 + lane), c2 = (uint32_t)r, c3 = inst;
                philox10(c0, c1, c2, c3, a.k0, a.k1);
                u = i == 0 ? c0 : (i == 1 ? c1 : (i == 2 ? c2 : c3));
              }
              th[t] = ((vmask[t] >> lane) & 1u) ? (int32_t)ceil_shift32(u, A) - 2 * dg[t] - Bk : INT_MIN;
            }
            qk = 0;
          }
          // ---- the test of one lane against the current fields
          auto accept = [&](int t) -> bool {
            const FT sw = ((Sm[p][t] >> lane) & 1u) ? w[t] : -w[t];
            if constexpr (FLT)
              return __fadd_rn(__fadd_rn(sw, __fmul_rn(2.0f, dg[t])), qk) < th[t];
            else
              return sw < th[t];
          };
          // ---- commit a flip of lane l of slot t (fields after earlier commits)
          auto commit = [&](FT wsel, FT dsel, uint32_t sbits, int j, int l) {
            const FT wj = __shfl_sync(ARP_FULL, wsel, l);
            const FT dj = __shfl_sync(ARP_FULL, dsel, l);
            const int so = ((sbits >> l) & 1u) ? 1 : -1;
            if constexpr (FLT)
              de = __fadd_rn(de, __fadd_rn(__fmul_rn((float)(4 * so), wj), __fmul_rn(8.0f, dj)));
            else
              de += 4LL * so * wj + 8LL * dj;
            const FT* gr = Gs + j * DP + lane;
#pragma unroll
            for (int t = 0; t < NS; ++t) {
              if constexpr (FLT)
                w[t] = __fadd_rn(w[t], __fmul_rn((float)(4 * so), gr[t * 32]));
              else
                w[t] += 4 * so * gr[t * 32];
            }
            ++flips;
          };
          if constexpr (!CHORD) {
            // the scan finishes slot t (positions 32 t .. 32 t + 31) before slot t + 1: a round accepts only after
            // the last flip, so a slot the scan has left has no candidate left this pass
            long long tt = 1;
#pragma unroll
            for (int t = 0; t < NS; ++t) {
              uint32_t rem = vmask[t];
              for (;;) {
                const uint32_t m = __ballot_sync(ARP_FULL, accept(t)) & rem;
                if (m == 0) break;
                const int l = __ffs(m) - 1;
                const int j = t * 32 + l;
                commit(w[t], dg[t], Sm[p][t], j, l);
                const uint32_t bit = 1u << l;
                Sm[p][t] ^= bit;
                rem &= ~((bit << 1) - 1u);
                if (j < D - 1) ++tt;
              }
            }
            tests += tt;
          } else {
            uint32_t am[NS];
#pragma unroll
            for (int t = 0; t < NS; ++t) am[t] = __ballot_sync(ARP_FULL, accept(t)) & vmask[t];
#pragma unroll
            for (int t = 0; t < NS; ++t) {
              uint32_t m = am[t];
              while (m) {
                const int l = __ffs(m) - 1;
                m &= m - 1u;
                commit(w[t], dg[t], Sm[p][t], t * 32 + l, l);
              }
              Sm[p][t] ^= am[t];
            }
            tests += 1;
          }
          if (de < best) {  // best state after each pass (arpeggio_fx.cu:90-93)
            best = de;
#pragma unroll
            for (int pp = 0; pp < P; ++pp)
#pragma unroll
              for (int t = 0; t < NS; ++t) Bm[pp][t] = Sm[pp][t];
          }
        }
      }
    }
    // ---- outputs (arpeggio_fx.cu:95-99)
    const size_t ar = (size_t)b * R + r;
    int8_t* os = a.out_s + ar * P * D;
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int t = 0; t < NS; ++t) {
        const int j = t * 32 + lane;
        if (j < D) os[p * D + j] = ((Bm[p][t] >> lane) & 1u) ? 1 : -1;
      }
    if (lane == 0) {
      reinterpret_cast<ET*>(a.out_de)[ar] = best;
      a.out_st[2 * ar] = flips;
      a.out_st[2 * ar + 1] = tests;
    }
  }
}

// Warps per block: a block holds one problem and its warps share the anneals, so fewer warps per block let
// more blocks (problems) share an SM.  Pick the width with the most resident warps per SM for this kernel's
// registers and shared memory (ties go to the wider block, which loads G fewer times per anneal).
template <typename K>
static int pick_warps(K kern, size_t smem, int R) {
  int best_w = 1, best_res = -1;
  for (int w = 1; w <= 8; w *= 2) {
    if (w > R && w > 1) break;
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, 32 * w, smem) != cudaSuccess) return R < 8 ? R : 8;
    const int res = nb * w;
    if (res >= best_res) {
      best_res = res;
      best_w = w;
    }
  }
  return best_w;
}

// Warps per block chosen by a caller's autotuner per (slots NS, copies P, policy: first accept, Chord round, warm
// first accept, FP32 fields); 0 = occupancy heuristic.  Process-wide, set through arp_anneal_tune.
static int g_tuned_warps[5][7][3][2];

int tuned_warps(int NS, int P, int policy, int precision) { return g_tuned_warps[NS][P][policy][precision]; }

template <int NS, int P, bool CHORD>
static cudaError_t launch_ns_p(const DDParams& a, int warps, cudaStream_t st) {
  const auto kern = k_anneal_dd<NS, P, CHORD, true, P * NS <= 8>;
  const size_t smem = (size_t)a.D * NS * 32 * 4;
  // Launch settings per device (the shared-memory limit raised by cudaFuncSetAttribute applies to the current
  // device only; occupancy and SM count are per device too), behind one lock per instantiation.
  struct Slot {
    size_t attr_smem = 48 * 1024, cached_smem = 0;
    int cached_w = 0, cached_nb = 0, sms = 0;
  };
  static Slot slots_by_dev[kMaxDevices];
  static std::mutex mu;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  int per_sm = 1, sms = 0;
  {
    std::lock_guard<std::mutex> lock(mu);
    Slot& sl = slots_by_dev[dev];
    if (smem > sl.attr_smem) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      sl.attr_smem = smem;
    }
    if (warps <= 0 && (sl.cached_w == 0 || sl.cached_smem != smem)) {
      sl.cached_w = pick_warps(kern, smem, 8);
      sl.cached_smem = smem;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&sl.cached_nb, kern, 32 * sl.cached_w, smem) != cudaSuccess)
        sl.cached_nb = 1;
      cudaDeviceGetAttribute(&sl.sms, cudaDevAttrMultiProcessorCount, dev);
    }
    per_sm = sl.cached_nb > 0 ? sl.cached_nb : 1;
    sms = sl.sms;
    if (warps <= 0) {
      warps = sl.cached_w;
      const int tw = tuned_warps(NS, P, CHORD ? 1 : 0, 1);
      if (tw > 0 && tw != warps) {  // same resident warps per SM, another width
        per_sm = sl.cached_nb * sl.cached_w / tw > 0 ? sl.cached_nb * sl.cached_w / tw : 1;
        warps = tw;
      }
      while (warps > 1 && warps > a.R) warps >>= 1;
    }
  }
  // Small batches: split each problem's anneals over several blocks so the batch still fills the GPU.
  DDParams b = a;
  b.split = 1;
  const long long slots = (long long)per_sm * (sms > 0 ? sms : 148);
  if ((long long)a.B < slots) {
    const int most = (a.R + warps - 1) / warps;
    long long sp = (slots + a.B - 1) / a.B;
    b.split = (int)(sp < most ? sp : most);
    if (b.split < 1) b.split = 1;
  }
  return launch_ex(kern, dim3((unsigned)((long long)a.B * b.split)), dim3(warps * 32), smem, st, false, b);
}

template <bool CHORD>
static cudaError_t launch_f32(const DDParams& a, int P, int warps, cudaStream_t st) {
  const int NS = (a.D + 31) / 32;
#define ARP_CASE(ns, pp) \
  if (NS == ns && P == pp) return launch_ns_p<ns, pp, CHORD>(a, warps, st);
  ARP_CASE(1, 2) ARP_CASE(1, 4) ARP_CASE(1, 6)
  ARP_CASE(2, 2) ARP_CASE(2, 4) ARP_CASE(2, 6)
  ARP_CASE(3, 2) ARP_CASE(3, 4) ARP_CASE(3, 6)
  ARP_CASE(4, 2) ARP_CASE(4, 4) ARP_CASE(4, 6)
#undef ARP_CASE
  return cudaErrorInvalidValue;
}

int check_dd(const void* Gt, const void* h, const void* T, int L, int P, int R, int D, int B,
                    const uint32_t* inst, int start, const int8_t* out_s, const void* out_de, const int64_t* out_st) {
  if (B < 0 || R < 1 || D < 1 || D > 128 || L < 1 || !(P == 2 || P == 4 || P == 6)) return ARP_ERR_SHAPE;
  if (start != 0 && start != 1) return ARP_ERR_ARG;
  if (B > 0 && (!Gt || !h || !T || !inst || !out_s || !out_de || !out_st)) return ARP_ERR_ARG;
  return ARP_OK;
}

int default_warps(int R) { return 0; }  // 0: chosen per kernel by occupancy (pick_warps)

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
  if (flt) return policy == 0 ? launch_f32<false>(a, P, warps, st) : launch_f32<true>(a, P, warps, st);
  if (warps <= 0) warps = tuned_warps((a.D + 31) / 32, P, policy, 0);
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

