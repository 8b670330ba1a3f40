// Integer anneals on compressed dDI problems, several anneals per warp: first accept (plain, warm-started) and the
// Chord round (Philox numbers, or the reference's C++ engine model's own).
//
// Problem (arpeggio_ref59.py:41-85, chord_ref.py:72-123): the dDI coupling over N = P D spins is
// J = -offdiag(G (x) 1 1^T), so one lane field per coordinate, w_j = h_j - 2 (G m)_j with m = sum of the P copies,
// serves every copy: the field of spin (p, j) is w_j + 2 G_jj s_pj.
//
// Mapping.  A warp runs A = 32 / LN anneals of one problem at once, LN lanes each; a lane holds C coordinates of its
// anneal, j = c LN + li for slot c, with the first coordinate of a slot on the highest lane of the group.  What a flip
// costs is mostly the scan around it (test, ballot, first set bit, broadcast: about 18 instructions of a warp,
// whatever the coordinates per lane) and what an idle pass costs is mostly its loop; holding more coordinates per lane
// lets one round of these serve a flip of every anneal of the warp.  Groups whose own slot has no candidate left idle
// in a round (it runs while any group has one), which bounds how far this goes.  Measured per 8192 32-user uses
// (32 anneals x 64 passes): one anneal per warp with two coordinates per lane 4.2 ms (the previous kernel; 3.7 ms in
// this form), two anneals with four 3.2 ms, four anneals with eight 2.9 ms; in instructions per anneal 14.6 k, 12.7 k
// (this form), 10.6 k, 9.76 k.  The issue slots bound it (79 % busy at 32 resident warps per SM).
//
// Margins.  For its copy's spin s a lane adds x = s ? ~e : e to w on entering a slot, with e = kappa - 2 G_jj - 1 and
// kappa = ceil(u 4T / 2^32) - q - 2T (+ c): then z = (w + x) XOR (s up ? 0 : -1) equals psi - kappa, psi = s w + 2 G_jj,
// in both cases.  The reference's decision u 4T > (s w + 2 G_jj + q + 2T) 2^32 (arpeggio_fx.cu:76-79) is psi < kappa,
// i.e. z < 0; a flip moves every field by 4 s_flipped G_ij, one multiply-add with a factor that is the same for the
// whole group, and the energy by 4 psi.  First accept: the ballot over the lanes below the last commit gives each group
// its first acceptance; rejected lanes stay rejected, as in the sequential scan, because their decision came before
// the flip, and a slot the scan has left has no candidate left this pass.  Chord: one snapshot of every slot, then the
// accepted lanes commit in index order with psi of the fields after the earlier commits.
//
// RNG: Philox4x32-10 with the reference's counters -- start (2^32-1, p*D+j, r, inst) word 0 ('rand') or
// (2^32-1, j, r, inst) ('bal'); pass k = n*P + p uses word n&3 of block (n>>2, p*D+j, r, inst).  One block serves four
// sweeps; the four sweeps' thresholds ceil(u 4T / 2^32) < 2^16 wait in shared memory, 16 bits each (eight coordinates
// x two copies x four sweeps would be 64 registers a lane as words), written and read by the same lane.
//
// Ranges.  |G| <= 2^18, |h| <= 2^28, |T|, |q|, |c| <= 2^26 keep every field, margin and threshold inside int32
// (ARP_ERR_RANGE otherwise).  Problems whose pass sums fit 32 bits (every fixed-point problem of to_fixed, where |G|,
// |h| <= 4096) and whose schedule has 0 <= T < 2^14 and at most kMaxSched passes run with the stored thresholds, and with a
// 32-bit running energy where that fits too; the others run the same scan with 64-bit energies and one Philox block per
// pass (WIDE).
#pragma once
#include <climits>
#include <mutex>
#include <type_traits>

#include "arp_common.cuh"
#include "arp_internal.h"

namespace arp {
namespace grp {

constexpr int32_t kMaxG = 1 << 18, kMaxH = 1 << 28, kMaxT = 1 << 26;
constexpr int kMaxSched = 8192;  // passes whose (4T, q + 2T - c) are staged in shared memory (64 KB)
constexpr int kFineSched = 1024;  // above, the room is rounded up to this many passes
constexpr int kMaxDevices = 64;

enum Rule { kFirst, kWarm, kChord, kEngine };

// The random numbers of the reference's C++ engine model run without Philox (arpeggio/sim/x3model/engine_model.cpp,
// philox = 0): murmur-style mixing steps for the per-anneal seed chain and the lane seeds, xorshift32 per lane.
__device__ __forceinline__ uint32_t eng_mix_a(uint32_t v) { return (v ^ (v >> 16)) * 0x85EBCA6Bu; }
__device__ __forceinline__ uint32_t eng_mix_b(uint32_t v) { return (v ^ (v >> 13)) * 0xC2B2AE35u; }
__device__ __forceinline__ uint32_t eng_fin(uint32_t v) { return v ^ (v >> 16); }
__device__ __forceinline__ uint32_t eng_xs32(uint32_t x) {
  x ^= x << 13;
  x ^= x >> 17;
  x ^= x << 5;
  return x;
}

// d = a b + c with a 32 x 32 -> 64-bit signed product.
__device__ __forceinline__ long long mad_wide_s32(int32_t a, int32_t b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}
// Index of the highest set bit, -1 (0xFFFFFFFF) for 0.
__device__ __forceinline__ int high_bit(uint32_t x) {
  int r;
  asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(x));
  return r;
}
__device__ __forceinline__ uint32_t sm32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// A row of G in shared memory holds a lane's C entries side by side, in planes of four slots (one 16-byte load), then
// two, then one: position of slot c of group lane ln.
template <int LN, int C>
__device__ __forceinline__ int row_pos(int c, int ln) {
  if (c < (C & ~3)) return (c >> 2) * 4 * LN + ln * 4 + (c & 3);
  if ((C & 2) && c < (C & ~1)) return (C & ~3) * LN + ln * 2 + (c & 1);
  return (C & ~1) * LN + ln;
}
// A lane's C entries of the row at shared address `row`.
template <int LN, int C>
__device__ __forceinline__ void load_row(uint32_t row, int ln, int32_t (&g)[C]) {
#pragma unroll
  for (int q = 0; q < C / 4; ++q)
    asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(g[4 * q]), "=r"(g[4 * q + 1]), "=r"(g[4 * q + 2]), "=r"(g[4 * q + 3])
                 : "r"(row + (uint32_t)ln * 16u + q * LN * 16));
  if constexpr (C & 2)
    asm volatile("ld.shared.v2.s32 {%0, %1}, [%2];"
                 : "=r"(g[C & ~3]), "=r"(g[(C & ~3) + 1])
                 : "r"(row + (uint32_t)ln * 8u + (C & ~3) * LN * 4));
  if constexpr (C & 1)
    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(g[C - 1]) : "r"(row + (uint32_t)ln * 4u + (C & ~1) * LN * 4));
}

// The block's anneals of problem b: warp `wid` of block share bs takes A at a time.  Rb: anneals to run (<= R).
template <int LN, int C, int P, Rule RULE, bool WIDE, bool SUM64 = WIDE>
__device__ __forceinline__ void run(const DDParams& a, const PhiloxKeys& K, const int b, const int bs,
                                    const int32_t* Gs, const int2* sched, uint32_t* words, const uint8_t* s_perm,
                                    const uint32_t inst, const int Rb) {
  constexpr int A = 32 / LN, DP = LN * C;
  constexpr bool CHORD = RULE == kChord || RULE == kEngine, WARM = RULE == kWarm, ENG = RULE == kEngine;
  // Margins of every slot formed before the scan, which is skipped when no lane has a candidate, instead of slot by
  // slot inside it: more registers for fewer serial steps.  Small problems, whose passes are mostly empty (8 users:
  // 0.82 -> 0.76 ms per 16384 uses), and the 512-thread blocks, which have the registers (64 users: 3.40 -> 3.31 ms per
  // 1024 uses); where 64 registers are the limit it loses (32 users: 2.94 -> 3.51 ms per 8192 uses).
  constexpr bool AHEAD = LN == 32 && !WIDE;
  constexpr bool HOIST = LN == 4 || LN * C > 64;
  // One anneal per warp: where its latency is what counts (up to two coordinates a lane), or the reduction would be of
  // 64 bits (five steps of two shuffles), a flip's psi goes to every lane by a shuffle beside its factor's and no
  // reduction stands between one pass and the next.  64 sweeps, chain of map, anneal and readout, with the reduction
  // against without: one 32-user frame 86.9 -> 81.4 us, one 8-user frame 37.1 -> 33.9, 40 9-user frames 58.9 -> 53.7.  By
  // Chord only with two copies and 32 bits: passes with many flips pay per flip (120 32-user uses of four copies, 16
  // anneals, 128 passes: 139 us with the reduction, 164 without).
  constexpr bool SPREAD = LN == 32 && (CHORD ? !WIDE && C <= 2 && P == 2 : WIDE || C <= 2);
  static_assert(P * C <= 32, "a lane's spins are one 32-bit word");
  static_assert(!ENG || WIDE, "the engine's numbers have no stored thresholds");
  using ET = typename std::conditional<WIDE, long long, int32_t>::type;   // a pass's sum
  using DT = typename std::conditional<SUM64, long long, int32_t>::type;  // the running energy and the best
  const int D = a.D, L = a.L, R = a.R, split = a.split;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int ln = lane & (LN - 1), grp = lane / LN;
  const int li = LN - 1 - ln;
  const uint32_t gmask = (LN == 32 ? ARP_FULL : ((1u << (LN & 31)) - 1u)) << (grp * LN);
  const int32_t* hg = reinterpret_cast<const int32_t*>(a.h) + (size_t)b * D;
  const int32_t* Tg = reinterpret_cast<const int32_t*>(a.T);
  const int32_t* cg = reinterpret_cast<const int32_t*>(a.c);
  uint32_t lmask = 0;  // the bits of coordinate D - 1 on its lane
  {
    const int cl = (D - 1) / LN;
    if (D - 1 - cl * LN == li)
#pragma unroll
      for (int p = 0; p < P; ++p) lmask |= 1u << (p * C + cl);
  }
  const uint32_t g0 = sm32(Gs) + (uint32_t)((LN - 1 + grp * LN) * DP * 4);
  const uint32_t wl = sm32(words) + (uint32_t)(wid * (P * C * 64) + lane) * 4u;
  const uint32_t sc = sm32(sched);
  for (int r0 = (bs + split * wid) * A; r0 < Rb; r0 += split * W * A) {
    const int r = r0 + grp;
    const bool live = r < Rb;
    // ---- start state (arpeggio_fx.cu:48-57): bit p C + c of dn is set where copy p of the lane's slot c is down
    uint32_t dn = 0;
    uint32_t es[ENG ? C : 1];  // the engine's per-coordinate generator states
    if constexpr (ENG) {  // (engine_model.cpp:185-194, 170-184, 142-163): bits 31, 30, ... start copies 0, 1, ...
      constexpr uint32_t PHI = 0x9E3779B9u;
      uint32_t f = eng_fin(eng_mix_b(eng_mix_a(a.k0 ^ inst)));
      f = eng_fin(eng_mix_b(eng_mix_a(f ^ a.k1)));
      f = eng_fin(eng_mix_b(eng_mix_a(f ^ (uint32_t)r)));
      const uint32_t seed = f + PHI;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const uint32_t v = eng_fin(eng_mix_b(eng_mix_a(seed + (uint32_t)(c * LN + li) * PHI)));
        es[c] = eng_xs32(v == 0 ? PHI : v);
#pragma unroll
        for (int p = 0; p < P; ++p)
          if (!((es[c] >> (31 - p)) & 1u)) dn |= 1u << (p * C + c);
      }
    } else if (WARM || a.start != 0) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int j = c * LN + li;
        uint32_t c0 = 0xFFFFFFFFu, c1 = (uint32_t)j, c2 = (uint32_t)r, c3 = inst;
        philox10(c0, c1, c2, c3, K);
        int mv = 0;  // spin sum: 0 takes the 'bal' pattern of the draw, else copies p < (m + P)/2 are up
        if constexpr (WARM) {
          if (j < D && r < a.warm_r) {
            if (a.cdf && r > 0) {  // a sampled start: the draw against the coordinate's thresholds
              const uint2 th = reinterpret_cast<const uint2*>(a.cdf)[(size_t)b * D + s_perm[j]];
              mv = c1 < th.x ? -2 : (c1 > th.y ? 2 : 0);
            } else {
              mv = a.m0[(size_t)b * D + s_perm[j]];
            }
          }
          mv = mv < -P ? -P : (mv > P ? P : mv);
        }
        const int pat = mv == 0 ? bal_pattern(P, (uint32_t)(((uint64_t)c0 * (uint64_t)bal_choose(P)) >> 32))
                                : (1 << ((mv + P) >> 1)) - 1;
#pragma unroll
        for (int p = 0; p < P; ++p)
          if (!((pat >> p) & 1)) dn |= 1u << (p * C + c);
      }
    } else {
#pragma unroll
      for (int p = 0; p < P; ++p)
#pragma unroll
        for (int c = 0; c < C; ++c) {
          uint32_t c0 = 0xFFFFFFFFu, c1 = (uint32_t)(p * D + c * LN + li), c2 = (uint32_t)r, c3 = inst;
          philox10(c0, c1, c2, c3, K);
          if (c0 < 0x80000000u) dn |= 1u << (p * C + c);
        }
    }
    // ---- fields w = h - 2 G m (arpeggio_fx.cu:58-66); dg = 2 G_jj + 1.  A padding coordinate (and every coordinate
    //      of a group without an anneal) keeps w = 0 and gets dg = 2^29 + 1, so its margin is above every threshold
    int32_t w[C], dg[C], m2[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int j = c * LN + li;
      int d = 0;
#pragma unroll
      for (int p = 0; p < P; ++p) d += (dn >> (p * C + c)) & 1u;
      const bool in = j < D;
      m2[c] = in ? 2 * (P - 2 * d) : 0;
      w[c] = in ? hg[WARM ? (int)s_perm[j] : j] : 0;
      dg[c] = (in && live ? 2 * Gs[j * DP + row_pos<LN, C>(c, ln)] : (1 << 29)) + 1;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
      // every spin sum of the slot 0 in every anneal of the warp ('bal' with two copies; most slots of a warm start):
      // nothing to add (3000 64-user uses from 'bal', 33 anneals x 24 sweeps, 3985 -> 3800 us); not asked of random starts
      // (65536 32-user uses, 32 anneals: 22.75 ms asking, 22.36 not), nor by Chord, whose passes are many and lose more to
      // the code it makes (700 18-user uses of six copies 334 -> 318 us, a 32-user use with T = 5 115 -> 108)
      if (!CHORD && (WARM || a.start != 0) && !__any_sync(ARP_FULL, m2[c] != 0)) continue;
#pragma unroll(LN == 32 ? 4 : 2)
      for (int i = 0; i < (LN == 32 ? min(LN, D - c * LN) : LN); ++i) {  // coordinate c LN + i, on lane LN - 1 - i
        const int32_t m = __shfl_sync(ARP_FULL, m2[c], LN - 1 - i, LN);
        int32_t g[C];
        load_row<LN, C>(sm32(Gs) + (uint32_t)((c * LN + i) * DP * 4), ln, g);
#pragma unroll
        for (int t = 0; t < C; ++t) w[t] -= m * g[t];
      }
    }
    if (!live) {
#pragma unroll
      for (int c = 0; c < C; ++c) w[c] = 0;
    }
    // energies in units of psi (a quarter of out_de); the engine's best register starts at 2^35 - 1
    DT de = 0, best = ENG ? (DT)(1LL << 33) : sizeof(DT) == 8 ? (DT)(1LL << 60) : (DT)INT_MAX;
    uint32_t bdn = dn;
    int32_t flips = 0, lastflips = 0, n1 = 0;
    int k = 0;
    for (int q4 = 0; k < L; ++q4) {
      if constexpr (!WIDE) {
        // thresholds ceil(u 4T / 2^32) of the quad's four sweeps, 16 bits each, sweeps (0, 1) and (2, 3) in a word
#pragma unroll(C * P <= 8 ? P : LN == 32 ? 2 : 1)
        for (int p = 0; p < P; ++p) {
          uint32_t t4[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(t4[i]) : "r"(sc + (uint32_t)((k + i * P + p) * 8)));
#pragma unroll
          for (int c = 0; c < C; ++c) {
            uint32_t x[4] = {(uint32_t)q4, (uint32_t)(p * D + c * LN + li), (uint32_t)r, inst};
            philox10(x[0], x[1], x[2], x[3], K);
            uint32_t hi[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) hi[i] = (uint32_t)(((uint64_t)x[i] * t4[i] + 0xFFFFFFFFull) >> 32);
            const uint32_t o = wl + (uint32_t)((p * C + c) * 256);
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(o), "r"(__byte_perm(hi[0], hi[1], 0x5410)) : "memory");
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(o + 128u), "r"(__byte_perm(hi[2], hi[3], 0x5410)) : "memory");
          }
        }
      }
      // one anneal per warp: the next pass's thresholds and B are loaded a pass ahead (nothing else hides their latency)
      int32_t hn[AHEAD ? C : 1], Bn = 0;
      auto ahead = [&](int i, int p, int kk) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          uint16_t hi;
          asm volatile("ld.shared.u16 %0, [%1];"
                       : "=h"(hi)
                       : "r"(wl + (uint32_t)((i & 1) * 2 + (i >> 1) * 128 + (p * C + c) * 256)));
          hn[AHEAD ? c : 0] = hi;
        }
        asm volatile("ld.shared.s32 %0, [%1];" : "=r"(Bn) : "r"(sc + (uint32_t)(kk * 8 + 4)));
      };
      if constexpr (AHEAD) ahead(0, 0, k);
      for (int i = 0; i < 4 && k < L; ++i) {
        const uint32_t wp = wl + (uint32_t)((i & 1) * 2 + (i >> 1) * 128);
        uint32_t fb = 0;  // the sweep's flips, bits as dn
#pragma unroll
        for (int p = 0; p < P; ++p) {
          if (k >= L) break;
          int32_t Bk, Tk = 0, hc[AHEAD ? C : 1];
          if constexpr (AHEAD) {
            Bk = Bn;
#pragma unroll
            for (int c = 0; c < C; ++c) hc[c] = hn[c];
            if (p + 1 < P)
              ahead(i, p + 1, k + 1);
            else if (i < 3)
              ahead(i + 1, 0, k + 1);
          } else if constexpr (WIDE) {
            Tk = Tg[k];
            Bk = a.qi + 2 * Tk - ((CHORD && cg) ? cg[k] : 0);
          } else {
            asm volatile("ld.shared.s32 %0, [%1];" : "=r"(Bk) : "r"(sc + (uint32_t)(k * 8 + 4)));
          }
          ET e = 0;
          auto kappa = [&](int c) -> int32_t {  // ceil(u 4T / 2^32) of slot c
            if constexpr (ENG) {  // advanced once per step, 16-bit draws: ceil(u 4T / 2^16) (engine_model.cpp:229-257)
              es[c] = eng_xs32(es[c]);
              return (int32_t)(((long long)(es[c] >> 16) * (4LL * Tk) + 0xFFFFLL) >> 16);
            } else if constexpr (WIDE) {
              // 4T as a 32-bit pattern: u A + 2^32 - 1 < 2^64, and for T < 0 the pattern adds u 2^32, taken back
              uint32_t c0 = (uint32_t)q4, c1 = (uint32_t)(p * D + c * LN + li), c2 = (uint32_t)r, c3 = inst;
              philox10(c0, c1, c2, c3, K);
              const uint32_t u = i == 0 ? c0 : (i == 1 ? c1 : (i == 2 ? c2 : c3));
              const uint32_t hi = (uint32_t)(((uint64_t)u * (4u * (uint32_t)Tk) + 0xFFFFFFFFull) >> 32);
              return (int32_t)(hi - (Tk < 0 ? u : 0u));
            } else if constexpr (AHEAD) {
              return hc[c];
            } else {
              uint16_t hi;
              asm volatile("ld.shared.u16 %0, [%1];" : "=h"(hi) : "r"(wp + (uint32_t)((p * C + c) * 256)));
              return (int32_t)hi;
            }
          };
          // whether the pass may have flipped (known for free with one anneal per warp and in the skipped scan)
          bool any = LN != 32 || k == 0;
          // one round of slot c: every group with a candidate (acc on some lane of m) flips its first
          auto commit = [&](int c, bool acc, uint32_t m, int32_t s4, int32_t psi, int& jl) {
            const int32_t v = acc ? s4 : 0;
            const int l = high_bit(m & gmask);  // -1 in a group without one: reads its last lane's v, which is 0
            const int32_t so4 = __shfl_sync(ARP_FULL, v, l, LN);
            int32_t g[C];
            load_row<LN, C>(g0 + c * LN * DP * 4 - (uint32_t)l * (DP * 4), ln, g);
#pragma unroll
            for (int t = 0; t < C; ++t) w[t] += so4 * g[t];
            if constexpr (SPREAD) {
              de += __shfl_sync(ARP_FULL, psi, l);
              if (lane == l) fb |= 1u << (p * C + c);
            } else if (lane == l) {
              if constexpr (WIDE)
                e = mad_wide_s32(psi, 1, e);
              else
                e += psi;
              fb |= 1u << (p * C + c);
            }
            jl = l;
            if constexpr (LN == 32 && !SPREAD) any = true;
          };
          if constexpr (!CHORD && HOIST) {
            int32_t x[C], zs = 0;
#pragma unroll
            for (int c = 0; c < C; ++c) {
              const int32_t sm = -(int32_t)((dn >> (p * C + c)) & 1u);
              x[c] = (kappa(c) - Bk - dg[c]) ^ ~sm;
              w[c] += x[c];
              zs |= w[c] ^ sm;
            }
            any = __any_sync(ARP_FULL, zs < 0) || k == 0;
            if (any) {
#pragma unroll
              for (int c = 0; c < C; ++c) {
                const int32_t sm = -(int32_t)((dn >> (p * C + c)) & 1u);
                const int32_t s4 = (sm & -8) ^ 4;
                int jl = 32;
                for (;;) {
                  const int32_t z = w[c] ^ sm;
                  const bool acc = z < 0 && lane < jl;
                  const uint32_t m = __ballot_sync(ARP_FULL, acc);
                  if (m == 0) break;
                  commit(c, acc, m, s4, z + (x[c] ^ ~sm) + dg[c], jl);
                }
              }
            }
#pragma unroll
            for (int c = 0; c < C; ++c) w[c] -= x[c];
          } else if constexpr (!CHORD) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
              const int32_t sm = -(int32_t)((dn >> (p * C + c)) & 1u);
              const int32_t hi = kappa(c);
              const int32_t x = (hi - Bk - dg[c]) ^ ~sm;
              const int32_t s4 = (sm & -8) ^ 4;
              w[c] += x;
              int jl = 32;
              for (;;) {
                const int32_t z = w[c] ^ sm;
                const bool acc = z < 0 && lane < jl;
                const uint32_t m = __ballot_sync(ARP_FULL, acc);
                if (m == 0) break;
                commit(c, acc, m, s4, z + hi - Bk, jl);
              }
              w[c] -= x;
            }
          } else {
            uint32_t snap = 0;
#pragma unroll
            for (int c = 0; c < C; ++c) {
              const int32_t sm = -(int32_t)((dn >> (p * C + c)) & 1u);
              const int32_t x = (kappa(c) - Bk - dg[c]) ^ ~sm;
              const int32_t z = (w[c] + x) ^ sm;
              if (z < 0) snap |= 1u << c;
            }
            uint32_t mb[C], ma = 0;  // one anneal per warp: the slots' ballots at once, a quiet pass takes one branch
            if constexpr (SPREAD) {
#pragma unroll
              for (int c = 0; c < C; ++c) ma |= mb[c] = __ballot_sync(ARP_FULL, (snap >> c) & 1u);
            }
            if (!SPREAD || ma != 0) {
#pragma unroll
              for (int c = 0; c < C; ++c) {
                const int32_t sm = -(int32_t)((dn >> (p * C + c)) & 1u);
                const int32_t s4 = (sm & -8) ^ 4;
                const bool sn = (snap >> c) & 1u;
                int jl = 32;
                if constexpr (LN == 32) {  // one anneal: its flips are the ballot's bits
                  for (uint32_t m = SPREAD ? mb[c] : __ballot_sync(ARP_FULL, sn); m != 0; m &= (1u << jl) - 1u)
                    commit(c, true, m, s4, (w[c] ^ sm) - sm + dg[c] - 1, jl);  // psi = s w + 2 G_jj
                } else {
                  for (;;) {
                    const bool acc = sn && lane < jl;
                    const uint32_t m = __ballot_sync(ARP_FULL, acc);
                    if (m == 0) break;
                    commit(c, acc, m, s4, (w[c] ^ sm) - sm + dg[c] - 1, jl);
                  }
                }
              }
            }
            if (a.out_n1) n1 += (__ballot_sync(ARP_FULL, (fb >> (p * C)) != 0) & gmask) != 0;
          }
          if (SPREAD || any) {
            if constexpr (LN == 32 && !SPREAD && !WIDE) {
              de += __reduce_add_sync(ARP_FULL, e);
            } else if constexpr (!SPREAD) {
#pragma unroll
              for (int o = LN / 2; o; o >>= 1) e += __shfl_xor_sync(ARP_FULL, e, o);
              de += e;
            }
            if (de < best) {  // best state after each pass (arpeggio_fx.cu:90-93)
              best = de;
              bdn = dn ^ fb;
            }
          }
          ++k;
        }
        dn ^= fb;
        flips += __popc(fb);
        lastflips += __popc(fb & lmask);
      }
    }
#pragma unroll
    for (int o = LN / 2; o; o >>= 1) {
      flips += __shfl_xor_sync(ARP_FULL, flips, o);
      lastflips += __shfl_xor_sync(ARP_FULL, lastflips, o);
    }
    if (live) {
      const size_t ar = (size_t)b * R + r;
      int8_t* os = a.out_s + ar * P * D;
#pragma unroll
      for (int p = 0; p < P; ++p)
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int j = c * LN + li;
          if (j < D) os[p * D + (WARM ? (int)s_perm[j] : j)] = ((bdn >> (p * C + c)) & 1u) ? -1 : 1;
        }
      if (ln == 0) {
        // every anneal runs all L passes; first accept reports flips + 1 tests per pass, less one when the last
        // coordinate flipped
        reinterpret_cast<long long*>(a.out_de)[ar] = (ENG && (long long)best == (1LL << 33)) ? (1LL << 35) - 1 : 4LL * best;
        a.out_st[2 * ar] = flips;
        a.out_st[2 * ar + 1] = CHORD ? L : L + flips - lastflips;
        if (CHORD && a.out_n1) a.out_n1[ar] = n1;
      }
    }
  }
}

// Dynamic shared memory: G (DP x DP), the schedule, the warps' thresholds.  A group without a candidate reads (and
// multiplies by zero) up to 33 - LN rows beyond G, so the block's allocation covers those.
template <int LN, int C>
__host__ __device__ constexpr size_t g_bytes() {
  return (size_t)LN * C * LN * C * 4;
}
template <int P>
__host__ __device__ inline size_t sched_bytes(int L) {
  constexpr int Q = 4 * P;  // a quad of sweeps
  return L <= kFineSched ? (size_t)((L + Q - 1) / Q * Q * 8)
         : L <= kMaxSched ? (size_t)((L + kFineSched - 1) / kFineSched * kFineSched + Q) * 8 : 0;
}
// STORED: with the thresholds' room (the engine's numbers have none).
template <int LN, int C, int P, bool STORED = true>
inline size_t smem_bytes(int L, int W) {
  const size_t s = g_bytes<LN, C>() + sched_bytes<P>(L) + (STORED ? (size_t)W * P * C * 256 : 0);
  const size_t rows = ((size_t)(C - 1) * LN + 33) * LN * C * 4;
  return s > rows ? s : rows;
}

// One problem b of a block: G and the schedule staged in shared memory, then the block's anneals.  Called by the
// per-launch kernel (one problem per block) and by the persistent mixed-size kernel (problems taken from a work
// counter, one after another).
template <int LN, int C, int P, Rule RULE>
__device__ __forceinline__ void problem(const DDParams& a, const PhiloxKeys& K, const int b, const int bs) {
  constexpr int DP = LN * C;
  constexpr bool CHORD = RULE == kChord || RULE == kEngine, WARM = RULE == kWarm;
  extern __shared__ __align__(16) unsigned char smem[];
  int32_t* Gs = reinterpret_cast<int32_t*>(smem);
  __shared__ int s_bad, s_wt;
  __shared__ uint32_t s_mg, s_mh;
  __shared__ uint8_t s_perm[WARM ? 128 : 1];
  const int D = a.D, L = a.L, R = a.R, bt = blockDim.x;
  int2* sched = reinterpret_cast<int2*>(smem + g_bytes<LN, C>());
  uint32_t* words = reinterpret_cast<uint32_t*>(smem + g_bytes<LN, C>() + sched_bytes<P>(L));
  if (threadIdx.x == 0) {
    s_bad = 0;
    s_mg = 0;
    s_mh = 0;
    s_wt = 0;
  }
  const int32_t* hg = reinterpret_cast<const int32_t*>(a.h) + (size_t)b * D;
  const int32_t* Tg = reinterpret_cast<const int32_t*>(a.T);
  const int32_t* cg = reinterpret_cast<const int32_t*>(a.c);
  const int32_t* Gg = reinterpret_cast<const int32_t*>(a.Gt) + (size_t)b * D * D;
  uint32_t mg = 0, mh = 0;  // largest |G|, |h| (as unsigned: |INT_MIN| = 2^31)
  bool bad = false;
  // G by 16-byte loads, eight in flight per thread.  By 4-byte loads, a row per warp, where the matrix is not 16-byte aligned
  // or D no multiple of 4 (an odd number of users); for one anneal per warp (small batches, whose instructions come cold
  // from L2 in every frame: less code, 1.5 us less for a 32-user frame than the unrolled loop); and for a scan order, where
  // a lane gathers its columns of each row.
  const bool vec = !WARM && LN < 32 && (D & 3) == 0 && (reinterpret_cast<uintptr_t>(Gg) & 15u) == 0;
  const int D4 = D >> 2, nv = vec ? D * D4 : 0;
  int4 v[8];
  auto fetch = [&](int x0) {
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (x0 + u * bt < nv) v[u] = reinterpret_cast<const int4*>(Gg)[x0 + u * bt];
  };
  fetch(threadIdx.x);
  // the first of the thread's h, T and c and the instance number travel beside G
  const int x1 = threadIdx.x;
  const int32_t h1 = x1 < D ? hg[x1] : 0, t1 = x1 < L ? Tg[x1] : 0, c1 = (CHORD && cg && x1 < L) ? cg[x1] : 0;
  const uint32_t inst = a.inst ? a.inst[b] : a.inst0 + (uint32_t)b;
  if constexpr (WARM) {
    // position j' of the scan holds coordinate perm[j']: G and h are gathered into that order
    for (int x = threadIdx.x; x < D; x += bt) {
      const uint8_t pv = a.perm[(size_t)b * D + x];
      bad |= pv >= D;  // reported as ARP_ERR_RANGE, never dereferenced
      s_perm[x] = pv < D ? pv : 0;
    }
  }
  __syncthreads();
  auto put = [&](int j, int i, int32_t g) {  // entry (j, i) into its place
    mg = max(mg, (uint32_t)abs(g));
    Gs[j * DP + row_pos<LN, C>(i / LN, LN - 1 - (i & (LN - 1)))] = g;
  };
  for (int x0 = threadIdx.x; x0 < nv; x0 += 8 * bt) {
    if (x0 != (int)threadIdx.x) fetch(x0);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int x = x0 + u * bt;
      if (x >= nv) break;
      const int j = D == DP ? x / (DP / 4) : x / D4, i = 4 * (x - j * D4);
      put(j, i, v[u].x);
      put(j, i + 1, v[u].y);
      put(j, i + 2, v[u].z);
      put(j, i + 3, v[u].w);
    }
  }
  if (WARM || LN == 32 || !vec) {  // a row per warp, four rows in flight
    constexpr int CW = (DP + 31) / 32;
    const int lane = threadIdx.x & 31, W = bt >> 5;
    int col[CW];
#pragma unroll
    for (int c = 0; c < CW; ++c) col[c] = WARM && c * 32 + lane < D ? s_perm[c * 32 + lane] : c * 32 + lane;
#pragma unroll 1
    for (int j0 = threadIdx.x >> 5; j0 < D; j0 += 4 * W) {
      int32_t g[4][CW];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = j0 + u * W, row = (WARM && j < D ? s_perm[j] : j) * D;
#pragma unroll
        for (int c = 0; c < CW; ++c) g[u][c] = (j < D && c * 32 + lane < D) ? Gg[row + col[c]] : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int c = 0; c < CW; ++c)
          if (j0 + u * W < D && c * 32 + lane < D) put(j0 + u * W, c * 32 + lane, g[u][c]);
    }
  }
  for (int x = threadIdx.x; x < D * (DP - D); x += bt) {  // padding columns
    const int j = x / (DP - D), i = D + x - j * (DP - D);
    Gs[j * DP + row_pos<LN, C>(i / LN, LN - 1 - (i & (LN - 1)))] = 0;
  }
  for (int x = x1; x < D; x += bt) mh = max(mh, (uint32_t)abs(x == x1 ? h1 : hg[x]));
  const int Lp = L <= kMaxSched ? (L + 4 * P - 1) / (4 * P) * 4 * P : L;
  for (int x = threadIdx.x; x < Lp; x += bt) {
    const int32_t t = x == x1 ? t1 : x < L ? Tg[x] : 0;
    const int32_t cv = x == x1 ? c1 : (x < L && CHORD && cg) ? cg[x] : 0;
    bad |= t > kMaxT || t < -kMaxT || cv > kMaxT || cv < -kMaxT;
    if (t < 0 || t >= (1 << 14)) s_wt = 1;
    if (L <= kMaxSched) sched[x] = make_int2(4 * t, a.qi + 2 * t - cv);
  }
  bad |= (a.qi > kMaxT || a.qi < -kMaxT);
  mg = __reduce_max_sync(ARP_FULL, mg);
  mh = __reduce_max_sync(ARP_FULL, mh);
  bad |= mg > (uint32_t)kMaxG || mh > (uint32_t)kMaxH;
  if (bad) s_bad = 1;
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&s_mg, mg);
    atomicMax(&s_mh, mh);
  }
  __syncthreads();
  if (s_bad) {
    if (threadIdx.x == 0) set_status(a.status, ARP_ERR_RANGE);
    return;
  }
  int Rb = R;
  if constexpr (WARM) {
    if (a.ra) {  // a per-problem anneal count: the skipped anneals report the guess
      const int v = a.ra[b], split = a.split;
      Rb = v < 1 ? 1 : (v > R ? R : v);
      for (int r = Rb + bs; r < R; r += split) {
        const size_t ar = (size_t)b * R + r;
        for (int x = threadIdx.x; x < P * D; x += blockDim.x) a.out_s[ar * P * D + x] = 0;
        if (threadIdx.x == 0) {
          reinterpret_cast<long long*>(a.out_de)[ar] = LLONG_MAX;
          a.out_st[2 * ar] = 0;
          a.out_st[2 * ar + 1] = 0;
        }
      }
    }
  }
  if constexpr (RULE == kEngine) {
    run<LN, C, P, RULE, true>(a, K, b, bs, Gs, sched, words, s_perm, inst, Rb);
  } else {
    // What max |G| = 4096, a fixed-point problem's, puts beyond 32 bits: (2 P D + 2) 4096 P D >= 2^30 from P D = 362, two
    // bits for the forms compiled (1: 32-bit sums, 2: 64-bit ones of 32-bit passes).  Six copies below 61 coordinates lose
    // 4 % with the wider sums (2000 30-user uses by Chord 829 -> 862 us), at 64 they gain (1409 -> 949; 64-bit throughout before).
    constexpr int SUMS = LN * C * P <= 361 ? 1 : (P == 6 && DP == 64) || (P == 4 && DP == 96) ? 3 : 2;
    // |psi| <= |h| + (2 P D + 2) max |G| at any state; a pass adds at most D of them and the energy of any state
    // stays within D P / 2 of them, so below 2^30 / (D P) every sum fits 32 bits, below 2^30 / D those of a pass
    const long long psi = (long long)s_mh + (2LL * P * D + 2) * s_mg;
    const bool pass = psi * D < (1LL << 30) && !s_wt && L <= kMaxSched;
    if ((SUMS & 1) && pass && psi * D * P < (1LL << 30))
      run<LN, C, P, RULE, false>(a, K, b, bs, Gs, sched, words, s_perm, inst, Rb);
    else if ((SUMS & 2) && pass)
      run<LN, C, P, RULE, false, true>(a, K, b, bs, Gs, sched, words, s_perm, inst, Rb);
    else
      run<LN, C, P, RULE, true>(a, K, b, bs, Gs, sched, words, s_perm, inst, Rb);
  }
}

template <int LN, int C>
constexpr int max_threads() {
  return LN == 16 && C > 4 ? 512 : 256;  // 64 KB of G at D = 128: one block of 16 warps per SM
}
// Resident blocks the registers are bounded for where the batch fills the GPU: 64 a thread, 128 for the 512-thread
// blocks and for one anneal per warp with three or more coordinates a lane.
template <int LN, int C>
constexpr int min_blocks() {
  return max_threads<LN, C>() == 512 ? 1 : LN == 32 && C >= 3 ? 2 : 4;
}

template <int LN, int C, int P, Rule RULE, int MB>
__global__ void __launch_bounds__(max_threads<LN, C>(), MB) k_anneal_grp(const DDParams a) {
  const int split = a.split, b = blockIdx.x / split, bs = blockIdx.x - b * split;
  pdl_trigger();
  pdl_wait();
  problem<LN, C, P, RULE>(a, *reinterpret_cast<const PhiloxKeys*>(a.rk0), b, bs);
}

// Per device: a kernel's resident blocks per SM at each block width (1, 2, 4, 8, 16 warps) for every shared-memory layout
// it was launched with (one per staged schedule length), and the dynamic shared memory it may use.  A launch with a
// layout met before asks the runtime nothing; nothing is allocated.
constexpr int kLayouts = kFineSched / 8 + kMaxSched / kFineSched + 1;
struct Widths {
  std::mutex mu;
  struct Dev {
    size_t limit = 0;  // 0: the 48 KB of every kernel
    int sms = 0;
    struct {
      bool known;
      int8_t nb[5];
    } layout[kLayouts] = {};
  } dev[kMaxDevices];
};
// The number of schedule length L's layout: its quads of sweeps or, of a long one, its thousands; 0 where it is not staged.
template <int P>
inline int layout_of(int L) {
  static_assert(P >= 2, "at least eight passes a quad");
  return L <= kFineSched  ? (L + 4 * P - 1) / (4 * P)
         : L <= kMaxSched ? kFineSched / 8 + (L + kFineSched - 1) / kFineSched : 0;
}
constexpr size_t kMinDynamic = 48 * 1024, kMaxDynamic = 226 * 1024;

// Launches kern for the A anneals per warp and blocks of at most WMAX warps it was compiled for; smem(W): its dynamic
// shared memory with blocks of W warps, layout: a number below kLayouts that differs where smem does.
template <int A, int WMAX, typename Kern, typename Smem>
static cudaError_t launch_widths(Widths& wd, Kern kern, int layout, Smem smem, const DDParams& a, int warps,
                                 cudaStream_t st) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(wd.mu);
  Widths::Dev& d = wd.dev[dev];
  const auto limit = [&](size_t bytes) {
    d.limit = bytes;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  auto& known = d.layout[layout];
  const int8_t* nb = known.nb;
  if (!known.known) {
    if ((e = cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const size_t was = d.limit;
    if ((e = limit(kMaxDynamic)) != cudaSuccess) return e;
    for (int i = 0; i < 5; ++i) {
      int n = 0;
      known.nb[i] = 0;
      if ((1 << i) > WMAX || smem(1 << i) > kMaxDynamic) continue;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, 32 << i, smem(1 << i));
      if (e != cudaSuccess) return e;
      known.nb[i] = (int8_t)n;
    }
    if ((e = limit(was > kMinDynamic ? was : kMinDynamic)) != cudaSuccess) return e;
    known.known = true;
  }
  const int sms = d.sms;
  // the width with the most resident warps per SM (ties: the wider block, which stages G fewer times per anneal),
  // or the caller's; no wider than the problem's anneals need
  int wi = 0;
  for (int i = 1; i < 5; ++i)
    if (nb[i] && (nb[i] << i) >= (nb[wi] << wi)) wi = i;
  if (warps > 0)
    for (wi = 4; wi > 0 && ((1 << wi) > warps || nb[wi] == 0);) --wi;
  while (wi > 0 && (1 << (wi - 1)) * A >= a.R) --wi;
  // one anneal per warp, every block resident at once: blocks of eight warps, or of four where those leave fewer warps on
  // the fullest SM (one 32-user frame: 44 us against 46 with eight; 37 26-user frames, 33 anneals a use, in the chain
  // of map, anneal and readout: 70 against 75; 64 32-user frames: 69 against 63 with eight); above 16 warps a SM not in a
  // programmatic launch, whose blocks wait beside the map's: 60 17-user uses of 33 in that chain 63.8 us with four, 56.7 with
  // eight (the kernel before 53.6), 64 32-user uses of 64 82.1 and 74.0 (104.1)
  const bool beside = a.B <= kPdlMaxB && a.B * (long long)((a.R + 7) / 8 * 8) > 16LL * sms;
  if (A == 1 && warps <= 0 && (wi == 2 || wi == 3) && a.R > 4 && !beside) {
    const auto fullest = [&](int W) { return (a.B * (long long)((a.R + W - 1) / W) + sms - 1) / sms; };
    if (fullest(8) <= nb[3] && fullest(4) <= nb[2]) wi = 4 * fullest(4) < 8 * fullest(8) ? 2 : 3;
  }
  if (nb[wi] == 0) return cudaErrorInvalidConfiguration;
  const int W = 1 << wi;
  // small batches: each problem's anneals over several blocks, as many as make the call shortest in anneals one after
  // another per warp times waves of blocks (each further block stages the problem once more)
  DDParams b = a;
  b.split = 1;
  const double slots = (double)nb[wi] * sms;
  const int most = (a.R + W * A - 1) / (W * A);
  double best = 0.0;
  for (int s = 1; a.B < 4 * slots && s <= most && s * (long long)a.B < 8 * slots + a.B; ++s) {
    // (per-problem counts: a second wave of a few long blocks counts whole; 473 49-user warm uses of 16, 128 passes, at low
    // SNR 1524 -> 1187 us, the kernel before 1235; 600 32-user ones of 32 379 -> 341, at high SNR 258 -> 236)
    const double full = a.B * s / slots, waves = a.ra && full > 1.0 && full <= 1.3 ? 2.0 : full;
    const double cost = ((a.R + W * A * s - 1) / (W * A * s)) * (waves > 1.0 ? waves : 1.0) + 0.02 * s;
    if (s == 1 || cost < best) {
      best = cost;
      b.split = s;
    }
  }
  if (smem(W) > (d.limit > kMinDynamic ? d.limit : kMinDynamic) && (e = limit(smem(W))) != cudaSuccess) return e;
  return launch_ex(kern, dim3((unsigned)((long long)a.B * b.split)), dim3(W * 32), smem(W), st, a.B <= kPdlMaxB, b);
}

template <int LN, int C, int P, Rule RULE, int MB = min_blocks<LN, C>()>
static cudaError_t launch(const DDParams& a, int warps, cudaStream_t st) {
  static Widths wd;
  return launch_widths<32 / LN, max_threads<LN, C>() / 32>(
      wd, k_anneal_grp<LN, C, P, RULE, MB>, layout_of<P>(a.L),
      [&](int W) { return smem_bytes<LN, C, P, RULE != kEngine>(a.L, W); }, a, warps, st);
}

// How many anneals share a warp is a matter of how many there are: A per warp need A times as many to fill the GPU.
// Warps of a call up to which one anneal per warp is the fastest: what the unbounded kernels (about 100 registers at two
// coordinates a lane) and the ones bound to 64 registers keep resident at once, 16 and 32 a SM; then anneals up to
// which half the full mapping's anneals per warp win, by coordinates.  32 anneals a use, one / two / four per warp at
// 64 coordinates: 64 uses 63 / 83 / 126 us, 148 uses 121 / 108 / 143, 600 uses 387 / 296 / 308, 1200 uses
// 727 / 522 / 512; one / two / four at 32: 156 uses 56 / 54 / 63, 312 uses 93 / 75 / 75, 625 uses 184 / 147 / 121;
// two / four / eight at 16: 156 uses 31 / 35 / 47, 625 uses 84 / 65 / 68, 1250 uses 133 / 106 / 103.  Above 16 coordinates one
// per warp keeps its lead into a short second wave (37 warps a SM for 32): 76 and 83 14-user uses of 64 anneals in the
// chain of map, anneal and readout 74 -> 67 and 79 -> 78 us, 120 21-user uses of 33 104 -> 93.
constexpr long long kLatWarps = 148LL * 16, kOnePerWarp = 148LL * 37;
// (by registers: 12 a SM with two coordinates a lane and four or six copies, 8 above 64 coordinates; 120 60-user uses of
// four copies, 16 anneals: 72 -> 57 us with the bound kernel; the kernel before 56)
template <int P>
inline long long lat_warps(int D) {
  return D > 64 ? kLatWarps / 2 : P > 2 && D > 32 ? kLatWarps * 3 / 4 : kLatWarps;
}
constexpr long long kMid16 = 30000, kMid32 = 10000, kMid64 = 148LL * 32 * 8;

// The mapping (LN lanes per anneal, C coordinates per lane) for D coordinates.  P = 6 keeps four coordinates a lane
// (24 spin bits); the engine's numbers use the same family.
template <int P, Rule RULE>
static cudaError_t dispatch(const DDParams& a, int warps, cudaStream_t st) {
  const int D = a.D;
  const long long n = (long long)a.B * a.R, w8 = (long long)a.B * ((a.R + 7) / 8 * 8);
  // (above 64 coordinates an unbounded block fills the SM's registers, half the warps; there one per warp at 128 registers)
  // Two anneals per warp fill the GPU with 2 kLatWarps of them, one per warp with half as many: just above a whole number
  // of the first's waves the finer steps of the second leave less of the last wave empty (5000 to 7100 anneals of 126
  // coordinates: Chord 248 -> 230 us, first accept 264 -> 253; of 90 coordinates 177 -> 168), at 64 anneals a use also
  // above the second wave (9600 to 14000: 431 -> 390, 275 -> 260; at 32 a use 386 against 396, so not there).
  const bool ragged = (w8 > 2 * kLatWarps && w8 <= 3 * kLatWarps) ||
                      (a.R >= 64 && w8 > 4 * kLatWarps && w8 <= 6 * kLatWarps);
  // And so for a count that fills its last block of 16 badly, at any size: 34000 anneals of 90 coordinates, 33 a use, Chord
  // 1200 -> 1060 us, first accept 1510 -> 1365; below 16 a use there are too few warps beside 64 KB of G.
  const bool waste = (a.R + 15) / 16 * 128 > a.R * 9;
  const bool start = RULE == kChord && w8 <= kLatWarps * 5 / 4;  // just above one per warp's first wave: 224 -> 207 us
  // Per-problem counts, most of them a few anneals in blocks of a few warps: the two-per-warp kernels of 128 coordinates,
  // bound for blocks of 16 warps, keep two of them an SM, one per warp four (3000 53-user uses, 16 anneals, easy ones 4:
  // 2667 -> 2420 us; 64-user ones 2705 -> 2440).  Up to 96 coordinates two per warp stay ahead (1790 against 1830).
  const bool counted = RULE == kWarm && a.ra && D > 96;
  // Four copies above 96 coordinates, up to 16 anneals: eight two-per-warp warps' thresholds (64 KB beside as much of G)
  // leave one block an SM, one per warp two (1000 64-user uses of 16: first accept 621 -> 479 us, Chord 1120 -> 856).
  const bool room = P == 4 && D > 96 && a.R <= 16;
  if constexpr (RULE != kEngine && P < 6)
    if (D > 64 && w8 > kLatWarps / 2 && (w8 <= kLatWarps || ragged || waste || start || counted || room))
      return D <= 96 ? launch<32, 3, P, RULE>(a, warps, st) : launch<32, 4, P, RULE>(a, warps, st);
  if (RULE != kEngine && w8 <= lat_warps<P>(D))
    return D <= 32   ? launch<32, 1, P, RULE, 1>(a, warps, st)
           : D <= 64 ? launch<32, 2, P, RULE, 1>(a, warps, st)
           : D <= 96 ? launch<32, 3, P, RULE, 1>(a, warps, st)
                     : launch<32, 4, P, RULE, 1>(a, warps, st);
  if (w8 <= (D > 16 ? kOnePerWarp : 148LL * 32) && D <= 64)
    return D <= 32 ? launch<32, 1, P, RULE>(a, warps, st) : launch<32, 2, P, RULE>(a, warps, st);
  // few anneals a use leave a wide block's warps without work: the half mapping below 16
  if (D <= 16 && (n <= kMid16 || a.R < 16)) return launch<8, 2, P, RULE>(a, warps, st);
  if (D <= 32 && D > 16 && (n <= kMid32 || a.R < 16)) return launch<16, 2, P, RULE>(a, warps, st);
  if (D <= 16) return launch<4, 4, P, RULE>(a, warps, st);
  if (D <= 32) return launch<8, 4, P, RULE>(a, warps, st);
  if constexpr (RULE == kEngine || P == 6) {
    return D <= 64   ? launch<16, 4, P, RULE>(a, warps, st)
           : D <= 96 ? launch<32, 3, P, RULE>(a, warps, st)
                     : launch<32, 4, P, RULE>(a, warps, st);
  } else {
    // (warm-started anneals: most problems run a few anneals each, which four to a warp would leave on one warp of the
    // block; 32768 32-user uses 8.28 -> 7.99 ms, 2741 uses 0.84 -> 0.78)
    if (D <= 64 && D > 48 && RULE == kWarm && a.R < 64) return launch<16, 4, P, RULE>(a, warps, st);
    if (D <= 64 && (n <= kMid64 || a.R < 16)) return launch<16, 4, P, RULE>(a, warps, st);
    return D <= 48   ? launch<8, 6, P, RULE>(a, warps, st)
           : D <= 64 ? launch<8, 8, P, RULE>(a, warps, st)
           : D <= 96 ? launch<16, 6, P, RULE>(a, warps, st)
                     : launch<16, 8, P, RULE>(a, warps, st);
  }
}

}  // namespace grp
}  // namespace arp
