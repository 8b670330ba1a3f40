// Trajectory soft output: Chord's synchronous rule as a sampler of the detection posterior on the RI map, with per-bit
// minima of ||y - H x||^2 over every visited state of every chain (the reference's mimo.chord_soft,
// arpeggio/mimo/mimo.py:332-394; the LLRs themselves are formed by arpeggio_b200.soft.trajectory_llr, mimo.py:397-413).
//
// Problem: N = nb D spins s = [s_MSB; s_LSB] (16-QAM, levels 2 s1 + s2) or N = D (QPSK), scaled J (B, N, N) with a
// zero diagonal, exploration field hf (the unregularised h0, or the RI field h), h0, scale and the distance constant
// c0 of ||y - H x||^2 = scale E0(s) + c0, E0(s) = -h0.s - s^T J s (mimo.energy0).
// Step k (temperature T[b][k], shared q): every spin tests the snapshot, z = s u + q against thr = (x/2^32 - 1/2) 4T
// with x the Philox word k & 3 of block (k >> 2, i, r, inst) (24-bit uniform, as the FP32 anneals), flips where
// z < thr; the flips commit in index order (u_i += -4 s_j J_ij, u_j after the earlier commits), E0 moving by
// 2 s_j (h0_j + u_j - hf_j) per flip.  After every step that flips (and step 0) the chain's distance
// d = scale E0 + c0 updates the minima m1 (bit = 1) and m0 (bit = 0) of each bit of the current levels (Gray bits:
// b1 = l > 0, b2 = |l| == 1, i.e. s1 > 0 and s1 != s2; QPSK b = s > 0) and the best state (lowest d; the earliest
// step, then the lowest chain, on ties).  One block per problem; the block reduces the minima over its chains.
//
// Mapping.  A step at the posterior's temperature flips a quarter to a half of the spins, and a flip is a serial round
// (find it, broadcast its field, one multiply-add per spin), so a warp runs A = 32 / LN chains at once, LN lanes each:
// lane li of a chain's group holds coordinates j = cc LN + li, as slot cc (the MSB spin j, or s) and, for 16-QAM, slot
// CD + cc (the LSB spin D + j), so slots and lanes ascend with the spin index and a coordinate's two spins share a
// lane.  A round commits one flip of every chain of the warp, and a slot's rounds are counted once (the largest number
// of flips among the chains) instead of voted on.  What bounds it is the rows of J: a flip reads one, two wavefronts
// of shared memory at 64 spins, and they keep its pipe 81 % busy (issue slots 67 %; 2018 instructions per step of four
// chains, 1826 per step of one before).  4096 16-user uses, 16 chains x 256 steps: 32.5 -> 11.1 ms.
// With few chains a problem's blocks are what is resident, so J takes a row per spin and columns to the next multiple of
// LN only (36 KB at 96 spins), and where it is large, or the problems few, four warps stage it though fewer run chains:
// 1400 24-user uses of one 64-step chain 2796 us with 64 KB rounded up to whole slots, 1927 with the rows (and four warps;
// one warp is as fast there, see launch_soft); of five 3171 and 2280.
// The reference draws its chains' start and tests from torch.rand; this sampler draws them from Philox counters of
// its own (start: word 0 of (2^32 - 1, i, r, inst), spin +1 iff >= 2^31), so its trajectories are its own while the
// rule, the visited-state bookkeeping and the LLR formation are the reference's.
#include <cfloat>
#include <climits>

#include "arp_common.cuh"
#include "arp_internal.h"

namespace arp {

struct SoftParams {
  const float *J, *hf, *h0, *scale, *c0, *T;  // T: (B, S) per-problem temperatures
  const int8_t* s0;                             // (B, N) start spins, or null: Philox
  float q;
  int S, R, N, D, M, B;
  const uint32_t* inst;
  float* m0;       // (B, D nb)
  float* m1;       // (B, D nb)
  float* best_d;   // (B)
  int8_t* best_l;  // (B, D)
  PhiloxKeys K;
};

constexpr int kSoftWarps = 8;

__device__ __forceinline__ int high_bit(uint32_t x) {  // -1 for 0
  int r;
  asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(x));
  return r;
}

// u[t] += cf g[t] where has != 0 (predicated: another chain's flip must not touch this one, not even by + 0 g; a branch
// around the row's loads and the sums costs more than the loads it saves, 4.5 -> 5.5 ms per 1024 uses).  cf is +-4, so
// the product is exact and the sum rounds once, as a multiply and an add (for |J| below 2^126).
template <int C>
__device__ __forceinline__ void axpy_if(int has, float cf, const float (&g)[C], float (&u)[C]) {
#pragma unroll
  for (int t = 0; t < C; t += 2)
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %4, 0;\n\t@p fma.rn.f32 %0, %5, %2, %0;\n\t@p fma.rn.f32 %1, %5, %3, %1;\n\t}"
        : "+f"(u[t]), "+f"(u[t + 1])
        : "f"(g[t]), "f"(g[t + 1]), "r"(has), "f"(cf));
}

template <int LN, int CD, bool QAM>
struct SoftMap {
  static constexpr int A = 32 / LN, C = QAM ? 2 * CD : CD, DP = LN * C, NB = QAM ? 2 : 1;
};

// A lane's C entries of a row lie side by side in planes of four slots (one 16-byte load), then two: position of slot c of
// group lane ln.
template <int LN, int C>
__device__ __forceinline__ int row_pos(int c, int ln) {
  return c < (C & ~3) ? (c >> 2) * 4 * LN + ln * 4 + (c & 3) : (C & ~3) * LN + ln * 2 + (c & 1);
}

template <int LN, int CD, bool QAM>
__global__ void __launch_bounds__(32 * kSoftWarps) k_traj_soft(const SoftParams a) {
  using M = SoftMap<LN, CD, QAM>;
  constexpr int A = M::A, C = M::C, DP = M::DP, NB = M::NB;
  extern __shared__ __align__(16) float sms[];
  const int N = a.N, D = a.D, S = a.S, R = a.R;
  // the first W warps run chains; a block of few chains has more, which help to stage J
  const int b = blockIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5, BW = blockDim.x >> 5;
  const int W = min(BW, (R + A - 1) / A);
  const int ln = lane & (LN - 1), grp = lane / LN, li = LN - 1 - ln;  // the first coordinate on the highest lane
  const uint32_t gmask = (LN == 32 ? ARP_FULL : (1u << (LN & 31)) - 1u) << (grp * LN);
  float* Js = sms;                          // N x DP: the spins' rows, columns by row_pos
  float* ws = Js + N * DP + wid * 4 * C * 32;  // the warp's scratch
  float* redm = Js + N * DP + W * 4 * C * 32;  // W x 2 x (CD NB) x LN: minima by group lane
  float* redb = redm + W * 2 * CD * NB * LN;  // W x 3: best d, step, chain
  uint32_t* redS = reinterpret_cast<uint32_t*>(redb + kSoftWarps * 3);  // W x LN: best spins
  // spin of slot c, group coordinate i
  auto spin = [&](int c, int i) { return QAM && c >= CD ? D + (c - CD) * LN + i : c * LN + i; };
  auto inside = [&](int c, int i) { return (QAM && c >= CD ? c - CD : c) * LN + i < D; };
  {  // a row per warp, four rows in flight
    constexpr int CW = (DP + 31) / 32;
    const float* Jb = a.J + (size_t)b * N * N;
    int pos[CW];  // place of the row's entry k 32 + lane; beyond the spins, of a column without one (zero)
#pragma unroll
    for (int k = 0; k < CW; ++k) {
      const int x = k * 32 + lane;
      int c, i;
      if (x < N) {
        const int j = QAM && x >= D ? x - D : x;
        c = j / LN + (QAM && x >= D ? CD : 0);
        i = j & (LN - 1);
      } else {  // columns without a spin, in order
        const int z = x - N, pad = CD * LN - D, h = QAM && z >= pad ? 1 : 0, j = D + z - h * pad;
        c = j / LN + h * CD;
        i = j & (LN - 1);
      }
      pos[k] = x < DP ? row_pos<LN, C>(c, LN - 1 - i) : 0;
    }
#pragma unroll 1
    for (int r0 = wid; r0 < N; r0 += 4 * BW) {
      float v[4][CW];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int k = 0; k < CW; ++k)
          v[u][k] = r0 + u * BW < N && k * 32 + lane < N ? Jb[(size_t)(r0 + u * BW) * N + k * 32 + lane] : 0.0f;
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int k = 0; k < CW; ++k)
          if (r0 + u * BW < N && k * 32 + lane < DP) Js[(r0 + u * BW) * DP + pos[k]] = v[u][k];
    }
  }
  __syncthreads();
  const uint32_t inst = a.inst[b];
  const float scale = a.scale[b], c0 = a.c0[b];
  const float* Tb = a.T + (size_t)b * S;
  float hfv[C], hd[C];  // hf and h0 - hf of the lane's spins
  uint32_t vm = 0;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const bool in = inside(c, li);
    const size_t o = (size_t)b * N + spin(c, li);
    hfv[c] = in ? a.hf[o] : 0.0f;
    hd[c] = in ? __fsub_rn(a.h0[o], hfv[c]) : 0.0f;
    if (in) vm |= 1u << c;
  }
  const float inf = __int_as_float(0x7f800000);
  float mn0[CD * NB], mn1[CD * NB];
#pragma unroll
  for (int c = 0; c < CD * NB; ++c) {
    mn0[c] = inf;
    mn1[c] = inf;
  }
  float wbest = inf;
  int wstep = INT_MAX, wchain = INT_MAX;
  uint32_t wup = 0;
  auto row = [&](int c, int l, float(&g)[C]) {  // row of slot c, group lane l
    const float* p = Js + spin(c, LN - 1 - l) * DP;
#pragma unroll
    for (int q = 0; q < C / 4; ++q) {
      const float4 v = *reinterpret_cast<const float4*>(p + ln * 4 + q * 4 * LN);
      g[4 * q] = v.x;
      g[4 * q + 1] = v.y;
      g[4 * q + 2] = v.z;
      g[4 * q + 3] = v.w;
    }
    if constexpr (C & 2) {
      const float2 v = *reinterpret_cast<const float2*>(p + ln * 2 + (C & ~3) * LN);
      g[C - 2] = v.x;
      g[C - 1] = v.y;
    }
  };
  for (int r0 = wid * A; r0 < R; r0 += W * A) {
    const int r = r0 + grp;
    const bool live = r < R;
    uint32_t up = 0;  // bit c: the lane's spin of slot c is +1
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int i = spin(c, li);
      bool u1 = false;
      if ((vm >> c) & 1u) {
        if (a.s0) {
          u1 = a.s0[(size_t)b * N + i] > 0;
        } else {
          uint32_t x0 = 0xFFFFFFFFu, x1 = (uint32_t)i, x2 = (uint32_t)r, x3 = inst;
          philox10(x0, x1, x2, x3, a.K);
          u1 = x0 >= 0x80000000u;
        }
      }
      if (u1) up |= 1u << c;
    }
    // u = hf + 2 J s (sum in spin order)
    float u[C];
#pragma unroll
    for (int c = 0; c < C; ++c) u[c] = 0.0f;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const uint32_t ub = __ballot_sync(ARP_FULL, (up >> c) & 1u);
      for (int l = LN - 1; l >= 0; --l) {
        if (!inside(c, LN - 1 - l)) break;
        const float sj = ((ub >> (grp * LN + l)) & 1u) ? 1.0f : -1.0f;
        float g[C];
        row(c, l, g);
#pragma unroll
        for (int t = 0; t < C; ++t) u[t] = __fadd_rn(u[t], __fmul_rn(g[t], sj));
      }
    }
#pragma unroll
    for (int c = 0; c < C; ++c) u[c] = __fadd_rn(hfv[c], __fmul_rn(2.0f, u[c]));
    // E0 = -sum_i s_i (h0_i + (u_i - hf_i) / 2): 32 partial sums (of spins v, v + 32, ...), then their binary tree in
    // v order; the terms cross lanes through the warp's scratch, which the thresholds overwrite later
    float E;
    {
      float* es = ws + grp * (C * LN);  // A C LN = 32 C <= 4 C 32 floats
      __syncwarp();
#pragma unroll
      for (int c = 0; c < C; ++c)
        if ((vm >> c) & 1u) {
          const int i = spin(c, li);
          const float si = ((up >> c) & 1u) ? 1.0f : -1.0f;
          es[i] = __fmul_rn(si, __fadd_rn(a.h0[(size_t)b * N + i], __fmul_rn(0.5f, __fsub_rn(u[c], hfv[c]))));
        }
      __syncwarp();
      float p[A];  // partial sums v = ln A .. ln A + A - 1
#pragma unroll
      for (int q = 0; q < A; ++q) {
        p[q] = 0.0f;
        for (int i = ln * A + q; i < N; i += 32) p[q] = __fsub_rn(p[q], es[i]);
      }
#pragma unroll
      for (int o = 1; o < A; o <<= 1)
#pragma unroll
        for (int q = 0; q + o < A; q += 2 * o) p[q] = __fadd_rn(p[q], p[q + o]);
      float e = p[0];
#pragma unroll
      for (int o = 1; o < LN; o <<= 1) e = __fadd_rn(e, __shfl_xor_sync(ARP_FULL, e, o));
      E = e;
      __syncwarp();
    }
    const uint32_t vr = live ? vm : 0u;
    float cbest = inf;
    int cstep = INT_MAX;
    uint32_t cup = up;
    for (int k = 0; k < S; ++k) {
      if ((k & 3) == 0) {  // the quad's thresholds (x / 2^32 - 1/2) 4T, word k & 3 of each spin's block
        float A4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) A4[i] = __fmul_rn(4.0f, k + i < S ? Tb[k + i] : 0.0f);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          uint32_t x[4] = {(uint32_t)(k >> 2), (uint32_t)spin(c, li), (uint32_t)r, inst};
          philox10(x[0], x[1], x[2], x[3], a.K);
#pragma unroll
          for (int i = 0; i < 4; ++i) ws[(c * 4 + i) * 32 + lane] = __fmul_rn(__fsub_rn(unit24(x[i]), 0.5f), A4[i]);
        }
      }
      uint32_t snap = 0;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const float su = ((up >> c) & 1u) ? u[c] : -u[c];
        if (__fadd_rn(su, a.q) < ws[(c * 4 + (k & 3)) * 32 + lane]) snap |= 1u << c;
      }
      snap &= vr;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        uint32_t mg = __ballot_sync(ARP_FULL, (snap >> c) & 1u) & gmask;
        const int rounds = __reduce_max_sync(ARP_FULL, __popc(mg));
        const bool su = (up >> c) & 1u;
        const float cfl = su ? -4.0f : 4.0f, s2 = su ? 2.0f : -2.0f;
        for (int t = 0; t < rounds; ++t) {
          // -1 without a flip left: the slot's first spin (the group's highest lane) is read, nothing is changed
          const int l = high_bit(mg);
          const int has = (int)mg;
          mg &= ~(1u << (l & 31));
          // dE0 = 2 s_j (h0_j + u_j - hf_j)
          const float dv = __shfl_sync(ARP_FULL, __fmul_rn(s2, __fadd_rn(hd[c], u[c])), l, LN);
          const float cf = __shfl_sync(ARP_FULL, cfl, l, LN);
          float g[C];
          row(c, l & (LN - 1), g);
          axpy_if<C>(has, cf, g, u);
          if (has) E = __fadd_rn(E, dv);
        }
      }
      up ^= snap;
      // the chain's distance after every step that flips (and step 0)
      const bool any = (__ballot_sync(ARP_FULL, snap != 0) & gmask) != 0 || k == 0;
      if (any && live) {
        const float d = __fadd_rn(__fmul_rn(scale, E), c0);
#pragma unroll
        for (int cc = 0; cc < CD; ++cc) {
          const bool s1 = (up >> cc) & 1u;
          mn1[NB * cc] = fminf(mn1[NB * cc], s1 ? d : inf);
          mn0[NB * cc] = fminf(mn0[NB * cc], s1 ? inf : d);
          if constexpr (QAM) {
            const bool b2 = s1 != (bool)((up >> (CD + cc)) & 1u);
            mn1[2 * cc + 1] = fminf(mn1[2 * cc + 1], b2 ? d : inf);
            mn0[2 * cc + 1] = fminf(mn0[2 * cc + 1], b2 ? inf : d);
          }
        }
        if (d < cbest) {
          cbest = d;
          cstep = k;
          cup = up;
        }
      }
    }
    // this chain's best against the group's: lowest d, then earliest step, then lowest chain
    if (live && (cbest < wbest || (cbest == wbest && (cstep < wstep || (cstep == wstep && r < wchain))))) {
      wbest = cbest;
      wstep = cstep;
      wchain = r;
      wup = cup;
    }
  }
  // ---- the minima and the best over the warp's groups, then over the chains' warps
#pragma unroll
  for (int o = LN; o < 32; o <<= 1) {
#pragma unroll
    for (int c = 0; c < CD * NB; ++c) {
      mn0[c] = fminf(mn0[c], __shfl_xor_sync(ARP_FULL, mn0[c], o));
      mn1[c] = fminf(mn1[c], __shfl_xor_sync(ARP_FULL, mn1[c], o));
    }
    const float ob = __shfl_xor_sync(ARP_FULL, wbest, o);
    const int os = __shfl_xor_sync(ARP_FULL, wstep, o), oc = __shfl_xor_sync(ARP_FULL, wchain, o);
    const uint32_t ou = __shfl_xor_sync(ARP_FULL, wup, o);
    if (ob < wbest || (ob == wbest && (os < wstep || (os == wstep && oc < wchain)))) {
      wbest = ob;
      wstep = os;
      wchain = oc;
      wup = ou;
    }
  }
  if (lane < LN && wid < W) {
#pragma unroll
    for (int c = 0; c < CD * NB; ++c) {
      redm[((wid * 2 + 0) * CD * NB + c) * LN + lane] = mn0[c];
      redm[((wid * 2 + 1) * CD * NB + c) * LN + lane] = mn1[c];
    }
    redS[wid * LN + lane] = wup;
  }
  if (lane == 0 && wid < W) {
    redb[wid * 3] = wbest;
    redb[wid * 3 + 1] = __int_as_float(wstep);
    redb[wid * 3 + 2] = __int_as_float(wchain);
  }
  __syncthreads();
  for (int x = threadIdx.x; x < D * NB; x += blockDim.x) {
    const int j = x / NB, o = ((j / LN) * NB + (x - j * NB)) * LN + (LN - 1 - (j & (LN - 1)));
    float v0 = inf, v1 = inf;
    for (int w = 0; w < W; ++w) {
      v0 = fminf(v0, redm[(w * 2) * CD * NB * LN + o]);
      v1 = fminf(v1, redm[(w * 2 + 1) * CD * NB * LN + o]);
    }
    a.m0[(size_t)b * D * NB + x] = v0;
    a.m1[(size_t)b * D * NB + x] = v1;
  }
  int bw = 0;
  for (int w = 1; w < W; ++w) {
    const float dw = redb[w * 3], db = redb[bw * 3];
    const int sw = __float_as_int(redb[w * 3 + 1]), sb = __float_as_int(redb[bw * 3 + 1]);
    const int cw2 = __float_as_int(redb[w * 3 + 2]), cb = __float_as_int(redb[bw * 3 + 2]);
    if (dw < db || (dw == db && (sw < sb || (sw == sb && cw2 < cb)))) bw = w;
  }
  if (threadIdx.x == 0) a.best_d[b] = redb[bw * 3];
  for (int j = threadIdx.x; j < D; j += blockDim.x) {
    const uint32_t w = redS[bw * LN + LN - 1 - (j & (LN - 1))];
    int l = ((w >> (j / LN)) & 1u) ? 1 : -1;
    if (QAM) l = 2 * l + (((w >> (CD + j / LN)) & 1u) ? 1 : -1);
    a.best_l[(size_t)b * D + j] = (int8_t)l;
  }
}

template <int LN, int CD, bool QAM>
static cudaError_t launch_soft(const SoftParams& a, cudaStream_t st) {
  using M = SoftMap<LN, CD, QAM>;
  // up to 64 spins, and up to 96 where the problems fill the GPU, the chains' warps stage J alone: more warps would hold
  // registers that other blocks' chains need (one chain each: 1400 uses of 64 spins 1345 us with one warp, 1547 with two;
  // 3000 of 72, with their LLRs, 10.4 ms with one, 11.8 with two, 12.7 with four; 3000 of 128 21.7 with four, 23.7 with two,
  // 27.8 with eight)
  const int W = min(kSoftWarps, (a.R + M::A - 1) / M::A), stage = a.N <= 64 || (a.N <= 96 && a.B > 296) ? 1 : 4;
  const size_t smem = 4 * ((size_t)a.N * M::DP + (size_t)W * 4 * M::C * 32 + (size_t)W * 2 * CD * M::NB * LN +
                           kSoftWarps * 3 + (size_t)W * LN);
  if (smem > 48 * 1024) {
    cudaError_t e =
        cudaFuncSetAttribute(k_traj_soft<LN, CD, QAM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  k_traj_soft<LN, CD, QAM><<<a.B, 32 * max(W, stage), smem, st>>>(a);
  return cudaGetLastError();
}

}  // namespace arp

using namespace arp;

extern "C" int arp_soft_trajectory(const float* J, const float* hf, const float* h0, const float* scale,
                                   const float* c0, const float* T, const int8_t* s0, float q, int S, int R, int D,
                                   int M, int B, const uint32_t* inst, uint32_t k0, uint32_t k1, float* m0, float* m1,
                                   float* best_d, int8_t* best_l, void* stream) {
  if (!(M == 4 || M == 16)) return ARP_ERR_SHAPE;
  const int N = M == 16 ? 2 * D : D;
  if (B < 0 || R < 1 || S < 1 || D < 1 || N > 128 || (N % 4)) return ARP_ERR_SHAPE;
  if (B == 0) return ARP_OK;
  if (!J || !hf || !h0 || !scale || !c0 || !T || !inst || !m0 || !m1 || !best_d || !best_l) return ARP_ERR_ARG;
  SoftParams a{J, hf, h0, scale, c0, T, s0, q, S, R, N, D, M, B, inst, m0, m1, best_d, best_l, philox_keys(k0, k1)};
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e;
  if (M == 16)
    e = D <= 16   ? launch_soft<8, 2, true>(a, st)
        : D <= 24 ? launch_soft<8, 3, true>(a, st)
        : D <= 32 ? launch_soft<8, 4, true>(a, st)
        : D <= 48 ? launch_soft<16, 3, true>(a, st)
                  : launch_soft<16, 4, true>(a, st);
  else
    e = D <= 32   ? launch_soft<8, 4, false>(a, st)
        : D <= 48 ? launch_soft<8, 6, false>(a, st)
        : D <= 64 ? launch_soft<8, 8, false>(a, st)
        : D <= 96 ? launch_soft<16, 6, false>(a, st)
                  : launch_soft<16, 8, false>(a, st);
  return e == cudaSuccess ? ARP_OK : ARP_ERR_LAUNCH;
}
