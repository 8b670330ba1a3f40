// FP32-field anneals on compressed dDI problems, several anneals per warp: first accept and the Chord round, with the
// lane mapping, scan and random numbers of the integer anneals (anneal_group.cuh).
//
// The float rule, one IEEE rounding per operation (the same operations in the same order for every anneal, so the
// mapping does not show in the results): th = ((x >> 8) 2^-24 - 1/2) 4T; accepted iff (s w_j + 2 G_jj) + (q - c) < th;
// a flip moves w_i by (4 s_j) G_ij and the energy by (4 s_j w_j) + 8 G_jj, w_j after the earlier flips; start fields
// are summed in j order over the coordinates with m != 0.  The products by powers of two are exact, so a multiply and
// an add are one fused multiply-add (for values below 2^126).  Each group adds its flips' energies in scan order.  A
// group without a flip in a round changes nothing (predicated, not a multiply by zero: 0 times an infinity is NaN).
//
// Bound by issue slots, as the integer anneals.  32 anneals x 24 sweeps, one anneal per warp (the previous kernel)
// against these: 4096 24-user uses 1.62 -> 1.03 ms, 4096 32-user 2.00 -> 1.44, 1024 64-user 2.00 -> 1.04, 16384 8-user
// 2.35 -> 0.99, one 32-user frame 51 -> 43 us; Chord 4096 32-user uses 1.54 -> 1.21 ms.
#pragma once
#include "anneal_group.cuh"

namespace arp {
namespace grpf {

using grp::high_bit;
using grp::Rule;
using grp::sm32;

template <int LN, int C>
__device__ __forceinline__ void load_rowf(uint32_t row, int ln, float (&g)[C]) {
  int32_t v[C];
  grp::load_row<LN, C>(row, ln, v);
#pragma unroll
  for (int c = 0; c < C; ++c) g[c] = __int_as_float(v[c]);
}

// w[t] += f g[t] and de += dv where has != 0.
template <int C>
__device__ __forceinline__ void flip_if(float has, float f, float dv, const float (&g)[C], float (&w)[C], float& de) {
  asm("{\n\t.reg .pred p;\n\tsetp.ne.f32 p, %1, 0f00000000;\n\t@p add.rn.f32 %0, %0, %2;\n\t}"
      : "+f"(de)
      : "f"(has), "f"(dv));
#pragma unroll
  for (int t = 0; t < C; ++t)
    asm("{\n\t.reg .pred p;\n\tsetp.ne.f32 p, %1, 0f00000000;\n\t@p fma.rn.f32 %0, %2, %3, %0;\n\t}"
        : "+f"(w[t])
        : "f"(has), "f"(f), "f"(g[t]));
}

template <int LN, int C, int P>
inline size_t smem_bytes(int W) {
  const size_t s = grp::g_bytes<LN, C>() + (size_t)W * P * C * 512;
  const size_t rows = ((size_t)(C - 1) * LN + 33) * LN * C * 4;
  return s > rows ? s : rows;
}

template <int LN, int C, int P, bool CHORD, int MB>
__global__ void __launch_bounds__(grp::max_threads<LN, C>(), MB) k_anneal_f32(const DDParams a) {
  constexpr int A = 32 / LN, DP = LN * C;
  static_assert(P * C <= 32, "a lane's spins are one 32-bit word");
  extern __shared__ __align__(16) unsigned char smem[];
  float* Gs = reinterpret_cast<float*>(smem);
  const PhiloxKeys& K = *reinterpret_cast<const PhiloxKeys*>(a.rk0);
  const int D = a.D, L = a.L, R = a.R;
  const int split = a.split, b = blockIdx.x / split, bs = blockIdx.x - b * split;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, W = blockDim.x >> 5, bt = blockDim.x;
  const int ln = lane & (LN - 1), grp = lane / LN, li = LN - 1 - ln;
  const uint32_t gmask = (LN == 32 ? ARP_FULL : ((1u << (LN & 31)) - 1u)) << (grp * LN);
  float* th = reinterpret_cast<float*>(smem + grp::g_bytes<LN, C>()) + wid * (P * C * 128) + lane;
  pdl_trigger();
  pdl_wait();
  const float* hg = reinterpret_cast<const float*>(a.h) + (size_t)b * D;
  const float* Tg = reinterpret_cast<const float*>(a.T);
  const float* cg = reinterpret_cast<const float*>(a.c);
  {
    const float* Gg = reinterpret_cast<const float*>(a.Gt) + (size_t)b * D * D;
    for (int x0 = threadIdx.x; x0 < D * DP; x0 += 4 * bt) {  // four loads in flight per thread
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int x = x0 + u * bt, j = x / DP, i = x - j * DP;
        v[u] = x < D * DP && i < D ? Gg[(size_t)j * D + i] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int x = x0 + u * bt, j = x / DP, i = x - j * DP;
        if (x < D * DP) Gs[j * DP + grp::row_pos<LN, C>(i / LN, LN - 1 - (i & (LN - 1)))] = v[u];
      }
    }
  }
  const uint32_t inst = a.inst ? a.inst[b] : a.inst0 + (uint32_t)b;
  __syncthreads();
  uint32_t lmask = 0, vm = 0;  // the bits of coordinate D - 1 on its lane; the lane's slots inside the problem
  {
    const int cl = (D - 1) / LN;
#pragma unroll
    for (int p = 0; p < P; ++p)
      if (D - 1 - cl * LN == li) lmask |= 1u << (p * C + cl);
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (c * LN + li < D) vm |= 1u << c;
  }
  const uint32_t g0 = sm32(Gs) + (uint32_t)((LN - 1 + grp * LN) * DP * 4);
  float dg[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int j = c * LN + li;
    dg[c] = j < D ? Gs[j * DP + grp::row_pos<LN, C>(c, ln)] : 0.0f;
  }
  for (int r0 = (bs + split * wid) * A; r0 < R; r0 += split * W * A) {
    const int r = r0 + grp;
    const bool live = r < R;
    // ---- start state (arpeggio_fx.cu:48-57): bit p C + c of dn is set where copy p of the lane's slot c is down
    uint32_t dn = 0;
    if (a.start != 0) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        uint32_t c0 = 0xFFFFFFFFu, c1 = (uint32_t)(c * LN + li), c2 = (uint32_t)r, c3 = inst;
        philox10(c0, c1, c2, c3, K);
        const int pat = bal_pattern(P, (uint32_t)(((uint64_t)c0 * (uint64_t)bal_choose(P)) >> 32));
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
    // ---- fields w = h - 2 G m (arpeggio_fx.cu:58-66), the sum in j order
    float w[C];
#pragma unroll
    for (int c = 0; c < C; ++c) w[c] = 0.0f;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      int d = 0;
#pragma unroll
      for (int p = 0; p < P; ++p) d += (dn >> (p * C + c)) & 1u;
      const float mc = ((vm >> c) & 1u) ? (float)(P - 2 * d) : 0.0f;
      if (!__any_sync(ARP_FULL, mc != 0.0f)) continue;  // as in the integer kernel
#pragma unroll 2
      for (int i = 0; i < LN; ++i) {
        if (c * LN + i >= D) break;
        const float m = __shfl_sync(ARP_FULL, mc, LN - 1 - i, LN);
        float g[C];
        load_rowf<LN, C>(sm32(Gs) + (uint32_t)((c * LN + i) * DP * 4), ln, g);
#pragma unroll
        for (int t = 0; t < C; ++t) {
          const float s = __fadd_rn(w[t], __fmul_rn(g[t], m));
          w[t] = m != 0.0f ? s : w[t];
        }
      }
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int j = c * LN + li;
      w[c] = __fsub_rn(j < D ? hg[j] : 0.0f, __fmul_rn(2.0f, w[c]));
    }
    const uint32_t vr = live ? vm : 0u;
    float de = 0.0f, best = __int_as_float(0x7f800000);
    uint32_t bdn = dn;
    int32_t flips = 0, lastflips = 0;
    int k = 0;
    for (int q4 = 0; k < L; ++q4) {
      // thresholds of the quad's four sweeps
#pragma unroll(C * P <= 8 ? P : LN == 32 ? 2 : 1)
      for (int p = 0; p < P; ++p) {
        float A4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) A4[i] = k + i * P + p < L ? __fmul_rn(4.0f, Tg[k + i * P + p]) : 0.0f;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          uint32_t x[4] = {(uint32_t)q4, (uint32_t)(p * D + c * LN + li), (uint32_t)r, inst};
          philox10(x[0], x[1], x[2], x[3], K);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            th[(p * C + c) * 128 + i * 32] = __fmul_rn(__fsub_rn(unit24(x[i]), 0.5f), A4[i]);
        }
      }
      for (int i = 0; i < 4 && k < L; ++i) {
        const float* thi = th + i * 32;
        uint32_t fb = 0;  // the sweep's flips, bits as dn
#pragma unroll
        for (int p = 0; p < P; ++p) {
          if (k >= L) break;
          const float qk = (CHORD && cg) ? __fsub_rn(a.qf, cg[k]) : a.qf;
          // one round of slot c: every group with a candidate (acc on some lane of m) flips its first
          auto commit = [&](int c, bool acc, uint32_t m, float s4, int& jl) {
            const int l = high_bit(m & gmask);  // -1 in a group without one: reads its last lane's f, which is 0
            const float f = __shfl_sync(ARP_FULL, acc ? s4 : 0.0f, l, LN);
            const float dv = __shfl_sync(ARP_FULL, __fadd_rn(__fmul_rn(s4, w[c]), __fmul_rn(8.0f, dg[c])), l, LN);
            float g[C];
            load_rowf<LN, C>(g0 + c * LN * DP * 4 - (uint32_t)l * (DP * 4), ln, g);
            flip_if<C>(f, f, dv, g, w, de);
            if (lane == l) fb |= 1u << (p * C + c);
            jl = l;
          };
          auto accept = [&](int c, uint32_t sb, float t) {  // sb: the sign bit of s w
            const float sw = __int_as_float(__float_as_int(w[c]) ^ (int)sb);
            return __fadd_rn(__fadd_rn(sw, __fmul_rn(2.0f, dg[c])), qk) < t;
          };
          if constexpr (!CHORD) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
              const uint32_t sb = ((dn >> (p * C + c)) & 1u) << 31;
              const float s4 = __int_as_float(0x40800000 | (int)sb);
              // nothing is below -inf: a padding coordinate, or a group without an anneal, never accepts
              const float t = ((vr >> c) & 1u) ? thi[(p * C + c) * 128] : __int_as_float(0xff800000);
              int jl = 32;
              for (;;) {
                const bool acc = lane < jl && accept(c, sb, t);
                const uint32_t m = __ballot_sync(ARP_FULL, acc);
                if (m == 0) break;
                commit(c, acc, m, s4, jl);
              }
            }
          } else {
            uint32_t snap = 0;
#pragma unroll
            for (int c = 0; c < C; ++c)
              if (accept(c, ((dn >> (p * C + c)) & 1u) << 31, thi[(p * C + c) * 128])) snap |= 1u << c;
            snap &= vr;
#pragma unroll
            for (int c = 0; c < C; ++c) {
              const float s4 = ((dn >> (p * C + c)) & 1u) ? -4.0f : 4.0f;
              const bool sn = (snap >> c) & 1u;
              int jl = 32;
              for (;;) {
                const bool acc = sn && lane < jl;
                const uint32_t m = __ballot_sync(ARP_FULL, acc);
                if (m == 0) break;
                commit(c, acc, m, s4, jl);
              }
            }
          }
          if (de < best) {  // best state after each pass (arpeggio_fx.cu:90-93)
            best = de;
            bdn = dn ^ fb;
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
          if (j < D) os[p * D + j] = ((bdn >> (p * C + c)) & 1u) ? -1 : 1;
        }
      if (ln == 0) {
        reinterpret_cast<float*>(a.out_de)[ar] = best;
        a.out_st[2 * ar] = flips;
        a.out_st[2 * ar + 1] = CHORD ? L : L + flips - lastflips;
      }
    }
  }
}

template <int LN, int C, int P, bool CHORD, int MB = grp::min_blocks<LN, C>()>
static cudaError_t launch(const DDParams& a, int warps, cudaStream_t st) {
  static grp::Widths wd;
  return grp::launch_widths<32 / LN, grp::max_threads<LN, C>() / 32>(
      wd, k_anneal_f32<LN, C, P, CHORD, MB>, 0, [](int W) { return smem_bytes<LN, C, P>(W); }, a, warps, st);
}

// The mapping for D coordinates, by the integer anneals' rule, except that 64 coordinates stay at two anneals per warp:
// the thresholds are 32 bits here, 8 KB a warp with eight coordinates a lane, which leaves half the warps (4096 32-user
// uses: 1.44 against 1.51-1.62 ms).  48 coordinates, six a lane, at 80 registers (1.03 ms per 4096 uses; bound to 64
// it spills, 1.16).
template <int P, bool CHORD>
static cudaError_t dispatch(const DDParams& a, int warps, cudaStream_t st) {
  const int D = a.D;
  const long long n = (long long)a.B * a.R, w8 = (long long)a.B * ((a.R + 7) / 8 * 8);
  // one anneal per warp, as in the integer kernel, for few anneals and for counts that fill their last block of 16 badly
  // (34000 of 126 coordinates, 33 a use: first accept 2211 -> 2119 us, Chord 1636 -> 1471); into a short second wave (81
  // uses of 32 anneals in the detector, first accept: 36 users 189 -> 156 us, 63 users 269 -> 230), by Chord above 96
  // coordinates only; and above 96 coordinates up to 16 anneals a use, which one block of eight two-per-warp warps holds
  const bool waste = (a.R + 15) / 16 * 128 > a.R * 9;
  const bool start = (!CHORD || D > 96) && w8 <= grp::kLatWarps * 5 / 4;
  if constexpr (P < 6)
    if (D > 64 && w8 > grp::kLatWarps / 2 && (w8 <= grp::kLatWarps || waste || start || (a.R <= 16 && D > 96)))
      return D <= 96 ? launch<32, 3, P, CHORD>(a, warps, st) : launch<32, 4, P, CHORD>(a, warps, st);
  if (w8 <= grp::lat_warps<P>(D))
    return D <= 32   ? launch<32, 1, P, CHORD, 1>(a, warps, st)
           : D <= 64 ? launch<32, 2, P, CHORD, 1>(a, warps, st)
           : D <= 96 ? launch<32, 3, P, CHORD, 1>(a, warps, st)
                     : launch<32, 4, P, CHORD, 1>(a, warps, st);
  if (w8 <= (D > 16 ? grp::kOnePerWarp : 148LL * 32) && D <= 64)
    return D <= 32 ? launch<32, 1, P, CHORD>(a, warps, st) : launch<32, 2, P, CHORD>(a, warps, st);
  if (D <= 16 && (n <= grp::kMid16 || a.R < 16)) return launch<8, 2, P, CHORD>(a, warps, st);
  if (D <= 32 && D > 16 && (n <= grp::kMid32 || a.R < 16)) return launch<16, 2, P, CHORD>(a, warps, st);
  if (D <= 16) return launch<4, 4, P, CHORD>(a, warps, st);
  if (D <= 32) return launch<8, 4, P, CHORD>(a, warps, st);
  if constexpr (P == 6) {
    return D <= 64   ? launch<16, 4, P, CHORD>(a, warps, st)
           : D <= 96 ? launch<32, 3, P, CHORD>(a, warps, st)
                     : launch<32, 4, P, CHORD>(a, warps, st);
  } else {
    if (D <= 48) return launch<8, 6, P, CHORD, 3>(a, warps, st);
    if (D <= 64) return launch<16, 4, P, CHORD>(a, warps, st);
    return D <= 96 ? launch<16, 6, P, CHORD>(a, warps, st) : launch<16, 8, P, CHORD>(a, warps, st);
  }
}

}  // namespace grpf
}  // namespace arp
