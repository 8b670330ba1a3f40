// C = A B^T for the warm-start network's large training products (bf16 operands, fp32 accumulation in TMEM): a
// persistent, warp-specialised tcgen05 kernel fed by TMA.
//
// Roles (576 threads, one CTA per SM):
//   warp 0     producer: one lane issues 2D tiled TMA loads (128-byte swizzle) of the A tile (128 rows) and the
//              B tile (BN rows) of each 64-wide k step into an S-slot shared-memory ring; a slot completes on its
//              `full` mbarrier by the loads' byte count;
//   warp 1     allocates TMEM for two BN-column accumulators; one lane issues the MMAs (M = 128, N = BN, K = 16,
//              four per k step) and commits them twice: to the slot's `empty` mbarrier (the slot may be refilled
//              once its MMAs have read it) and, after a work item's last k step, to the accumulator's `tfull`;
//   warps 2-17 epilogue: warp w reads TMEM lane quarter w % 4 (rows 32 (w % 4) ..), part (w - 2) / 4 of the
//              columns, of the finished accumulator with tcgen05.ld, applies the fused epilogue, stores through a
//              staging tile to global memory and releases the accumulator (`tempty`), so the MMAs of the next work
//              item run while this one drains.
// Work items (128-row tile, BN-column tile, K split) are dealt round-robin to the persistent CTAs.
// Every wait is bounded (ARP_ERR_TIMEOUT).  After a timeout every role stops issuing; before TMEM is released the
// producer waits (bounded) for the loads it has in flight and the MMA lane for the MMAs it has issued.
//
// Shared-memory layouts (every load fills this CTA's own shared memory only): a K-major operand box {64 k, R rows} lands as R rows of 128 bytes
// (SBO 1024); an MN-major operand is loaded as boxes {64 of M or N, 64 k}, 64 rows of 128 bytes each (SBO 1024
// between 8-k groups, LBO 8192 between the 64-element blocks).
#include <cuda.h>

#include <mutex>

#include "../../include/arpeggio_b200.h"
#include "arp_common.cuh"
#include "gemm.cuh"
#include "umma.cuh"

namespace arp {
namespace tmagemm {

constexpr int kEpiWarps = 16;
constexpr int kThreads = 64 + 32 * kEpiWarps;  // producer warp, MMA warp, the epilogue warps
constexpr uint32_t kABytes = 128 * 128;  // 128 rows x 64 k x 2 bytes
constexpr uint32_t kStageOut = 2048;  // per epilogue warp: 32 rows x 64 bytes of its output tile

template <int BN>
__host__ __device__ constexpr int stages() {
  return (192 * 1024) / (int)(kABytes + BN * 128) > 8 ? 8 : (192 * 1024) / (int)(kABytes + BN * 128);
}
template <int BN>
__host__ __device__ constexpr size_t smem_bytes() {
  return (size_t)stages<BN>() * (kABytes + BN * 128) + kEpiWarps * kStageOut + 1024;  // + to align the ring to 1024
}

struct Work {
  int items, gx, gy, nkt, kt_per;
};

__device__ __forceinline__ void decode(const Work& w, int item, int& m0, int& n0, int& z, int& kt0, int& kt1, int BN) {
  // column tiles fastest: CTAs running at the same time share their A tile through L2
  const int nt = item % w.gy, rest = item / w.gy;
  n0 = nt * BN;
  m0 = (rest % w.gx) * 128;
  z = rest / w.gx;
  kt0 = z * w.kt_per;
  kt1 = min(w.nkt, kt0 + w.kt_per);
}

// One epilogue warp's 32 x 32 tile of C at (row0, n), its rows in the lanes' registers, goes through 2 KB of shared
// memory so that a store instruction covers 64 contiguous bytes of eight rows; a lane storing its own row writes 16
// bytes every ldc elements, half a sector at a time over 32 rows.  Row r's 16-byte groups sit at j ^ (r / 2 % 4), so
// neither side has bank conflicts.  The mask's activations ax are read in the same layout.  The values and roundings
// are epilogue()'s.  With sixteen epilogue warps instead of eight (eight left a quarter of the issue slots in use, each
// warp a serial chain of TMEM read, bias, convert, store), 65,536 x 256 x 256: ReLU forward 28.7 -> 19.2 us, input
// gradient with the mask 38.7 -> 24.8.
struct OutTile {
  int n, j, r, left;  // first column, this lane's 16-byte group, its first row of the tile, rows of C from there on
  size_t off, offx;   // element offsets of (row0 + r, n + the group) in C and in aux (bf16)
};

__device__ __forceinline__ uint4* slot(uint4* st, int row, int j) { return st + row * 4 + (j ^ ((row >> 1) & 3)); }

__device__ __forceinline__ void load_aux(const GemmParams& p, const OutTile& t, uint4 (&ax)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (8 * i < t.left && t.n + 8 * t.j < p.N)
      ax[i] = *reinterpret_cast<const uint4*>(p.aux + t.offx + (size_t)(8 * i) * p.ldaux);
}

__device__ __forceinline__ void store_bf16(const GemmParams& p, const OutTile& t, uint32_t (&v)[32], uint4* st,
                                           const uint4 (&ax)[4]) {
  const int lane = threadIdx.x & 31;
  if (p.epi == EPI_BIAS_RELU_BF16) {
    // the tile's biases, one per lane, handed round through the staging rows
    float* sb = reinterpret_cast<float*>(st);
    sb[lane] = t.n + lane < p.N ? p.bias[t.n + lane] : 0.0f;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 b = reinterpret_cast<const float4*>(sb)[i];
      v[4 * i] = __float_as_uint(__uint_as_float(v[4 * i]) + b.x);
      v[4 * i + 1] = __float_as_uint(__uint_as_float(v[4 * i + 1]) + b.y);
      v[4 * i + 2] = __float_as_uint(__uint_as_float(v[4 * i + 2]) + b.z);
      v[4 * i + 3] = __float_as_uint(__uint_as_float(v[4 * i + 3]) + b.w);
    }
    __syncwarp();
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t pk[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 h2 =
          __floats2bfloat162_rn(__uint_as_float(v[8 * j + 2 * i]), __uint_as_float(v[8 * j + 2 * i + 1]));
      if (p.epi == EPI_BIAS_RELU_BF16) h2 = __hmax2(h2, __nv_bfloat162(0.0f, 0.0f));  // the rounding keeps the sign
      pk[i] = *reinterpret_cast<const uint32_t*>(&h2);
    }
    *slot(st, lane, j) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
  }
  __syncwarp();
  if (t.n + 8 * t.j < p.N) {
    bf16* o = reinterpret_cast<bf16*>(p.C) + t.off;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 u = *slot(st, t.r + 8 * i, t.j);
      uint32_t w[4] = {u.x, u.y, u.z, u.w};
      if (p.epi == EPI_MASK_BF16) {  // ReLU backward through the stored activation
        const uint32_t a[4] = {ax[i].x, ax[i].y, ax[i].z, ax[i].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (!(__uint_as_float(a[k] << 16) > 0.0f)) w[k] &= 0xFFFF0000u;
          if (!(__uint_as_float(a[k] & 0xFFFF0000u) > 0.0f)) w[k] &= 0x0000FFFFu;
        }
      }
      if (8 * i < t.left)
        *reinterpret_cast<uint4*>(o + (size_t)(8 * i) * p.ldc) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  __syncwarp();  // read before the next tile is staged
}

__device__ __forceinline__ void store_f32(const GemmParams& p, const OutTile& t, const uint32_t (&v)[32], int z,
                                          uint4* st) {
  const int lane = threadIdx.x & 31;
  float* o = reinterpret_cast<float*>(p.C) + t.off;
  if (p.epi == EPI_F32_PART) o += (size_t)z * p.M * p.ldc;
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) {  // 16 columns at a time
    const int nn = t.n + 16 * hf;
    if (nn >= p.N) break;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *slot(st, lane, j) = make_uint4(v[16 * hf + 4 * j], v[16 * hf + 4 * j + 1], v[16 * hf + 4 * j + 2],
                                      v[16 * hf + 4 * j + 3]);
    float b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (p.epi == EPI_BIAS_F32)
#pragma unroll
      for (int i = 0; i < 4; ++i) b[i] = p.bias[nn + 4 * t.j + i];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 u = *slot(st, t.r + 8 * i, t.j);
      float4 f = make_float4(__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w));
      if (p.epi == EPI_BIAS_F32) f = make_float4(f.x + b[0], f.y + b[1], f.z + b[2], f.w + b[3]);
      if (8 * i < t.left) *reinterpret_cast<float4*>(o + 16 * hf + (size_t)(8 * i) * p.ldc) = f;
    }
    __syncwarp();
  }
}

template <int BN, bool AMN, bool BMN>
__global__ void __launch_bounds__(kThreads, 1)
    k_gemm_tma(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
               const GemmParams p, const Work wk) {
  constexpr int S = stages<BN>();
  constexpr uint32_t BBYTES = BN * 128, SBYTES = kABytes + BBYTES;
  constexpr uint32_t NCOL = 2 * BN < 32 ? 32 : 2 * BN;  // two accumulators
  constexpr uint32_t IDESC = umma::idesc_bf16(BN, AMN, BMN);
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t full[S], empty[S], tfull[2], tempty[2], done;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t ring = (umma::su32(smem) + 1023u) & ~1023u;
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      umma::mbar_init(&full[s], 1);
      umma::mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      umma::mbar_init(&tfull[a], 1);
      umma::mbar_init(&tempty[a], kEpiWarps);
    }
    umma::mbar_init(&done, 1);
    umma::fence_mbar_init();
    s_abort = 0;
    umma::tma_prefetch(&tma_a);
    umma::tma_prefetch(&tma_b);
  }
  if (warp == 1) umma::tmem_alloc(&s_tmem, NCOL);
  umma::tc_before_sync();
  __syncthreads();
  umma::tc_after_sync();
  const uint32_t tmem = s_tmem;
  // One column tile and a K that fits the ring: B is the same for every item, so its k tile kt is loaded once, with
  // the CTA's first item, into slot kt and stays there.  Reading the same few KB
  // from every SM for every tile cost more than A's stream: 151,552 x 256 x 16 with ReLU 39.2 -> 30.5 us, with the
  // mask 50.0 -> 41.9.
  const bool keep_b = wk.gy == 1 && wk.kt_per == wk.nkt && wk.nkt <= S;

  if (warp == 0) {
    if (lane == 0) {
      // ---- producer
      int slot = 0, armed[S];
      uint32_t ph = 0;
      for (int s = 0; s < S; ++s) armed[s] = 0;
      for (int item = blockIdx.x; item < wk.items && !s_abort; item += gridDim.x) {
        int m0, n0, z, kt0, kt1;
        decode(wk, item, m0, n0, z, kt0, kt1, BN);
        for (int kt = kt0; kt < kt1; ++kt) {
          if (s_abort) break;
          if (!umma::mbar_wait(&empty[slot], ph ^ 1u)) {
            s_abort = 1;
            break;
          }
          const uint32_t sa = ring + (uint32_t)slot * SBYTES, sb = sa + kABytes;
          const int k0 = kt * 64;
          const bool load_b = !keep_b || item == (int)blockIdx.x;
          umma::expect_tx(&full[slot], load_b ? SBYTES : kABytes);
          if constexpr (AMN) {
            umma::tma_load_2d(sa, &tma_a, m0, k0, &full[slot]);
            umma::tma_load_2d(sa + 8192, &tma_a, m0 + 64, k0, &full[slot]);
          } else {
            umma::tma_load_2d(sa, &tma_a, k0, m0, &full[slot]);
          }
          if (load_b) {
            if constexpr (BMN) {
#pragma unroll
              for (int c = 0; c < BN / 64; ++c)
                umma::tma_load_2d(sb + (uint32_t)c * 8192, &tma_b, n0 + 64 * c, k0, &full[slot]);
            } else {
              umma::tma_load_2d(sb, &tma_b, k0, n0, &full[slot]);
            }
          }
          ++armed[slot];
          if (++slot == S) {
            slot = 0;
            ph ^= 1u;
          }
        }
      }
      // every load issued has landed before the CTA may leave (bounded)
      for (int s = 0; s < S; ++s)
        if (armed[s] > 0 && !umma::mbar_wait(&full[s], (uint32_t)((armed[s] - 1) & 1))) s_abort = 1;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      // ---- MMA issue
      const int whole = p.K >> 6;  // k tiles without zeros past K
      int slot = 0, it = 0;
      uint32_t ph = 0;
      for (int item = blockIdx.x; item < wk.items && !s_abort; item += gridDim.x, ++it) {
        int m0, n0, z, kt0, kt1;
        decode(wk, item, m0, n0, z, kt0, kt1, BN);
        const int ab = it & 1;
        const uint32_t aph = (uint32_t)((it >> 1) & 1);
        if (!umma::mbar_wait(&tempty[ab], aph ^ 1u)) {
          s_abort = 1;
          break;
        }
        umma::tc_after_sync();
        const uint32_t acc = tmem + (uint32_t)(ab * BN);
        bool ok = true;
        for (int kt = kt0; kt < kt1; ++kt) {
          if (!umma::mbar_wait(&full[slot], ph)) {
            ok = false;
            break;
          }
          umma::tc_after_sync();
          const uint32_t sa = ring + (uint32_t)slot * SBYTES;
          const uint32_t sb = ring + (uint32_t)(keep_b ? kt : slot) * SBYTES + kABytes;
          auto mma = [&](int kk) {
            const uint64_t ad = AMN ? umma::sdesc_sw128(sa + kk * 2048, 8192, 1024) : umma::sdesc_sw128(sa + kk * 32, 16, 1024);
            const uint64_t bd = BMN ? umma::sdesc_sw128(sb + kk * 2048, 8192, 1024) : umma::sdesc_sw128(sb + kk * 32, 16, 1024);
            umma::mma(acc, ad, bd, IDESC, (kt > kt0 || kk > 0) ? 1u : 0u);
          };
          if (kt < whole) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) mma(kk);
          } else {  // past K the tiles hold zeros
#pragma unroll 1
            for (int kk = 0; kt * 64 + kk * 16 < p.K; ++kk) mma(kk);
          }
          umma::commit(&empty[slot]);
          if (++slot == S) {
            slot = 0;
            ph ^= 1u;
          }
        }
        umma::commit(&tfull[ab]);  // arrives even on a timeout, so the epilogue is not left waiting
        if (!ok) {
          s_abort = 1;
          break;
        }
      }
      // every MMA issued has completed before TMEM is released (bounded)
      umma::commit(&done);
      if (!umma::mbar_wait(&done, 0)) s_abort = 1;
    }
    __syncwarp();
  } else {
    // ---- epilogue: warp w drains TMEM lane quarter w % 4, the (w - 2) / 4-th part of the columns
    constexpr int CPW = BN / 4 < 32 ? 32 : BN / 4;  // BN = 64: two of the four parts
    const int q = warp & 3, c_lo = ((warp - 2) >> 2) * CPW;
    uint4* st = reinterpret_cast<uint4*>(smem + (ring - umma::su32(smem)) + S * SBYTES + (warp - 2) * kStageOut);
    const bool wide = p.epi == EPI_BIAS_RELU_BF16 || p.epi == EPI_MASK_BF16;
    int it = 0;
    for (int item = blockIdx.x; item < wk.items && !s_abort; item += gridDim.x, ++it) {
      int m0, n0, z, kt0, kt1;
      decode(wk, item, m0, n0, z, kt0, kt1, BN);
      const int ab = it & 1;
      const int row0 = m0 + q * 32;
      OutTile t;
      t.n = n0 + c_lo;
      t.j = lane & 3;
      t.r = lane >> 2;
      t.left = p.M - (row0 + t.r);
      t.off = (size_t)(row0 + t.r) * p.ldc + t.n + (wide ? 8 : 4) * t.j;
      t.offx = (size_t)(row0 + t.r) * p.ldaux + t.n + 8 * t.j;
      uint4 ax[4];
      if (p.epi == EPI_MASK_BF16 && c_lo < BN) load_aux(p, t, ax);  // on its way while the tensor core works
      const bool ok = umma::mbar_wait(&tfull[ab], (uint32_t)((it >> 1) & 1));
      umma::tc_after_sync();
      if (ok && !s_abort) {
#pragma unroll 1
        for (int c = c_lo; c < c_lo + CPW && c < BN; c += 32) {
          if (t.n >= p.N) break;
          uint32_t v[32];
          umma::tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(ab * BN + c), v);
          if (wide)
            store_bf16(p, t, v, st, ax);
          else if (p.epi != EPI_F32_ACC)
            store_f32(p, t, v, z, st);
          else if (row0 + lane < p.M)
            epilogue<32>(p, row0 + lane, t.n, v, z);
          t.n += 32;
          t.off += 32;
          t.offx += 32;
          if (p.epi == EPI_MASK_BF16 && c + 32 < c_lo + CPW) load_aux(p, t, ax);
        }
      } else {
        s_abort = 1;
      }
      umma::tc_before_sync();
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(&tempty[ab]);
      if (!ok) break;
    }
  }
  umma::tc_before_sync();
  __syncthreads();
  if (tid == 0 && s_abort) set_status(p.status, ARP_ERR_TIMEOUT);
  if (warp == 1) umma::tmem_free(tmem, NCOL);
}

}  // namespace tmagemm
}  // namespace arp

namespace arp {
namespace tmagemm {

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, looked up once through the runtime (no link against the driver library).
static EncodeTiled encoder() {
  static EncodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(f);
  });
  return fn;
}

// A 2D bf16 tensor (inner x outer elements, rows ld elements apart) tiled in boxes of box_inner x box_outer with
// 128-byte swizzle; elements outside the tensor read as zero.
static bool tensor_map(CUtensorMap* m, const bf16* base, int inner, int outer, int ld, int box_inner, int box_outer) {
  const EncodeTiled enc = encoder();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
  const cuuint32_t es[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(base), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr int kMaxDevices = 64;

template <int BN, bool AMN, bool BMN>
static cudaError_t launch(const GemmParams& p, const Work& w, cudaStream_t st) {
  CUtensorMap ta, tb;
  // A: 128 rows x 64 k per step (K-major: one box; MN-major: two boxes of 64 rows); B: BN rows x 64 k
  const bool ok_a = AMN ? tensor_map(&ta, p.A, p.M, p.K, p.lda, 64, 64) : tensor_map(&ta, p.A, p.K, p.M, p.lda, 64, 128);
  const bool ok_b = BMN ? tensor_map(&tb, p.B, p.N, p.K, p.ldb, 64, 64) : tensor_map(&tb, p.B, p.K, p.N, p.ldb, 64, BN);
  if (!ok_a || !ok_b) return cudaErrorNotSupported;
  constexpr size_t smem = smem_bytes<BN>();
  static bool attr[kMaxDevices];
  static int sms[kMaxDevices];
  static std::mutex mu;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!attr[dev]) {
      e = cudaFuncSetAttribute(k_gemm_tma<BN, AMN, BMN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      e = cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
      if (e != cudaSuccess) return e;
      attr[dev] = true;
    }
  }
  const int grid = w.items < sms[dev] ? w.items : sms[dev];
  k_gemm_tma<BN, AMN, BMN><<<grid, kThreads, smem, st>>>(ta, tb, p, w);
  return cudaGetLastError();
}

template <int BN>
static cudaError_t launch_bn(const GemmParams& p, const Work& w, bool amn, bool bmn, cudaStream_t st) {
  if (!amn && !bmn) return launch<BN, false, false>(p, w, st);
  if (!amn && bmn) return launch<BN, false, true>(p, w, st);
  if (amn && !bmn) return launch<BN, true, false>(p, w, st);
  return launch<BN, true, true>(p, w, st);
}

}  // namespace tmagemm

// Everything with a full row tile, narrow and short products too: their zero-filled boxes cost less than the cp.async
// kernel's one CTA per tile without overlap (65,536 x 256 x 16 with ReLU 39.3 -> 18.8 us, with the mask 52.6 -> 18.8;
// 65,536 x 16 x 256 21.9 -> 14.3; 512 x 256 x 16 13.0 -> 6.4).  Accumulating products stay with it below N = 64:
// there it splits K twice as fine, and the shorter fp32 chains are the more exact ones.
bool gemm_tma_fits(const GemmParams& p) { return p.M >= 128 && p.N >= 16 && p.K >= 16 && (p.epi != EPI_F32_ACC || (p.N >= 64 && p.K >= 64)); }

// Column tile width and K split from a small cost model: the operand bytes the tiles pull through L2
// (tiles x k steps x (A tile + B tile)) over the SMs that work at once (items per wave, at ~60 GB/s each), plus,
// for a split-K product, its partial tiles written and summed through HBM (~6 TB/s).  Wider tiles read A fewer
// times; narrower ones cover more SMs in short products and need fewer splits in long ones.
static int plan(const GemmParams& p, int sms, tmagemm::Work& out) {
  using namespace tmagemm;
  double best = 1e30;
  int best_bn = 64;
  for (int BN = 256; BN >= 64; BN >>= 1) {
    if (BN > 64 && BN > p.N) continue;
    Work w;
    w.gx = (p.M + 127) / 128;
    w.gy = (p.N + BN - 1) / BN;
    w.nkt = (p.K + 63) / 64;
    int split = 1;
    if (p.epi == EPI_F32_ACC) {  // split K until the work items fill the SMs once
      const int want = sms / (w.gx * w.gy);
      split = want < w.nkt ? want : w.nkt;
      if (split < 1) split = 1;
    }
    w.kt_per = (w.nkt + split - 1) / split;
    split = (w.nkt + w.kt_per - 1) / w.kt_per;
    w.items = w.gx * w.gy * split;
    const double waves = (double)((w.items + sms - 1) / sms);
    const double busy = w.items / waves;  // CTAs at work per wave, on average
    const double bytes = (double)w.gx * w.gy * w.nkt * (kABytes + BN * 128.0);
    double t = bytes / (busy * 60e9);
    if (split > 1) t += (double)split * p.M * p.N * 8.0 / 6e12;
    if (t < best) {
      best = t;
      best_bn = BN;
      out = w;
    }
  }
  return best_bn;
}

cudaError_t gemm_tma(const GemmParams& p0, bool amn, bool bmn, cudaStream_t st) {
  using namespace tmagemm;
  GemmParams p = p0;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    sms = 148;
  Work w;
  const int BN = plan(p, sms, w);
  const int split = w.items / (w.gx * w.gy);
  auto run = [&](const GemmParams& q) {
    return BN == 256 ? launch_bn<256>(q, w, amn, bmn, st)
                     : (BN == 128 ? launch_bn<128>(q, w, amn, bmn, st) : launch_bn<64>(q, w, amn, bmn, st));
  };
  if (split == 1) return run(p);
  // split K: each split's partial tile to the workspace, then C += the partials in a fixed order
  Partials ws;
  cudaError_t e = ws.get(p.ws, p.ws_bytes, (size_t)p.M * p.N * split * sizeof(float), st);
  if (e != cudaSuccess) return e;
  GemmParams q = p;
  q.epi = EPI_F32_PART;
  q.C = ws.p;
  q.ldc = p.N;
  e = run(q);
  if (e == cudaSuccess) e = sum_splits(ws.p, split, p.M, p.N, reinterpret_cast<float*>(p.C), p.ldc, st);
  const cudaError_t ef = ws.put(st);
  return e != cudaSuccess ? e : ef;
}

}  // namespace arp
