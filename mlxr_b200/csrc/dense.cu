// Quantized linear for many tokens: the weights are converted to 16 bits once, then multiplied by a dense
// GEMM on the 5th-generation tensor cores.
//
//   Y[M, N] = X[M, K] * dequant(W)[N, K]^T (+ bias),  X, Y fp16 or bf16, W in MLXR's Q4_K, Q4_0 or Q8_0
//   layout or NF4; or Y = SiLU(X gate^T) * (X up^T).
//
// The kernel that converts inside the GEMM (widem.cu) converts every weight once per 256 tokens beside the
// MMAs and draws power for it; from some number of tokens on (14336 x 4096: 1950 of Q8_0, 2500 to 3000 of the other
// formats, by how the last wave comes out; 4096 x 14336: 2200 to 3500 of Q8_0, 4000 and more of the others), one pass that writes 16-bit
// weights (2.6 bytes of traffic per weight: 27 us for 14336 x 4096, 23 at HBM's rate) costs less than the conversions it saves, and
// the GEMM behind it leaves the CUDA cores to the epilogue and runs at the tensor pipe's rate, which
// under the power cap also means a higher clock.  It takes the rows in slices of at most kSliceBytes so
// that the workspace is bounded.
//
// * weights16_kernel: a warp per row and 4096 weights of it, a lane per eight: loads and 16-byte stores are coalesced.
//   Values are rounded once to T (fp16: the reference shader's half arithmetic).
// * gemm16_kernel: pairs of CTAs (cta_group::2), 256 tokens x nt weight rows per tile, nt a multiple of 32
//   chosen so that the last wave of tiles is nearly full; persistent; six stages of 64-wide K-blocks by TMA
//   (32 KB each and CTA), two accumulators in tensor memory so that the epilogue of a tile runs beside the
//   next one's MMAs; results leave through shared memory and TMA stores.
// * Gate/up: 16 gate rows and 16 up rows alternate in the 16-bit buffer, so a thread of the epilogue holds
//   both factors of its outputs.
// * Waits on mbarriers are bounded and reported as in the other tensor-core kernels; every barrier is waited on by one
//   role in phase order.  `dead` is a CTA's own: a CTA whose partner has given up runs into its own limits, once per role.
//   Without a limit: the cluster barriers (a cluster's CTAs start together, and each role's loop ends by its last tile or its
//   first give-up), tcgen05.alloc (the shared memory leaves room for one such CTA per SM, and one that leaves has freed its
//   columns), tcgen05.wait::ld (its own loads), cp.async.bulk.wait_group (its own stores), griddepcontrol.wait (the previous kernel's end;
//   all of a launch's CTAs have started before the next launch's may, so none waits for room that a later launch holds).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "kernels.h"
#include "tc_common.cuh"
#include "weight_convert.cuh"
#include "weight_maps.h"

namespace mlxr {
namespace dense {

using namespace tc;
using namespace wconv;

constexpr size_t kSliceBytes = (size_t)256 << 20;
constexpr int kPassWords = 512;          // words (eight weights) of a row that one warp converts

// ---- 16-bit weights ------------------------------------------------------------------------------
// Eight consecutive weights, word w of a row (element 8 w ..): its bytes, then its conversion, so that the
// loads of several words are in flight together.
template <int QT> struct Word8 { uint32_t q[QT == MLXR_Q8_0 ? 2 : 1], h[QT == MLXR_Q4_K ? 3 : 1]; };

__device__ __forceinline__ uint32_t ld_u32_2b(const uint8_t* p) { return (uint32_t)ld_u16(p) | ((uint32_t)ld_u16(p + 2) << 16); }

template <int QT> __device__ __forceinline__ Word8<QT> load8w(const uint8_t* row, int w) {
  Word8<QT> o;
  if constexpr (QT == MLXR_Q4_K) {
    const uint8_t* b = row + (size_t)(w >> 5) * 144;
    const uint4 h = __ldg(reinterpret_cast<const uint4*>(b));
    o.h[0] = h.x; o.h[1] = h.y; o.h[2] = h.z;
    o.q[0] = __ldg(reinterpret_cast<const uint32_t*>(b + 16) + (w & 31));
  } else if constexpr (QT == MLXR_Q4_0) {
    const uint8_t* b = row + (size_t)(w >> 2) * 18;
    o.h[0] = ld_u16(b);
    o.q[0] = ld_u32_2b(b + 2 + 4 * (w & 3));
  } else if constexpr (QT == MLXR_Q8_0) {
    const uint8_t* b = row + (size_t)(w >> 2) * 34;
    o.h[0] = ld_u16(b);
    o.q[0] = ld_u32_2b(b + 2 + 8 * (w & 3));
    o.q[1] = ld_u32_2b(b + 6 + 8 * (w & 3));
  } else {
    const uint8_t* b = row + (size_t)(w >> 3) * 34;
    o.h[0] = ld_u16(b);
    o.q[0] = ld_u32_2b(b + 2 + 4 * (w & 7));
  }
  return o;
}

template <int QT, int BF> __device__ __forceinline__ uint4 convert8w(const Word8<QT>& o, int w, const float* nf4) {
  uint32_t r[4] = {}, lo = 0;
  if constexpr (QT == MLXR_Q4_K) {
    // sub-blocks 0, 2, 3 / 1 / 4, 6, 7 / 5 share (scale, min) pairs 0 / 1 / 2 / 3: 6-bit fields from bit 12 p
    const int s = (w >> 2) & 7, p = (s >> 2) * 2 + ((s & 3) == 1 ? 1 : 0);
    const uint32_t f = p == 3 ? o.h[2] >> 4 : p == 2 ? __funnelshift_r(o.h[1], o.h[2], 24) : o.h[1] >> (12 * p);
    const __half d = h_from_bits((uint16_t)(o.h[0] & 0xFFFFu)), dmin = h_from_bits((uint16_t)(o.h[0] >> 16));
    const __half ss = __hmul_rn(__int2half_rn((int)(f & 63u)), d), sm = __hmul_rn(__int2half_rn((int)((f >> 6) & 63u)), dmin);
    if constexpr (BF == 0) exact8_f16(o.q[0], dup_f16(ss), dup_f16(sm), r);
    else { const float sf = __half2float(ss); return dequant8_bf16(o.q[0], sf, fmaf(-136.0f, sf, __half2float(sm))); }
  } else if constexpr (QT == MLXR_Q4_0) {
    const __half d = h_from_bits((uint16_t)o.h[0]);
    if constexpr (BF == 0) exact8_f16(o.q[0], dup_f16(d), 0u, r);
    else { const float sf = __half2float(d); return dequant8_bf16(o.q[0], sf, -136.0f * sf); }
  } else if constexpr (QT == MLXR_Q8_0) {
    const float d = __half2float(h_from_bits((uint16_t)o.h[0]));
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t u = o.q[j >> 1] >> (16 * (j & 1));
      emit<BF, kRound>((float)(int)(int8_t)(u & 0xFFu) * d, (float)(int)(int8_t)((u >> 8) & 0xFFu) * d, r[j], lo);
    }
  } else {
    const float a = __half2float(h_from_bits((uint16_t)o.h[0]));
#pragma unroll
    for (int j = 0; j < 4; j++) emit<BF, kRound>(nf4[(o.q[0] >> (8 * j)) & 15u] * a, nf4[(o.q[0] >> (8 * j + 4)) & 15u] * a, r[j], lo);
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}

// out [rows][K] of T.  Row r is weight row row0 + r, or with w2 the 16 + 16 alternation of w's and w2's rows.
template <int QT, int BF>
__global__ void __launch_bounds__(256) weights16_kernel(const uint8_t* __restrict__ w, const uint8_t* __restrict__ w2, uint4* __restrict__ out,
                                                        int row0, int rows, int N, int K, size_t row_bytes) {
  __shared__ float nf4[16];
  if (QT == MLXR_NF4 && threadIdx.x < 16) nf4[threadIdx.x] = kNF4[threadIdx.x];
  if (QT == MLXR_NF4) __syncthreads();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, words = K >> 3;
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5);
  // the buffer may still be read by the previous GEMM of the stream
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (r >= rows) return;
  const int R = row0 + r, n = w2 ? 16 * (R >> 5) + (R & 15) : R;
  if (n >= N) return;
  const uint8_t* row = ((w2 && (R & 16)) ? w2 : w) + (size_t)n * row_bytes;
  uint4* dst = out + (size_t)r * words;
  const int end = min(words, (int)(blockIdx.y + 1) * kPassWords);
  for (int i = blockIdx.y * kPassWords + lane; i < end; i += 128) {
    Word8<QT> q[4];
#pragma unroll
    for (int u = 0; u < 4; u++) if (i + 32 * u < end) q[u] = load8w<QT>(row, i + 32 * u);
#pragma unroll
    for (int u = 0; u < 4; u++) if (i + 32 * u < end) dst[i + 32 * u] = convert8w<QT, BF>(q[u], i + 32 * u, nf4);
  }
}

// ---- dense GEMM ----------------------------------------------------------------------------------
constexpr int kRows = 128, kBK = 64, kStages = 6;
constexpr int kATile = kRows * kBK * 2;                 // this CTA's 128 tokens of a K-block
constexpr int kStageBytes = 2 * kATile;                 // and its half of the weight rows (up to 128)
constexpr int kOutBytes = 32 * 64;                      // a warp's 32 tokens x 32 columns on their way out
constexpr int kWarpTma = 4, kWarpMma = 5, kThreads = 6 * 32;
constexpr int kTileGroup = 8;                           // token tiles that share a sweep over the weights

struct Params {
  const void* bias;
  void* y;
  int M, N, K;                 // N, and the columns of Y this launch writes: [col0, N)
  int col0, ldy;
  int nt, mtiles, ntiles;      // weight rows per tile; token tiles, weight tiles
  int tma_store;               // Y's rows start on 16 bytes
  int* status;
};
struct Maps { CUtensorMap x, w, y; };
struct Shared {
  uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int dead;
};
constexpr size_t kSmem = (size_t)kStages * kStageBytes + 4 * 2 * kOutBytes + sizeof(Shared) + 1024;
static_assert(kSmem <= 227 * 1024, "shared memory");

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(src), "r"(x), "r"(y) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

template <typename T, bool SWIGLU>
__global__ void __launch_bounds__(kThreads, 1) gemm16_kernel(const __grid_constant__ Maps maps, const Params P) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
  uint8_t* ring = smem_raw + pad;
  uint8_t* outs = ring + (size_t)kStages * kStageBytes;
  Shared* sh = reinterpret_cast<Shared*>(outs + 4 * 2 * kOutBytes);
  volatile int* dead = &sh->dead;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int rank = (int)cluster_rank(), pairs = gridDim.x >> 1, pair = blockIdx.x >> 1;
  if (tid < (P.tma_store ? 3 : 2)) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tid == 0 ? &maps.x : tid == 1 ? &maps.w : &maps.y)) : "memory");
  if (tid == 0) {
    sh->dead = 0;
    for (int s = 0; s < kStages; s++) {
      mbar_init(smem_u32(&sh->full[s]), 1);
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(smem_u32(&sh->acc_full[a]), 1);
      mbar_init(smem_u32(&sh->acc_empty[a]), 8);       // epilogue warps of both CTAs (the first CTA's barrier is used)
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  cluster_arrive();       // both CTAs run and have their barriers before either signals the other or allocates in both SMs' tensor memory
  cluster_wait();
  if (warp == kWarpMma) tmem_alloc_pair(smem_u32(&sh->tmem_base), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&sh->tmem_base);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");      // X, the 16-bit weights and Y

  const int nkb = (P.K + kBK - 1) / kBK, ntile = P.mtiles * P.ntiles;
  // token tile and weight tile of tile t: groups of kTileGroup token tiles, weight tiles inside a group
  auto tile_of = [&](int t, int& mt, int& wt) {
    const int per = P.ntiles * kTileGroup, g = t / per, r = t - g * per, gs = min(kTileGroup, P.mtiles - g * kTileGroup);
    wt = r / gs;
    mt = g * kTileGroup + r - wt * gs;
  };

  if (warp == kWarpTma) {
    // ===== copies: this CTA's 128 tokens and its half of the tile's weight rows; both CTAs' complete on the
    // first one's barrier =====
    if (lane == 0) {
      int i = 0;
      bool ok = true;
      for (int t = pair; t < ntile && ok; t += pairs) {
        int mt, wt;
        tile_of(t, mt, wt);
        const int xrow = 256 * mt + kRows * rank, wrow = P.nt * wt + (P.nt / 2) * rank;
        for (int kb = 0; kb < nkb; kb++, i++) {
          const int s = i % kStages;
          ok = mbar_wait(smem_u32(&sh->empty[s]), (uint32_t)((i / kStages) & 1) ^ 1u, dead);
          if (!ok) break;
          const uint32_t bar = smem_u32(&sh->full[s]), cbar = cluster_map(bar, 0), dst = smem_u32(ring + (size_t)s * kStageBytes);
          if (rank == 0) mbar_expect_tx(bar, 2u * kATile + (uint32_t)P.nt * kBK * 2);
          tma_load_2d_pair(dst, &maps.x, kb * kBK, xrow, cbar);
          tma_load_2d_pair(dst + kATile, &maps.w, kb * kBK, wrow, cbar);
        }
      }
      if (*dead) {
        // a give-up: copies in flight must land before either CTA exits; time is given to them (they take microseconds)
        if (i > 0) for (int k = 0; k < 100; k++) __nanosleep(2000);
      } else {
        // the stages' last releases come from the pair's issuer: none may still be on its way when this CTA exits, or it would
        // arrive in the shared memory of whatever runs here next
        for (int k = max(0, i - kStages); k < i; k++) mbar_wait(smem_u32(&sh->empty[k % kStages]), (uint32_t)(k / kStages) & 1u, dead);
      }
    }
  } else if (warp == kWarpMma) {
    if (rank == 0) {
      // ===== MMA issuer of the pair: the whole warp walks the loop, one elected lane issues =====
      const uint32_t idesc = instr_desc(Fmt<T>::v, Fmt<T>::v, 2 * kRows, P.nt);
      const uint64_t desc_hi = smem_desc_sw128(0);
      const uint32_t base = (smem_u32(ring) & 0x3FFFFu) >> 4, tm = __shfl_sync(0xffffffffu, tmem, 0);
      int i = 0, part = 0;
      bool ok = true;
      for (int t = pair; t < ntile && ok; t += pairs, part++) {
        const int ab = part & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->acc_empty[ab]), (uint32_t)((part >> 1) & 1) ^ 1u, dead));
        for (int kb = 0; kb < nkb && ok; kb++, i++) {
          const int s = i % kStages;
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->full[s]), (uint32_t)(i / kStages) & 1u, dead));
          if (!ok) break;
          tc_fence_after();
          const uint64_t adesc = desc_hi | (uint64_t)(base + (uint32_t)s * (kStageBytes >> 4)), bdesc = adesc + (kATile >> 4);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < kBK / kUmmaK; k++)
              umma_f16_pair(tm + (uint32_t)(ab * 256), adesc + (uint64_t)(k * (kUmmaK * 2 >> 4)), bdesc + (uint64_t)(k * (kUmmaK * 2 >> 4)), idesc, (kb > 0 || k > 0) ? 1u : 0u);
            umma_commit_pair(smem_u32(&sh->empty[s]));
            if (kb == nkb - 1) umma_commit_pair(smem_u32(&sh->acc_full[ab]));
          }
          __syncwarp();
        }
      }
    }
  } else {
    // ===== epilogue: warp q owns TMEM lanes 32 q .. 32 q + 31 = 32 tokens of this CTA's 128 =====
    const uint32_t acc_free[2] = {cluster_map(smem_u32(&sh->acc_empty[0]), 0), cluster_map(smem_u32(&sh->acc_empty[1]), 0)};
    constexpr int kCols = SWIGLU ? 16 : 32;                // columns of Y per 32 accumulator columns
    const T* bias = reinterpret_cast<const T*>(P.bias);
    T* y = reinterpret_cast<T*>(P.y);
    int part = 0, buf = 0;
    for (int t = pair; t < ntile; t += pairs, part++) {
      const int ab = part & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->acc_full[ab]), (uint32_t)(part >> 1) & 1u, dead))) break;
      tc_fence_after();
      int mt, wt;
      tile_of(t, mt, wt);
      const int m0 = 256 * mt + kRows * rank + 32 * warp;
#pragma unroll 1
      for (int c = 0; c < P.nt; c += 32) {
        const int n0 = P.col0 + (SWIGLU ? (P.nt * wt + c) / 2 : P.nt * wt + c);
        if (m0 >= P.M || n0 >= P.N) break;
        uint32_t r[32];
        tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(ab * 256 + c), r);
        uint32_t o[kCols / 2];
#pragma unroll
        for (int e = 0; e < kCols / 2; e++) {
          T v[2];
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const int j = 2 * e + k;
            if constexpr (SWIGLU) {
              const float g = Act<T>::to_f(Act<T>::from_f(__uint_as_float(r[j]))), u = Act<T>::to_f(Act<T>::from_f(__uint_as_float(r[16 + j])));
              v[k] = Act<T>::from_f(swish_h(g) * u);
            } else {
              v[k] = Act<T>::from_f(__uint_as_float(r[j]) + (bias && n0 + j < P.N ? Act<T>::to_f(bias[n0 + j]) : 0.0f));
            }
          }
          o[e] = (uint32_t)*reinterpret_cast<const uint16_t*>(&v[0]) | ((uint32_t)*reinterpret_cast<const uint16_t*>(&v[1]) << 16);
        }
        uint8_t* dst = outs + (size_t)(warp * 2 + buf) * kOutBytes;
        if (P.tma_store) {
          // the store that last read this buffer must be done with it
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          __syncwarp();
#pragma unroll
          for (int p = 0; p < kCols / 8; p++) {
            // 16-byte piece p of the row; 64-byte rows with the 64-byte swizzle, 32-byte rows plain
            const int at = SWIGLU ? p : p ^ ((lane >> 1) & 3);
            *reinterpret_cast<uint4*>(dst + lane * (kCols * 2) + at * 16) = make_uint4(o[4 * p], o[4 * p + 1], o[4 * p + 2], o[4 * p + 3]);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) tma_store_2d(&maps.y, smem_u32(dst), n0, m0);
          buf ^= 1;
        } else {
          // rows of Y start anywhere: turn in shared memory (rows 4 bytes apart from a multiple of 64), a
          // row's columns by consecutive lanes
          uint16_t* turn = reinterpret_cast<uint16_t*>(outs + (size_t)warp * 2 * kOutBytes);
          constexpr int kPitch = kCols + 2;
#pragma unroll
          for (int e = 0; e < kCols / 2; e++) *reinterpret_cast<uint32_t*>(turn + lane * kPitch + 2 * e) = o[e];
          __syncwarp();
          const int col = lane % kCols, rr0 = lane / kCols;
#pragma unroll 4
          for (int rr = rr0; rr < 32; rr += 32 / kCols)
            if (m0 + rr < P.M && n0 + col < P.N) y[(size_t)(m0 + rr) * P.ldy + n0 + col] = *reinterpret_cast<const T*>(turn + rr * kPitch + col);
          __syncwarp();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_free[ab]);
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();         // neither CTA's memory is read or signalled by the other any more
  cluster_wait();
  if (warp == kWarpMma) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, 512);
  }
  __syncwarp();
  cluster_arrive();         // and neither leaves while the other still frees columns in both SMs
  cluster_wait();
  if (tid == 0 && sh->dead) atomicExch(P.status, MLXR_ERR_TIMEOUT);
}

}  // namespace dense

// ---- host side -----------------------------------------------------------------------------------
// K = 32 mod 64 stays with the generic kernel, which multiplies the float32 weights (rounded to 16 bits the result is 1.4
// times as far from the exact one)
bool dense_supported(int qt, int M, int N, int K, int dtype, const void* x, const void* w) {
  if (qt != MLXR_Q4_K && qt != MLXR_Q4_0 && qt != MLXR_Q8_0 && qt != MLXR_NF4) return false;
  if (dtype != MLXR_F16 && dtype != MLXR_BF16) return false;
  if (M < 9 || N < 1 || K < 64 || K % 64 != 0 || K % block_elems(qt) != 0) return false;
  if (qt == MLXR_Q4_K && (((uintptr_t)w) & 15u)) return false;      // 16-byte headers
  return (((uintptr_t)x) & 15u) == 0;
}

// Weight rows per tile, rows per slice of the 16-bit buffer, and an estimate of the time.  A tile takes K / 16
// MMAs of about 60 + 0.3 nt cycles each (fitted: 137 at 256 rows, where the pipe allows 128; 98 at 128, where
// it allows 64 but reading the tokens' operand again for every tile sets the pace), so wide tiles are better
// unless their last wave over the pairs of SMs is nearly empty (2048 tokens x 14336 rows x 4096: 448 tiles of
// 256 rows are 6.05 waves on 74 pairs, 184 us; 512 tiles of 224 are 6.92 waves, 176 us).
int dense_plan(int M, int rows, int K, DensePlan* out) {
  int sms = 0;
  if (int r = device_sms(&sms)) return r;
  const int pairs = sms / 2, mtiles = (M + 255) / 256;
  const size_t row_bytes = (size_t)K * 2;
  const int most = (int)std::max<size_t>(256, (dense::kSliceBytes / row_bytes) & ~(size_t)255);
  const int slices = (rows + most - 1) / most;
  const int slice = slices == 1 ? rows : ((rows + slices - 1) / slices + 255) / 256 * 256;
  double best = 1e300;
  for (int nt = 256; nt >= 128; nt -= 32) {
    const long long tiles = (long long)mtiles * ((slice + nt - 1) / nt);
    const double waves = (double)((tiles + pairs - 1) / pairs);
    const double c = waves * (K / 16.0 * (60.0 + 0.3 * nt) + 300.0) + 3000.0;
    if (c < best) { best = c; out->nt = nt; }
  }
  out->slice = slice;
  out->bytes = (size_t)slice * row_bytes;
  // short launches take less than the sum of their parts, which overlap; long ones more, at the clock that the power cap leaves and with X
  // that does not stay in L2 (to 20 us 0.95 to 1.0 of it, 100 us 1.2, 250 us 1.3, 800 us 1.37 in runs of half a second each).  Rows that do not start
  // on 16 bytes leave by plain stores
  const double us = slices * (best / 1700.0 + 3.0) + (double)rows * K * 2.6 / 5.0e6 + 3.0;
  out->cost_us = us * (0.65 + 0.1 * std::log(us)) * (rows % 8 ? 1.1 : 1.0);
  return MLXR_OK;
}

// programmatic stream serialization, clusters of `cluster` CTAs
static void launch_config(dim3 grid, int threads, size_t smem, int cluster, cudaStream_t st, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
  *cfg = {};
  cfg->gridDim = grid;
  cfg->blockDim = dim3(threads);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = st;
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = overlap_launches() ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg->attrs = at;
  cfg->numAttrs = cluster > 1 ? 2 : 1;
}

template <int QT, int BF>
static int launch_weights16(const void* w, const void* w2, void* out, int row0, int rows, int N, int K, cudaStream_t st) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  auto kern = dense::weights16_kernel<QT, BF>;
  launch_config(dim3((rows + 7) / 8, (K / 8 + dense::kPassWords - 1) / dense::kPassWords), 256, 0, 1, st, &cfg, at);
  const size_t row_bytes = (size_t)(K / block_elems(QT)) * block_bytes(QT);
  MLXR_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, (const uint8_t*)w, (const uint8_t*)w2, (uint4*)out, row0, rows, N, K, row_bytes));
  count_launch();
  return MLXR_OK;
}

template <typename T, bool SWIGLU>
static int launch_gemm16(const dense::Maps& maps, const dense::Params& P, cudaStream_t st) {
  using namespace dense;
  auto kern = gemm16_kernel<T, SWIGLU>;
  static std::atomic<bool> attr_done[64] = {};
  int dev = 0, sms = 0;
  MLXR_CUDA_TRY(cudaGetDevice(&dev));
  if (!attr_done[dev & 63].load(std::memory_order_acquire)) {
    MLXR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    attr_done[dev & 63].store(true, std::memory_order_release);
  }
  if (int r = device_sms(&sms)) return r;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  launch_config(dim3(2 * std::min(sms / 2, P.mtiles * P.ntiles)), kThreads, kSmem, 2, st, &cfg, at);
  MLXR_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, maps, P));
  count_launch();
  return MLXR_OK;
}

// buf: plan.bytes of scratch for the 16-bit weights.  w2 == nullptr: Y = X W^T (+ bias); otherwise gate / up.
int launch_dense(const void* x, const void* w, const void* w2, const void* bias, void* y, int M, int N, int K, int qt, int dtype,
                 int* status, void* buf, const DensePlan& plan, cudaStream_t st) {
  const bool swiglu = w2 != nullptr;
  const int rows = swiglu ? 32 * ((N + 15) / 16) : N;
  dense::Maps maps;
  dense::Params P;
  memset(&maps, 0, sizeof(maps));
  memset(&P, 0, sizeof(P));
  if (int r = activation_map(x, M, K, dtype, dense::kRows, &maps.x)) return r;
  P.tma_store = N % 8 == 0 && ((uintptr_t)y & 15u) == 0;
  if (P.tma_store)
    if (int r = result_map(y, M, N, dtype, swiglu ? 16 : 32, 32, &maps.y)) return r;
  P.bias = bias;
  P.y = y;
  P.M = M; P.N = N; P.K = K;
  P.ldy = N;
  P.nt = plan.nt;
  P.mtiles = (M + 255) / 256;
  P.status = status;
  for (int row0 = 0; row0 < rows; row0 += plan.slice) {
    const int n = std::min(plan.slice, rows - row0);
    int rc = MLXR_ERR_UNSUPPORTED;
#define MLXR_W16(QTV) rc = dtype == MLXR_F16 ? launch_weights16<QTV, 0>(w, w2, buf, row0, n, N, K, st) : launch_weights16<QTV, 1>(w, w2, buf, row0, n, N, K, st)
    switch (qt) {
      case MLXR_Q4_K: MLXR_W16(MLXR_Q4_K); break;
      case MLXR_Q4_0: MLXR_W16(MLXR_Q4_0); break;
      case MLXR_Q8_0: MLXR_W16(MLXR_Q8_0); break;
      case MLXR_NF4: MLXR_W16(MLXR_NF4); break;
      default: set_error("dense path: no conversion for %s", mlxr_quant_type_name(qt)); break;
    }
#undef MLXR_W16
    if (rc) return rc;
    if (int r = activation_map(buf, n, K, dtype, plan.nt / 2, &maps.w)) return r;
    P.col0 = swiglu ? row0 / 2 : row0;
    P.ntiles = (n + plan.nt - 1) / plan.nt;
    P.N = swiglu ? std::min(N, (row0 + n) / 2) : row0 + n;      // the slice's columns end here
    if (dtype == MLXR_F16) rc = swiglu ? launch_gemm16<__half, true>(maps, P, st) : launch_gemm16<__half, false>(maps, P, st);
    else rc = swiglu ? launch_gemm16<__nv_bfloat16, true>(maps, P, st) : launch_gemm16<__nv_bfloat16, false>(maps, P, st);
    if (rc) return rc;
  }
  return MLXR_OK;
}

}  // namespace mlxr
