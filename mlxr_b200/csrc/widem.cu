// Quantized linear for 65 and more tokens, as long as dense.cu is not faster (14336 x 4096: to 2000 .. 3000, by format), on the 5th-generation
// tensor cores, every weight converted once per 256 tokens:
//
//   Y[M, N] = X[M, K] * dequant(W)[N, K]^T (+ bias),  X, Y fp16 or bf16, W in MLXR's Q4_K, Q4_0 or
//   Q8_0 layout or NF4 (q_gemm_dequant.metal:142-260 for the formats).
//
// The form of the small-batch kernel (smallm.cu) for more tokens, on pairs of CTAs: 2 x 128 weight rows are
// the M side of a cta_group::2 MMA and live in the two SMs' tensor memories as its A operand, up to 256
// tokens are its N side, half of them in each SM's shared memory.  Shared memory then carries 64
// bytes a cycle (X written by TMA and read by the MMAs) of the 128 it can, and an SM fetches 32 bytes a
// cycle of X from L2; one CTA per tile asked for twice that and ran at half the tensor rate, and
// converted tiles in shared memory (the form before) for 170 bytes a cycle.
//
// * Tiles are (256 weight rows) x (nt tokens), nt a multiple of 16 chosen with the number of token
//   tiles so that the last one is not padding (333 tokens: two tiles of 176, not 512 rows of which 179
//   are empty).  Work units are (tile, 256-wide super-block of K), weight tile-major with token tiles
//   inside, so a weight tile's second reading comes from L2.  (Taken back: tiles of up to 384 tokens, which convert a weight once for 333 tokens, 70.1 us
//   instead of 65.4 on 22016 x 4096 Q4_0; the last wave's tiles shared by up to six pairs, 67.8: under the power cap idle SMs cost
//   little, parts' trips through L2 more.)
//   Token tiles go in groups of eight, weight tiles inside a group, so that a group's X stays in L2.
// * With few tiles per pair the units are dealt to the pairs in equal contiguous ranges and shared tiles
//   are added up by the CTA that delivers the last part; with many, every pair takes whole tiles.
// * Four groups of four producer warps convert a 64-wide k-block of the unit each, double-buffered in
//   tensor memory; two k-blocks' weights and X tiles share a stage and with it one barrier each way; one warp of the pair's first CTA issues.
// * Weights are rounded once to the activation dtype (fp16: the reference shader's half arithmetic).
// * Waits are bounded and reported as in smallm.cu; every barrier is waited on by one role in phase order.
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
namespace widem {

using namespace tc;
using namespace wconv;

constexpr int kRows = 128, kBK = 64;
constexpr int kGroups = 4;                 // producer groups of four warps; group g converts k-block g of every unit
constexpr int kSlots = 2;                  // converted k-blocks per group
// A stage is half a unit, two k-blocks: their converted weights (two groups' slots) and their X tiles (one copy), with one
// barrier each way.  What a hand-over costs the warps that copy X and issue MMAs is the same for one k-block as for two:
// with a stage and a copy for each k-block the copy warp needed 500 cycles for one (time stamps; the conversion 400),
// 2050 a unit whatever the number of tokens.
constexpr int kBlocks = 2;
constexpr int kHalves = kGroups / kBlocks;
constexpr int kStages = kHalves * kSlots;  // stage (unit & 1) * kHalves + half
constexpr int kSlotCols = kBK / 2;         // tensor-memory columns of one: two 16-bit elements each
[[maybe_unused]] constexpr int kWarpMma = 0, kWarpRaw = 1, kWarpX = 2, kWarpFix = 3, kWarpEpi0 = 4, kWarpProd0 = 8;
constexpr int kThreads = (kWarpProd0 + 4 * kGroups) * 32;
constexpr int kTileGroup = 8;              // token tiles that share a sweep over the weights
constexpr int kSmemMax = 227 * 1024;
constexpr int kMaxRawStages = 4;

struct Params {
  const void* bias;
  void* y;
  int M, N, K;
  int nsb;             // super-blocks per row = K / 256
  int nt, ntt;         // tokens per tile, token tiles
  int wtiles;          // 256-row weight tiles (gate/up: 128 output columns)
  int ntiles;          // weight tiles * ntt
  int whole;           // every pair takes whole tiles
  int vec_stores;      // rows of Y start on 16 bytes
  int odd_shift;       // NF4: byte offset of odd rows within their tensor map (0 or 8)
  int* status;
  float* partials;     // [grid][2][nt][128] fp32: a CTA's first tile's part, its last tile's part
  uint32_t* counters;  // two per tile (one per CTA of the pair), self-clearing
};
struct Maps { CUtensorMap x, w[4]; };

struct Shared {
  uint64_t full[kStages];       // (first CTA) both CTAs' producer warps have written their k-blocks, both halves of X have landed
  uint64_t empty[kStages];      // the MMAs that read it are done
  uint64_t raw_full[kMaxRawStages], raw_empty[kMaxRawStages];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int dead, epi_fail;
  int ntodo, todo_tile[2], todo_first[2], todo_parts[2];
  alignas(16) uint32_t turn[4][16 * 32];    // epilogue warps: 32 tokens' results on their way to 16-byte stores
};

// The table that a format's producers look codes up in (weight_convert.cuh), behind the rings.  Up to 128 tokens a
// tile the conversion sets the pace (1530 cycles a unit of fp16 Q4_0 with arithmetic alone, 128 tokens' MMAs 1024); the
// wider tiles' X leaves no room for a table, and their MMAs take 2048.
struct LevelTable : Levels {
  static constexpr int kBytes = 64;
  __device__ __forceinline__ LevelTable(const uint8_t* table, int) : Levels{reinterpret_cast<const float*>(table)} {}
  static __device__ __forceinline__ void fill(uint8_t* table, int tid, int) { if (tid < 16) reinterpret_cast<float*>(table)[tid] = kNF4[tid]; }
};
template <int QT, int BF, int NMAX> struct TableOf { using type = LevelTable; };
template <int BF> struct TableOf<MLXR_NF4, BF, 128> { using type = LanePairLevels; };
template <> struct TableOf<MLXR_Q4_K, 0, 128> { using type = CodePairs<0>; };
template <> struct TableOf<MLXR_Q4_0, 0, 128> { using type = CodePairs<0>; };
template <> struct TableOf<MLXR_Q4_K, 1, 128> { using type = CodePairs32; };
template <> struct TableOf<MLXR_Q4_0, 1, 128> { using type = CodePairs32; };

template <int QT, int BF, int NMAX> struct Rings {
  static constexpr int kRawBytes = kRows * Geo<QT>::kStage;
  static constexpr int kXStage = kBlocks * NMAX / 2 * kBK * 2;               // this CTA's half of the tokens, two tiles of nt / 2 rows
  static constexpr int kRawStages = QT != MLXR_Q8_0 ? 4 : 2;
  using Tab = typename TableOf<QT, BF, NMAX>::type;
  static constexpr size_t kBytes = Tab::kBytes + (size_t)kStages * kXStage + (size_t)kRawStages * kRawBytes;
  static constexpr int kBufs = NMAX == 128 ? 2 : 1;
  static constexpr uint32_t kA0 = 256, kCols = 512;                          // accumulators in columns 0 .. 255
};

// first unit of pair c, and the pair that owns unit u, when U units are dealt to G pairs
__device__ inline long long unit_begin(long long U, int G, int c) { return (U * c) / G; }
__device__ inline int unit_owner(long long U, int G, long long u) { return (int)(((u + 1) * G - 1) / U); }

// SiLU(gate) * up of two outputs held by a pair of lanes FAR apart: the lower lane has both gates, the upper one both ups.
// Each of the two computes one output (the upper lane the second): with SiLU on one lane for both the block of 333 tokens,
// 4096 x 11008, took 9 % more when that was measured (138 us and 127, of the 107 it takes now).
template <typename T> struct Pair { T value; int second; };
template <typename T, int FAR> __device__ __forceinline__ Pair<T> swiglu_pair(float a, float b, int lane) {
  const bool up = (lane & FAR) != 0;
  const float o = __shfl_xor_sync(0xffffffffu, up ? a : b, FAR);
  const float g = Act<T>::to_f(Act<T>::from_f(up ? o : a)), u = Act<T>::to_f(Act<T>::from_f(up ? b : o));
  return {Act<T>::from_f(swish_h(g) * u), up ? 1 : 0};
}

// two values rounded to T in one word, the first in its low half
template <typename T> __device__ __forceinline__ uint32_t pack2(float a, float b) {
  if constexpr (Act<T>::kDtype == MLXR_F16) { const __half2 v = __floats2half2_rn(a, b); return *reinterpret_cast<const uint32_t*>(&v); }
  else { const __nv_bfloat162 v = __floats2bfloat162_rn(a, b); return *reinterpret_cast<const uint32_t*>(&v); }
}

// weight tile and token tile of tile t
struct Tile { int wt, tt; };
__device__ __forceinline__ Tile tile_of(const Params& P, int t) {
  const int per = P.wtiles * kTileGroup, g = t / per, r = t - g * per, gs = min(kTileGroup, P.ntt - g * kTileGroup);
  const int wt = r / gs;
  return {wt, g * kTileGroup + r - wt * gs};
}

__device__ __forceinline__ void epi_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// SWIGLU: a tile's rows are 16 gate rows and 16 up rows per TMEM lane quarter, Y = SiLU(gate) * up with
// both rounded to T first, N = the number of gate rows; a tile covers 64 output columns.
template <int QT, typename T, int NMAX, bool SWIGLU>
__global__ void __launch_bounds__(kThreads, 1)
qgemm_widem_kernel(const __grid_constant__ Maps maps, const Params P) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  constexpr int BF = Fmt<T>::v;
  constexpr bool kSplitRows = QT == MLXR_NF4;
  if (threadIdx.x < 5) {
    const CUtensorMap* m = threadIdx.x == 4 ? &maps.x : &maps.w[threadIdx.x];
    if (threadIdx.x == 4 || threadIdx.x < (SWIGLU ? 2 : 1) * (kSplitRows ? 2 : 1))
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
  }
  using R = Rings<QT, BF, NMAX>;
  using Tab = typename R::Tab;
  constexpr int kRawStages = R::kRawStages, kXStage = R::kXStage, kRawBytes = R::kRawBytes;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw & 1023u)) & 1023u;
  uint8_t* xring = smem_raw + pad;
  uint8_t* rawring = xring + (size_t)kStages * kXStage;
  uint8_t* table = rawring + (size_t)kRawStages * kRawBytes;
  Shared* sh = reinterpret_cast<Shared*>(table + Tab::kBytes);
  volatile int* dead = &sh->dead;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int rank = (int)cluster_rank(), G = gridDim.x >> 1, pair = blockIdx.x >> 1, cta = blockIdx.x;
  const long long U = (long long)P.ntiles * P.nsb;

  // this pair's units [u0, u1): unit u = (tile u / nsb, super-block u % nsb)
  const long long u0 = P.whole ? unit_begin(P.ntiles, G, pair) * P.nsb : unit_begin(U, G, pair);
  const long long u1 = P.whole ? unit_begin(P.ntiles, G, pair + 1) * P.nsb : unit_begin(U, G, pair + 1);
  const int nunits = (int)(u1 - u0);
  const int t_first = (int)(u0 / P.nsb), sb_first = (int)(u0 - (long long)t_first * P.nsb);

  // packed rows of unit (t, sb) into stage r: one box (two for gate/up; for NF4 one per row parity)
  auto load_raw = [&](int t, int sb, int r) {
    constexpr int nbox = (SWIGLU ? 2 : 1) * (kSplitRows ? 2 : 1);
    const uint32_t bar = smem_u32(&sh->raw_full[r]);
    mbar_expect_tx(bar, kRawBytes);
    const int row0 = (SWIGLU ? 64 : kRows) * (2 * tile_of(P, t).wt + rank);
#pragma unroll
    for (int b = 0; b < nbox; b++) {
      int x = Geo<QT>::kUnit / 8 * sb, y = row0;
      if constexpr (kSplitRows) { x = ((136 * sb + ((b & 1) ? P.odd_shift : 0)) & ~15) >> 3; y = row0 >> 1; }
      tma_load_2d(smem_u32(rawring + (size_t)r * kRawBytes + (size_t)b * (kRawBytes / nbox)), &maps.w[b], x, y, bar);
    }
  };
  int raw_t = t_first, raw_sb = sb_first, raw_issued = 0;     // copy warp: the next unit to request
  if (tid == kWarpRaw * 32) {
    for (int r = 0; r < kRawStages; r++) {
      mbar_init(smem_u32(&sh->raw_full[r]), 1);
      mbar_init(smem_u32(&sh->raw_empty[r]), 4 * kGroups);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (; raw_issued < min(nunits, kRawStages); raw_issued++) {
      load_raw(raw_t, raw_sb, raw_issued);
      if (++raw_sb == P.nsb) { raw_sb = 0; raw_t++; }
    }
  }
  if (tid == 0) {
    sh->dead = 0;
    sh->ntodo = 0;
    sh->epi_fail = 0;
    for (int s = 0; s < kStages; s++) {
      mbar_init(smem_u32(&sh->full[s]), kBlocks * 4 * 2 + 1);    // the groups' four warps of both CTAs, the copy warp's byte count
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(smem_u32(&sh->acc_full[a]), 1);
      mbar_init(smem_u32(&sh->acc_empty[a]), 8);       // epilogue warps of both CTAs
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  Tab::fill(table, tid, kThreads);
  __syncthreads();
  cluster_arrive();       // both CTAs run and have their barriers before either signals the other or allocates in both SMs' tensor memory
  cluster_wait();
  if (warp == kWarpMma) tmem_alloc_pair(smem_u32(&sh->tmem_base), R::kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&sh->tmem_base);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp >= kWarpProd0) {
    // ===== producers: k-block g of every unit =====
    const int g = (warp - kWarpProd0) >> 2, p = (warp & 3) * 32 + lane;
    const int local = SWIGLU ? 16 * (warp & 3) + (lane & 15) : p;     // row within the matrix's part of the tile
    const int mrows = SWIGLU ? 64 : 128;
    const int mat_off = (SWIGLU && lane >= 16) ? 64 : 0;
    const int row_off = (kSplitRows ? mat_off + (local & 1) * (mrows / 2) + (local >> 1) : mat_off + local) * Geo<QT>::kStage;
    const uint32_t col = tmem + R::kA0 + (uint32_t)(g * kSlots * kSlotCols) + ((uint32_t)((warp & 3) * 32) << 16);
    const int half = g / kBlocks;
    const uint32_t full[2] = {cluster_map(smem_u32(&sh->full[half]), 0), cluster_map(smem_u32(&sh->full[kHalves + half]), 0)};
    const Tab levels(table, lane);
    int r = 0, sb = sb_first;
    uint32_t rpar = 0;
    for (int i = 0; i < nunits; i++) {
      const int q = i & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->raw_full[r]), rpar, dead))) break;   // warp-uniform
      const uint8_t* row = rawring + (size_t)r * kRawBytes + row_off;
      if constexpr (kSplitRows) row += (136 * sb + ((local & 1) ? P.odd_shift : 0)) & 8;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->empty[q * kHalves + half]), (uint32_t)((i >> 1) & 1) ^ 1u, dead))) break;
      tc_fence_after();
      convert64<QT, BF, kRound>(row, g, levels, [&](auto H, const uint32_t (&a)[16], const uint32_t (&)[16]) {
        tmem_st16(col + q * kSlotCols + 16 * decltype(H)::value, a);
      });
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { mbar_arrive_cluster(full[q]); mbar_arrive(smem_u32(&sh->raw_empty[r])); }
      if (++r == kRawStages) { r = 0; rpar ^= 1u; }
      if (++sb == P.nsb) sb = 0;
    }
  } else if (warp == kWarpMma) {
   if (rank == 0) {
    // ===== MMA issuer of the pair: the whole warp walks the loop, one elected lane issues =====
    const uint32_t idesc = instr_desc(BF, BF, 2 * kRows, P.nt);
    const uint64_t desc_hi = smem_desc_sw128(0);
    const uint32_t x_lo0 = (smem_u32(xring) & 0x3FFFFu) >> 4, tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t x_tile = (uint32_t)P.nt * (kBK >> 4);         // nt / 2 rows of 128 bytes, in units of 16 bytes
    bool ok = true;
    for (int i0 = 0, part = 0, cnt; i0 < nunits && ok; i0 += cnt, part++) {
      cnt = min(part == 0 ? P.nsb - sb_first : P.nsb, nunits - i0);
      const int ab = part % R::kBufs;
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->acc_empty[ab]), ((part / R::kBufs) & 1) ^ 1u, dead));
      const uint32_t dcol = tm + (uint32_t)(ab * NMAX);
      for (int i = i0; i < i0 + cnt && ok; i++) {
        const int q = i & 1;
#pragma unroll
        for (int h = 0; h < kHalves; h++) {
          const int st = q * kHalves + h;
          ok = __all_sync(0xffffffffu, ok && mbar_wait(smem_u32(&sh->full[st]), (uint32_t)(i >> 1) & 1u, dead));
          if (!ok) break;
          tc_fence_after();
          const uint32_t acol = tm + R::kA0 + (uint32_t)((h * kBlocks * kSlots + q) * kSlotCols);
          const uint64_t xdesc = desc_hi | (uint64_t)(x_lo0 + (uint32_t)st * (kXStage >> 4));
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < kBlocks * kBK / kUmmaK; k++) {
              const int kb = k / (kBK / kUmmaK), kk = k % (kBK / kUmmaK);
              umma_f16_ts_pair(dcol, acol + kb * kSlots * kSlotCols + kk * (kUmmaK / 2), xdesc + (uint64_t)(kb * x_tile + kk * (kUmmaK * 2 >> 4)), idesc,
                               (i > i0 || h > 0 || k > 0) ? 1u : 0u);
            }
            umma_commit_pair(smem_u32(&sh->empty[st]));
          }
          __syncwarp();
        }
      }
      if (ok && elect_one()) umma_commit_pair(smem_u32(&sh->acc_full[ab]));
      __syncwarp();
    }
   }
  } else if (warp == kWarpRaw) {
    // ===== packed weights: the ring was filled once above =====
    if (lane == 0) {
      for (int i = raw_issued; i < nunits; i++) {
        const int r = i % kRawStages;
        if (!mbar_wait(smem_u32(&sh->raw_empty[r]), (uint32_t)(i / kRawStages - 1) & 1u, dead)) break;
        load_raw(raw_t, raw_sb, r);
        raw_issued = i + 1;
        if (++raw_sb == P.nsb) { raw_sb = 0; raw_t++; }
      }
      if (*dead) {   // copies in flight must land before the CTA may exit (bounded)
        for (int i = max(0, raw_issued - kRawStages); i < raw_issued; i++) {
          const uint32_t bar = smem_u32(&sh->raw_full[i % kRawStages]);
          for (uint32_t sp = 0; sp < kSpin; sp++) if (mbar_try(bar, (i / kRawStages) & 1)) break;
        }
      }
    }
  } else if (warp == kWarpX) {
    // ===== activations: this CTA's half of two X tiles [nt rows, 64 columns] per stage, one copy; both CTAs' complete on the
    // first one's barrier.  The whole warp walks the loop, one elected lane issues. =====
    int issued = 0, t = t_first, hb = kHalves * sb_first;
    int tok = tile_of(P, t).tt * P.nt + rank * (P.nt / 2);
    const uint32_t bytes = kBlocks * (uint32_t)P.nt * kBK * 2;
    asm volatile("griddepcontrol.wait;" ::: "memory");      // X may be the previous kernel's output
    for (int i = 0; i < kHalves * nunits; i++) {
      const int st = i % kStages;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->empty[st]), (uint32_t)((i / kStages) & 1) ^ 1u, dead))) break;
      const uint32_t bar = smem_u32(&sh->full[st]);
      if (elect_one()) {
        if (rank == 0) mbar_expect_tx(bar, bytes);
        tma_load_3d_pair(smem_u32(xring + (size_t)st * kXStage), &maps.x, 0, tok, kBlocks * hb, cluster_map(bar, 0));
      }
      __syncwarp();
      issued = i + 1;
      if (++hb == kHalves * P.nsb && i + 1 < kHalves * nunits) { hb = 0; t++; tok = tile_of(P, t).tt * P.nt + rank * (P.nt / 2); }
    }
    if (*dead) {
      // a give-up: copies in flight must land before either CTA exits; their barrier also counts the producers,
      // so time is given to them instead (a copy takes microseconds)
      if (issued > 0) for (int i = 0; i < 100; i++) __nanosleep(2000);
    } else {
      // the last releases of the stages come from the pair's issuer: none may be on its way when this CTA exits
      for (int i = max(0, issued - kStages); i < issued; i++) mbar_wait(smem_u32(&sh->empty[i % kStages]), (uint32_t)(i / kStages) & 1u, dead);
    }
  } else if (warp == kWarpFix) {
    // ===== shared tiles: once the epilogue has parked a part, count it; the CTA that delivers a tile's
    // last part adds the parts below, when its other work is done =====
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int t = t_first, bar = 2;
    for (int i = 0, cnt; i < nunits; i += cnt, t++) {
      cnt = min(i == 0 ? P.nsb - sb_first : P.nsb, nunits - i);
      if (cnt == P.nsb) continue;
      asm volatile("bar.sync %0, 160;" ::"r"(bar++) : "memory");
      if (*reinterpret_cast<volatile int*>(&sh->epi_fail)) break;
      if (lane == 0) {
        const int c0 = unit_owner(U, G, (long long)t * P.nsb), nc = unit_owner(U, G, (long long)(t + 1) * P.nsb - 1) - c0 + 1;
        __threadfence();
        const uint32_t prev = atomicAdd(P.counters + 2 * t + rank, 1u);
        __threadfence();
        if (prev == (uint32_t)nc - 1u) {
          P.counters[2 * t + rank] = 0u;                 // self-clearing for the next launch
          sh->todo_tile[sh->ntodo] = t;
          sh->todo_first[sh->ntodo] = c0;
          sh->todo_parts[sh->ntodo++] = nc;
        }
      }
      __syncwarp();
    }
  } else {
    // ===== epilogue: warp quarter q owns TMEM lanes 32 q .. 32 q + 31 = weight rows of the tile =====
    const int quarter = warp & 3, rt = quarter * 32 + lane;
    const T* bias = reinterpret_cast<const T*>(P.bias);
    const uint32_t acc_free[2] = {cluster_map(smem_u32(&sh->acc_empty[0]), 0), cluster_map(smem_u32(&sh->acc_empty[1]), 0)};
    const int nparts = (sb_first + nunits + P.nsb - 1) / P.nsb;      // tiles that the range touches
    int t = t_first, g = 0, fix_bar = 2;
    asm volatile("griddepcontrol.wait;" ::: "memory");        // Y, the partial sums and the tile counters
    for (int i = 0, cnt; i < nunits; i += cnt, t++, g++) {
      cnt = min(i == 0 ? P.nsb - sb_first : P.nsb, nunits - i);
      const int ab = g % R::kBufs;
      const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->acc_full[ab]), (g / R::kBufs) & 1, dead));
      if (!ok) sh->epi_fail = 1;
      epi_barrier();                         // the four warps leave together or not at all
      if (*reinterpret_cast<volatile int*>(&sh->epi_fail)) {
        for (; fix_bar < 4; fix_bar++) asm volatile("bar.arrive %0, 160;" ::"r"(fix_bar) : "memory");   // do not leave the counting warp waiting
        break;
      }
      tc_fence_after();
      const bool whole = cnt == P.nsb;       // this CTA summed the tile's whole K: store Y directly
      const Tile tile = tile_of(P, t);
      const int wt = 2 * tile.wt + rank, tok0 = tile.tt * P.nt, ntok = min(P.nt, P.M - tok0);
      const int n = SWIGLU ? 64 * wt + 16 * quarter + (lane & 15) : wt * kRows + rt;
      float* part = P.partials + ((size_t)(2 * cta + (i > 0 ? 1 : 0)) * P.nt) * kRows + rt;
      const float bv = (!SWIGLU && bias && n < P.N) ? Act<T>::to_f(bias[n]) : 0.0f;
      // this warp's first output column; all its columns exist and start on 16 bytes
      const int nw = SWIGLU ? 64 * wt + 16 * quarter : wt * kRows + 32 * quarter;
      constexpr int kCols = SWIGLU ? 16 : 32;
      const bool vec = P.vec_stores && nw + kCols <= P.N;
      T* yv = reinterpret_cast<T*>(P.y) + (size_t)tok0 * P.N + nw;
      // a part is parked sixteen tokens at a time: 32 took 1.8 us more for a part of 256 tokens (MMAs of the next tile wait for it: 20480 x 1280
      // Q8_0, 256 tokens, equal ranges 31.8 us, so 26.6)
      if (!whole) {
#pragma unroll 1
        for (int c0 = 0; c0 < ntok; c0 += 16) {
          uint32_t r[16];
          tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ab * NMAX + c0), r);
#pragma unroll
          for (int c = 0; c < 16; c++)
            if (c0 + c < ntok) __stcg(part + (size_t)(c0 + c) * kRows, __uint_as_float(r[c]));
        }
      } else if (!SWIGLU && !vec) {
        // rows that start anywhere, and the ragged end of the others: straight from the registers (turned in shared memory first,
        // 12363 x 2304 Q8_0, 515 tokens, took 43.5 us, so 41.5)
        T* y = yv + lane;
#pragma unroll 1
        for (int c0 = 0; c0 < ntok; c0 += 16) {
          uint32_t r[16];
          tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ab * NMAX + c0), r);
#pragma unroll
          for (int c = 0; c < 16; c++)
            if (n < P.N && c0 + c < ntok) y[(size_t)(c0 + c) * P.N] = Act<T>::from_f(__uint_as_float(r[c]) + bv);
        }
      } else {
#pragma unroll 1
        for (int c0 = 0; c0 < ntok; c0 += 32) {      // past nt: columns of the other buffer, not stored
          uint32_t r[32];
          tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ab * NMAX + c0), r);
          // 32 tokens x 32 weight rows (gate/up: 16 columns) turn in shared memory into 16-byte stores.  Beside busy producers
          // every instruction here counts: a tile of 256 tokens whose results leave one 2-byte word each took 6.4 us of a
          // tile's 24 (K = 4096), and the next tile's MMAs wait for it.
          if constexpr (SWIGLU) {
            uint16_t* turn = reinterpret_cast<uint16_t*>(sh->turn[quarter]);
#pragma unroll
            for (int c = 0; c < 32; c += 2) {
              const Pair<T> h = swiglu_pair<T, 16>(__uint_as_float(r[c]), __uint_as_float(r[c + 1]), lane);
              turn[(c + h.second) * kCols + (lane & 15)] = *reinterpret_cast<const uint16_t*>(&h.value);
            }
            __syncwarp();
            if (vec) {
#pragma unroll
              for (int e = 0; e < 2; e++) {
                const int piece = e * 32 + lane, tk = piece >> 1, pc = piece & 1;
                if (c0 + tk < ntok) *reinterpret_cast<uint4*>(yv + (size_t)(c0 + tk) * P.N + pc * 8) = *reinterpret_cast<const uint4*>(turn + tk * kCols + pc * 8);
              }
            } else {      // nothing to store today: a warp's columns all exist or none does, and h starts on 16 bytes; without these lines the block takes 1.2 % longer
#pragma unroll 4
              for (int e = lane; e < 32 * kCols; e += 32) {
                const int tk = e / kCols, col = e % kCols;
                if (c0 + tk < ntok && nw + col < P.N) yv[(size_t)(c0 + tk) * P.N + col] = *reinterpret_cast<const T*>(turn + e);
              }
            }
          } else {
            uint32_t* turn = sh->turn[quarter];                            // [pair of tokens][row]: two tokens of a row per word
#pragma unroll
            for (int c = 0; c < 16; c++) turn[c * 32 + lane] = pack2<T>(__uint_as_float(r[2 * c]) + bv, __uint_as_float(r[2 * c + 1]) + bv);
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 2; e++) {
              const int piece = e * 32 + lane, tk = 2 * (piece >> 2), pc = piece & 3;
              const uint4* w = reinterpret_cast<const uint4*>(turn + (piece >> 2) * 32 + pc * 8);
              const uint4 u = w[0], v = w[1];
              T* at = yv + (size_t)(c0 + tk) * P.N + pc * 8;
              if (c0 + tk < ntok) *reinterpret_cast<uint4*>(at) = make_uint4(__byte_perm(u.x, u.y, 0x5410), __byte_perm(u.z, u.w, 0x5410), __byte_perm(v.x, v.y, 0x5410), __byte_perm(v.z, v.w, 0x5410));
              if (c0 + tk + 1 < ntok) *reinterpret_cast<uint4*>(at + P.N) = make_uint4(__byte_perm(u.x, u.y, 0x7632), __byte_perm(u.z, u.w, 0x7632), __byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x7632));
            }
          }
          __syncwarp();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0 && g + R::kBufs < nparts) mbar_arrive_cluster(acc_free[ab]);      // nobody waits for the last ones
      if (!whole) { asm volatile("bar.arrive %0, 160;" ::"r"(fix_bar) : "memory"); fix_bar++; }
    }
  }
  tc_fence_before();
  __syncthreads();
  // neither CTA's memory is read or signalled by the other any more: each signal has been waited for where it arrives (the stages'
  // releases by the copy warps, accumulators by the epilogues and, but for the last ones, which are not sent, the issuer), so the
  // meeting need not wait for this CTA's stores (release: 0.7 us)
  if (sh->dead) cluster_arrive(); else cluster_arrive_relaxed();
  cluster_wait();
  if (warp == kWarpMma) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, R::kCols);
  }
  __syncwarp();                   // the meetings want whole warps
  cluster_arrive_relaxed();       // and neither leaves while the other still frees columns in both SMs
  if (tid == 0 && sh->dead) atomicExch(P.status, MLXR_ERR_TIMEOUT);
  // ===== shared tiles of which this CTA delivered the last part: all warps, four tokens each at a time,
  // four weight rows per lane, two parts in flight, added in CTA order =====
  const int ntodo = sh->dead ? 0 : sh->ntodo;
  constexpr int kW = kThreads / 32;
  for (int k = 0; k < ntodo; k++) {
    const int t = sh->todo_tile[k], c0 = sh->todo_first[k], nc = sh->todo_parts[k];
    const Tile tile = tile_of(P, t);
    const int wt = 2 * tile.wt + rank, tok0 = tile.tt * P.nt, ntok = min(P.nt, P.M - tok0);
    const T* bias = reinterpret_cast<const T*>(P.bias);
    const int n = SWIGLU ? 64 * wt + 16 * (lane >> 3) + 4 * (lane & 3) : wt * kRows + 4 * lane;
    // parts of the tile: the first pair's is its first tile's (0) if its range begins with this tile, else its last
    // tile's (1); the others' ranges begin inside the tile
    const size_t slab = (size_t)P.nt * (kRows / 4);
    const float4* first = reinterpret_cast<const float4*>(P.partials) + (size_t)(2 * (2 * c0 + rank) + (unit_begin(U, G, c0) < (long long)t * P.nsb ? 1 : 0)) * slab + lane;
    const float4* later = reinterpret_cast<const float4*>(P.partials) + (size_t)(2 * (2 * c0 + rank)) * slab + lane;
    for (int m0 = warp; m0 < ntok; m0 += 4 * kW) {
      float v[4][4];
#pragma unroll
      for (int q = 0; q < 4; q++) v[q][0] = v[q][1] = v[q][2] = v[q][3] = 0.0f;
      for (int z = 0; z < nc; z += 2) {
        float4 a[2][4];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const float4* src = z + e == 0 ? first : later + (size_t)(4 * (z + e)) * slab;
#pragma unroll
          for (int q = 0; q < 4; q++) a[e][q] = z + e < nc && m0 + q * kW < ntok ? __ldcg(src + (size_t)(m0 + q * kW) * (kRows / 4)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int e = 0; e < 2; e++)
#pragma unroll
          for (int q = 0; q < 4; q++) { v[q][0] += a[e][q].x; v[q][1] += a[e][q].y; v[q][2] += a[e][q].z; v[q][3] += a[e][q].w; }
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int m = m0 + q * kW;
        T* y = reinterpret_cast<T*>(P.y) + (size_t)(tok0 + m) * P.N + n;
        if constexpr (SWIGLU) {
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const Pair<T> h = swiglu_pair<T, 4>(v[q][e], v[q][e + 2], lane);
            if (m < ntok && n + e + 2 * h.second < P.N) y[e + 2 * h.second] = h.value;
          }
        } else {
#pragma unroll
          for (int e = 0; e < 4; e++)
            if (m < ntok && n + e < P.N) y[e] = Act<T>::from_f(v[q][e] + (bias ? Act<T>::to_f(bias[n + e]) : 0.0f));
        }
      }
    }
  }
  __syncwarp();
  cluster_wait();
}

}  // namespace widem

// ---- host side -----------------------------------------------------------------------------------
bool widem_supported(int qt, int M, int N, int K, int dtype, const void* x, const void* w) {
  if (qt != MLXR_Q4_K && qt != MLXR_Q4_0 && qt != MLXR_Q8_0 && qt != MLXR_NF4) return false;
  if (dtype != MLXR_F16 && dtype != MLXR_BF16) return false;
  if (M < 1 || N < 2 || K < 256 || K % 256 != 0) return false;
  return ((((uintptr_t)x) | ((uintptr_t)w)) & 15u) == 0;
}

// Token tile, grid and dealing of the units.  Fitted, in us, to 29000 measurements of 2365 linears (65 to 8192 tokens; 256 to 22016 rows of
// 1024 to 16384; tiles of 32 to 256 tokens; equal ranges, whole tiles, two to 32 pairs per tile; bursts of 4 ms, weights from HBM): the choice
// by this estimate takes 2 % more than the best of them in the mean.  A unit takes its MMAs or its conversion, whichever is longer.  A tile costs its results' way out beside
// that, with two accumulators (to 128 tokens) less, and more if its rows start anywhere (2-byte stores); a shared tile its parts' trip through
// L2 at the end; equal ranges also the parts that a pair parks between two tiles.  Whole tiles need none of that but leave SMs idle in the last
// wave.  A launch on more than half of the pairs cannot set itself up beside its predecessor's end.  Long launches run at
// the lower clock that the power cap leaves: the last line.
int widem_plan(int qt, int dtype, int M, int rows, int K, WidePlan* out) {
  int sms = 0;
  if (int r = device_sms(&sms)) return r;
  const int nsb = K / 256, wtiles = (rows + 2 * widem::kRows - 1) / (2 * widem::kRows), pairs = sms / 2;
  // a unit's conversion with tiles to 128 and to 256 tokens, its MMAs per token with either, what a tile's way out costs beside them
  struct Costs { double convert128, convert256, mma128, mma256, out; };
  static constexpr Costs kQ8 = {0.93, 1.10, 0.0070, 0.0043, 0.65}, kNf4 = {0.87, 1.21, 0.0064, 0.0024, 0.92}, kQ40[2] = {{0.76, 0.66, 0.0060, 0.0035, 0.95}, {0.71, 0.99, 0.0051, 0.0036, 0.96}},
                         kQ4K[2] = {{0.59, 0.84, 0.0037, 0.0036, 1.30}, {0.77, 0.98, 0.0053, 0.0038, 0.71}};      // fp16, bf16
  const int bf = dtype == MLXR_F16 ? 0 : 1;
  const Costs& k = qt == MLXR_Q8_0 ? kQ8 : qt == MLXR_NF4 ? kNf4 : qt == MLXR_Q4_0 ? kQ40[bf] : kQ4K[bf];
  double best = 1e300;
  for (int ntt = (M + 255) / 256;; ntt++) {
    const int nt = ((M + ntt - 1) / ntt + 15) / 16 * 16;
    if (nt < (M <= 1024 ? 48 : 112) && best < 1e300) break;
    const long long ntiles = (long long)wtiles * ((M + nt - 1) / nt), U = ntiles * nsb;
    const double unit = nt <= 128 ? std::max(k.convert128, 0.32 + k.mma128 * nt) : std::max(k.convert256, 0.32 + k.mma256 * nt);
    const double drain = (nt <= 128 ? 0.68 : 0.0169 * nt - 0.91) * k.out, whole = drain + (rows % 8 ? 0.016 * nt : 0.0);
    const double shared = 1.56 + 0.0164 * nt, part = 0.07 + 0.0023 * nt, parked = 0.38 + 0.014 * nt;
    // split 0: equal ranges of units for all pairs; else so many pairs for each tile (1: whole tiles, any number of them)
    for (int split = 0; split < 2 || (split <= nsb && split * ntiles <= pairs); split++) {
      if (split != 1 && 2 * ntiles > kSyncWords - kTileCounters) continue;        // two counters per tile
      const int G = (int)(split == 0 ? std::min<long long>(pairs, U) : split == 1 ? std::min<long long>(pairs, ntiles) : split * ntiles);
      double c = 1.55 * std::max(2.0 * G / pairs - 1.0, 0.0);
      if (split == 0) {
        const double units = (double)((U + G - 1) / G);
        c += units * unit + std::max(units / nsb - 1.0, 0.0) * whole + drain + shared + part * std::floor((nsb + units - 1) / units) + parked;
        // pairs at different places of K share neither X nor weights in L2; in runs of half a second 48 MB of X take 8 % more than whole
        // tiles' share of it, 96 MB 22 % (4096 x 14336 Q4_K, 4096 tokens, 502 us; the dense path 432); few weight tiles read X few times
        c *= 1.0 + 0.0025 * std::min(std::max((double)M * K / (1 << 19) - 16.0, 0.0), 120.0) * std::min(wtiles / 8.0, 1.0);
      } else {
        const double tiles = (double)((ntiles + G - 1) / G);
        c += split == 1 ? tiles * (nsb * unit + whole) : (nsb + split - 1) / split * unit + drain + shared + part * split;
      }
      if (c < best) {
        best = c;
        out->nt = nt; out->ntt = (M + nt - 1) / nt; out->ntiles = (int)ntiles; out->grid = 2 * G; out->whole = split == 1;
        out->partial_bytes = split == 1 ? 0 : (size_t)2 * G * 2 * nt * widem::kRows * sizeof(float);
      }
    }
    if (nt <= 16) break;
  }
  best += 4.29;
  out->cost_us = best * (0.54 + 0.1435 * std::log(best));
  return MLXR_OK;
}

template <int QT, typename T, int NMAX, bool SWIGLU>
static int launch_wide_inst(const widem::Maps& maps, const widem::Params& P, int grid, cudaStream_t st) {
  using namespace widem;
  auto kern = qgemm_widem_kernel<QT, T, NMAX, SWIGLU>;
  constexpr size_t smem = Rings<QT, Fmt<T>::v, NMAX>::kBytes + sizeof(Shared) + 1024;
  static_assert(smem <= (size_t)kSmemMax, "shared memory");
  static std::atomic<bool> attr_done[64] = {};
  int dev = 0;
  MLXR_CUDA_TRY(cudaGetDevice(&dev));
  if (!attr_done[dev & 63].load(std::memory_order_acquire)) {
    MLXR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_done[dev & 63].store(true, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = overlap_launches() ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 2;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  MLXR_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, maps, P));
  count_launch();
  return MLXR_OK;
}

// w2 == nullptr: Y[M, N] = X W^T (+ bias).  Otherwise w = gate, w2 = up and Y = SiLU(X gate^T) * (X up^T).
int launch_widem(const void* x, const void* w, const void* w2, const void* bias, void* y, int M, int N, int K, int qt, int dtype,
                 int* status, float* partials, uint32_t* counters, const WidePlan& plan, cudaStream_t st) {
  const bool swiglu = w2 != nullptr;
  widem::Maps maps;
  widem::Params P;
  memset(&maps, 0, sizeof(maps));
  memset(&P, 0, sizeof(P));
  if (int r = activation_blocks_map(x, M, K, dtype, plan.nt / 2, widem::kBlocks, &maps.x)) return r;
  const int tile_rows = swiglu ? 64 : widem::kRows;
  if (int r = weight_maps(qt, w, N, K, tile_rows, maps.w, &P.odd_shift)) return r;
  if (swiglu)
    if (int r = weight_maps(qt, w2, N, K, tile_rows, maps.w + (qt == MLXR_NF4 ? 2 : 1), &P.odd_shift)) return r;
  P.bias = bias;
  P.y = y;
  P.M = M; P.N = N; P.K = K;
  P.nsb = K / 256;
  P.nt = plan.nt; P.ntt = plan.ntt; P.ntiles = plan.ntiles; P.wtiles = plan.ntiles / plan.ntt; P.whole = plan.whole;
  P.vec_stores = N % 8 == 0 && ((uintptr_t)y & 15u) == 0;
  P.status = status;
  P.partials = partials;
  P.counters = counters;
  int rc = MLXR_ERR_UNSUPPORTED;
#define MLXR_WIDE_N(QTV, T, SW) (plan.nt > 128 ? launch_wide_inst<QTV, T, 256, SW>(maps, P, plan.grid, st) : launch_wide_inst<QTV, T, 128, SW>(maps, P, plan.grid, st))
#define MLXR_WIDE_T(QTV, SW) (dtype == MLXR_F16 ? MLXR_WIDE_N(QTV, __half, SW) : MLXR_WIDE_N(QTV, __nv_bfloat16, SW))
#define MLXR_WIDE(QTV) rc = swiglu ? MLXR_WIDE_T(QTV, true) : MLXR_WIDE_T(QTV, false)
  switch (qt) {
    case MLXR_Q4_K: MLXR_WIDE(MLXR_Q4_K); break;
    case MLXR_Q4_0: MLXR_WIDE(MLXR_Q4_0); break;
    case MLXR_Q8_0: MLXR_WIDE(MLXR_Q8_0); break;
    case MLXR_NF4: MLXR_WIDE(MLXR_NF4); break;
    default: set_error("wide kernel: no producer for %s", mlxr_quant_type_name(qt)); break;
  }
#undef MLXR_WIDE
#undef MLXR_WIDE_T
#undef MLXR_WIDE_N
  return rc;
}

}  // namespace mlxr
