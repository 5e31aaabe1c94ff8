// Small-batch quantized linear (M <= 64 rows of X; few of them as far as gemv.cu and gemv_tokens.cu are not faster) on the 5th-generation tensor cores.
//
//   Y[M, N] = X[M, K] * dequant(W)[N, K]^T (+ bias),  X, Y fp16 or bf16, W in MLXR's Q4_K, Q4_0 or
//   Q8_0 layout, NF4 or the canonical ggml Q4_K layout (q_gemm_dequant.metal:142-260 and
//   q_gemm_dequant_primitive.mm:186-203 for the formats and the host contract).
//
// At these batch sizes the linear is bound by the stream of packed weights from HBM, and the
// work per byte is the conversion of the weights, not the product.  The roles of the operands
// are therefore swapped against the usual GEMM: 128 WEIGHT rows are the M side of a tcgen05.mma
// (the TMEM lanes), the batch (padded to 16, 32 or 64) is its N side, and every weight is converted
// exactly once.
//
// * Work units are (tile of 128 weight rows, 256-wide super-block of K).  All units of the
//   linear, tile-major, are dealt to the CTAs in equal contiguous ranges (one CTA per SM), so
//   every SM streams the same number of bytes whatever N and K are.  A CTA's range may cover
//   the end of one tile, whole tiles and the start of another; the sums of a tile that several
//   CTAs share are parked as fp32 partials, and the CTA that delivers a tile's last part (a counter
//   per tile, nobody waits) adds the parts in CTA order with all its warps when its own range is done.
// * TMA boxes bring a unit's packed rows into a ring (six units, 110 KB in flight per SM; three of Q8_0).
//   The converted weights go to TENSOR MEMORY (tcgen05.st: a thread's row is its lane) and are
//   the A operand of the MMA from there.  Shared memory sees neither their stores nor the MMA's
//   reads of them, so all of it is left to the ring and to X; the previous form, converted tiles
//   in swizzled shared memory, spent 343 instructions per 64 weights on the conversion, its
//   addresses and its proxy fences.  Three groups of four producer warps take units in turn, each
//   with four 64-wide k-blocks of tensor memory of its own; a thread converts a whole unit of its
//   row, so the row's header is decoded once per 256 weights.
// * Two issuer warps take units in turn, each with an accumulator of its own; X tiles (128-byte
//   swizzle) come a unit at a time by TMA; four epilogue warps add the two accumulators and drain
//   them, double-buffered up to batch 32.
// * Gate/up form: a tile holds 16 gate rows and 16 up rows per TMEM lane quarter (boxes of 64 rows
//   from two matrices) and the epilogue stores SiLU(gate) * up.
// * Launched with programmatic stream serialization: set-up, the weight stream and the
//   conversion start while the previous kernel of the stream drains; the X loads and everything
//   the epilogue reads or writes wait for griddepcontrol.wait.
// * Every wait is bounded (tc::mbar_wait); a role that gives up sets a flag that the others
//   poll, copies in flight are awaited, tensor memory is freed, and the status word reports
//   MLXR_ERR_TIMEOUT.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>

#include "common.cuh"
#include "kernels.h"
#include "tc_common.cuh"
#include "weight_convert.cuh"
#include "weight_maps.h"

namespace mlxr {
namespace smallm {

using namespace tc;
using namespace wconv;

constexpr int kRows = 128;                 // weight rows per tile (MMA M, TMEM lanes)
constexpr int kBK = 64;                    // K of one X tile (a 128-byte swizzle row) and of one slot of converted weights
constexpr int kGroups = 3;                 // producer groups of four warps; group g converts units g, g + 3, ..
constexpr int kSlots = 2;                  // slots of converted weights per group, two 64-wide k-blocks each (kSplit:
                                           // the leading parts and the residuals of one)
constexpr int kBlockCols = kBK / 2;        // tensor-memory columns of a k-block: two 16-bit elements each
// Warp roles: single-warp roles first, four epilogue warps (warp % 4 = TMEM lane quarter), producers
[[maybe_unused]] constexpr int kWarpMma = 0, kWarpRaw = 2, kWarpX = 3, kWarpEpi0 = 4, kWarpProd0 = 8;   // two issuer warps: 0 and 1
constexpr int kWarpFix = kWarpProd0 + 4 * kGroups;                                     // counts shared tiles
constexpr int kThreads = (kWarpFix + 1) * 32;
constexpr int kMaxXStages = 4, kMaxXBars = 6, kMaxRawStages = 2 * kGroups;
constexpr int kSmemMax = 227 * 1024;

struct Params {
  const void* bias;
  int M, K;
  // matrices stacked along the tiles (q / k / v; one otherwise): rows of each, the tile after its last, its Y
  int rows[3], end[3];
  void* y[3];
  int nsb;             // super-blocks per row = K / 256
  int ntiles;          // ceil(rows / 128)
  int maxc;            // most CTAs that share one tile
  int odd_shift;       // NF4: byte offset of odd rows within their tensor map (0 or 8)
  int vec_stores;      // bit i: rows of y[i] start on 16 bytes
  long long U;         // units = ntiles * nsb
  int* status;
  float* partials;     // [ntiles][maxc][NPAD][128] fp32
  uint32_t* counters;  // one per tile, self-clearing
  // kSplit: X and the packed matrices (gate, up for kSwiglu), for the rows that the two-part products cannot give
  const void* x;
  const uint8_t* w[3];
  size_t row_bytes;
};

// Tensor maps of the packed weights: one per stacked matrix, or [0] gate, [1] up; NF4 (rows only 8-byte
// aligned): two of each, for its even and its odd rows.
struct Maps { CUtensorMap x, w[6]; };

// One matrix, gate and up with SiLU(gate) * up, or matrices stacked along the tiles.  (A kernel for all three, which
// finds every tile's matrix, took 1.1 us longer on one: 8.9 us instead of 7.8 at 16 x 4096 x 4096.)
enum Form { kPlain, kSwiglu, kStacked };

// the matrix of tile t and the tile's number in it
struct Place { int mat, tile; };
template <int FORM>
__device__ __forceinline__ Place place_of(const Params& P, int t) {
  if (FORM != kStacked || t < P.end[0]) return {0, t};
  return t < P.end[1] ? Place{1, t - P.end[0]} : Place{2, t - P.end[1]};
}

struct Shared {
  // The group's four warps have written the slot.  Consecutive units of a group belong to different
  // issuers, so even and odd units signal through barriers of their own: a barrier is waited on by one
  // issuer, which sees every phase of it in turn.  (With one barrier per slot an issuer a unit ahead
  // of the other would take the parity of the phase before last for completion.)
  uint64_t full_a[kGroups][kSlots][2];
  uint64_t empty_a[kGroups][kSlots];   // the MMAs that read it are done
  uint64_t x_full[kMaxXBars];          // the four X tiles of a unit have landed
  uint64_t x_empty[kMaxXStages];
  uint64_t raw_full[kMaxRawStages];
  uint64_t raw_empty[kMaxRawStages];
  uint64_t acc_full[2];         // all MMAs of a tile part are done (both issuers')
  uint64_t acc_empty[2];        // the epilogue has read the accumulator out
  uint32_t tmem_base;
  int dead;
  int ntodo;                    // shared tiles of which this CTA delivered the last part (the first and the last of its range)
  int todo_tile[2], todo_parts[2];
  int epi_fail;
  int bad;                      // kSplit: some sum was not finite
  alignas(16) uint16_t turn[4][16 * 32];    // epilogue warps: sixteen tokens' results on their way to 16-byte stores
};

// The table that a format's producers look codes up in, behind the rings: NF4, and 4-bit codes that are multiplied in
// 16-bit arithmetic.  The latter with a copy per lane leaves three instructions per pair of codes where the arithmetic takes four or
// five (14336 x 4096 Q4_K, 16 tokens: 12.6 us with arithmetic, 10.6 so), but 64 KB less for the rings: at batch 64 X needs
// them.  (NF4's pairs are of float32 and take two cycles of shared memory each, which is its limit: a copy per lane gains nothing.)
struct NoTable {
  static constexpr int kBytes = 0;
  __device__ __forceinline__ NoTable(const uint8_t*, int) {}
  static __device__ __forceinline__ void fill(uint8_t*, int, int) {}
};
template <int QT, int BF, int NPAD, int MODE> struct TableOf { using type = NoTable; };
template <int BF, int NPAD, int MODE> struct TableOf<MLXR_NF4, BF, NPAD, MODE> { using type = PairLevels; };
template <int BF> struct TableOf<MLXR_Q4_K, BF, 16, kFast> { using type = CodePairs<BF>; };
template <int BF> struct TableOf<MLXR_Q4_K, BF, 32, kFast> { using type = CodePairs<BF>; };
template <int BF> struct TableOf<MLXR_Q4_0, BF, 16, kFast> { using type = CodePairs<BF>; };
template <int BF> struct TableOf<MLXR_Q4_0, BF, 32, kFast> { using type = CodePairs<BF>; };

// first unit of CTA c, and the CTA that owns unit u, when U units are dealt to G CTAs
__host__ __device__ inline long long unit_begin(long long U, int G, int c) { return (U * c) / G; }
__host__ __device__ inline int unit_owner(long long U, int G, long long u) { return (int)(((u + 1) * G - 1) / U); }

// SiLU with the sign-split sigmoid of swiglu_mlp_fused.metal:92-99, on the fast exponential and
// reciprocal (relative error 1e-6 to |x| = 5, 7e-6 at 50: 2 + 1.17 |x| units of 2^-24 for the exponential; the
// rounding to the activation dtype that follows is 5e-4 or more): the epilogue applies it to every batch row in turn, one thread per output column, and
// the exact expf and division made that serial chain several times longer than the tile's MMAs.
__device__ __forceinline__ float swish_fast(float x) {
  const float e = __expf(-fabsf(x));
  const float s = __fdividef(1.0f, 1.0f + e);      // sigmoid(|x|)
  return x * (x >= 0.0f ? s : e * s);
}

// kSplit: a leading part beyond fp16's range is infinite and its residual the opposite infinity, and an infinite activation
// meets residuals of the other sign: their sum is NaN where the float32 product is finite or an infinity.  Sums that
// are not finite are computed again from the float32 weights, a warp per sum; such values are rare, and a
// row of them takes about as long as the generic kernel's.
// Added to by every sum that is to be stored: stays 0 as long as all are finite
__device__ __forceinline__ void note_bad(float& t, float v) { t = fmaf(v, 0.0f, t); }

__device__ __forceinline__ void epi_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

template <int QT, int NPAD, int TABLE> struct Rings {
  static constexpr int kRawBytes = kRows * Geo<QT>::kStage;                 // packed rows of one unit
  static constexpr int kXTile = NPAD * kBK * 2;                             // one k-block of X
  static constexpr int kXUnit = 4 * kXTile;                                 // the four k-blocks of a unit
  static constexpr int kTable = TABLE;
  static constexpr int kXStages = NPAD == 64 ? 2 : NPAD == 32 && TABLE > 32768 ? 3 : 4;
  // barriers of the X stages' arrival: as units alternate between the issuers, an odd number of stages needs two of each (see
  // Shared::full_a)
  static constexpr int kXBars = kXStages % 2 ? 2 * kXStages : kXStages;
  static constexpr int kFree = kSmemMax - kXStages * kXUnit - kTable - (int)sizeof(Shared) - 1024;
  // a multiple of the number of groups, so that a stage's barrier is always waited on by one group
  static constexpr int kRawStages = kFree / kRawBytes >= 2 * kGroups ? 2 * kGroups : kGroups;
  static constexpr size_t kBytes = (size_t)kXStages * kXUnit + (size_t)kRawStages * kRawBytes + kTable;
  // tensor-memory columns: accumulators [buffer][issuer][NPAD], then the converted weights; the widest
  // batch has no room for a second buffer
  static constexpr int kBufs = NPAD == 64 ? 1 : 2;
  static constexpr uint32_t kAcc0 = 0, kA0 = kBufs * 2 * NPAD;
  static constexpr uint32_t kColsUsed = kA0 + kGroups * kSlots * 2 * kBlockCols;
  static constexpr uint32_t kCols = 512;
  static_assert(kRawStages * kRawBytes <= kFree && kColsUsed <= kCols, "ring or tensor memory does not fit");
};

// SWIGLU: the tile's rows are 16 gate rows and 16 up rows per TMEM lane quarter (from two weight
// matrices), Y = SiLU(gate) * up with gate and up rounded to T first, N = the number of gate rows; a
// tile then covers 64 output columns.
template <int QT, typename T, int NPAD, int MODE, int FORM>
__global__ void __launch_bounds__(kThreads, 1)
qgemm_smallm_kernel(const __grid_constant__ Maps maps, const Params P) {
  constexpr bool SWIGLU = FORM == kSwiglu;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  constexpr int BF = Fmt<T>::v;
  constexpr bool kSplitRows = QT == MLXR_NF4;                 // even and odd rows come through maps of their own
  // the TMA unit fetches a tensor map on first use: ask for them before anything else
  if (threadIdx.x < 7) {
    const CUtensorMap* m = threadIdx.x == 6 ? &maps.x : &maps.w[threadIdx.x];
    constexpr int mats = FORM == kPlain ? 1 : FORM == kSwiglu ? 2 : 3;
    if (threadIdx.x == 6 || threadIdx.x < mats * (kSplitRows ? 2 : 1))
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
  }
  using Tab = typename TableOf<QT, BF, NPAD, MODE>::type;
  using R = Rings<QT, NPAD, Tab::kBytes>;
  constexpr int kXStages = R::kXStages, kXBars = R::kXBars, kRawStages = R::kRawStages, kXTile = R::kXTile, kXUnit = R::kXUnit, kRawBytes = R::kRawBytes;
  constexpr int kSteps = MODE == kSplit ? 4 : 2;              // slots filled per unit
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw & 1023u)) & 1023u;       // X tiles need 1024-byte alignment (128-byte swizzle)
  uint8_t* xring = smem_raw + pad;
  uint8_t* rawring = xring + (size_t)kXStages * kXUnit;
  uint8_t* table = rawring + (size_t)kRawStages * kRawBytes;       // in front of the rings the tables cost 2 to 5 % of a launch
  Shared* sh = reinterpret_cast<Shared*>(table + R::kTable);
  volatile int* dead = &sh->dead;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int G = gridDim.x, cta = blockIdx.x;

  // this CTA's units [u0, u1): unit u = (tile u / nsb, super-block u % nsb)
  const long long u0 = unit_begin(P.U, G, cta), u1 = unit_begin(P.U, G, cta + 1);
  const int nunits = (int)(u1 - u0);
  const int t_first = (int)(u0 / P.nsb), sb_first = (int)(u0 - (long long)t_first * P.nsb);

  // packed rows of unit (t, sb) into stage r: one box (two for gate/up; for NF4 one per row parity)
  auto load_raw = [&](int t, int sb, int r) {
    constexpr int nbox = (SWIGLU ? 2 : 1) * (kSplitRows ? 2 : 1);
    const uint32_t bar = smem_u32(&sh->raw_full[r]);
    mbar_expect_tx(bar, kRawBytes);
    const Place at = place_of<FORM>(P, t);
    const int row0 = (SWIGLU ? 64 : kRows) * at.tile;
#pragma unroll
    for (int b = 0; b < nbox; b++) {
      int x = Geo<QT>::kUnit / 8 * sb, y = row0;
      if constexpr (kSplitRows) { x = ((136 * sb + ((b & 1) ? P.odd_shift : 0)) & ~15) >> 3; y = row0 >> 1; }
      tma_load_2d(smem_u32(rawring + (size_t)r * kRawBytes + (size_t)b * (kRawBytes / nbox)), &maps.w[at.mat * nbox + b], x, y, bar);
    }
  };
  int raw_t = t_first, raw_sb = sb_first, raw_issued = 0;     // copy warp: the next unit to request
  if (tid == kWarpRaw * 32) {
    // the copy warp owns the ring's barriers and fills the ring before the CTA's other set-up is done
    for (int r = 0; r < kRawStages; r++) {
      mbar_init(smem_u32(&sh->raw_full[r]), 1);
      mbar_init(smem_u32(&sh->raw_empty[r]), 4);       // the group that converts the unit
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
    sh->bad = 0;
    for (int g = 0; g < kGroups; g++)
      for (int s = 0; s < kSlots; s++) {
        mbar_init(smem_u32(&sh->full_a[g][s][0]), 4);
        mbar_init(smem_u32(&sh->full_a[g][s][1]), 4);
        mbar_init(smem_u32(&sh->empty_a[g][s]), 1);
      }
    for (int r = 0; r < kXBars; r++) mbar_init(smem_u32(&sh->x_full[r]), 1);
    for (int r = 0; r < kXStages; r++) mbar_init(smem_u32(&sh->x_empty[r]), 1);
    for (int a = 0; a < 2; a++) {
      mbar_init(smem_u32(&sh->acc_full[a]), 2);
      mbar_init(smem_u32(&sh->acc_empty[a]), 4);       // the four epilogue warps
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  Tab::fill(table, tid, kThreads);
  if (warp == kWarpMma) tmem_alloc(smem_u32(&sh->tmem_base), R::kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&sh->tmem_base);

  // Under a programmatic-overlap launch the next kernel of the stream may start its set-up and its
  // weight stream now; whatever it reads or writes that this launch produces waits below
  // (griddepcontrol.wait).  Without the launch attribute both instructions do nothing.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  [[maybe_unused]] float bad = 0.0f;    // kSplit, see note_bad
  if (warp >= kWarpProd0 && warp < kWarpFix) {
    // ===== producers =====
    const int g = (warp - kWarpProd0) >> 2, p = (warp & 3) * 32 + lane;       // group, weight row of the tile = TMEM lane
    // where this row lies in a stage: matrix (gate / up), then for NF4 the parity of the row
    const int local = SWIGLU ? 16 * (warp & 3) + (lane & 15) : p;     // row within the matrix's part of the tile
    const int mrows = SWIGLU ? 64 : 128;
    const int mat_off = (SWIGLU && lane >= 16) ? 64 : 0;
    const int row_off = (kSplitRows ? mat_off + (local & 1) * (mrows / 2) + (local >> 1) : mat_off + local) * Geo<QT>::kStage;
    const uint32_t a_col = tmem + R::kA0 + (uint32_t)(g * kSlots * 2 * kBlockCols) + ((uint32_t)((warp & 3) * 32) << 16);
    int r = g;
    const Tab levels(table, lane);
    uint32_t rpar = 0, use = 0;         // use: how often this group's slots have been filled
    for (int i = g; i < nunits; i += kGroups) {
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->raw_full[r]), rpar, dead))) break;   // warp-uniform
      const uint8_t* row = rawring + (size_t)r * kRawBytes + row_off;
      if constexpr (kSplitRows) {
        const int sb = (int)((sb_first + i) % P.nsb);
        row += (136 * sb + ((local & 1) ? P.odd_shift : 0)) & 8;
      }
      bool ok = true;
      // k-block kb: half of slot kb / 2, or for kSplit (leading part and residual) all of slot kb & 1
      auto step = [&](auto KB) {
        const int kb = block_of(KB);
        const int st = MODE == kSplit ? kb : kb >> 1, q = st & 1;
        if (MODE == kSplit || (kb & 1) == 0) {
          const uint32_t u = use * (kSteps / kSlots) + st / kSlots;     // how often the slot has been filled before
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->empty_a[g][q]), (u & 1u) ^ 1u, dead));
          if (!ok) return;
          tc_fence_after();
        }
        const uint32_t col = a_col + (MODE == kSplit ? q * 2 * kBlockCols : kb * kBlockCols);
        convert64<QT, BF, MODE>(row, KB, levels, [&](auto H, const uint32_t (&a)[16], const uint32_t (&b)[16]) {
          tmem_st16(col + 16 * decltype(H)::value, a);
          if constexpr (MODE == kSplit) tmem_st16(col + kBlockCols + 16 * decltype(H)::value, b);
        });
        if (MODE == kSplit || (kb & 1) == 1) {
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sh->full_a[g][q][use & 1u]));
        }
      };
      if constexpr (MODE == kSplit) {
#pragma unroll 1
        for (int kb = 0; kb < 4 && ok; kb++) step(kb);
      } else {
        step(Int<0>{});
        if (ok) step(Int<1>{});
        if (ok) step(Int<2>{});
        if (ok) step(Int<3>{});
      }
      if (!ok) break;
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh->raw_empty[r]));
      use++;
      r += kGroups;
      if (r >= kRawStages) { r -= kRawStages; rpar ^= 1u; }
    }
  } else if (warp < kWarpMma + 2) {
    // ===== MMA issuers: issuer w takes every other unit into an accumulator of its own (one warp's
    // waits, issues and commits cost about 1100 cycles per unit beside busy producers; HBM brings a
    // unit in 820).  The whole warp walks the loop, one elected lane issues. =====
    const int w = warp - kWarpMma;
    constexpr uint32_t idesc = instr_desc(BF, BF, kRows, NPAD);
    // shared-memory descriptors differ only in their start-address field (bits 0-13, in 16-byte units)
    const uint64_t desc_hi = smem_desc_sw128(0);
    const uint32_t x_lo0 = (smem_u32(xring) & 0x3FFFFu) >> 4, tm = __shfl_sync(0xffffffffu, tmem, 0);
    bool ok = true;
    for (int i0 = 0, part = 0, cnt; i0 < nunits && ok; i0 += cnt, part++) {
      cnt = min(part == 0 ? P.nsb - sb_first : P.nsb, nunits - i0);
      const int ab = part % R::kBufs;
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->acc_empty[ab]), ((part / R::kBufs) & 1) ^ 1u, dead));
      const uint32_t dcol = tm + R::kAcc0 + (uint32_t)((ab * 2 + w) * NPAD);
      const int first = i0 + ((i0 ^ w) & 1);
      for (int i = first; i < i0 + cnt && ok; i += 2) {
        const int g = i % kGroups, xs = i % kXStages;
        const uint32_t use = (uint32_t)(i / kGroups);
        ok = mbar_wait(smem_u32(&sh->x_full[i % kXBars]), (uint32_t)(i / kXBars) & 1u, dead);
        const uint32_t acol = tm + R::kA0 + (uint32_t)(g * kSlots * 2 * kBlockCols);
        const uint64_t xdesc = desc_hi | (uint64_t)(x_lo0 + (uint32_t)xs * (kXUnit >> 4));
#pragma unroll
        for (int s = 0; s < kSteps; s++) {
          const int q = s % kSlots;
          const uint32_t u = (use >> 1) * (kSteps / kSlots) + s / kSlots;      // phase of this unit parity's barrier
          ok = __all_sync(0xffffffffu, ok && mbar_wait(smem_u32(&sh->full_a[g][q][use & 1u]), u & 1u, dead));   // warp-uniform
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < 2 * kBK / kUmmaK; k++) {
              const int kb = MODE == kSplit ? s : 2 * s + k / 4;        // k-block of X
              umma_f16_ts(dcol, acol + q * 2 * kBlockCols + k * (kUmmaK / 2), xdesc + (uint64_t)((kb * kXTile >> 4) + (k & 3) * (kUmmaK * 2 >> 4)), idesc,
                          (i != first || s > 0 || k > 0) ? 1u : 0u);
            }
            umma_commit(smem_u32(&sh->empty_a[g][q]));
            if (s == kSteps - 1) umma_commit(smem_u32(&sh->x_empty[xs]));
          }
          __syncwarp();
        }
      }
      if (ok && first < i0 + cnt && elect_one()) {
        umma_commit(smem_u32(&sh->acc_full[ab]));
        if (cnt == 1) umma_commit(smem_u32(&sh->acc_full[ab]));     // the other issuer has no unit of this part
      }
      __syncwarp();
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
    // ===== activations: per unit the four X tiles [NPAD rows, 64 columns] of its super-block (one copy of all four
    // took NF4 at 64 tokens, 4096 x 14336, from 18.9 to 19.8 us).  The whole warp walks the loop, one elected lane issues. =====
    int issued = 0, sb = sb_first;
    asm volatile("griddepcontrol.wait;" ::: "memory");      // X may be the previous kernel's output
    for (int i = 0; i < nunits; i++) {
      const int xs = i % kXStages;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->x_empty[xs]), ((uint32_t)(i / kXStages) & 1u) ^ 1u, dead))) break;
      if (elect_one()) {
        const uint32_t bar = smem_u32(&sh->x_full[i % kXBars]);
        mbar_expect_tx(bar, kXUnit);
#pragma unroll
        for (int jj = 0; jj < 4; jj++)
          tma_load_2d(smem_u32(xring + (size_t)xs * kXUnit + (size_t)jj * kXTile), &maps.x, (4 * sb + jj) * kBK, 0, bar);
      }
      __syncwarp();
      issued = i + 1;
      if (++sb == P.nsb) sb = 0;
    }
    if (*dead) {
      for (int i = max(0, issued - kXStages); i < issued; i++) {
        const uint32_t bar = smem_u32(&sh->x_full[i % kXBars]);
        for (uint32_t sp = 0; sp < kSpin; sp++) if (mbar_try(bar, (i / kXBars) & 1)) break;
      }
    }
  } else if (warp == kWarpFix) {
    // ===== shared tiles: once the epilogue has parked a part, count it (release); the CTA that
    // delivers a tile's last part adds the parts below, when its other work is done.  A warp of its own,
    // so that the epilogue does not wait for the fence and the counter's round trip. =====
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int t = t_first, bar = 2;
    for (int i = 0, cnt; i < nunits; i += cnt, t++) {
      cnt = min(i == 0 ? P.nsb - sb_first : P.nsb, nunits - i);
      if (cnt == P.nsb) continue;
      asm volatile("bar.sync %0, 160;" ::"r"(bar++) : "memory");
      if (*reinterpret_cast<volatile int*>(&sh->epi_fail)) break;
      if (lane == 0) {
        const int nc = unit_owner(P.U, G, (long long)(t + 1) * P.nsb - 1) - unit_owner(P.U, G, (long long)t * P.nsb) + 1;
        __threadfence();
        const uint32_t prev = atomicAdd(P.counters + t, 1u);
        __threadfence();
        if (prev == (uint32_t)nc - 1u) {
          P.counters[t] = 0u;                 // self-clearing for the next launch
          sh->todo_tile[sh->ntodo] = t;
          sh->todo_parts[sh->ntodo++] = nc;
        }
      }
      __syncwarp();
    }
  } else {
    // ===== epilogue: warp quarter q owns TMEM lanes 32 q .. 32 q + 31 = weight rows of the tile =====
    const int quarter = warp & 3;
    const int rt = quarter * 32 + lane;      // row within the tile
    const T* bias = reinterpret_cast<const T*>(P.bias);
    int t = t_first, sb = sb_first, g = 0, fix_bar = 2;
    asm volatile("griddepcontrol.wait;" ::: "memory");        // Y, the partial sums and the tile counters
    for (int i = 0; i < nunits; g++) {
      const int cnt = min(P.nsb - sb, nunits - i);
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
      // output column of this lane: its weight row, or for SWIGLU the gate row that lanes l and l + 16 share
      const Place at = place_of<FORM>(P, t);
      const int N = P.rows[at.mat], n = SWIGLU ? 64 * at.tile + 16 * quarter + (lane & 15) : at.tile * kRows + rt;
      T* y = reinterpret_cast<T*>(P.y[at.mat]);
      const int slot = whole ? 0 : cta - unit_owner(P.U, G, (long long)t * P.nsb);
      float* part = P.partials + (((size_t)t * P.maxc + slot) * NPAD) * kRows + rt;
      const float bv = (!SWIGLU && bias && n < N) ? Act<T>::to_f(bias[n]) : 0.0f;
      // this warp's first output column; all its columns exist and start on 16 bytes
      constexpr int kCols = SWIGLU ? 16 : 32;
      const int nw = SWIGLU ? 64 * at.tile + 16 * quarter : at.tile * kRows + 32 * quarter;
      const bool vec = ((P.vec_stores >> at.mat) & 1) && nw + kCols <= N;
      // the sums of sixteen tokens: both issuers' accumulators
      auto sums = [&](int c0, uint32_t (&r)[16]) {
        const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + R::kAcc0 + (uint32_t)(ab * 2 * NPAD + c0);
        if (cnt == 1) {
          tmem_ld16(acc + (uint32_t)((i & 1) * NPAD), r);
        } else {
          uint32_t q[16];
          tmem_ld16(acc, r);
          tmem_ld16(acc + NPAD, q);
#pragma unroll
          for (int c = 0; c < 16; c++) r[c] = __float_as_uint(__uint_as_float(r[c]) + __uint_as_float(q[c]));
        }
        if constexpr (MODE == kSplit) {
#pragma unroll
          for (int c = 0; c < 16; c++) note_bad(bad, __uint_as_float(r[c]));
        }
      };
      auto park = [&](int c0, const uint32_t (&r)[16]) {
#pragma unroll
        for (int c = 0; c < 16; c++)
          if (c0 + c < P.M) __stcg(part + (size_t)(c0 + c) * kRows, __uint_as_float(r[c]));
      };
      auto out = [&](int c0, const uint32_t (&r)[16]) {
        if (!SWIGLU && !vec) {
          // rows that start anywhere, and the ragged end of the others (turned in shared memory first, 3333 x 1536 Q4_0, 64 tokens, took
          // 9.2 us, so 8.6)
#pragma unroll
          for (int c = 0; c < 16; c++)
            if (c0 + c < P.M && n < N) y[(size_t)(c0 + c) * N + n] = Act<T>::from_f(__uint_as_float(r[c]) + bv);
          return;
        }
        // sixteen tokens x 32 weight rows (gate/up: 16 columns, SiLU of every other token on the upper lanes; a warp's columns there all exist or
        // none does) turn in shared memory into 16-byte stores: with a 2-byte store per lane and token a round of sixteen took 1400 cycles
        uint16_t* turn = sh->turn[quarter];
        if constexpr (SWIGLU) {
          const bool up = lane >= 16;
#pragma unroll
          for (int c = 0; c < 16; c += 2) {
            const float a = __uint_as_float(r[c]), b = __uint_as_float(r[c + 1]);
            const float o = __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
            const float gv = Act<T>::to_f(Act<T>::from_f(up ? o : a)), uv = Act<T>::to_f(Act<T>::from_f(up ? b : o));
            const T h = Act<T>::from_f(swish_fast(gv) * uv);
            turn[(c + (up ? 1 : 0)) * kCols + (lane & 15)] = *reinterpret_cast<const uint16_t*>(&h);
          }
        } else {
#pragma unroll
          for (int c = 0; c < 16; c++) {
            const T o = Act<T>::from_f(__uint_as_float(r[c]) + bv);
            turn[c * kCols + lane] = *reinterpret_cast<const uint16_t*>(&o);
          }
        }
        __syncwarp();
        if (vec) {
          constexpr int kPer = kCols / 8;                                // 16-byte pieces per token
#pragma unroll
          for (int e = 0; e < 16 * kPer / 32; e++) {
            const int piece = e * 32 + lane, tk = piece / kPer, pc = piece % kPer;
            if (c0 + tk < P.M) *reinterpret_cast<uint4*>(y + (size_t)(c0 + tk) * N + nw + pc * 8) = *reinterpret_cast<const uint4*>(turn + tk * kCols + pc * 8);
          }
        }
        __syncwarp();
      };
      // Rounds of sixteen tokens.  Where there are several, a loop for each way out: with both in one, parking took 1 to 2 % of a short launch
      // more (and with a single round a loop of each takes 1 % of a launch more: 14336 x 4096 NF4, 16 tokens, 16.1 us and 15.9)
      uint32_t r[16];
      if constexpr (NPAD == 16) {
        sums(0, r);
        if (!whole) park(0, r); else out(0, r);
      } else if (!whole) {
#pragma unroll 1
        for (int c0 = 0; c0 < NPAD && c0 < P.M; c0 += 16) { sums(c0, r); park(c0, r); }
      } else {
#pragma unroll 1
        for (int c0 = 0; c0 < NPAD && c0 < P.M; c0 += 16) { sums(c0, r); out(c0, r); }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh->acc_empty[ab]));
      if (!whole) { asm volatile("bar.arrive %0, 160;" ::"r"(fix_bar) : "memory"); fix_bar++; }
      i += cnt;
      sb = 0;
      t++;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kWarpMma) {
    tc_fence_after();
    tmem_dealloc(tmem, R::kCols);
  }
  if (tid == 0 && sh->dead) atomicExch(P.status, MLXR_ERR_TIMEOUT);
  // ===== shared tiles of which this CTA delivered the last part: all warps, four weight rows per lane, parts
  // added in CTA order.  Bound by L2 latency and by fetching this code, which runs once: a warp has as many batch rows in
  // work at a time as the padded batch gives it, with four parts of each in flight (eight of a single row).  With sixteen
  // loads in flight at any batch, in two forms, 32 tokens of Q8_0, 4096 x 11008, took 47.6 us instead of 45.9; with eight at
  // batch 64, 4402 x 6144 canonical Q4_K, 18.2 instead of 17.8 =====
  const int ntodo = sh->dead ? 0 : sh->ntodo;
  constexpr int kW = kThreads / 32;
  for (int k = 0; k < ntodo; k++) {
    const int t = sh->todo_tile[k], nc = sh->todo_parts[k];
    const T* bias = reinterpret_cast<const T*>(P.bias);
    const Place at = place_of<FORM>(P, t);
    const int N = P.rows[at.mat];
    T* y = reinterpret_cast<T*>(P.y[at.mat]);
    const int n = SWIGLU ? 64 * at.tile + 16 * (lane >> 3) + 4 * (lane & 3) : at.tile * kRows + 4 * lane;
    const bool writer = !SWIGLU || (lane & 4) == 0;
    const float4* parts = reinterpret_cast<const float4*>(P.partials + (size_t)t * P.maxc * NPAD * kRows) + lane;
    auto store = [&](int m, const float (&v)[4]) {
#pragma unroll
      for (int e = 0; e < 4; e++) {
        T o;
        if constexpr (MODE == kSplit) note_bad(bad, v[e]);
        if constexpr (SWIGLU) {
          const float up = __shfl_xor_sync(0xffffffffu, v[e], 4);      // lanes 0-3 of eight: gate, lanes 4-7: up
          o = Act<T>::from_f(swish_fast(Act<T>::to_f(Act<T>::from_f(v[e]))) * Act<T>::to_f(Act<T>::from_f(up)));
        } else {
          o = Act<T>::from_f(v[e] + (bias && n + e < N ? Act<T>::to_f(bias[n + e]) : 0.0f));
        }
        if (writer && n + e < N) y[(size_t)m * N + n + e] = o;
      }
    };
    auto sum = [&](auto RC, int m0) {
      constexpr int R = decltype(RC)::value, Z = R == 1 ? 8 : 4;       // batch rows m0, m0 + kW, .. and parts at a time
      float v[R][4] = {};
      for (int z = 0; z < nc; z += Z) {
        float4 a[R][Z];
#pragma unroll
        for (int q = 0; q < R; q++)
#pragma unroll
          for (int e = 0; e < Z; e++)
            a[q][e] = z + e < nc && m0 + q * kW < P.M ? __ldcg(parts + ((size_t)(z + e) * NPAD + m0 + q * kW) * (kRows / 4)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int q = 0; q < R; q++)
#pragma unroll
          for (int e = 0; e < Z; e++) { v[q][0] += a[q][e].x; v[q][1] += a[q][e].y; v[q][2] += a[q][e].z; v[q][3] += a[q][e].w; }
      }
#pragma unroll
      for (int q = 0; q < R; q++)
        if (m0 + q * kW < P.M) store(m0 + q * kW, v[q]);
    };
    static_assert(kW >= 16 && 2 * kW >= 32 && 4 * kW >= 64, "a round covers the batch");
    if (warp < P.M) sum(Int<NPAD / 16>{}, warp);
  }
  if constexpr (MODE == kSplit) {
    // ===== results that are not finite, in the tiles that this CTA stored: again, from the float32 weights (with the
    // repair beside the stores the kernel took 1.2 us more) =====
    if (bad != 0.0f) sh->bad = 1;
    __syncthreads();
    if (__builtin_expect(*reinterpret_cast<volatile int*>(&sh->bad) && !sh->dead, 0)) {
      const T* bias = reinterpret_cast<const T*>(P.bias);
      const T* x = reinterpret_cast<const T*>(P.x);
#pragma unroll 1
      for (int i = 0, t = t_first, cnt; i < nunits; i += cnt, t++) {
        cnt = min(i == 0 ? P.nsb - sb_first : P.nsb, nunits - i);
        bool mine = cnt == P.nsb;
        for (int k = 0; k < ntodo; k++) mine = mine || sh->todo_tile[k] == t;
        if (!mine) continue;
        const Place at = place_of<FORM>(P, t);
        constexpr int kCols = SWIGLU ? 64 : kRows;                       // columns of Y in a tile
        const int N = P.rows[at.mat], n0 = kCols * at.tile;
        T* y = reinterpret_cast<T*>(P.y[at.mat]);
#pragma unroll 1
        for (int e = warp; e < P.M * (kCols / 32); e += kW) {
          const int m = e / (kCols / 32), n = n0 + 32 * (e % (kCols / 32)) + lane;
          const bool lost = n < N && !(fabsf(Act<T>::to_f(y[(size_t)m * N + n])) <= 3.402823466e38f);
#pragma unroll 1
          for (unsigned left = __ballot_sync(0xffffffffu, lost); left; left &= left - 1) {
            const int row = n - lane + __ffs(left) - 1;
            const float g = exact_sum<QT, T>(P.w[at.mat] + (size_t)row * P.row_bytes, x + (size_t)m * P.K, P.K, lane);
            T o;
            if constexpr (SWIGLU) {
              const float u = exact_sum<QT, T>(P.w[1] + (size_t)row * P.row_bytes, x + (size_t)m * P.K, P.K, lane);
              o = Act<T>::from_f(swish_fast(Act<T>::to_f(Act<T>::from_f(g))) * Act<T>::to_f(Act<T>::from_f(u)));
            } else {
              o = Act<T>::from_f(g + (bias ? Act<T>::to_f(bias[row]) : 0.0f));
            }
            if (lane == 0) y[(size_t)m * N + row] = o;
          }
        }
      }
    }
  }
}

}  // namespace smallm

// ---- host side -----------------------------------------------------------------------------------
static int smallm_npad(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : 64; }

void smallm_partition(long long units, int ctas, int cta, long long unit, long long* begin, long long* end, int* owner) {
  if (begin) *begin = smallm::unit_begin(units, ctas, cta);
  if (end) *end = smallm::unit_begin(units, ctas, cta + 1);
  if (owner) *owner = smallm::unit_owner(units, ctas, unit);
}

// Every format but Q4_1 and canonical ggml Q4_0; NF4 rows come as pairs, so N >= 2.
bool smallm_supported(int qt, int M, int N, int K, int dtype, const void* x, const void* w) {
  if (qt != MLXR_Q4_K && qt != MLXR_Q4_0 && qt != MLXR_Q8_0 && qt != MLXR_NF4 && qt != MLXR_GGML_Q4_K) return false;
  if (dtype != MLXR_F16 && dtype != MLXR_BF16) return false;
  if (M < 1 || M > 64 || N < 2 || K < 256 || K % 256 != 0) return false;
  if ((((uintptr_t)x) | ((uintptr_t)w)) & 15u) return false;
  if ((N + smallm::kRows - 1) / smallm::kRows > kSyncWords - kTileCounters) return false;   // one counter per tile
  return true;
}

int smallm_plan(int qt, bool stacked, int M, int rows, int K, int* grid, int* maxc, size_t* partial_bytes) {
  const int N = rows;
  int sms = 0;
  if (int r = device_sms(&sms)) return r;
  const int nsb = K / 256, ntiles = (N + smallm::kRows - 1) / smallm::kRows;
  const long long U = (long long)ntiles * nsb;
  // Either all SMs get equal ranges, which cross tiles, or every tile gets c CTAs of its own (the same formula with
  // c * ntiles CTAs).  Fitted, in us, to 13700 measurements of 2524 linears (five formats; 3 to 64 tokens; 256 to 22016 rows of 1024 to
  // 16384; the choice by this estimate takes 0.6 % more than the best one in the mean, 13 % at most; by one fitted to 1500 and more rows of 2048 and
  // more, 2.5 % and up to 58 %: 8192 x 1024 Q8_0, 16 tokens, 6.4 us with two CTAs a tile, 4.2 with one).  A unit takes what its conversion does, about half as much
  // again if a CTA has only one (the groups of producers take units in turn), and more from the seventh on: the first six's bytes have come while the
  // previous kernel ended.  A shared tile costs its parts' trip through L2, which all CTAs make at the same time, and something for
  // each part; a range that crosses tiles more, because its CTA parks two parts.
  struct Costs { double unit[4], late[4], one, shared, together, ranges, part; };      // unit, late: 4-bit, Q8_0, NF4, weights in two parts
  static constexpr Costs kCosts[3] = {{{0.40, 0.52, 0.64, 1.20}, {0.1, 0.3, 0.0, 0.1}, 1.34, 1.93, 1.12, 0.57, 0.063},        // to 16 tokens
                                      {{0.44, 0.52, 0.71, 1.42}, {0.1, 0.3, 0.1, 0.2}, 1.54, 2.15, 1.18, 0.95, 0.109},        // to 32
                                      {{0.62, 0.62, 0.66, 1.57}, {0.1, 0.2, 0.1, 0.0}, 1.46, 2.48, 1.15, 1.18, 0.196}};       // to 64
  const Costs& k = kCosts[M <= 16 ? 0 : M <= 32 ? 1 : 2];
  const bool split = qt == MLXR_GGML_Q4_K || (M <= 8 && (stacked || qt == MLXR_Q8_0 || qt == MLXR_NF4));     // weights in two parts
  const int f = split ? 3 : qt == MLXR_NF4 ? 2 : qt == MLXR_Q8_0 ? 1 : 0;
  auto units = [&](double n) { return std::max(n, k.one) * k.unit[f] + std::max(n - 6.0, 0.0) * k.late[f]; };
  auto shared = [&](int G, double parts) { return k.shared + k.together * G / sms + k.part * parts; };
  // q/k/v: RMSNorm before it and RoPE behind it set themselves up beside it on the SMs that it leaves to them, if it leaves one for each
  // token, to 18 (hidden size 3584, 24 tokens of NF4: 15.6 us with 144 CTAs, 11.9 with 108; 2560, five tokens 10.6 with 140, 11.9 with 112)
  const double need = std::min(18, M);
  auto crowded = [&](int G) { return stacked ? 3.0 * std::max((G - (sms - need)) / need, 0.0) : 0.0; };
  int G = (int)std::min<long long>(sms, U);
  double best = units(std::ceil((double)U / G)) + (U % G == 0 && U / G % nsb == 0 ? 0.0 : shared(G, (double)nsb * G / U + 1.0) + k.ranges) + crowded(G);
  for (int c = 1; c <= nsb && (long long)c * ntiles <= sms; c++) {
    const double cost = units((nsb + c - 1) / c) + (c > 1 ? shared(c * ntiles, c) : 0.0) + crowded(c * ntiles);
    if (cost < best) { best = cost; G = c * ntiles; }
  }
  int mc = 1;
  for (int t = 0; t < ntiles; t++)
    mc = std::max(mc, smallm::unit_owner(U, G, (long long)(t + 1) * nsb - 1) - smallm::unit_owner(U, G, (long long)t * nsb) + 1);
  *grid = G;
  *maxc = mc;
  *partial_bytes = (size_t)ntiles * mc * smallm_npad(M) * smallm::kRows * sizeof(float);
  return MLXR_OK;
}

template <int QT, typename T, int NPAD, int MODE, int FORM>
static int launch_inst(const smallm::Maps& maps, const smallm::Params& P, int grid, cudaStream_t st) {
  using namespace smallm;
  auto kern = qgemm_smallm_kernel<QT, T, NPAD, MODE, FORM>;
  constexpr size_t smem = Rings<QT, NPAD, TableOf<QT, tc::Fmt<T>::v, NPAD, MODE>::type::kBytes>::kBytes + sizeof(Shared) + 1024;
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
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = overlap_launches() ? 1 : 0;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  MLXR_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, maps, P));
  count_launch();
  return MLXR_OK;
}

// One matrix, or three [rows[i], K] stacked: y[i] [M, rows[i]] = X w[i]^T (+ bias, one matrix only).  Or swiglu: w[0] = gate,
// w[1] = up (both [rows[0], K]) and y[0] = SiLU(X gate^T) * (X up^T), the two products rounded to the
// activation dtype first.
int launch_smallm(const void* x, const void* const* w, const int* rows, int nmat, bool swiglu, const void* bias, void* const* y, int M, int K, int qt, int dtype,
                  int* status, float* partials, uint32_t* counters, int grid, int maxc, cudaStream_t st) {
  const int npad = smallm_npad(M), form = swiglu ? smallm::kSwiglu : nmat == 1 ? smallm::kPlain : smallm::kStacked;
  smallm::Maps maps;
  smallm::Params P;
  memset(&maps, 0, sizeof(maps));
  memset(&P, 0, sizeof(P));
  if (int r = activation_map(x, M, K, dtype, npad, &maps.x)) return r;
  const int tile_rows = swiglu ? 64 : smallm::kRows, per = qt == MLXR_NF4 ? 2 : 1;
  for (int i = 0; i < nmat; i++)
    if (int r = weight_maps(qt, w[i], rows[swiglu ? 0 : i], K, tile_rows, maps.w + per * i, &P.odd_shift)) return r;
  for (int i = 0; i < 3; i++) {
    if (i < (swiglu ? 1 : nmat)) {
      P.rows[i] = rows[i];
      P.y[i] = y[i];
      if (rows[i] % 8 == 0 && ((uintptr_t)y[i] & 15u) == 0) P.vec_stores |= 1 << i;
      P.ntiles += (rows[i] + tile_rows - 1) / tile_rows;
    }
    P.end[i] = P.ntiles;
  }
  if (swiglu && (rows[0] % 16 || !P.vec_stores)) { set_error("small-batch kernel: gate / up wants outputs of a multiple of 16 columns, on 16 bytes"); return MLXR_ERR_UNSUPPORTED; }
  P.bias = bias;
  P.M = M; P.K = K;
  P.nsb = K / 256;
  P.maxc = maxc;
  P.U = (long long)P.ntiles * P.nsb;
  P.status = status;
  P.partials = partials;
  P.counters = counters;
  P.x = x;
  for (int i = 0; i < nmat; i++) P.w[i] = (const uint8_t*)w[i];
  P.row_bytes = (size_t)(K / block_elems(qt)) * block_bytes(qt);
  int rc = MLXR_ERR_UNSUPPORTED;
#define MLXR_SMALLM_BY_NPAD(QTV, T, MODE, SW)                                            \
  do {                                                                                   \
    if (npad == 16) rc = launch_inst<QTV, T, 16, MODE, SW>(maps, P, grid, st);           \
    else if (npad == 32) rc = launch_inst<QTV, T, 32, MODE, SW>(maps, P, grid, st);      \
    else rc = launch_inst<QTV, T, 64, MODE, SW>(maps, P, grid, st);                      \
  } while (0)
#define MLXR_SMALLM_BY_DTYPE(QTV, MODE, SW)                                              \
  do {                                                                                   \
    if (dtype == MLXR_F16) MLXR_SMALLM_BY_NPAD(QTV, __half, MODE, SW);                   \
    else MLXR_SMALLM_BY_NPAD(QTV, __nv_bfloat16, MODE, SW);                              \
  } while (0)
#define MLXR_SMALLM(QTV, MODE)                                                           \
  do {                                                                                   \
    if (form == smallm::kSwiglu) MLXR_SMALLM_BY_DTYPE(QTV, MODE, smallm::kSwiglu);       \
    else if (form == smallm::kPlain) MLXR_SMALLM_BY_DTYPE(QTV, MODE, smallm::kPlain);    \
    else MLXR_SMALLM_BY_DTYPE(QTV, MODE, smallm::kStacked);                              \
  } while (0)
  // Q8_0 and NF4 at batch <= 8, canonical Q4_K at any, and stacked Q4_K and Q4_0 at batch <= 8 keep the precision of
  // the float32 weights (wconv::kSplit).  Stacked, that is what the integer kernel of decode.cu (K >= 512) multiplies
  // with, and hidden size 4096 at 8 tokens takes 17.4 us so instead of 12.2 with weights rounded by kFast (33.4 there).
#define MLXR_SMALLM_SPLIT_BY_DTYPE(QTV, FORM)                                            \
  do {                                                                                   \
    if (dtype == MLXR_F16) rc = launch_inst<QTV, __half, 16, wconv::kSplit, FORM>(maps, P, grid, st);    \
    else rc = launch_inst<QTV, __nv_bfloat16, 16, wconv::kSplit, FORM>(maps, P, grid, st);               \
  } while (0)
#define MLXR_SMALLM_SPLIT(QTV)                                                           \
  do {                                                                                   \
    if (M > 8) MLXR_SMALLM(QTV, wconv::kRound);                                          \
    else if (form == smallm::kSwiglu) MLXR_SMALLM_SPLIT_BY_DTYPE(QTV, smallm::kSwiglu);  \
    else if (form == smallm::kPlain) MLXR_SMALLM_SPLIT_BY_DTYPE(QTV, smallm::kPlain);    \
    else MLXR_SMALLM_SPLIT_BY_DTYPE(QTV, smallm::kStacked);                              \
  } while (0)
  switch (qt) {
    case MLXR_Q4_K:
      if (form == smallm::kStacked && M <= 8 && K >= 512) MLXR_SMALLM_SPLIT_BY_DTYPE(MLXR_Q4_K, smallm::kStacked);
      else MLXR_SMALLM(MLXR_Q4_K, wconv::kFast);
      break;
    case MLXR_Q4_0:
      if (form == smallm::kStacked && M <= 8 && K >= 512) MLXR_SMALLM_SPLIT_BY_DTYPE(MLXR_Q4_0, smallm::kStacked);
      else MLXR_SMALLM(MLXR_Q4_0, wconv::kFast);
      break;
    case MLXR_Q8_0: MLXR_SMALLM_SPLIT(MLXR_Q8_0); break;
    case MLXR_NF4: MLXR_SMALLM_SPLIT(MLXR_NF4); break;
    case MLXR_GGML_Q4_K: MLXR_SMALLM(MLXR_GGML_Q4_K, wconv::kSplit); break;
    default: set_error("small-batch kernel: no producer for %s", mlxr_quant_type_name(qt)); break;
  }
#undef MLXR_SMALLM_SPLIT
#undef MLXR_SMALLM_SPLIT_BY_DTYPE
#undef MLXR_SMALLM
#undef MLXR_SMALLM_BY_DTYPE
#undef MLXR_SMALLM_BY_NPAD
  return rc;
}

}  // namespace mlxr
