// Linears for one or two tokens (Q4_K, Q4_0, Q8_0), single, stacked along N (q / k / v) or gate / up.
//
// Roofline: HBM.  What kept the earlier kernels at 0.4 of it was a meeting of all warps for every 16 rows and
// unequal numbers of tiles per CTA.  Here
//   * a CTA (one per SM) owns a contiguous range of rows (in granules of four: 14336 rows are 24 or 25
//     granules each on 148 SMs); its work units, (16-row tile, stage of K), go to the sixteen warps in turn, so that
//     what a CTA has in flight is contiguous (a stream of 400 MB: 6.5 TB/s; 6.0 to 6.25 when every warp has a range of
//     units of its own).  Every warp keeps its own sums of a tile, and the warps meet once in up to 32 tiles, when
//     their sums lie in shared memory and are added in the order of K (deterministic);
//   * every warp fills its own ring of two stages with 2-D tensor TMA (four boxes of 4 rows per stage) and drains it, so
//     nothing inside the stream waits on another warp (147 KB in flight per SM; with three stages, 221 KB, the same
//     stream of 400 MB falls to 5.9 TB/s);
//   * under programmatic stream serialization the launch's CTAs fill their rings while the previous launch's
//     last CTAs finish, and only the activations wait for its end.
// 8B-shaped block of one token (two launches): 34.9 us with the persistent kernel of decode.cu, 22.9 here (25.2 with the
// units in ranges, 64-bit divisions before the first copy and a serial addition of the warps' sums); 2048 x 5632 Q4_0
// 12.7 -> 9.9.  Small Q4_K and Q8_0 matrices, which do not repay the fixed part, are on stream_gemv.cu and gemv_rows_kernel.
// What is left beside the stream, per launch: its CTAs start when the previous one's leave the SMs, request weights 0.8 us
// later and learn of its end 1.1 us after it; activations, their conversion and a meeting 2 to 3 us (the ring
// fills meanwhile), the last sums and the epilogue 0.7 us; the slowest SM ends 1 us after the median one.
// Eight warps in half an SM's resources, so that the next launch's CTA could sit beside, took 36.8 us: two CTAs of the next
// launch came to lie on one SM.  Requests into L2 for the weights that the next launch reads first, sent behind the last of
// gate / up's own, took the block from 24.2 to 25.8 us.
//
// Arithmetic, 4-bit formats: activations as 16-bit fixed point per 256 elements, split in a high and a low
// signed byte; raw nibbles multiplied as unsigned bytes by mma.sync.m16n8k32 (the 16 MMA rows are weight
// rows); scales and the offset term in float32.  Q8_0: q is exact in fp16, so are the activations (bf16 ones
// times a power of two per segment), mma.sync.m16n8k16 with float32 accumulation, the block's scale on the sum.  In both the MMA's columns
// keep apart what has a scale of its own: a thread's part of the K range is one block (or (scale, min) pair)
// and its B fragment is zero outside that block's columns, so each thread ends up with the sums of the block
// whose scale it holds and no shuffles are needed before the end.
#include <atomic>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "decode_kernel.cuh"
#include "kernels.h"
#include "weight_maps.h"

namespace mlxr {
namespace gemv {

using decode::bounded_wait;
using decode::imma16832;
using decode::load8;
using decode::mbar_arrive_expect_tx;
using decode::mbar_init;
using decode::mbar_wait;
using decode::smem_u32;
using decode::tma_load_2d;

constexpr int kWarps = 16, kThreads = kWarps * 32;
constexpr int kMaxStages = 2;
constexpr int kMaxChunk = 32, kMinChunk = 8;     // tiles between two meetings: as many as shared memory has places for
constexpr int kSmemMax = 227 * 1024;

// Bytes of 256 weights of a row, 256-element segments per stage, and sums of the activations kept per segment
template <int QT> struct Geo {
  static constexpr int kSeg = QT == MLXR_Q8_0 ? 272 : 144;
  static constexpr int kSegs = QT == MLXR_Q8_0 ? 1 : 2;
  static constexpr int kPitch = kSeg * kSegs;
  static constexpr int kBox = (4 * kPitch + 127) & ~127;     // four rows; TMA wants 128-byte aligned places in shared memory
  static constexpr int kStage = 4 * kBox;
  static constexpr int kAux = QT == MLXR_Q4_K ? 4 : QT == MLXR_Q4_0 ? 8 : 0;
};

struct Params {
  alignas(64) CUtensorMap map[3];
  int rows[3];
  int nmat, interleave;      // interleave: map[0] gate, map[1] up; y[0] = h [M, rows[0]]
  int n_total;               // rows (h elements)
  int granules, gbase, gextra;      // granules of four rows: in all, per CTA, and CTAs with one more
  int K, nseg, nst;          // nst: stages per row
  int step_tiles, step_st;   // kWarps units on: so many tiles and stages
  int chunk;                 // tiles between two meetings of the warps
  int M;
  const void* x;
  const void* gamma;
  float eps;
  int round_n;               // see DecodeLinear
  void* y[3];
  const void* bias[3];
  int epi[3];                // decode::Epilogue
  const __half* cos_t;
  const __half* sin_t;
  const int32_t* positions;
  int head_dim, max_seq, pos_offset;
  int* status;
  unsigned long long wait_ns;
  int stages, x_stride;
  int off_x, off_aux, off_delta, off_parts, off_misc;
};
struct Misc {
  unsigned long long full[kWarps][kMaxStages];
  float red[kWarps * 2];
  float rinv[2];             // 1 / rms of the batch rows
  int dead;
};

// Fixed-point words of one (batch row, segment): v holds this lane's eight activations.  x ~ dl * xi with xi = v * inv,
// |xi| <= 32000, xi = 256 hi + lo as two signed-byte rows in MMA k order, and the exact integer sums of xi that
// the offset / min terms need.  1.5 * 2^23 + 2^15 added in the multiply leaves xi + 2^15, rounded to nearest, in the low bits.
// Returns the lane's sum of xi.
template <int QT>
__device__ __forceinline__ int emit_words(uint8_t* smem, const Params& P, int m, int sg, int lane, const float (&v)[8], float dl, float inv) {
  uint32_t t[8], sum = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) { t[i] = __float_as_uint(fmaf(v[i], inv, 12582912.0f + 32768.0f)); sum += t[i]; }
  const int ssum = (int)(sum - 8u * 0x4B408000u);
  // bytes of an 8-group are stored as (e0,e2,e4,e6 | e1,e3,e5,e7): the MMA k order.  xi + 32768 in 16 bits: its low
  // byte is the low part; plus 128, its high byte is the high part plus 128.
  uint8_t* row = smem + P.off_x + (size_t)(2 * m) * P.x_stride + sg * 256 + lane * 8;
  const uint32_t p02 = __byte_perm(t[0], t[2], 0x5410), p46 = __byte_perm(t[4], t[6], 0x5410), p13 = __byte_perm(t[1], t[3], 0x5410), p57 = __byte_perm(t[5], t[7], 0x5410);
  const uint32_t lo_e = __byte_perm(p02, p46, 0x6420), lo_o = __byte_perm(p13, p57, 0x6420);
  const uint32_t hi_e = __byte_perm(p02 + 0x00800080u, p46 + 0x00800080u, 0x7531) ^ 0x80808080u, hi_o = __byte_perm(p13 + 0x00800080u, p57 + 0x00800080u, 0x7531) ^ 0x80808080u;
  *reinterpret_cast<uint2*>(row) = make_uint2(hi_e, hi_o);
  *reinterpret_cast<uint2*>(row + P.x_stride) = make_uint2(lo_e, lo_o);
  float* aux = reinterpret_cast<float*>(smem + P.off_aux) + ((size_t)m * P.nseg + sg) * Geo<QT>::kAux;
  if (lane == 0) reinterpret_cast<float*>(smem + P.off_delta)[m * P.nseg + sg] = dl;
  // sums per sub-block of 32 (four lanes)
  int s4 = ssum;
  s4 += __shfl_xor_sync(0xffffffffu, s4, 1);
  s4 += __shfl_xor_sync(0xffffffffu, s4, 2);
  if constexpr (QT == MLXR_Q4_0) {
    if ((lane & 3) == 0) aux[lane >> 2] = (float)s4;
  } else {
    // per (scale, min) pair: sub-blocks {0,2,3}, {1}, {4,6,7}, {5} (q_gemm_dequant.metal:222-242)
    const int base = lane & 16;
    const int a = __shfl_sync(0xffffffffu, s4, base), b = __shfl_sync(0xffffffffu, s4, base + 4);
    const int c = __shfl_sync(0xffffffffu, s4, base + 8), d = __shfl_sync(0xffffffffu, s4, base + 12);
    if ((lane & 15) == 0) *reinterpret_cast<float2*>(aux + (lane >> 3)) = make_float2((float)(a + c + d), (float)b);
  }
  return ssum;
}
// The conversion as it nearly always is, in few instructions (every launch fetches them anew: with the rare cases in
// line 4096 x 14336 took 1.5 us more).  True if the segment has to be done again by emit_any: a largest value
// outside the range of the fast division (it returns 0 for divisors above 2^126 and overflows below 2^-113), or
// an infinity or a NaN, whose "words" put the sum far outside +- 8 * 32000 however many there are.
template <int QT>
__device__ __forceinline__ bool emit_fixed(uint8_t* smem, const Params& P, int m, int sg, int lane, const float (&v)[8]) {
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; i++) amax = fmaxf(amax, fabsf(v[i]));
  amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));     // non-negative floats order like their bit patterns
  const int ssum = emit_words<QT>(smem, P, m, sg, lane, v, amax * (1.0f / 32000.0f), amax > 0.0f ? __fdividef(32000.0f, amax) : 0.0f);
  return (uint32_t)(ssum + 8 * 32000) > 16u * 32000u || amax > 0x1p100f || (amax < 0x1p-100f && amax > 0.0f);
}
template <int QT>
__device__ __forceinline__ void emit_any(uint8_t* smem, const Params& P, int m, int sg, int lane, float (&v)[8]) {
  float dl, inv;
  decode::fixed_scale(v, dl, inv);
  emit_words<QT>(smem, P, m, sg, lane, v, dl, inv);
}

// Eight activations as they lie in memory (16-bit types: four registers)
template <typename T> struct Raw8 {
  uint4 q[sizeof(T) / 2];
  __device__ __forceinline__ void load(const T* p) {
    if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
#pragma unroll
      for (int i = 0; i < (int)(sizeof(T) / 2); i++) q[i] = __ldcg(reinterpret_cast<const uint4*>(p) + i);
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) reinterpret_cast<T*>(q)[i] = __ldcg(p + i);
    }
  }
  __device__ __forceinline__ float f(int i) const { return Act<T>::to_f(reinterpret_cast<const T*>(q)[i]); }
};

// Per-thread constants of the MMA mapping: lane = 4 g + c
struct Lane {
  int g, c, rg;              // MMA rows g and g + 8 are tile rows rg and rg + 8 (rows two apart lie 16 banks apart)
  bool keep0, keep1;         // this thread's B fragment belongs to its column (first / second half of the segment)
  int sh1, sh2;
};
__device__ __forceinline__ Lane make_lane(int lane, int qt) {
  Lane L;
  L.g = lane >> 2;
  L.c = lane & 3;
  // Q8_0: eight threads that read together have rows 16 bytes apart modulo 32
  L.rg = qt == MLXR_Q8_0 ? L.g : (L.g & 4) | ((L.g & 1) << 1) | ((L.g >> 1) & 1);
  if (qt == MLXR_Q4_K) {
    // sub-block s belongs to pair {0,1,0,0,2,3,2,2}[s]; MMA column g stands for pair g >> 1
    L.keep0 = (int)((0x22320010u >> (4 * L.c)) & 7u) == (L.g >> 1);
    L.keep1 = (int)((0x22320010u >> (4 * (L.c + 4))) & 7u) == (L.g >> 1);
  } else {
    L.keep0 = L.keep1 = (L.g >> 1) == L.c;    // columns 2 c and 2 c + 1 stand for thread c's own block
  }
  L.sh1 = L.c < 2 ? 12 * L.c : 24;
  L.sh2 = L.c == 3 ? 12 : 0;
  return L;
}

// One segment (256 weights) of 16 rows.  rl / rh: rows rg and rg + 8 in the stage at the segment; sg: segment of K.
// tot[j][h] gets this thread's part of batch row j, tile row rg + 8 h.
//
// Q4_K: thread c feeds the words of sub-block c, then 4 + c; columns 2 p + part stand for (scale, min) pair p, and
// the thread ends up with pair c's sums.  High nibbles stay in place (w & 0xf0f0f0f0 = 16 x nibble) and
// accumulate apart: two logic operations per word and two independent MMA chains.
template <int NT>
__device__ __forceinline__ void seg_q4k(const uint8_t* rl, const uint8_t* rh, const uint8_t* smem, const Params& P, int sg, const Lane& L, float (&tot)[NT][2]) {
  const uint4 hl = *reinterpret_cast<const uint4*>(rl), hh = *reinterpret_cast<const uint4*>(rh);
  int lo[NT][4] = {}, hi[NT][4] = {};
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const bool keep = h ? L.keep1 : L.keep0;
    const uint4 wl = *reinterpret_cast<const uint4*>(rl + 16 + 64 * h + 16 * L.c), wh = *reinterpret_cast<const uint4*>(rh + 16 + 64 * h + 16 * L.c);
    uint4 xa[NT], xb[NT];
#pragma unroll
    for (int j = 0; j < NT; j++) {
      xa[j] = xb[j] = make_uint4(0u, 0u, 0u, 0u);
      if (keep) {
        const uint8_t* xr = smem + P.off_x + (size_t)(2 * j + (L.g & 1)) * P.x_stride + sg * 256 + 128 * h + 32 * L.c;
        xa[j] = *reinterpret_cast<const uint4*>(xr);
        xb[j] = *reinterpret_cast<const uint4*>(xr + 16);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const uint32_t wa = i == 0 ? wl.x : wl.z, wb = i == 0 ? wl.y : wl.w, va = i == 0 ? wh.x : wh.z, vb = i == 0 ? wh.y : wh.w;
#pragma unroll
      for (int j = 0; j < NT; j++) {
        const uint4 xv = i == 0 ? xa[j] : xb[j];
        imma16832(lo[j], wa & 0x0f0f0f0fu, va & 0x0f0f0f0fu, wb & 0x0f0f0f0fu, vb & 0x0f0f0f0fu, xv.x, xv.z);
        imma16832(hi[j], wa & 0xf0f0f0f0u, va & 0xf0f0f0f0u, wb & 0xf0f0f0f0u, vb & 0xf0f0f0f0u, xv.y, xv.w);
      }
    }
  }
  // pair c of both rows: 6-bit fields at bit 12 c (scale) and 12 c + 6 (min) of scales[0..5]; sub-block scale =
  // rn16(sc * d), min = rn16(m * dmin); w = (q - 8) ss + sm = q ss + (sm - 8 ss)
  const uint32_t ul = __funnelshift_r(hl.y, hl.z, L.sh1) >> L.sh2, uh = __funnelshift_r(hh.y, hh.z, L.sh1) >> L.sh2;
  const __half2 dl2 = *reinterpret_cast<const __half2*>(&hl.x), dh2 = *reinterpret_cast<const __half2*>(&hh.x);
  const float ss_l = __half2float(__hmul(__int2half_rn((int)(ul & 63u)), __low2half(dl2)));
  const float ss_h = __half2float(__hmul(__int2half_rn((int)(uh & 63u)), __low2half(dh2)));
  const float sm_l = __half2float(__hmul(__int2half_rn((int)((ul >> 6) & 63u)), __high2half(dl2)));
  const float sm_h = __half2float(__hmul(__int2half_rn((int)((uh >> 6) & 63u)), __high2half(dh2)));
  const float of_l = fmaf(-8.0f, ss_l, sm_l), of_h = fmaf(-8.0f, ss_h, sm_h);
#pragma unroll
  for (int j = 0; j < NT; j++) {
    const float sx = reinterpret_cast<const float*>(smem + P.off_aux)[((size_t)j * P.nseg + sg) * 4 + L.c];
    const float dl = reinterpret_cast<const float*>(smem + P.off_delta)[j * P.nseg + sg];
    // the high-nibble sums are exact multiples of 16
    const float v0 = (float)((lo[j][0] + (hi[j][0] >> 4)) * 256 + (lo[j][1] + (hi[j][1] >> 4)));
    const float v1 = (float)((lo[j][2] + (hi[j][2] >> 4)) * 256 + (lo[j][3] + (hi[j][3] >> 4)));
    tot[j][0] = fmaf(dl, fmaf(ss_l, v0, of_l * sx), tot[j][0]);
    tot[j][1] = fmaf(dl, fmaf(ss_h, v1, of_h * sx), tot[j][1]);
  }
}

// N words from a 2-byte aligned place whose first word also holds the 16 bits before them: odd = the scale is the
// high half of the first word and the words follow whole, else it is the low half and they are 16 bits off
template <int N> __device__ __forceinline__ void words_after_scale(const uint8_t* p, bool odd, __half& d, uint32_t (&v)[N]) {
  const uint32_t* q = reinterpret_cast<const uint32_t*>(p - (odd ? 2 : 0));
  uint32_t w[N + 1];
#pragma unroll
  for (int i = 0; i <= N; i++) w[i] = q[i];
  d = __ushort_as_half((unsigned short)(odd ? w[0] >> 16 : w[0] & 0xFFFFu));
#pragma unroll
  for (int i = 0; i < N; i++) v[i] = __funnelshift_rc(w[i], w[i + 1], odd ? 32 : 16);
}

// Q4_0: thread c feeds block 4 i + c (18 bytes), columns 2 c and 2 c + 1 stand for the high and low bytes of its x
template <int NT>
__device__ __forceinline__ void seg_q40(const uint8_t* rl, const uint8_t* rh, const uint8_t* smem, const Params& P, int sg, const Lane& L, float (&tot)[NT][2]) {
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int at = 72 * i + 18 * L.c;
    __half dl, dh;
    uint32_t wl[4], wh[4];
    words_after_scale<4>(rl + at, L.c & 1, dl, wl);
    words_after_scale<4>(rh + at, L.c & 1, dh, wh);
#pragma unroll
    for (int j = 0; j < NT; j++) {
      uint4 xa = make_uint4(0u, 0u, 0u, 0u), xb = xa;
      if (L.keep0) {
        const uint8_t* xr = smem + P.off_x + (size_t)(2 * j + (L.g & 1)) * P.x_stride + sg * 256 + 128 * i + 32 * L.c;
        xa = *reinterpret_cast<const uint4*>(xr);
        xb = *reinterpret_cast<const uint4*>(xr + 16);
      }
      int lo[4] = {}, hi[4] = {};
      imma16832(lo, wl[0] & 0x0f0f0f0fu, wh[0] & 0x0f0f0f0fu, wl[1] & 0x0f0f0f0fu, wh[1] & 0x0f0f0f0fu, xa.x, xa.z);
      imma16832(hi, wl[0] & 0xf0f0f0f0u, wh[0] & 0xf0f0f0f0u, wl[1] & 0xf0f0f0f0u, wh[1] & 0xf0f0f0f0u, xa.y, xa.w);
      imma16832(lo, wl[2] & 0x0f0f0f0fu, wh[2] & 0x0f0f0f0fu, wl[3] & 0x0f0f0f0fu, wh[3] & 0x0f0f0f0fu, xb.x, xb.z);
      imma16832(hi, wl[2] & 0xf0f0f0f0u, wh[2] & 0xf0f0f0f0u, wl[3] & 0xf0f0f0f0u, wh[3] & 0xf0f0f0f0u, xb.y, xb.w);
      const float sx = reinterpret_cast<const float*>(smem + P.off_aux)[((size_t)j * P.nseg + sg) * 8 + 4 * i + L.c];
      const float dx = reinterpret_cast<const float*>(smem + P.off_delta)[j * P.nseg + sg];
      const float v0 = (float)((lo[0] + (hi[0] >> 4)) * 256 + (lo[1] + (hi[1] >> 4)));
      const float v1 = (float)((lo[2] + (hi[2] >> 4)) * 256 + (lo[3] + (hi[3] >> 4)));
      tot[j][0] = fmaf(dx * __half2float(dl), fmaf(-8.0f, sx, v0), tot[j][0]);
      tot[j][1] = fmaf(dx * __half2float(dh), fmaf(-8.0f, sx, v1), tot[j][1]);
    }
  }
}

// Block 4 I + c of a Q8_0 segment: its 34 bytes begin 2 c (+ 8 for I = 1) bytes behind a 16-byte boundary and are read as three
// 16-byte words.  (Word by word, 36 loads a unit with four-way bank conflicts, they were what bound the
// stream: 14336 x 4096 16.9 us, 15.0 so.)
template <int I> __device__ __forceinline__ void block_q80(const uint8_t* r, int c, __half& d, uint32_t (&v)[8]) {
  const uint4* q = reinterpret_cast<const uint4*>(r + ((136 * I + 34 * c) & ~15));
  const uint4 a = q[0], b = q[1], e = q[2];
  const uint32_t w[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, e.x, e.y, e.z, e.w};
  uint32_t t[9];
#pragma unroll
  for (int j = 0; j < 9; j++) t[j] = (c & 2) ? w[2 * I + j + 1] : w[2 * I + j];
  const bool odd = c & 1;
  d = __ushort_as_half((unsigned short)(odd ? t[0] >> 16 : t[0] & 0xFFFFu));
#pragma unroll
  for (int j = 0; j < 8; j++) v[j] = __funnelshift_rc(t[j], t[j + 1], odd ? 32 : 16);
}

// Q8_0: thread c feeds block 4 i + c (34 bytes); columns 2 c and 2 c + 1 stand for its two batch rows
template <bool SCALED, int NT>
__device__ __forceinline__ void seg_q80(const uint8_t* rl, const uint8_t* rh, const uint8_t* smem, const Params& P, int sg, const Lane& L, float (&tot)[NT][2]) {
  const bool keep = L.keep0 && (L.g & 1) < NT;
  auto half = [&](auto I) {
    constexpr int i = decltype(I)::value;
    __half dl, dh;
    uint32_t wl[8], wh[8];
    block_q80<i>(rl, L.c, dl, wl);
    block_q80<i>(rh, L.c, dh, wh);
    float acc[2][4] = {};
    const uint8_t* xr = smem + P.off_x + (size_t)(L.g & 1) * P.x_stride + (sg * 256 + 128 * i + 32 * L.c) * 2;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      uint4 xv = make_uint4(0u, 0u, 0u, 0u);
      if (keep) xv = *reinterpret_cast<const uint4*>(xr + 16 * q);
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const uint32_t ul = wl[2 * q + k] ^ 0x80808080u, uh = wh[2 * q + k] ^ 0x80808080u;
        hmma16816(acc[k], pair_of_bytes<0>(ul), pair_of_bytes<0>(uh), pair_of_bytes<1>(ul), pair_of_bytes<1>(uh), k ? xv.z : xv.x, k ? xv.w : xv.y);
      }
    }
#pragma unroll
    for (int j = 0; j < NT; j++) {
      const float dx = SCALED ? reinterpret_cast<const float*>(smem + P.off_delta)[j * P.nseg + sg] : 1.0f;
      tot[j][0] = fmaf(__half2float(dl) * dx, acc[0][j] + acc[1][j], tot[j][0]);
      tot[j][1] = fmaf(__half2float(dh) * dx, acc[0][2 + j] + acc[1][2 + j], tot[j][1]);
    }
  };
  half(std::integral_constant<int, 0>{});
  half(std::integral_constant<int, 1>{});
}

template <int QT, typename T, int NT>
__global__ void __launch_bounds__(kThreads, 1) gemv_kernel(const __grid_constant__ Params P) {
  using G_ = Geo<QT>;
  extern __shared__ __align__(128) uint8_t smem[];
  Misc* misc = reinterpret_cast<Misc*>(smem + P.off_misc);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int D = P.stages, S = P.nst;

  // This CTA's granules and tiles.  Unit u = (tile u / S, stage u % S); warp w takes units w, w + 16, ..
  const int cta = blockIdx.x, g0 = cta * P.gbase + min(cta, P.gextra), g1 = g0 + P.gbase + (cta < P.gextra ? 1 : 0);
  const int gpt = P.interleave ? 2 : 4, ntiles = (g1 - g0 + gpt - 1) >> (P.interleave ? 1 : 2), mine = (ntiles * S - warp + kWarps - 1) / kWarps;
  int tile0 = 0, st0 = warp;
  if (S <= warp) { tile0 = warp / S; st0 = warp - tile0 * S; }
  auto advance = [&](int& tile, int& st) {
    tile += P.step_tiles;
    st += P.step_st;
    if (st >= S) { st -= S; tile++; }
  };

  // ---- this warp's copy stream; weights are constants of the model, so it starts before the activations are there ----
  const uint32_t ring = smem_u32(smem) + warp * D * G_::kStage;
  int i_tile = tile0, i_st = st0, i_slot = 0, i_left = mine;
  auto issue = [&]() {
    if (i_left <= 0) return;
    i_left--;
    const int first = g0 + i_tile * gpt, have = min(gpt, g1 - first);
    const uint32_t bar = smem_u32(&misc->full[warp][i_slot]);
    if (lane == 0) mbar_arrive_expect_tx(bar, (uint32_t)(P.interleave ? 2 * have : have) * (4 * G_::kPitch));
    __syncwarp();
    if (lane < 4) {
      const int k = P.interleave ? (lane & 1) : lane;
      if (k < have) {
        int m = 0, row = 4 * (first + k);
        if (P.interleave) m = lane >> 1;
        else if (P.nmat > 1 && row >= P.rows[0]) { row -= P.rows[0]; m = 1; if (P.nmat > 2 && row >= P.rows[1]) { row -= P.rows[1]; m = 2; } }
        tma_load_2d(ring + i_slot * G_::kStage + lane * G_::kBox, &P.map[m], i_st * (G_::kPitch / 8), row, bar);
      }
    }
    if (++i_slot == D) i_slot = 0;
    advance(i_tile, i_st);
  };
  if (lane == 0) {
    for (int s = 0; s < D; s++) mbar_init(smem_u32(&misc->full[warp][s]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 0) misc->dead = 0;
  }
  __syncwarp();
  // Half of the ring now, the rest once the activations' loads are on their way: requested behind a full ring
  // of every SM (22 MB), they came 3 us after the previous kernel's end instead of 1.5.  A CTA whose units all fit the ring
  // does not have that much to request (2048 x 5632: 10.4 us in halves, 9.8 at once).
  int held = ntiles * S <= D * kWarps ? 0 : D - D / 2;
  for (int i = held; i < D; i++) issue();
  auto issue_held = [&]() { for (; held > 0; held--) issue(); };
  // The activations' and the norm weight's lines and pages are asked for, into L2 only: the data itself is
  // read after griddepcontrol.wait.
  {
    const int xl = (int)(((size_t)NT * P.K * sizeof(T) + 127) >> 7), gl = P.gamma ? (int)(((size_t)P.K * sizeof(T) + 127) >> 7) : 0;
    for (int i = tid; i < xl + gl; i += kThreads)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(i < xl ? (const char*)P.x + (size_t)i * 128 : (const char*)P.gamma + (size_t)(i - xl) * 128));
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // ---- activations: a warp per segment of 256 ----
  const T* xg = reinterpret_cast<const T*>(P.x);
  const T* gam = reinterpret_cast<const T*>(P.gamma);
  // up to four segments (v) of batch row m from s0 on, kWarps apart
  auto load_x = [&](int m, int s0, float (&v)[4][8]) {
#pragma unroll
    for (int u = 0; u < 4; u++) if (s0 + u * kWarps < P.nseg) load8(xg + (size_t)m * P.K + (s0 + u * kWarps) * 256 + lane * 8, v[u]);
  };
  auto load_raw = [&](const T* row, int s0, Raw8<T> (&r)[4]) {
#pragma unroll
    for (int u = 0; u < 4; u++) if (s0 + u * kWarps < P.nseg) r[u].load(row + (s0 + u * kWarps) * 256 + lane * 8);
  };
  float rinv[NT];
  bool rare = false;                                                    // see emit_fixed
  if constexpr (QT == MLXR_Q8_0) {
    // fp16 as they are; bf16 times a power of two per segment that brings its largest value to 2^14 .. 2^15, as fp16:
    // exact for every value above 2^-31 of the largest, so the products are those of the bf16 values and the
    // weights need only the cheaper conversion to fp16.  An infinity or a NaN stays what it is and does not set the scale,
    // or the finite values beside it would leave fp16's range.  With RMSNorm the norm is rounded to T first, so the
    // row's sum of squares comes before.
#pragma unroll
    for (int m = 0; m < NT; m++) {
      rinv[m] = 1.0f;
      if (gam) {
        float ss = 0.0f;
        for (int s0 = warp; s0 < P.nseg; s0 += 4 * kWarps) {
          float v[4][8];
          load_x(m, s0, v);
          issue_held();
#pragma unroll
          for (int u = 0; u < 4; u++)
            if (s0 + u * kWarps < P.nseg)
#pragma unroll
              for (int i = 0; i < 8; i++) ss = fmaf(v[u][i], v[u][i], ss);
        }
        ss = warp_sum(ss);
        if (lane == 0) misc->red[warp * NT + m] = ss;
      }
    }
    if (gam) {
      __syncthreads();
#pragma unroll
      for (int m = 0; m < NT; m++) {
        float tot = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; w++) tot += misc->red[w * NT + m];
        rinv[m] = 1.0f / sqrtf(tot / (float)P.K + P.eps);
      }
    }
#pragma unroll
    for (int m = 0; m < NT; m++)
      for (int s0 = warp; s0 < P.nseg; s0 += 4 * kWarps) {
        float v[4][8];
        load_x(m, s0, v);
        issue_held();
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int sg = s0 + u * kWarps;
          if (sg >= P.nseg) break;
          if (gam) {
            float gv[8];
            load8(gam + sg * 256 + lane * 8, gv);
#pragma unroll
            for (int i = 0; i < 8; i++) v[u][i] = Act<T>::to_f(Act<T>::from_f(__fmul_rn(__fmul_rn(v[u][i], rinv[m]), gv[i])));
          }
          float scale = 1.0f;
          if constexpr (Act<T>::kDtype == MLXR_BF16) {
            float amax = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; i++) amax = fabsf(v[u][i]) <= 3.4e38f ? fmaxf(amax, fabsf(v[u][i])) : amax;
            const int e = (int)(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)) >> 23);     // biased exponent
            const int se = e == 0 ? 127 : min(254, 268 - e);                                        // 2^14 / 2^(e - 127)
            scale = __int_as_float(se << 23);
            if (lane == 0) reinterpret_cast<float*>(smem + P.off_delta)[m * P.nseg + sg] = 1.0f / scale;
          }
          __half o[8];
#pragma unroll
          for (int i = 0; i < 8; i++) o[i] = __float2half_rn(v[u][i] * scale);
          *reinterpret_cast<uint4*>(smem + P.off_x + (size_t)m * P.x_stride + (sg * 256 + lane * 8) * 2) = *reinterpret_cast<const uint4*>(o);
        }
      }
  } else if (gam && P.round_n) {
    // n rounded to T before its conversion, so the row's sum of squares comes first.  A warp's first four segments
    // and their norm weights wait for it in registers: up to K = 16384 nothing is read twice.
    Raw8<T> v[NT][4], gv[4];
#pragma unroll
    for (int m = 0; m < NT; m++) load_raw(xg + (size_t)m * P.K, warp, v[m]);
    load_raw(gam, warp, gv);
    issue_held();
#pragma unroll
    for (int m = 0; m < NT; m++) {
      float ss = 0.0f;
      auto add = [&](int s0, const Raw8<T> (&a)[4]) {
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (s0 + u * kWarps < P.nseg)
#pragma unroll
            for (int i = 0; i < 8; i++) ss = fmaf(a[u].f(i), a[u].f(i), ss);
      };
      add(warp, v[m]);
      for (int s0 = warp + 4 * kWarps; s0 < P.nseg; s0 += 4 * kWarps) {
        Raw8<T> a[4];
        load_raw(xg + (size_t)m * P.K, s0, a);
        add(s0, a);
      }
      ss = warp_sum(ss);
      if (lane == 0) misc->red[warp * NT + m] = ss;
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < NT; m++) {
      float tot = 0.0f;
#pragma unroll
      for (int w = 0; w < kWarps; w++) tot += misc->red[w * NT + m];
      rinv[m] = 1.0f / sqrtf(tot / (float)P.K + P.eps);
    }
    for (int s0 = warp; s0 < P.nseg; s0 += 4 * kWarps) {
      if (s0 != warp) load_raw(gam, s0, gv);
#pragma unroll
      for (int m = 0; m < NT; m++) {
        if (s0 != warp) load_raw(xg + (size_t)m * P.K, s0, v[m]);
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int sg = s0 + u * kWarps;
          if (sg >= P.nseg) break;
          float n[8];
#pragma unroll
          for (int i = 0; i < 8; i++) n[i] = Act<T>::to_f(Act<T>::from_f(__fmul_rn(__fmul_rn(v[m][u].f(i), rinv[m]), gv[u].f(i))));
          rare |= emit_fixed<QT>(smem, P, m, sg, lane, n);
        }
      }
    }
  } else {
    // fixed point; the block scaling is independent of a factor common to the row, so 1 / rms multiplies the sums at
    // the end and the conversion does not wait for the sum of squares
#pragma unroll
    for (int m = 0; m < NT; m++) {
      float ss = 0.0f;
      Raw8<T> cur[4], next[4];
      load_raw(xg + (size_t)m * P.K, warp, cur);
#pragma unroll 1
      for (int s0 = warp; s0 < P.nseg; s0 += 4 * kWarps) {
        load_raw(xg + (size_t)m * P.K, s0 + 4 * kWarps, next);      // on their way while these are converted
        if (!gam) issue_held();
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int sg = s0 + u * kWarps;
          if (sg >= P.nseg) break;
          float v[8];
#pragma unroll
          for (int i = 0; i < 8; i++) v[i] = cur[u].f(i);
          if (gam) {
            float gv[8];
            load8(gam + sg * 256 + lane * 8, gv);
            issue_held();
#pragma unroll
            for (int i = 0; i < 8; i++) { ss = fmaf(v[i], v[i], ss); v[i] *= gv[i]; }
          }
          rare |= emit_fixed<QT>(smem, P, m, sg, lane, v);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) cur[u] = next[u];
      }
      if (gam) {
        ss = warp_sum(ss);
        if (lane == 0) misc->red[warp * NT + m] = ss;
      }
    }
  }
  issue_held();
  if constexpr (QT != MLXR_Q8_0) {
    if (__builtin_expect(__any_sync(0xffffffffu, rare), 0)) {
#pragma unroll 1
      for (int i = 0; i < NT * ((P.nseg - warp + kWarps - 1) / kWarps); i++) {
        const int m = i % NT, sg = warp + (i / NT) * kWarps;
        float v[8], gv[8];
        load8(xg + (size_t)m * P.K + sg * 256 + lane * 8, v);
        if (gam) load8(gam + sg * 256 + lane * 8, gv);
        const float r = NT == 1 || m == 0 ? rinv[0] : rinv[NT - 1];
#pragma unroll
        for (int e = 0; e < 8; e++)
          if (gam) v[e] = P.round_n ? Act<T>::to_f(Act<T>::from_f(__fmul_rn(__fmul_rn(v[e], r), gv[e]))) : v[e] * gv[e];
        emit_any<QT>(smem, P, m, sg, lane, v);
      }
    }
  }
  __syncthreads();
  const bool scale_sums = QT != MLXR_Q8_0 && gam && !P.round_n;     // 1 / rms still to be applied
  if (scale_sums && tid >= kThreads - NT) {
    const int m = kThreads - 1 - tid;
    float tot = 0.0f;
#pragma unroll
    for (int w = 0; w < kWarps; w++) tot += misc->red[w * NT + m];
    misc->rinv[m] = 1.0f / sqrtf(tot / (float)P.K + P.eps);
  }

  // ---- the stream ----
  const Lane L = make_lane(lane, QT);
  float* parts = reinterpret_cast<float*>(smem + P.off_parts);          // [tiles of a chunk][warp][16][NT]
  float tot[NT][2] = {};
  int tile = tile0, st = st0, slot = 0, left = mine;
  uint32_t par = 0;
  const int row_end = min(4 * g1, P.n_total);
  for (int t0 = 0;; t0 += P.chunk) {
    const int t1 = min(t0 + P.chunk, ntiles);
    while (left > 0 && tile < t1) {
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&misc->full[warp][slot]), par, &misc->dead, P.wait_ns))) break;
      const uint8_t* stage = smem + (size_t)(warp * D + slot) * G_::kStage;
      const uint8_t *rl = stage + (L.rg >> 2) * G_::kBox + (L.rg & 3) * G_::kPitch, *rh = rl + 2 * G_::kBox;
      const int sg = st * G_::kSegs;
      if constexpr (QT == MLXR_Q8_0) {
        seg_q80<Act<T>::kDtype == MLXR_BF16, NT>(rl, rh, smem, P, sg, L, tot);
      } else {
#pragma unroll
        for (int k = 0; k < 2; k++) {
          if (k && sg + 1 >= P.nseg) break;
          if constexpr (QT == MLXR_Q4_K) seg_q4k<NT>(rl + k * 144, rh + k * 144, smem, P, sg + k, L, tot);
          else seg_q40<NT>(rl + k * 144, rh + k * 144, smem, P, sg + k, L, tot);
        }
      }
      if (++slot == D) { slot = 0; par ^= 1u; }
      __syncwarp();
      issue();      // refill the stage that was just drained
      left--;
      const int was = tile;
      advance(tile, st);
      if (tile != was || left == 0) {
        // the quad's four parts of (row, batch) go to shared memory
        float* dst = parts + ((was - t0) * kWarps + warp) * 16 * NT;
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            float v = tot[j][h];
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            if (L.c == 0) dst[(L.rg + 8 * h) * NT + j] = v;
            tot[j][h] = 0.0f;
          }
      }
    }
    __syncthreads();
    if (misc->dead) {       // some sums are missing: nothing is stored; the copies in flight must land before the CTA may exit (bounded)
      if (lane == 0)
        for (int i = mine - left; i < mine - i_left; i++)
          bounded_wait([&] { return decode::mbar_try_wait(smem_u32(&misc->full[warp][i % D]), (uint32_t)(i / D) & 1u); }, 1000000000ull);
      __syncwarp();
      if (tid == 0) atomicExch(P.status, MLXR_ERR_TIMEOUT);
      return;
    }

    // ---- rows of these tiles: a thread per row and batch row adds the warps' parts in the order of K; a row's partner (the
    // up row of a gate row, the other row of a RoPE pair) is a lane of the same warp ----
    const int n = (t1 - t0) * 16 * NT;
    for (int e0 = warp * 32; e0 < n; e0 += kThreads) {
      const int e = e0 + lane, tl = e / (16 * NT), r = (e / NT) & 15, m = e % NT;
      float v = 0.0f;
      if (e < n) {
        const float* p = parts + tl * (kWarps * 16 * NT) + r * NT + m;
        const int first = (t0 + tl) * S;
        float a[kWarps];
#pragma unroll
        for (int k = 0; k < kWarps; k++) a[k] = k < S ? p[((first + k) & (kWarps - 1)) * (16 * NT)] : 0.0f;
#pragma unroll
        for (int k = 0; k < kWarps; k++) v += a[k];
        if (scale_sums) v *= misc->rinv[m];
      }
      if (P.interleave) {
        const float up = __shfl_xor_sync(0xffffffffu, v, 8 * NT);
        const int col = 4 * g0 + 8 * (t0 + tl) + r;
        if (e < n && r < 8 && col < row_end) {
          const float gv = Act<T>::to_f(Act<T>::from_f(v)), uv = Act<T>::to_f(Act<T>::from_f(up));
          reinterpret_cast<T*>(P.y[0])[(size_t)m * P.n_total + col] = Act<T>::from_f(swish_f(gv) * uv);
        }
        continue;
      }
      int R = 4 * g0 + 16 * (t0 + tl) + r;
      const bool store = e < n && R < row_end;
      int mat = 0;
      if (P.nmat > 1 && R >= P.rows[0]) { R -= P.rows[0]; mat = 1; if (P.nmat > 2 && R >= P.rows[1]) { R -= P.rows[1]; mat = 2; } }
      const T* bias = reinterpret_cast<const T*>(P.bias[mat]);
      if (bias && store) v += Act<T>::to_f(bias[R]);
      const float other = __shfl_xor_sync(0xffffffffu, v, NT);
      if (!store) continue;
      const size_t at = (size_t)m * P.rows[mat] + R;
      if (P.epi[mat] == decode::kEpiF32) {
        reinterpret_cast<float*>(P.y[mat])[at] = v;
        continue;
      }
      T* out = reinterpret_cast<T*>(P.y[mat]) + at;
      if (P.epi[mat] == decode::kEpiRope) {
        const float own = Act<T>::to_f(Act<T>::from_f(v)), oth = Act<T>::to_f(Act<T>::from_f(other));
        const long long pos = (long long)P.positions[m] + P.pos_offset;
        if (pos < 0 || pos >= P.max_seq) { atomicExch(P.status, MLXR_ERR_SHAPE); continue; }
        const int pairs = P.head_dim >> 1, pi = (R % P.head_dim) >> 1;
        const float cs = __half2float(P.cos_t[(size_t)pos * pairs + pi]), sn = __half2float(P.sin_t[(size_t)pos * pairs + pi]);
        *out = Act<T>::from_f((R & 1) ? __fadd_rn(__fmul_rn(own, cs), __fmul_rn(oth, sn)) : __fsub_rn(__fmul_rn(own, cs), __fmul_rn(oth, sn)));
      } else {
        *out = Act<T>::from_f(v);
      }
    }
    if (t1 == ntiles) break;
    __syncthreads();        // the parts' places are free again
  }
}

}  // namespace gemv

using namespace gemv;

static size_t unit_bytes(int qt) { return qt == MLXR_Q8_0 ? 272 : 144; }

// Shared-memory layout for a launch; the total, or 0 if it does not fit an SM
template <int QT> static size_t layout(Params* P, int M, int grid) {
  using G = Geo<QT>;
  const int per = P->interleave ? 2 : 4, most = (P->granules + grid - 1) / grid, tiles = (most + per - 1) / per;
  P->x_stride = (QT == MLXR_Q8_0 ? 2 * P->K : P->K) + 16;
  for (P->stages = kMaxStages; P->stages >= 1; P->stages--)
    for (P->chunk = kMaxChunk; P->chunk >= kMinChunk; P->chunk /= 2) {
      size_t o = (size_t)kWarps * P->stages * G::kStage;
      auto take = [&](size_t n) { const size_t at = o; o += (n + 15) & ~(size_t)15; return (int)at; };
      P->off_x = take((size_t)(QT == MLXR_Q8_0 ? M : 2 * M) * P->x_stride);
      P->off_aux = take((size_t)M * P->nseg * G::kAux * 4);
      P->off_delta = take((size_t)M * P->nseg * 4);
      P->off_parts = take((size_t)std::min(tiles, P->chunk) * kWarps * 16 * M * 4);
      P->off_misc = take(sizeof(Misc));
      if (o <= (size_t)kSmemMax) return o;
    }
  return 0;
}

bool gemv_supported(int qt, int M, int K, int rows, int dtype, const void* const* w, int nmat) {
  if (qt != MLXR_Q4_K && qt != MLXR_Q4_0 && !(qt == MLXR_Q8_0 && dtype != MLXR_F32)) return false;
  if (M < 1 || M > 2 || K < 256 || K % 256 != 0 || K > 32768 || rows < 1 || rows > (1 << 19)) return false;
  // Q4_0 rows of one segment are gemv_rows_kernel's, which multiplies the float32 activations (K = 256, float32: 8e-8 of
  // the result there, 2.6e-5 with 16-bit fixed point)
  if (qt == MLXR_Q4_0 && K < 512) return false;
  // Shared memory: the ring (74 KB per stage of all warps), the activations, the sums of a CTA's rows.  Two tokens of more
  // than about 20000 elements leave room for one stage.  As single or stacked rows and as gate / up.
  int sms = 0;
  if (device_sms(&sms)) return false;
  Params P;
  memset(&P, 0, sizeof(P));
  P.K = K;
  P.nseg = K / 256;
  for (P.interleave = 0; P.interleave < 2; P.interleave++) {
    P.granules = (rows / (P.interleave + 1) + 3) / 4;
    const int grid = std::max(1, std::min(sms, P.granules));
    if (!(qt == MLXR_Q4_K ? layout<MLXR_Q4_K>(&P, M, grid) : qt == MLXR_Q4_0 ? layout<MLXR_Q4_0>(&P, M, grid) : layout<MLXR_Q8_0>(&P, M, grid))) return false;
  }
  for (int i = 0; i < nmat; i++)
    if (((uintptr_t)w[i]) & 15u) return false;
  return true;
}

template <int QT, typename T, int NT>
static int launch_gemv_inst(Params& P, int grid, cudaStream_t st) {
  auto kern = gemv_kernel<QT, T, NT>;
  const size_t smem = layout<QT>(&P, NT, grid);
  if (!smem) { set_error("gemv: K = %d does not fit shared memory", P.K); return MLXR_ERR_UNSUPPORTED; }
  static std::atomic<bool> attr_done[64] = {};
  int dev = 0;
  MLXR_CUDA_TRY(cudaGetDevice(&dev));
  if (!attr_done[dev & 63].load(std::memory_order_acquire)) {
    MLXR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
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
  MLXR_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, P));
  count_launch();
  return MLXR_OK;
}

// L: see DecodeLinear (no tagged hand-over: chained linears are separate launches)
int launch_gemv(const DecodeLinear& L, int M, int qt, int dtype, int* status, cudaStream_t st) {
  int sms = 0;
  if (int r = device_sms(&sms)) return r;
  Params P;
  memset(&P, 0, sizeof(P));
  int total = 0;
  for (int j = 0; j < L.nmat; j++) {
    P.rows[j] = L.rows[j];
    total += L.rows[j];
    if (L.nmat > 1 && !L.interleave && L.rows[j] % 4 != 0) {
      set_error("gemv: stacked matrices need row counts that are multiples of 4");
      return MLXR_ERR_UNSUPPORTED;
    }
    const size_t rb = (size_t)(L.K / 256) * unit_bytes(qt);
    if (int r = rows_map(L.w[j], L.rows[j], rb, (int)(qt == MLXR_Q8_0 ? Geo<MLXR_Q8_0>::kPitch : Geo<MLXR_Q4_K>::kPitch), 4, &P.map[j])) return r;
  }
  for (int j = 0; j < 3; j++) { P.y[j] = L.y[j]; P.bias[j] = L.bias[j]; P.epi[j] = L.epi[j]; }
  P.nmat = L.nmat;
  P.interleave = L.interleave;
  P.n_total = L.interleave ? L.rows[0] : total;
  P.granules = (P.n_total + 3) / 4;
  P.K = L.K;
  P.nseg = L.K / 256;
  P.nst = qt == MLXR_Q8_0 ? P.nseg : (P.nseg + 1) / 2;
  P.M = M;
  P.x = L.x;
  P.gamma = L.gamma;
  P.eps = L.eps;
  P.round_n = L.round_n;
  P.cos_t = (const __half*)L.cos_t;
  P.sin_t = (const __half*)L.sin_t;
  P.positions = L.positions;
  P.head_dim = L.head_dim;
  P.max_seq = L.max_seq;
  P.pos_offset = L.pos_offset;
  P.status = status;
  P.wait_ns = wait_limit_ns();
  if (P.granules < 1) return MLXR_OK;
  const int grid = P.granules < sms ? P.granules : sms;
  P.gbase = P.granules / grid;
  P.gextra = P.granules % grid;
  P.step_tiles = kWarps / P.nst;
  P.step_st = kWarps % P.nst;
#define MLXR_GEMV_T(QTV, T) return M == 1 ? launch_gemv_inst<QTV, T, 1>(P, grid, st) : launch_gemv_inst<QTV, T, 2>(P, grid, st)
#define MLXR_GEMV_4(QTV)                                                       \
  do {                                                                         \
    if (dtype == MLXR_F16) MLXR_GEMV_T(QTV, __half);                           \
    if (dtype == MLXR_BF16) MLXR_GEMV_T(QTV, __nv_bfloat16);                   \
    MLXR_GEMV_T(QTV, float);                                                   \
  } while (0)
  if (qt == MLXR_Q4_K) MLXR_GEMV_4(MLXR_Q4_K);
  if (qt == MLXR_Q4_0) MLXR_GEMV_4(MLXR_Q4_0);
  if (qt == MLXR_Q8_0) { if (dtype == MLXR_F16) MLXR_GEMV_T(MLXR_Q8_0, __half); MLXR_GEMV_T(MLXR_Q8_0, __nv_bfloat16); }
#undef MLXR_GEMV_4
#undef MLXR_GEMV_T
  set_error("gemv: no code for %s", mlxr_quant_type_name(qt));
  return MLXR_ERR_UNSUPPORTED;
}

}  // namespace mlxr
