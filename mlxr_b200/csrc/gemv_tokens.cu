// Linears of up to eight tokens of 16-bit activations (canonical ggml Q4_K from one token on, Q8_0, Q4_K and Q4_0 from
// three), single, stacked along N (q / k / v) or gate / up, with products of the weights as they are.
//
// Roofline: HBM, but most of these calls are small and a launch's fixed part decides.  The small-batch kernel (smallm.cu) converts
// every weight to two 16-bit parts, hands them to tensor memory and two issuers, and adds parked parts of shared
// tiles at the end: [5, 4096] x [4096, 4096]^T canonical Q4_K took 11.1 us there for 1.5 us of weights.  Here the weights go from
// a warp's TMA ring straight into mma.sync fragments as gemv.cu does it (the same CTAs, rows, units and rings), with the
// eight columns of m16n8k16 for the tokens:
//   * a code of four bits, less 8, becomes an fp16 integer where it lies: (w & 0x000f000f) | 0x64006400 is 1024 + code,
//     w & 0x00f000f0 likewise 16 times the code, and one subtraction of pairs is exact; Q8_0's bytes as in gemv.cu.  (Codes left
//     as the subnormal numbers that they are need no subtraction, but the MMA then aligns its products some seven bits
//     too high and drops as many bits of the sum: the results of [1, 1536] x [1318, 1536]^T with some activations 1000 times the others
//     were 7.5e-6 off before their rounding, 4e-7 so.  It takes 5 to 19 % longer: 4 tokens, 7424 x 14336, 24.6 us and 29.2.)
//   * activations are fp16 as they are, bf16 ones times a power of two per 256 elements that brings the largest to 2^14 .. 2^15: exact
//     down to 2^-31 of it, fewer bits below that, zero below 2^-40 (which shows where the large ones meet weights of zero only);
//     they are stored so that a thread's 16 bytes are the B fragments of the eight weights it holds;
//   * a block's sum over its 32 weights is complete in the accumulators of two MMAs: scale, minimum and the sum of the
//     block's activations are applied in float32, so the products are those of the float32 weights.
// Sums of the warps meet in shared memory and are added in the order of K.  A sum that is not finite is computed again from
// the float32 weights (a code times an infinite activation is not what the weight's offset makes of it).
#include <atomic>
#include <cstring>
#include <type_traits>

#include "decode_kernel.cuh"
#include "kernels.h"
#include "weight_maps.h"

namespace mlxr {
namespace gemvt {

using decode::bounded_wait;
using decode::mbar_arrive_expect_tx;
using decode::mbar_init;
using decode::mbar_wait;
using decode::smem_u32;
using decode::tma_load_2d;

constexpr int kWarps = 16, kThreads = kWarps * 32, kMaxStages = 2, kTokens = 8;
constexpr int kMaxChunk = 16;
constexpr int kSmemMax = 227 * 1024;

template <int QT> struct Geo {
  static constexpr int kSeg = QT == MLXR_Q8_0 ? 272 : 144, kSegs = QT == MLXR_Q8_0 ? 1 : 2, kPitch = kSeg * kSegs;
  static constexpr int kBox = (4 * kPitch + 127) & ~127, kStage = 4 * kBox;
  static constexpr bool kSums = QT == MLXR_GGML_Q4_K || QT == MLXR_Q4_K;      // formats with an offset per block
};

struct Params {
  alignas(64) CUtensorMap map[3];
  int rows[3];
  int nmat, interleave;      // interleave: map[0] gate, map[1] up; y[0] = h [M, rows[0]]
  int n_total, granules, gbase, gextra;
  int K, nseg, nst, step_tiles, step_st, chunk, M;
  const void* x;
  void* y[3];
  const void* bias;          // one matrix only
  const uint8_t* w[3];
  size_t row_bytes;
  int* status;
  unsigned long long wait_ns;
  int stages, x_stride;
  int off_x, off_sum, off_delta, off_parts, off_misc;
};
struct Misc {
  unsigned long long full[kWarps][kMaxStages];
  int dead, bad;
};

// Byte J of v as a float, exactly: 2^23 + b is 0x4B000000 | b
template <int J> __device__ __forceinline__ float byte_f(uint32_t v) { return __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440u | J)) - 8388608.0f; }
__device__ __forceinline__ float lo_f(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)(v & 0xFFFFu))); }
__device__ __forceinline__ float hi_f(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)(v >> 16))); }

// The order in which eight consecutive activations are stored (element numbers, four bits each): the order of the weights in
// a thread's fragments of two MMAs
template <int QT> constexpr uint32_t kOrder = QT == MLXR_GGML_Q4_K ? 0x75643120u : QT == MLXR_Q8_0 ? 0x76543210u : 0x73516240u;

// The low nibbles of bytes 0 and 2 less 8; their high nibbles, 16 times that
__device__ __forceinline__ uint32_t codes_lo(uint32_t w) { return sub_half2((w & 0x000F000Fu) | 0x64006400u, 0x64086408u); }
__device__ __forceinline__ uint32_t codes_hi(uint32_t w) { return sub_half2((w & 0x00F000F0u) | 0x64006400u, 0x64806480u); }

// One segment (256 weights) of 16 rows.  rl / rh: this thread's two rows at the segment; x: its token's row at the segment
// (+ 16 c bytes); s: sums of the activations per block of 32 of its two tokens, [block][8].  a[2 h + t]: row h, token t.
template <int QT> __device__ __forceinline__ void seg(const uint8_t* rl, const uint8_t* rh, const uint8_t* x, const float* s, int c, float (&a)[4]) {
  auto xblock = [&](int b) { return *reinterpret_cast<const uint4*>(x + 64 * b); };
  auto sblock = [&](int b) { return *reinterpret_cast<const float2*>(s + 8 * b); };
  // a += scale d + offset sum
  auto add = [&](const float (&d)[4], float sl, float sh, float ol, float oh, float2 sm) {
    a[0] = fmaf(sl, d[0], fmaf(ol, sm.x, a[0]));
    a[1] = fmaf(sl, d[1], fmaf(ol, sm.y, a[1]));
    a[2] = fmaf(sh, d[2], fmaf(oh, sm.x, a[2]));
    a[3] = fmaf(sh, d[3], fmaf(oh, sm.y, a[3]));
  };
  if constexpr (QT == MLXR_GGML_Q4_K) {
    // w = (d sc) (q - 8) + (8 d sc - dmin m); chunk j: low nibbles of its 32 bytes are block 2 j, high nibbles block 2 j + 1
    const uint4 hl = *reinterpret_cast<const uint4*>(rl), hh = *reinterpret_cast<const uint4*>(rh);
    const float dl = lo_f(hl.x), ml = -hi_f(hl.x), dh = lo_f(hh.x), mh = -hi_f(hh.x);
    auto half = [&](auto H) {
      constexpr int h = decltype(H)::value;
      const uint32_t scl = h ? (hl.w & 0x0F0F0F0Fu) | ((hl.y >> 2) & 0x30303030u) : hl.y & 0x3F3F3F3Fu, mnl = h ? ((hl.w >> 4) & 0x0F0F0F0Fu) | ((hl.z >> 2) & 0x30303030u) : hl.z & 0x3F3F3F3Fu;
      const uint32_t sch = h ? (hh.w & 0x0F0F0F0Fu) | ((hh.y >> 2) & 0x30303030u) : hh.y & 0x3F3F3F3Fu, mnh = h ? ((hh.w >> 4) & 0x0F0F0F0Fu) | ((hh.z >> 2) & 0x30303030u) : hh.z & 0x3F3F3F3Fu;
      auto chunk = [&](auto J) {
        constexpr int j = decltype(J)::value, b = 4 * h + 2 * j;
        const uint2 wl = *reinterpret_cast<const uint2*>(rl + 16 + 16 * b + 8 * c), wh = *reinterpret_cast<const uint2*>(rh + 16 + 16 * b + 8 * c);
        const uint4 xa = xblock(b), xb = xblock(b + 1);
        float lo[4] = {}, hi[4] = {};
        hmma16816(lo, codes_lo(wl.x), codes_lo(wh.x), codes_lo(wl.x >> 8), codes_lo(wh.x >> 8), xa.x, xa.y);
        hmma16816(hi, codes_hi(wl.x), codes_hi(wh.x), codes_hi(wl.x >> 8), codes_hi(wh.x >> 8), xb.x, xb.y);
        hmma16816(lo, codes_lo(wl.y), codes_lo(wh.y), codes_lo(wl.y >> 8), codes_lo(wh.y >> 8), xa.z, xa.w);
        hmma16816(hi, codes_hi(wl.y), codes_hi(wh.y), codes_hi(wl.y >> 8), codes_hi(wh.y >> 8), xb.z, xb.w);
        auto finish = [&](const float (&d)[4], float part, float sl, float sh, float nl, float nh, float2 sm) {
          add(d, sl * part, sh * part, fmaf(8.0f, sl, ml * nl), fmaf(8.0f, sh, mh * nh), sm);
        };
        finish(lo, 1.0f, dl * byte_f<2 * j>(scl), dh * byte_f<2 * j>(sch), byte_f<2 * j>(mnl), byte_f<2 * j>(mnh), sblock(b));
        finish(hi, 0x1p-4f, dl * byte_f<2 * j + 1>(scl), dh * byte_f<2 * j + 1>(sch), byte_f<2 * j + 1>(mnl), byte_f<2 * j + 1>(mnh), sblock(b + 1));
      };
      chunk(std::integral_constant<int, 0>{});
      chunk(std::integral_constant<int, 1>{});
    };
    half(std::integral_constant<int, 0>{});
    half(std::integral_constant<int, 1>{});
  } else if constexpr (QT == MLXR_Q4_K) {
    // (scale, min) pairs of blocks {0, 2, 3}, {1}, {4, 6, 7}, {5} (q_gemm_dequant.metal:222-242); scale rn16(sc d), min
    // rn16(m dmin); w = (q - 8) ss + sm
    const uint4 hl = *reinterpret_cast<const uint4*>(rl), hh = *reinterpret_cast<const uint4*>(rh);
    auto block = [&](int b, float (&d)[4]) {
      const uint32_t wl = *reinterpret_cast<const uint32_t*>(rl + 16 + 16 * b + 4 * c), wh = *reinterpret_cast<const uint32_t*>(rh + 16 + 16 * b + 4 * c);
      const uint4 xv = xblock(b);
      hmma16816(d, codes_lo(wl), codes_lo(wh), codes_lo(wl >> 8), codes_lo(wh >> 8), xv.x, xv.y);
      hmma16816(d, codes_lo(wl >> 4), codes_lo(wh >> 4), codes_lo(wl >> 12), codes_lo(wh >> 12), xv.z, xv.w);
    };
    auto finish = [&](int p, const float (&d)[4], float2 sm) {
      auto pair = [&](const uint4& h, float& sc, float& of) {
        const uint32_t f = p == 3 ? h.z >> 4 : p == 2 ? __funnelshift_r(h.y, h.z, 24) : h.y >> (12 * p);
        const __half2 dd = *reinterpret_cast<const __half2*>(&h.x);
        sc = __half2float(__hmul(__int2half_rn((int)(f & 63u)), __low2half(dd)));
        of = __half2float(__hmul(__int2half_rn((int)((f >> 6) & 63u)), __high2half(dd)));
      };
      float sl, ol, sh, oh;
      pair(hl, sl, ol);
      pair(hh, sh, oh);
      add(d, sl, sh, ol, oh, sm);
    };
#pragma unroll
    for (int h = 0; h < 2; h++) {
      float d[4] = {}, e[4] = {};
      block(4 * h, d);
      block(4 * h + 1, e);
      block(4 * h + 2, d);
      block(4 * h + 3, d);
      const float2 s0 = sblock(4 * h), s2 = sblock(4 * h + 2), s3 = sblock(4 * h + 3);
      finish(2 * h, d, make_float2(s0.x + s2.x + s3.x, s0.y + s2.y + s3.y));
      finish(2 * h + 1, e, sblock(4 * h + 1));
    }
  } else if constexpr (QT == MLXR_Q4_0) {
#pragma unroll
    for (int b = 0; b < 8; b++) {      // 18 bytes: fp16 d, 16 bytes of nibbles; odd blocks begin 2 bytes off a word
      uint32_t w[2];
      float d2[2];
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const uint8_t* p = (r ? rh : rl) + 18 * b;
        d2[r] = __half2float(*reinterpret_cast<const __half*>(p));
        const uint32_t* q = reinterpret_cast<const uint32_t*>(p + (b & 1 ? 2 : 0) + 4 * c);
        w[r] = b & 1 ? q[0] : __funnelshift_r(q[0], q[1], 16);
      }
      const uint4 xv = xblock(b);
      float d[4] = {};
      hmma16816(d, codes_lo(w[0]), codes_lo(w[1]), codes_lo(w[0] >> 8), codes_lo(w[1] >> 8), xv.x, xv.y);
      hmma16816(d, codes_lo(w[0] >> 4), codes_lo(w[1] >> 4), codes_lo(w[0] >> 12), codes_lo(w[1] >> 12), xv.z, xv.w);
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = fmaf(d2[i >> 1], d[i], a[i]);
    }
  } else {
#pragma unroll
    for (int b = 0; b < 8; b++) {      // 34 bytes: fp16 d, 32 signed bytes; even blocks' bytes begin 2 bytes off a word
      uint32_t w[2][2];
      float d2[2];
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const uint8_t* p = (r ? rh : rl) + 34 * b;
        d2[r] = __half2float(*reinterpret_cast<const __half*>(p));
        const uint32_t* q = reinterpret_cast<const uint32_t*>(p + (b & 1 ? 2 : 0) + 8 * c);
        w[r][0] = (b & 1 ? q[0] : __funnelshift_r(q[0], q[1], 16)) ^ 0x80808080u;
        w[r][1] = (b & 1 ? q[1] : __funnelshift_r(q[1], q[2], 16)) ^ 0x80808080u;
      }
      const uint4 xv = xblock(b);
      float d[4] = {};
      hmma16816(d, pair_of_bytes<0>(w[0][0]), pair_of_bytes<0>(w[1][0]), pair_of_bytes<1>(w[0][0]), pair_of_bytes<1>(w[1][0]), xv.x, xv.y);
      hmma16816(d, pair_of_bytes<0>(w[0][1]), pair_of_bytes<0>(w[1][1]), pair_of_bytes<1>(w[0][1]), pair_of_bytes<1>(w[1][1]), xv.z, xv.w);
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = fmaf(d2[i >> 1], d[i], a[i]);
    }
  }
}

template <int QT, typename T>
__global__ void __launch_bounds__(kThreads, 1) gemv_tokens_kernel(const __grid_constant__ Params P) {
  using G_ = Geo<QT>;
  constexpr bool kScaled = Act<T>::kDtype == MLXR_BF16, kSums = Geo<QT>::kSums;
  extern __shared__ __align__(128) uint8_t smem[];
  Misc* misc = reinterpret_cast<Misc*>(smem + P.off_misc);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  const int D = P.stages, S = P.nst, M = P.M;

  // Granules, tiles, units and the ring: as in gemv.cu
  const int cta = blockIdx.x, g0 = cta * P.gbase + min(cta, P.gextra), g1 = g0 + P.gbase + (cta < P.gextra ? 1 : 0);
  const int gpt = P.interleave ? 2 : 4, ntiles = (g1 - g0 + gpt - 1) >> (P.interleave ? 1 : 2), mine = (ntiles * S - warp + kWarps - 1) / kWarps;
  int tile0 = 0, st0 = warp;
  if (S <= warp) { tile0 = warp / S; st0 = warp - tile0 * S; }
  auto advance = [&](int& tile, int& st) {
    tile += P.step_tiles;
    st += P.step_st;
    if (st >= S) { st -= S; tile++; }
  };
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
    if (warp == 0) misc->dead = misc->bad = 0;
  }
  __syncwarp();
  int held = ntiles * S <= D * kWarps ? 0 : D - D / 2;
  for (int i = held; i < D; i++) issue();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // ---- activations: a warp per (token, segment of 256), four of them on their way at a time ----
  const T* xg = reinterpret_cast<const T*>(P.x);
  const int items = M * P.nseg;
  auto load = [&](int i0, uint4 (&q)[4]) {
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (i0 + u * kWarps < items) q[u] = __ldcg(reinterpret_cast<const uint4*>(xg) + (size_t)(i0 + u * kWarps) * 32 + lane);
  };
  uint4 cur[4], next[4];
  load(warp, cur);
  for (; held > 0; held--) issue();
#pragma unroll 1
  for (int i0 = warp; i0 < items; i0 += 4 * kWarps) {
    load(i0 + 4 * kWarps, next);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = i0 + u * kWarps;
      if (i >= items) break;
      const int m = i / P.nseg, sg = i - m * P.nseg;
      const T* v = reinterpret_cast<const T*>(&cur[u]);
      __half o[8];
      if constexpr (kScaled) {
        float amax = 0.0f, f[8];
#pragma unroll
        for (int e = 0; e < 8; e++) { f[e] = Act<T>::to_f(v[e]); amax = fabsf(f[e]) <= 3.4e38f ? fmaxf(amax, fabsf(f[e])) : amax; }
        const int ex = (int)(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)) >> 23), se = ex == 0 ? 127 : min(254, 268 - ex);
        const float scale = __int_as_float(se << 23);
        if (lane == 0) reinterpret_cast<float*>(smem + P.off_delta)[sg * kTokens + m] = 1.0f / scale;
#pragma unroll
        for (int e = 0; e < 8; e++) o[e] = __float2half_rn(f[e] * scale);
      } else {
#pragma unroll
        for (int e = 0; e < 8; e++) o[e] = reinterpret_cast<const __half*>(v)[e];
      }
      if constexpr (kSums) {
        float sum = 0.0f;
#pragma unroll
        for (int e = 0; e < 8; e++) sum += __half2float(o[e]);
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if ((lane & 3) == 0) reinterpret_cast<float*>(smem + P.off_sum)[(sg * 8 + (lane >> 2)) * kTokens + m] = sum;
      }
      __half r[8];
#pragma unroll
      for (int e = 0; e < 8; e++) r[e] = o[(kOrder<QT> >> (4 * e)) & 7u];
      *reinterpret_cast<uint4*>(smem + P.off_x + (size_t)m * P.x_stride + (sg * 256 + lane * 8) * 2) = *reinterpret_cast<const uint4*>(r);
    }
#pragma unroll
    for (int u = 0; u < 4; u++) cur[u] = next[u];
  }
  __syncthreads();

  // ---- the stream ----
  const int rg = QT == MLXR_Q8_0 ? g : (g & 4) | ((g & 1) << 1) | ((g >> 1) & 1);      // conflict-free reads: see gemv.cu
  const uint8_t* xrow = smem + P.off_x + (size_t)min(g, M - 1) * P.x_stride + 16 * c;
  const float* sums = reinterpret_cast<const float*>(smem + P.off_sum) + 2 * c;
  float* parts = reinterpret_cast<float*>(smem + P.off_parts);          // [tiles of a chunk][warp][16][M]
  const int tile_floats = kWarps * 16 * M;
  float tot[4] = {};
  int tile = tile0, st = st0, slot = 0, left = mine;
  uint32_t par = 0;
  const int row_end = min(4 * g1, P.n_total);
  for (int t0 = 0;; t0 += P.chunk) {
    const int t1 = min(t0 + P.chunk, ntiles);
    while (left > 0 && tile < t1) {
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&misc->full[warp][slot]), par, &misc->dead, P.wait_ns))) break;
      const uint8_t* stage = smem + (size_t)(warp * D + slot) * G_::kStage;
      const uint8_t *rl = stage + (rg >> 2) * G_::kBox + (rg & 3) * G_::kPitch, *rh = rl + 2 * G_::kBox;
#pragma unroll 1
      for (int k = 0; k < G_::kSegs; k++) {
        const int sg = st * G_::kSegs + k;
        if (sg >= P.nseg) break;
        float a[4] = {};
        seg<QT>(rl + k * G_::kSeg, rh + k * G_::kSeg, xrow + sg * 512, sums + sg * 64, c, a);
        float2 dx = make_float2(1.0f, 1.0f);
        if constexpr (kScaled) dx = *reinterpret_cast<const float2*>(reinterpret_cast<const float*>(smem + P.off_delta) + sg * kTokens + 2 * c);
        tot[0] = fmaf(dx.x, a[0], tot[0]);
        tot[1] = fmaf(dx.y, a[1], tot[1]);
        tot[2] = fmaf(dx.x, a[2], tot[2]);
        tot[3] = fmaf(dx.y, a[3], tot[3]);
      }
      if (++slot == D) { slot = 0; par ^= 1u; }
      __syncwarp();
      issue();
      left--;
      const int was = tile;
      advance(tile, st);
      if (tile != was || left == 0) {
        float* dst = parts + (was - t0) * tile_floats + (warp * 16 + rg) * M + 2 * c;
#pragma unroll
        for (int i = 0; i < 4; i++) {
          if (2 * c + (i & 1) < M) dst[(i >> 1) * 8 * M + (i & 1)] = tot[i];
          tot[i] = 0.0f;
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

    // ---- a thread per row and token adds the warps' parts in the order of K ----
    const int n = (t1 - t0) * 16 * M;
    bool bad = false;
    for (int e = tid; e < n; e += kThreads) {
      const int row = e / M, m = e - row * M, tl = row >> 4, r = row & 15, first = (t0 + tl) * S;
      float* p = parts + tl * tile_floats + r * M + m;
      float a[kWarps], v = 0.0f;
#pragma unroll
      for (int k = 0; k < kWarps; k++) a[k] = k < S ? p[((first + k) & (kWarps - 1)) * 16 * M] : 0.0f;
#pragma unroll
      for (int k = 0; k < kWarps; k++) v += a[k];
      if (P.interleave) {
        if (4 * g0 + 8 * (t0 + tl) + (r & 7) < row_end) bad = bad || !(fabsf(v) <= 3.402823466e38f);
        p[(first & (kWarps - 1)) * 16 * M] = v;      // only this thread reads that place
        continue;
      }
      int R = 4 * g0 + 16 * (t0 + tl) + r;
      if (R >= row_end) continue;
      bad = bad || !(fabsf(v) <= 3.402823466e38f);
      int mat = 0;
      if (P.nmat > 1 && R >= P.rows[0]) { R -= P.rows[0]; mat = 1; if (P.nmat > 2 && R >= P.rows[1]) { R -= P.rows[1]; mat = 2; } }
      if (P.bias) v += Act<T>::to_f(reinterpret_cast<const T*>(P.bias)[R]);
      reinterpret_cast<T*>(P.y[mat])[(size_t)m * P.rows[mat] + R] = Act<T>::from_f(v);
    }
    if (bad) misc->bad = 1;
    __syncthreads();
    if (P.interleave) {
      for (int e = tid; e < n / 2; e += kThreads) {
        const int pr = e / M, m = e - pr * M, tl = pr >> 3, r = pr & 7, first = (t0 + tl) * S, col = 4 * g0 + 8 * (t0 + tl) + r;
        if (col >= row_end) continue;
        const float* p = parts + tl * tile_floats + (first & (kWarps - 1)) * 16 * M + r * M + m;
        const float gv = Act<T>::to_f(Act<T>::from_f(p[0])), uv = Act<T>::to_f(Act<T>::from_f(p[8 * M]));
        reinterpret_cast<T*>(P.y[0])[(size_t)m * P.n_total + col] = Act<T>::from_f(swish_f(gv) * uv);
      }
      __syncthreads();
    }
    if (__builtin_expect(misc->bad, 0)) {
      // ---- some sum of these tiles is not finite: results that are not, again from the float32 weights, a warp each ----
      const int per = P.interleave ? 8 : 16, cols = (t1 - t0) * per;
#pragma unroll 1
      for (int e = warp; e < cols * M; e += kWarps) {
        const int m = e / cols, q = e - m * cols, tl = q / per, r = q - tl * per;
        int R = 4 * g0 + per * (t0 + tl) + r, mat = 0;
        if (R >= row_end) continue;
        if (!P.interleave && P.nmat > 1 && R >= P.rows[0]) { R -= P.rows[0]; mat = 1; if (P.nmat > 2 && R >= P.rows[1]) { R -= P.rows[1]; mat = 2; } }
        T* y = reinterpret_cast<T*>(P.y[mat]) + (size_t)m * P.rows[mat] + R;
        if (fabsf(Act<T>::to_f(*y)) <= 3.402823466e38f) continue;
        const T* x = xg + (size_t)m * P.K;
        const float s0 = exact_sum<QT, T>(P.w[mat] + (size_t)R * P.row_bytes, x, P.K, lane);
        T o;
        if (P.interleave) {
          const float s1 = exact_sum<QT, T>(P.w[1] + (size_t)R * P.row_bytes, x, P.K, lane);
          o = Act<T>::from_f(swish_f(Act<T>::to_f(Act<T>::from_f(s0))) * Act<T>::to_f(Act<T>::from_f(s1)));
        } else {
          o = Act<T>::from_f(s0 + (P.bias ? Act<T>::to_f(reinterpret_cast<const T*>(P.bias)[R]) : 0.0f));
        }
        __syncwarp();
        if (lane == 0) *y = o;
      }
      __syncthreads();
      if (tid == 0) misc->bad = 0;
      __syncthreads();
    }
    if (t1 == ntiles) break;
  }
}

}  // namespace gemvt

using namespace gemvt;

// Shared-memory layout for a launch; the total, or 0 if it does not fit an SM
template <int QT> static size_t layout(Params* P, int grid) {
  using G = Geo<QT>;
  const int per = P->interleave ? 2 : 4, most = (P->granules + grid - 1) / grid, tiles = (most + per - 1) / per;
  P->x_stride = 2 * P->K + 64;       // two tokens lie 64 bytes apart modulo 128: a quad's reads and the next token's do not conflict
  for (P->stages = kMaxStages; P->stages >= 1; P->stages--)
    for (P->chunk = kMaxChunk; P->chunk >= 1; P->chunk /= 2) {
      if (P->chunk < 4 && P->chunk < tiles) continue;       // a meeting of the warps for every few tiles
      size_t o = (size_t)kWarps * P->stages * G::kStage;
      auto take = [&](size_t n) { const size_t at = o; o += (n + 15) & ~(size_t)15; return (int)at; };
      P->off_x = take((size_t)P->M * P->x_stride);
      P->off_sum = take(G::kSums ? (size_t)P->nseg * 8 * kTokens * 4 : 0);
      P->off_delta = take((size_t)P->nseg * kTokens * 4);
      P->off_parts = take((size_t)std::min(tiles, P->chunk) * kWarps * 16 * P->M * 4);
      P->off_misc = take(sizeof(Misc));
      if (o <= (size_t)kSmemMax) return o;
    }
  return 0;
}
static size_t layout(int qt, Params* P, int grid) {
  switch (qt) {
    case MLXR_GGML_Q4_K: return layout<MLXR_GGML_Q4_K>(P, grid);
    case MLXR_Q4_K: return layout<MLXR_Q4_K>(P, grid);
    case MLXR_Q4_0: return layout<MLXR_Q4_0>(P, grid);
    default: return layout<MLXR_Q8_0>(P, grid);
  }
}

// Where this kernel is the faster one of the two that take these calls (the other: smallm.cu, which splits K over CTAs).  Every CTA
// here converts all M * K activations and multiplies whole rows, so few rows of many activations are the other's; bf16 ones
// cost more to convert.  Device times, weights rotating through more than L2, this / the other in us:
//   canonical Q4_K  bf16 5 tokens 1000 x 4096 6.1 / 6.6, 1000 x 5632 7.6 / 7.5, 1000 x 8192 9.8 / 9.1, 4096 x 8192 15.2 / 17.6, 14336 x 4096 17.4 / 28.5;
//                   3 tokens 256 x 16384 14.2 / 9.5, 3000 x 14336 21.1 / 20.7, 4096 x 16384 24.2 / 30.6; one 256 x 24576 14.2 / 12.2.  fp16
//                   6 tokens 1000 x 8192 7.8 / 9.1; 2 tokens 256 x 16384 10.7 / 9.5.  One token of 1000 x 256 3.3 / 3.0 (the generic kernel)
//   Q8_0            bf16 3 tokens 1000 x 11008 10.8 / 10.9, 1000 x 16384 16.3 / 12.3, 4096 x 14336 25.8 / 28.4; 8 tokens 1000 x 3072 5.8 / 6.8,
//                   1000 x 5632 9.7 / 7.4, 3000 x 5632 13.9 / 12.3, 4096 x 5632 14.7 / 14.8
//   Q4_K, Q4_0      (one 16-bit part per weight over there, 1.75 times as far from the exact result: left to it where it gains an eighth and more)
//                   Q4_K 3 tokens 1000 x 768 3.6 / 3.3, 4096 x 1024 3.7 / 3.8, 6144 x 1024 4.4 / 4.0, 4096 x 1536 4.5 / 5.7, 8192 x 1536 5.7 / 5.1, 8192 x
//                   2048 6.8 / 7.6, 1000 x 4096 5.0 / 5.1, 1000 x 8192 8.0 / 6.3; 8 tokens 1000 x 1024 4.0 / 3.7, 1000 x 2048 4.9 / 5.1, 1000 x
//                   4096 7.2 / 5.3.  Q4_0 5 tokens 1000 x 3072 4.9 / 5.3
//   gate / up       Q4_K 5 tokens of hidden size 1024: block of 2048 9.7 / 11.4
//   q / k / v       Q4_K bf16 8 tokens of hidden size 2048 (3072 rows) 0.96 of the other's time, 2560 (3584) 1.10, 3072 (4096) 1.04,
//                   4096 (4352) 1.05, (6144) 0.91, 5120 (5376) 1.08; canonical 5120 (6144) 0.91; Q4_0, 6 tokens and fp16 at most 1.04
// To 2368 rows (16 for each of 148 SMs) a CTA has one tile of rows; from 1800 on the other's CTAs have as much to do as at 2368.
bool gemv_tokens_faster(int qt, int M, int K, int rows, int form, int dtype) {
  const long long acts = (long long)M * K;
  const bool bf16 = dtype == MLXR_BF16, one_full = rows >= 1800 && rows <= 2368, two = rows > 2368;
  if (form == kTokensStacked) return !(bf16 && qt != MLXR_Q4_0 && M >= 7 && K > 2048 && K < 4096 && 2ll * rows < 3ll * K);
  if (qt == MLXR_Q4_K || qt == MLXR_Q4_0) {
    const long long most = qt == MLXR_Q4_K ? 18432 : 20480;
    if (form == kTokensPlain && ((K < 1536 && rows > 4096) || (K < 2048 && rows > 6144))) return false;
    // a block whose down rows are the other kernel's too: 6 tokens of 1024 x 3584 12.6 us in turns, 11.5 both there
    if (form == kTokensGateUp && K < 1536 && rows > 6144 && (long long)M * rows > 2 * most) return false;
    return acts * rows <= 3ll << 24 && acts <= most;
  }
  if (rows >= 3500) return true;
  if (qt == MLXR_Q8_0) return acts <= (bf16 ? (one_full ? 39000 : two ? 34000 : 28000 + 3 * rows) : (one_full ? 49152 : two ? 36500 : 38000 + rows));
  if (M == 1 && K <= 512 && rows <= 1024) return false;
  if (one_full && M <= 3) return true;
  if (!bf16) return rows >= 3000 || K <= 8192 || (rows >= 1500 && M <= 2) || (M + 2ll) * K <= 58000 + 20ll * rows;      // 8192: one stage for each of the 16 warps
  return acts <= (one_full ? 46000 : two ? 33500 : M == 1 ? 13500 + 12 * rows : 26000 + 4 * rows);
}

bool gemv_tokens_supported(int qt, int M, int K, int rows, int form, int dtype, const void* x, const void* const* w, int nmat) {
  if (dtype != MLXR_F16 && dtype != MLXR_BF16) return false;
  if (qt != MLXR_GGML_Q4_K && qt != MLXR_Q8_0 && qt != MLXR_Q4_K && qt != MLXR_Q4_0) return false;
  // One linear or gate / up of MLXR's 4-bit formats and fp16 activations multiplies weights in the shader's half arithmetic
  if ((qt == MLXR_Q4_K || qt == MLXR_Q4_0) && dtype == MLXR_F16 && form != kTokensStacked) return false;
  if (M < (qt == MLXR_GGML_Q4_K ? 1 : 3) || M > kTokens || K < 256 || K % 256 != 0 || rows < 1 || rows > (1 << 19)) return false;
  if (M * (long long)K > 49152 || !gemv_tokens_faster(qt, M, K, rows, form, dtype)) return false;
  int sms = 0;
  if (device_sms(&sms)) return false;
  Params P;
  memset(&P, 0, sizeof(P));
  P.K = K;
  P.M = M;
  P.nseg = K / 256;
  P.interleave = form == kTokensGateUp;
  P.granules = (rows / (P.interleave + 1) + 3) / 4;
  if (!layout(qt, &P, std::max(1, std::min(sms, P.granules)))) return false;
  for (int i = 0; i < nmat; i++)
    if (((uintptr_t)w[i]) & 15u) return false;
  return (((uintptr_t)x) & 15u) == 0;
}

template <int QT, typename T> static int launch_tokens_inst(Params& P, int grid, cudaStream_t st) {
  auto kern = gemv_tokens_kernel<QT, T>;
  const size_t smem = layout<QT>(&P, grid);
  if (!smem) { set_error("gemv_tokens: K = %d does not fit shared memory", P.K); return MLXR_ERR_UNSUPPORTED; }
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

int launch_gemv_tokens(const void* x, const void* const* w, const int* rows, int nmat, int form, const void* bias, void* const* y, int M, int K, int qt, int dtype,
                       int* status, cudaStream_t st) {
  int sms = 0;
  if (int r = device_sms(&sms)) return r;
  Params P;
  memset(&P, 0, sizeof(P));
  P.interleave = form == kTokensGateUp;
  P.nmat = nmat;
  P.row_bytes = (size_t)(K / block_elems(qt)) * block_bytes(qt);
  for (int j = 0; j < nmat; j++) {
    P.rows[j] = P.interleave ? rows[0] : rows[j];
    P.n_total += P.interleave && j ? 0 : P.rows[j];
    P.y[j] = P.interleave && j ? nullptr : y[j];
    P.w[j] = (const uint8_t*)w[j];
    if (form == kTokensStacked && P.rows[j] % 4 != 0) { set_error("gemv_tokens: stacked matrices need row counts that are multiples of 4"); return MLXR_ERR_UNSUPPORTED; }
    if (int r = rows_map(w[j], P.rows[j], P.row_bytes, qt == MLXR_Q8_0 ? Geo<MLXR_Q8_0>::kPitch : Geo<MLXR_Q4_K>::kPitch, 4, &P.map[j])) return r;
  }
  P.granules = (P.n_total + 3) / 4;
  P.K = K;
  P.nseg = K / 256;
  P.nst = qt == MLXR_Q8_0 ? P.nseg : (P.nseg + 1) / 2;
  P.M = M;
  P.x = x;
  P.bias = bias;
  P.status = status;
  P.wait_ns = wait_limit_ns();
  const int grid = std::min(P.granules, sms);
  P.gbase = P.granules / grid;
  P.gextra = P.granules % grid;
  P.step_tiles = kWarps / P.nst;
  P.step_st = kWarps % P.nst;
#define MLXR_TOKENS(QTV) return dtype == MLXR_F16 ? launch_tokens_inst<QTV, __half>(P, grid, st) : launch_tokens_inst<QTV, __nv_bfloat16>(P, grid, st)
  switch (qt) {
    case MLXR_GGML_Q4_K: MLXR_TOKENS(MLXR_GGML_Q4_K);
    case MLXR_Q4_K: MLXR_TOKENS(MLXR_Q4_K);
    case MLXR_Q4_0: MLXR_TOKENS(MLXR_Q4_0);
    case MLXR_Q8_0: MLXR_TOKENS(MLXR_Q8_0);
    default: set_error("gemv_tokens: no code for %s", mlxr_quant_type_name(qt)); return MLXR_ERR_UNSUPPORTED;
  }
#undef MLXR_TOKENS
}

}  // namespace mlxr
