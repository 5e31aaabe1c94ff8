// Packed weights in shared memory -> 16-bit MMA operands in registers, for the tensor-core kernels
// that hold the weight tile in tensor memory.
//
// One thread owns one weight row.  A work unit is 256 consecutive weights of a row ("super-block"
// whatever the format), staged by TMA; convert32 turns 32 of them into 16 registers of packed pairs,
// element order = K order, ready for tcgen05.st (a 32-bit tensor-memory column holds two
// consecutive K elements of the row that is its lane).
#pragma once
#include "common.cuh"
#include "tc_common.cuh"

namespace mlxr {
namespace wconv {

using tc::dequant8_bf16;

// How a weight becomes a 16-bit number:
//   kFast    bf16 Q4_K / Q4_0: scale and min rounded to bf16, bf16 arithmetic (about 3e-3 relative on
//            the product); everything else as kRound
//   kRound   the exact value rounded once (fp16 Q4_K / Q4_1: the reference shader's half arithmetic)
//   kSplit   a leading and a residual 16-bit part, both multiplied: the weight keeps 16 (bf16) or 22
//            (fp16) significant bits.  For the formats whose small-batch products have always used
//            the float32 value of the weight
enum Mode { kFast = 0, kRound = 1, kSplit = 2 };

// Bytes that 256 weights of a row occupy, and the bytes staged for them.  NF4's 136 bytes are not a
// multiple of the 16 that TMA coordinates and boxes need: 144 bytes from the 16-byte boundary at or
// below them are staged and the row starts at byte 0 or 8 of the stage row.
template <int QT> struct Geo {
  static constexpr int kUnit = QT == MLXR_Q8_0 ? 272 : QT == MLXR_NF4 ? 136 : 144;
  static constexpr int kStage = QT == MLXR_NF4 ? 144 : kUnit;
};

template <int ALIGN> struct Vec;
template <> struct Vec<16> { using T = uint4; };
template <> struct Vec<8> { using T = uint2; };

// The 32-bit words covering bytes [OFF, OFF + LEN) of a row, fetched with ALIGN-byte shared-memory
// loads; word(k) is the (possibly half-word shifted) word at byte OFF + 4 k.
template <int OFF, int LEN, int ALIGN> struct Span {
  static constexpr int kFirst = OFF / ALIGN, kCount = (OFF + LEN + ALIGN - 1) / ALIGN - kFirst;
  uint32_t w[kCount * (ALIGN / 4)];
  __device__ __forceinline__ explicit Span(const uint8_t* row) {
#pragma unroll
    for (int i = 0; i < kCount; i++) {
      const typename Vec<ALIGN>::T v = *reinterpret_cast<const typename Vec<ALIGN>::T*>(row + (kFirst + i) * ALIGN);
      if constexpr (ALIGN == 16) { w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w; }
      else { w[2 * i] = v.x; w[2 * i + 1] = v.y; }
    }
  }
  template <int BYTE> __device__ __forceinline__ uint32_t word() const {   // BYTE is even
    constexpr int rel = BYTE - kFirst * ALIGN, i = rel / 4;
    if constexpr (rel % 4 == 0) return w[i];
    else return __funnelshift_r(w[i], w[i + 1], 16);
  }
  template <int BYTE> __device__ __forceinline__ __half half() const {
    constexpr int rel = BYTE - kFirst * ALIGN;
    return __ushort_as_half((unsigned short)((rel & 2) ? (w[rel / 4] >> 16) : (w[rel / 4] & 0xFFFFu)));
  }
};

// Per-row constants of a unit, decoded once for its 256 weights: scale and min of the four (scale,
// min) pairs of a Q4_K super-block in the form the conversion wants, or the packed header of a
// canonical ggml super-block.
struct Hdr { uint32_t s[4], m[4]; };

__device__ __forceinline__ uint32_t dup_bf16(float f) {
  const __nv_bfloat162 v = __float2bfloat162_rn(f);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t dup_f16(__half h) {
  const __half2 v = __half2half2(h);
  return *reinterpret_cast<const uint32_t*>(&v);
}

template <int QT, int BF, int MODE>
__device__ __forceinline__ Hdr load_header(const uint8_t* row) {
  Hdr h = {};
  if constexpr (QT == MLXR_Q4_K) {
    // d, dmin (fp16), scales[12] of which the shader reads six bytes: eight consecutive 6-bit fields,
    // scale and min of pairs 0 .. 3 (q_gemm_dequant.metal:222-242); sub-block scale = rn16(sc * d),
    // sub-block min = rn16(m * dmin)
    const uint4 q = *reinterpret_cast<const uint4*>(row);
    const __half d = __ushort_as_half((unsigned short)(q.x & 0xFFFFu)), dmin = __ushort_as_half((unsigned short)(q.x >> 16));
    const uint32_t f[4] = {q.y, q.y >> 12, __funnelshift_r(q.y, q.z, 24), q.z >> 4};
#pragma unroll
    for (int p = 0; p < 4; p++) {
      // 1024 + n as fp16 is 0x6400 | n: the exact half of a 6-bit field without a conversion instruction
      const __half k1024 = __ushort_as_half((unsigned short)0x6400);
      const __half sc = __hsub(__ushort_as_half((unsigned short)(0x6400u | (f[p] & 63u))), k1024);
      const __half mn = __hsub(__ushort_as_half((unsigned short)(0x6400u | ((f[p] >> 6) & 63u))), k1024);
      const __half ss = __hmul_rn(sc, d), sm = __hmul_rn(mn, dmin);
      if constexpr (BF == 0) { h.s[p] = dup_f16(ss); h.m[p] = dup_f16(sm); }
      else if constexpr (MODE == kFast) { h.s[p] = dup_bf16(__half2float(ss)); h.m[p] = dup_bf16(__half2float(sm)); }
      else { const float s = __half2float(ss); h.s[p] = __float_as_uint(s); h.m[p] = __float_as_uint(fmaf(-136.0f, s, __half2float(sm))); }
    }
  } else if constexpr (QT == MLXR_GGML_Q4_K) {
    const uint4 q = *reinterpret_cast<const uint4*>(row);
    h.s[0] = q.x; h.s[1] = q.y; h.s[2] = q.z; h.s[3] = q.w;
  }
  return h;
}

// Nibbles 2 j and 2 j + 1 of word v (consecutive weights) as a pair of 16-bit floats n0 - 8, n1 - 8:
// one byte permute, one and-or with the exponent of a number whose last mantissa bits are free, one
// fused multiply-add (exact).  The integer pipe is what bounds these kernels, so the second nibble stays
// where its byte has it: 1024 + 16 n1 in fp16, 128 + 8 n1 in bf16 (of v1 = v >> 1, whose nibble fits
// bf16's seven mantissa bits), and the multiply-add takes the factor out.  Written as instructions:
// the same operations through __byte_perm were rewritten by the compiler into half as many again.
template <int J> __device__ __forceinline__ uint32_t nibble_pair(uint32_t v, uint32_t v1, uint32_t mask, uint32_t magic) {
  uint32_t t;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(t) : "r"(v), "r"(v1), "n"(J | (J << 4) | ((4 + J) << 8) | ((4 + J) << 12)));
  asm("lop3.b32 %0, %0, %1, %2, 0xEA;" : "+r"(t) : "r"(mask), "r"(magic));   // (t & mask) | magic
  return t;
}
__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t v) { return *reinterpret_cast<const __nv_bfloat162*>(&v); }
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }

// Eight consecutive weights (one word of nibbles) as four bf16 pairs, bf16 arithmetic throughout: n - 8
// exactly, then one fused multiply-add with the sub-block's scale and min (both rounded to bf16).
__device__ __forceinline__ void fast8_bf16(uint32_t v, uint32_t ss_, uint32_t sm_, uint32_t* out) {
  const __nv_bfloat162 ss = as_bf162(ss_), sm = as_bf162(sm_);
  const __nv_bfloat162 f = as_bf162(0x3E003F80u), c = as_bf162(0xC1C0C308u);     // {1, 1/8}, {-136, -24}
  const uint32_t v1 = v >> 1;
  const uint32_t t[4] = {nibble_pair<0>(v, v1, 0x0078000Fu, 0x43004300u), nibble_pair<1>(v, v1, 0x0078000Fu, 0x43004300u),
                         nibble_pair<2>(v, v1, 0x0078000Fu, 0x43004300u), nibble_pair<3>(v, v1, 0x0078000Fu, 0x43004300u)};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const __nv_bfloat162 r = __hfma2(__hfma2(as_bf162(t[j]), f, c), ss, sm);
    out[j] = *reinterpret_cast<const uint32_t*>(&r);
  }
}
// The same for fp16 with the shader's arithmetic (q_gemm_dequant.metal:244-256): rn16(rn16((n - 8) ss) + sm)
__device__ __forceinline__ void exact8_f16(uint32_t v, uint32_t ss_, uint32_t sm_, uint32_t* out) {
  const __half2 ss = as_half2(ss_), sm = as_half2(sm_);
  const __half2 f = as_half2(0x2C003C00u), c = as_half2(0xD480E408u);            // {1, 1/16}, {-1032, -72}
  const uint32_t t[4] = {nibble_pair<0>(v, v, 0x00F0000Fu, 0x64006400u), nibble_pair<1>(v, v, 0x00F0000Fu, 0x64006400u),
                         nibble_pair<2>(v, v, 0x00F0000Fu, 0x64006400u), nibble_pair<3>(v, v, 0x00F0000Fu, 0x64006400u)};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const __half2 r = __hadd2_rn(__hmul2_rn(__hfma2(as_half2(t[j]), f, c), ss), sm);
    out[j] = *reinterpret_cast<const uint32_t*>(&r);
  }
}

__device__ __forceinline__ void put(const uint4& v, uint32_t* out) { out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w; }

// A pair of float32 weights -> one register (kSplit: leading part and residual)
template <int BF, int MODE>
__device__ __forceinline__ void emit(float a, float b, uint32_t& hi, uint32_t& lo) {
  if constexpr (BF == 0) {
    const __half2 h = __floats2half2_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    if constexpr (MODE == kSplit) {
      const __half2 l = __floats2half2_rn(a - __low2float(h), b - __high2float(h));
      lo = *reinterpret_cast<const uint32_t*>(&l);
    }
  } else {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    if constexpr (MODE == kSplit) {
      const __nv_bfloat162 l = __floats2bfloat162_rn(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xFFFF0000u));
      lo = *reinterpret_cast<const uint32_t*>(&l);
    }
  }
}

// Weights 32 S .. 32 S + 31 of the unit at `row` (shared memory) -> hi[16] (and lo[16] for kSplit).
// nf4: the 16 codebook levels in shared memory (one word per bank: lookups never conflict).
template <int QT, int BF, int MODE, int S>
__device__ __forceinline__ void convert32(const uint8_t* row, const Hdr& h, const float* nf4, uint32_t (&hi)[16], uint32_t (&lo)[16]) {
  if constexpr (QT == MLXR_Q4_K) {
    constexpr int p = S == 1 ? 1 : S == 5 ? 3 : S < 4 ? 0 : 2;     // sub-blocks 0, 2, 3 / 1 / 4, 6, 7 / 5 share a pair
    const Span<16 + 16 * S, 16, 16> q(row);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if constexpr (BF == 0) exact8_f16(q.w[i], h.s[p], h.m[p], hi + 4 * i);
      else if constexpr (MODE == kFast) fast8_bf16(q.w[i], h.s[p], h.m[p], hi + 4 * i);
      else put(dequant8_bf16(q.w[i], __uint_as_float(h.s[p]), __uint_as_float(h.m[p])), hi + 4 * i);
    }
  } else if constexpr (QT == MLXR_Q4_0) {       // 18-byte blocks: fp16 d, 16 bytes of nibbles (q_gemm_dequant.metal:142-161)
    const Span<18 * S, 18, 16> q(row);
    const __half d = q.template half<18 * S>();
    const uint32_t w[4] = {q.template word<18 * S + 2>(), q.template word<18 * S + 6>(), q.template word<18 * S + 10>(), q.template word<18 * S + 14>()};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if constexpr (BF == 0) exact8_f16(w[i], dup_f16(d), 0u, hi + 4 * i);
      else if constexpr (MODE == kFast) fast8_bf16(w[i], dup_bf16(__half2float(d)), 0u, hi + 4 * i);
      else { const float s = __half2float(d); put(dequant8_bf16(w[i], s, -136.0f * s), hi + 4 * i); }
    }
  } else if constexpr (QT == MLXR_Q8_0) {       // 34-byte blocks: fp16 d, 32 int8 (q_gemm_dequant.metal:190-201)
    const Span<34 * S, 34, 16> q(row);
    const __half d = q.template half<34 * S>();
    const float df = __half2float(d);
    const uint32_t w[8] = {q.template word<34 * S + 2>(),  q.template word<34 * S + 6>(),  q.template word<34 * S + 10>(), q.template word<34 * S + 14>(),
                           q.template word<34 * S + 18>(), q.template word<34 * S + 22>(), q.template word<34 * S + 26>(), q.template word<34 * S + 30>()};
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t u = w[i] ^ 0x80808080u;    // bytes q + 128
#pragma unroll
      for (int j = 0; j < 2; j++) {
        if constexpr (BF == 0 && MODE != kSplit) {
          // 1024 + (q + 128) as fp16 is 0x6400 | byte; minus 1152 is q exactly; one rounding of q * d
          const uint32_t bits = __byte_perm(u, 0x64646464u, j == 0 ? 0x4140 : 0x4342);
          const __half2 r = __hmul2_rn(__hsub2(*reinterpret_cast<const __half2*>(&bits), __half2half2(__ushort_as_half((unsigned short)0x6480))), __half2half2(d));
          hi[2 * i + j] = *reinterpret_cast<const uint32_t*>(&r);
        } else {
          // byte b one byte up in 0x4300'0000 is the fp32 number 128 + b / 256:
          // (128 + b / 256) * 256 d - (32768 + 128) d = (b - 128) d
          const float fe = __uint_as_float(__byte_perm(u, 0x00004300u, 0x5606u | ((uint32_t)(2 * j) << 4)));
          const float fo = __uint_as_float(__byte_perm(u, 0x00004300u, 0x5606u | ((uint32_t)(2 * j + 1) << 4)));
          const float s256 = 256.0f * df, c = -32896.0f * df;
          emit<BF, MODE>(fmaf(fe, s256, c), fmaf(fo, s256, c), hi[2 * i + j], lo[2 * i + j]);
        }
      }
    }
  } else if constexpr (QT == MLXR_NF4) {        // 34-byte blocks of 64: fp16 absmax, 32 bytes of codes
    constexpr int B = 34 * (S / 2), Q = B + 2 + 16 * (S & 1);
    const Span<B, 34, 8> q(row);
    const float a = __half2float(q.template half<B>());
    const uint32_t w[4] = {q.template word<Q>(), q.template word<Q + 4>(), q.template word<Q + 8>(), q.template word<Q + 12>()};
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float e = nf4[(w[i] >> (8 * j)) & 15u], o = nf4[(w[i] >> (8 * j + 4)) & 15u];
        emit<BF, MODE>(e * a, o * a, hi[4 * i + j], lo[4 * i + j]);
      }
  } else if constexpr (QT == MLXR_GGML_Q4_K) {
    // sub-block S of 64-element chunk S / 2: low (S even) or high nibbles of its 32 bytes; eight
    // 6-bit (scale, min) pairs; w = (d sc) q - dmin m in float32 (both products are exact)
    const Span<16 + 32 * (S / 2), 32, 16> q(row);
    uint32_t sc, mn;
    if constexpr (S < 4) { sc = (h.s[1] >> (8 * S)) & 63u; mn = (h.s[2] >> (8 * S)) & 63u; }
    else {
      constexpr int t = 8 * (S - 4);
      sc = ((h.s[3] >> t) & 15u) | (((h.s[1] >> (t + 6)) & 3u) << 4);
      mn = ((h.s[3] >> (t + 4)) & 15u) | (((h.s[2] >> (t + 6)) & 3u) << 4);
    }
    const float d = __half2float(__ushort_as_half((unsigned short)(h.s[0] & 0xFFFFu))), dmin = __half2float(__ushort_as_half((unsigned short)(h.s[0] >> 16)));
    const float ds = d * (float)sc, dm = dmin * (float)mn;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t n = (S & 1) ? (q.w[i] >> 4) & 0x0F0F0F0Fu : q.w[i] & 0x0F0F0F0Fu;
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        // byte n in the low byte of 0x4B00'0000 is the fp32 number 2^23 + n: exact difference
        const float f = __uint_as_float(__byte_perm(n, 0x4B000000u, 0x7440u | (uint32_t)j)) - 8388608.0f;
        v[j] = __fsub_rn(__fmul_rn(ds, f), dm);
      }
      emit<BF, MODE>(v[0], v[1], hi[2 * i], lo[2 * i]);
      emit<BF, MODE>(v[2], v[3], hi[2 * i + 1], lo[2 * i + 1]);
    }
  }
}

}  // namespace wconv
}  // namespace mlxr
