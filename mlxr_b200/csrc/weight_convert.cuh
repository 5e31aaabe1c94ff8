// Packed weights in shared memory -> 16-bit MMA operands in registers, for the tensor-core kernels
// that hold the weight tile in tensor memory.
//
// One thread owns one weight row.  A work unit is 256 consecutive weights of a row ("super-block"
// whatever the format), staged by TMA; convert64 turns 64 of them into 2 x 16 registers of packed pairs,
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
//            (fp16) significant bits.  For the products that use the float32 value of the weight: Q8_0 and
//            NF4 up to 8 tokens, canonical Q4_K, and the q / k / v projections of 4-bit formats up to 8 tokens
enum Mode { kFast = 0, kRound = 1, kSplit = 2 };

// Bytes that 256 weights of a row occupy, and the bytes staged for them.  NF4's 136 bytes are not a
// multiple of the 16 that TMA coordinates and boxes need: 144 bytes from the 16-byte boundary at or
// below them are staged and the row starts at byte 0 or 8 of the stage row.
template <int QT> struct Geo {
  static constexpr int kUnit = QT == MLXR_Q8_0 ? 272 : QT == MLXR_NF4 ? 136 : 144;
  static constexpr int kStage = QT == MLXR_NF4 ? 144 : kUnit;
};

__device__ __forceinline__ uint32_t dup_bf16(float f) {
  const __nv_bfloat162 v = __float2bfloat162_rn(f);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t dup_f16(__half h) {
  const __half2 v = __half2half2(h);
  return *reinterpret_cast<const uint32_t*>(&v);
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

// Both members times f, one instruction (fmul.f32x2)
__device__ __forceinline__ float2 mul2(float2 v, float f) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmul.rn.f32x2 c, a, b;\n\tmov.b64 {%0, %1}, c;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(v.x), "f"(v.y), "f"(f));
  return r;
}
__device__ __forceinline__ float2 fma2(float2 v, float f, float c) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 c, {%5, %5};\n\tfma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(v.x), "f"(v.y), "f"(f), "f"(c));
  return r;
}
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

// N consecutive words of a row in shared memory from byte PER * kb (rounded down to a word).  A run-time kb takes
// word loads; a compile-time one (tc::Int) the widest loads that the row's alignment of ALIGN bytes allows, and
// the bytes around the words go unused.
template <int PER, int ALIGN, int N> __device__ __forceinline__ void lds_words(const uint8_t* row, int kb, uint32_t (&w)[N]) {
  const uint32_t* p = reinterpret_cast<const uint32_t*>(row + ((PER * kb) & ~3));
#pragma unroll
  for (int i = 0; i < N; i++) w[i] = p[i];
}
template <int PER, int ALIGN, int N, int KB> __device__ __forceinline__ void lds_words(const uint8_t* row, tc::Int<KB>, uint32_t (&w)[N]) {
  constexpr int at = (PER * KB) & ~3, first = at / ALIGN, count = (at + 4 * N + ALIGN - 1) / ALIGN - first, skip = (at - first * ALIGN) / 4, per = ALIGN / 4;
  uint32_t v[count * per];
#pragma unroll
  for (int i = 0; i < count; i++) {
    if constexpr (ALIGN == 16) {
      const uint4 q = *reinterpret_cast<const uint4*>(row + (first + i) * 16);
      v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
    } else {
      const uint2 q = *reinterpret_cast<const uint2*>(row + (first + i) * 8);
      v[2 * i] = q.x; v[2 * i + 1] = q.y;
    }
  }
#pragma unroll
  for (int i = 0; i < N; i++) w[i] = v[skip + i];
}
template <int KB> __device__ __forceinline__ constexpr int block_of(tc::Int<KB>) { return KB; }
__device__ __forceinline__ int block_of(int kb) { return kb; }
__device__ __forceinline__ __half low_half(uint32_t v) { return __ushort_as_half((unsigned short)(v & 0xFFFFu)); }
__device__ __forceinline__ __half high_half(uint32_t v) { return __ushort_as_half((unsigned short)(v >> 16)); }
// 1024 + n as fp16 is 0x6400 | n: the exact half of a 6-bit field without a conversion instruction
__device__ __forceinline__ __half half_of6(uint32_t n) {
  return __hsub(__ushort_as_half((unsigned short)(0x6400u | n)), __ushort_as_half((unsigned short)0x6400));
}

// Tables in shared memory that turn a byte (two codes) into a pair of numbers, a copy for each lane so that lookups never
// conflict; rows are 256 bytes apart, so that one byte permute makes the place: the code in byte 1, the lane's copy in byte 0.
template <int BYTES> struct TableBase {
  const uint8_t* t;
  uint32_t mine;
  __device__ __forceinline__ TableBase(const uint8_t* table, int lane) : t(table), mine(BYTES * (uint32_t)lane) {}
  template <int J> __device__ __forceinline__ const uint8_t* at(uint32_t v) const {
    uint32_t o;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(o) : "r"(v), "r"(mine), "n"(0x5504 | (J << 4)));
    return t + o;
  }
};
// Pairs n0 - 8, n1 - 8 of the two nibbles of a byte, in fp16 (BF 0) or bf16
template <int BF> struct CodePairs : TableBase<4> {
  static constexpr int kBytes = 256 * 256;
  using TableBase<4>::TableBase;
  template <int J> __device__ __forceinline__ uint32_t pair(uint32_t v) const { return *reinterpret_cast<const uint32_t*>(at<J>(v)); }
  // by all threads of the CTA; a barrier must follow
  static __device__ __forceinline__ void fill(uint8_t* table, int tid, int threads) {
    for (int i = tid; i < 256 * 8; i += threads) {
      const float a = (float)((i >> 3) & 15) - 8.0f, b = (float)(i >> 7) - 8.0f;
      uint32_t w;
      if constexpr (BF == 0) { const __half2 h = __floats2half2_rn(a, b); w = *reinterpret_cast<const uint32_t*>(&h); }
      else { const __nv_bfloat162 h = __floats2bfloat162_rn(a, b); w = *reinterpret_cast<const uint32_t*>(&h); }
      *reinterpret_cast<uint4*>(table + (i >> 3) * 256 + (i & 7) * 16) = make_uint4(w, w, w, w);
    }
  }
};
// The same pairs in float32, for bf16 weights that are rounded once.  Two cycles of shared memory per lookup: only two words of
// four take the table, the others the arithmetic, so that neither the one nor the other pipe is the limit.
struct CodePairs32 : TableBase<8> {
  static constexpr int kBytes = 256 * 256;
  using TableBase<8>::TableBase;
  template <int J> __device__ __forceinline__ float2 pair(uint32_t v) const { return *reinterpret_cast<const float2*>(at<J>(v)); }
  static __device__ __forceinline__ void fill(uint8_t* table, int tid, int threads) {
    for (int i = tid; i < kBytes / 16; i += threads) {
      const float a = (float)((i >> 4) & 15) - 8.0f, b = (float)(i >> 8) - 8.0f;
      reinterpret_cast<float4*>(table)[i] = make_float4(a, b, a, b);
    }
  }
};
// Eight weights of one word from the table: the same values as fast8_bf16 and exact8_f16 (MIN: the format has a min)
template <int BF, bool MIN> __device__ __forceinline__ void table8(uint32_t v, uint32_t ss, uint32_t sm, const CodePairs<BF>& t, uint32_t* out) {
  const uint32_t q[4] = {t.template pair<0>(v), t.template pair<1>(v), t.template pair<2>(v), t.template pair<3>(v)};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if constexpr (BF == 0) {
      __half2 r = __hmul2_rn(as_half2(q[j]), as_half2(ss));
      if constexpr (MIN) r = __hadd2_rn(r, as_half2(sm));
      out[j] = *reinterpret_cast<const uint32_t*>(&r);
    } else {
      const __nv_bfloat162 r = MIN ? __hfma2(as_bf162(q[j]), as_bf162(ss), as_bf162(sm)) : __hmul2_rn(as_bf162(q[j]), as_bf162(ss));
      out[j] = *reinterpret_cast<const uint32_t*>(&r);
    }
  }
}

// Eight weights q ss + sm of one word of nibbles (q = n - 8), in the form MODE asks for
template <int BF, int MODE> struct Scale { uint32_t s, m; float min = 0.0f; };      // packed pair, or float32 bits (kRound in bf16: m = min - 136 s)
template <int BF, int MODE> __device__ __forceinline__ Scale<BF, MODE> make_scale(__half ss, __half sm) {
  if constexpr (MODE == kSplit) return {__float_as_uint(__half2float(ss)), __float_as_uint(__half2float(sm))};
  else if constexpr (BF == 0) return {dup_f16(ss), dup_f16(sm)};
  else if constexpr (MODE == kFast) return {dup_bf16(__half2float(ss)), dup_bf16(__half2float(sm))};
  else { const float f = __half2float(ss), m = __half2float(sm); return {__float_as_uint(f), __float_as_uint(fmaf(-136.0f, f, m)), m}; }
}
template <int BF, int MODE, bool MIN> __device__ __forceinline__ void nibbles8(int, uint32_t v, const Scale<BF, MODE>& c, const CodePairs<BF>& t, uint32_t* out, uint32_t*) {
  table8<BF, MIN>(v, c.s, c.m, t, out);
}
// i: the word's number in its block, a constant
template <int BF, int MODE, bool MIN> __device__ __forceinline__ void nibbles8(int i, uint32_t v, const Scale<BF, MODE>& c, const CodePairs32& t, uint32_t* out, uint32_t*) {
  const float s = __uint_as_float(c.s), m = __uint_as_float(c.m);
  if (i & 1) return put(dequant8_bf16(v, s, m), out);
  const float2 q[4] = {t.template pair<0>(v), t.template pair<1>(v), t.template pair<2>(v), t.template pair<3>(v)};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const float2 w = MIN ? fma2(q[j], s, c.min) : mul2(q[j], s);
    const __nv_bfloat162 b = __floats2bfloat162_rn(w.x, w.y);
    out[j] = *reinterpret_cast<const uint32_t*>(&b);
  }
}
template <int BF, int MODE, bool MIN, typename L> __device__ __forceinline__ void nibbles8(int, uint32_t v, const Scale<BF, MODE>& c, const L&, uint32_t* out, uint32_t* res) {
  if constexpr (MODE == kSplit) {
    const uint32_t lo = v & 0x0F0F0F0Fu, hi = (v >> 4) & 0x0F0F0F0Fu;
    const float s = __uint_as_float(c.s), m = __uint_as_float(c.m);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      // byte n in the low byte of 0x4B00'0000 is the fp32 number 2^23 + n: n - 8 exactly, one rounding of the sum
      const float fe = __uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7440u | (uint32_t)j)) - 8388616.0f;
      const float fo = __uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7440u | (uint32_t)j)) - 8388616.0f;
      emit<BF, MODE>(fmaf(fe, s, m), fmaf(fo, s, m), out[j], res[j]);
    }
  } else if constexpr (BF == 0) exact8_f16(v, c.s, c.m, out);
  else if constexpr (MODE == kFast) fast8_bf16(v, c.s, c.m, out);
  else put(dequant8_bf16(v, __uint_as_float(c.s), __uint_as_float(c.m)), out);
}

// NF4 levels of the codes in byte J of v, from tables in shared memory.  Levels: the 16 levels, one word per bank, so that lookups
// never conflict.  PairLevels: the two levels of every byte, once for each thread of a half warp, whose eight bytes lie
// in banks of their own: half the address arithmetic and loads per weight.
struct Levels {
  const float* t;
  template <int J> __device__ __forceinline__ float2 pair(uint32_t v) const { return make_float2(t[(v >> (8 * J)) & 15u], t[(v >> (8 * J + 4)) & 15u]); }
};
struct PairLevels {
  static constexpr int kBytes = 256 * 16 * 8;
  uint32_t t;                 // shared address of this thread's copy
  __device__ __forceinline__ PairLevels(const void* table, int lane) : t(tc::smem_u32(table) + 8u * (uint32_t)(lane & 15)) {}
  template <int J> __device__ __forceinline__ float2 pair(uint32_t v) const {
    float2 r;
    asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(r.x), "=f"(r.y) : "r"(__byte_perm(v, 0u, 0x4440u | J) * 128u + t));
    return r;
  }
  // by all threads of the CTA; a barrier must follow
  static __device__ __forceinline__ void fill(void* table, int tid, int threads) {
    for (int i = tid; i < kBytes / 16; i += threads) {
      const float lo = kNF4[(i >> 3) & 15], hi = kNF4[i >> 7];
      reinterpret_cast<float4*>(table)[i] = make_float4(lo, hi, lo, hi);
    }
  }
};

// PairLevels with a copy for every lane: one instruction for the address instead of two, 64 KB instead of 32
struct LanePairLevels : TableBase<8> {
  static constexpr int kBytes = 256 * 256;
  using TableBase<8>::TableBase;
  template <int J> __device__ __forceinline__ float2 pair(uint32_t v) const { return *reinterpret_cast<const float2*>(at<J>(v)); }
  static __device__ __forceinline__ void fill(uint8_t* table, int tid, int threads) {
    for (int i = tid; i < kBytes / 16; i += threads) {
      const float lo = kNF4[(i >> 4) & 15], hi = kNF4[i >> 8];
      reinterpret_cast<float4*>(table)[i] = make_float4(lo, hi, lo, hi);
    }
  }
};

// Weights 64 kb .. 64 kb + 63 of the unit at `row` (shared memory): out(Int<0>, hi, lo) gets the first 32,
// out(Int<1>, hi, lo) the others (lo only for kSplit).  nf4: Levels, PairLevels or LanePairLevels; CodePairs, or else nothing of use, for
// the other formats.  KB is int or tc::Int.  With a run-time kb the body stays at a few hundred
// instructions that every producer warp shares; unrolled over a unit of the long conversions (kSplit), or
// specialised per group, the warps of a scheduler fetch more code than its instruction cache holds and
// wait for it (the largest stall by far: canonical Q4_K [16, 4096] x [37888, 4096]^T 90.9 us unrolled, 52.5
// us rolled).  The short conversions fit unrolled and are faster so (Q4_K, same size: 27.8 rolled, 24.7).
template <int QT, int BF, int MODE, typename KB, typename L, typename F>
__device__ __forceinline__ void convert64(const uint8_t* row, KB KBV, const L& nf4, F&& out) {
  const int kb = block_of(KBV);
  uint32_t a[16], b[16];
  if constexpr (QT == MLXR_Q4_K) {
    // d, dmin (fp16), scales[12] of which the shader reads six bytes: (scale, min) pairs 0 .. 3 as eight 6-bit
    // fields (q_gemm_dequant.metal:222-242); sub-block 2 kb takes the first pair of its half, sub-block
    // 2 kb + 1 the second one for even kb.  Sub-block scale = rn16(sc * d), min = rn16(m * dmin).
    const uint4 h = *reinterpret_cast<const uint4*>(row);
    const uint4 q0 = *reinterpret_cast<const uint4*>(row + 16 + 32 * kb), q1 = *reinterpret_cast<const uint4*>(row + 32 + 32 * kb);
    const uint32_t f = (kb & 2) ? __funnelshift_r(h.y, h.z, 24) : h.y, g = (kb & 1) ? f : f >> 12;
    const __half d = low_half(h.x), dmin = high_half(h.x);
    const auto c0 = make_scale<BF, MODE>(__hmul_rn(half_of6(f & 63u), d), __hmul_rn(half_of6((f >> 6) & 63u), dmin));
    const auto c1 = make_scale<BF, MODE>(__hmul_rn(half_of6(g & 63u), d), __hmul_rn(half_of6((g >> 6) & 63u), dmin));
    const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
    for (int i = 0; i < 4; i++) nibbles8<BF, MODE, true>(i, w[i], c0, nf4, a + 4 * i, b + 4 * i);
    out(tc::Int<0>{}, a, b);
#pragma unroll
    for (int i = 0; i < 4; i++) nibbles8<BF, MODE, true>(i, w[4 + i], c1, nf4, a + 4 * i, b + 4 * i);
    out(tc::Int<1>{}, a, b);
  } else if constexpr (QT == MLXR_Q4_0) {       // two 18-byte blocks: fp16 d, 16 bytes of nibbles (q_gemm_dequant.metal:142-161)
    uint32_t w[9];
    lds_words<36, 16>(row, KBV, w);
    const __half zero = __ushort_as_half((unsigned short)0);
    const auto c0 = make_scale<BF, MODE>(low_half(w[0]), zero), c1 = make_scale<BF, MODE>(high_half(w[4]), zero);
#pragma unroll
    for (int i = 0; i < 4; i++) nibbles8<BF, MODE, false>(i, __funnelshift_r(w[i], w[i + 1], 16), c0, nf4, a + 4 * i, b + 4 * i);
    out(tc::Int<0>{}, a, b);
#pragma unroll
    for (int i = 0; i < 4; i++) nibbles8<BF, MODE, false>(i, w[5 + i], c1, nf4, a + 4 * i, b + 4 * i);
    out(tc::Int<1>{}, a, b);
  } else if constexpr (QT == MLXR_Q8_0) {       // two 34-byte blocks: fp16 d, 32 int8 (q_gemm_dequant.metal:190-201)
    uint32_t w[17];
    lds_words<68, 16>(row, KBV, w);
    auto block = [&](auto S) {
      constexpr int s = decltype(S)::value;
      const __half d = s ? high_half(w[8]) : low_half(w[0]);
      const float df = __half2float(d);
      [[maybe_unused]] const float s256 = 256.0f * df, c = -32896.0f * df;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t u = (s ? w[9 + i] : __funnelshift_r(w[i], w[i + 1], 16)) ^ 0x80808080u;    // bytes q + 128
#pragma unroll
        for (int j = 0; j < 2; j++) {
          if constexpr (BF == 0 && MODE != kSplit) {
            // 1024 + (q + 128) as fp16 is 0x6400 | byte; minus 1152 is q exactly; one rounding of q * d
            const uint32_t bits = __byte_perm(u, 0x64646464u, j == 0 ? 0x4140 : 0x4342);
            const __half2 r = __hmul2_rn(__hsub2(as_half2(bits), __half2half2(__ushort_as_half((unsigned short)0x6480))), __half2half2(d));
            a[2 * i + j] = *reinterpret_cast<const uint32_t*>(&r);
          } else {
            // byte b one byte up in 0x4300'0000 is the fp32 number 128 + b / 256:
            // (128 + b / 256) * 256 d - (32768 + 128) d = (b - 128) d
            const float fe = __uint_as_float(__byte_perm(u, 0x00004300u, 0x5606u | ((uint32_t)(2 * j) << 4)));
            const float fo = __uint_as_float(__byte_perm(u, 0x00004300u, 0x5606u | ((uint32_t)(2 * j + 1) << 4)));
            emit<BF, MODE>(fmaf(fe, s256, c), fmaf(fo, s256, c), a[2 * i + j], b[2 * i + j]);
          }
        }
      }
      out(S, a, b);
    };
    block(tc::Int<0>{});
    block(tc::Int<1>{});
  } else if constexpr (QT == MLXR_NF4) {        // one 34-byte block: fp16 absmax, 32 bytes of codes; odd blocks start 2 bytes off a word
    uint32_t w[9];
    lds_words<34, 8>(row, KBV, w);
    const uint32_t sh = (kb & 1) ? 16 : 0;
    const float am = __half2float((kb & 1) ? high_half(w[0]) : low_half(w[0]));
    // codes from byte 2 of the block: shifted by 16 bits for even blocks, whole words for odd ones
    auto block = [&](auto S) {
      constexpr int s = decltype(S)::value;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t v = sh ? w[4 * s + i + 1] : __funnelshift_r(w[4 * s + i], w[4 * s + i + 1], 16);
        const float2 l[4] = {nf4.template pair<0>(v), nf4.template pair<1>(v), nf4.template pair<2>(v), nf4.template pair<3>(v)};
#pragma unroll
        for (int j = 0; j < 4; j++) emit<BF, MODE>(l[j].x * am, l[j].y * am, a[4 * i + j], b[4 * i + j]);
      }
      out(S, a, b);
    };
    block(tc::Int<0>{});
    block(tc::Int<1>{});
  } else if constexpr (QT == MLXR_GGML_Q4_K) {
    // chunk kb: low nibbles of its 32 bytes are sub-block 2 kb, high nibbles sub-block 2 kb + 1; eight 6-bit
    // (scale, min) pairs, unpacked here four at a time; w = (d sc) q - dmin m in float32 (both products are exact)
    const uint4 h = *reinterpret_cast<const uint4*>(row);
    const uint4 q0 = *reinterpret_cast<const uint4*>(row + 16 + 32 * kb), q1 = *reinterpret_cast<const uint4*>(row + 32 + 32 * kb);
    const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    const uint32_t sc4 = (kb & 2) ? (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u) : h.y & 0x3F3F3F3Fu;
    const uint32_t mn4 = (kb & 2) ? ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u) : h.z & 0x3F3F3F3Fu;
    const float d = __half2float(low_half(h.x)), dmin = __half2float(high_half(h.x));
    auto block = [&](auto S) {
      constexpr int s = decltype(S)::value;
      const int at = 16 * (kb & 1) + 8 * s;
      const float ds = d * (float)((sc4 >> at) & 0xFFu), dm = dmin * (float)((mn4 >> at) & 0xFFu);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t n = (w[i] >> (4 * s)) & 0x0F0F0F0Fu;
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          // byte n in the low byte of 0x4B00'0000 is the fp32 number 2^23 + n: exact difference
          const float f = __uint_as_float(__byte_perm(n, 0x4B000000u, 0x7440u | (uint32_t)j)) - 8388608.0f;
          v[j] = __fsub_rn(__fmul_rn(ds, f), dm);
        }
        emit<BF, MODE>(v[0], v[1], a[2 * i], b[2 * i]);
        emit<BF, MODE>(v[2], v[3], a[2 * i + 1], b[2 * i + 1]);
      }
      out(S, a, b);
    };
    block(tc::Int<0>{});
    block(tc::Int<1>{});
  }
}

}  // namespace wconv
}  // namespace mlxr
