// RMSNorm, SwiGLU and RoPE as standalone kernels: the primitives called on their own, and RMSNorm and RoPE
// around the linears of three and more tokens (the kernels for fewer carry their own copies of this arithmetic).
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace mlxr {

// ---- RMSNorm ---------------------------------------------------------------------------
// One CTA per row: y = (x * rsqrt(mean(x^2) + eps)) * w (+ residual), fp32 throughout, one
// rounding at the store (rmsnorm.metal:105-156, :165-217).  The row is read once from
// HBM and kept in registers for the second pass (the reference reads it twice).
template <typename T, int THREADS, int PER_THREAD>
__global__ void __launch_bounds__(THREADS) rmsnorm_kernel(const T* x,
                                                          const T* __restrict__ w,
                                                          const T* res,
                                                          T* y, int hidden,
                                                          float eps) {
  __shared__ float red[THREADS / 32];
  // A kernel launched behind this one with programmatic stream serialization (the linears of the
  // MLP block) may start its set-up and its weight stream now; it waits for this kernel's
  // completion before it reads y.  Without such a dependent the instruction does nothing.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const size_t row = blockIdx.x;
  const T* xr = x + row * hidden;
  float v[PER_THREAD];
  float ss = 0.0f;
#pragma unroll
  for (int i = 0; i < PER_THREAD; i++) {
    const int c = threadIdx.x + i * THREADS;
    v[i] = c < hidden ? Act<T>::to_f(xr[c]) : 0.0f;
    ss = fmaf(v[i], v[i], ss);
  }
  // columns beyond THREADS * PER_THREAD (very wide rows) are streamed without caching
  for (int c = threadIdx.x + PER_THREAD * THREADS; c < hidden; c += THREADS) {
    const float t = Act<T>::to_f(xr[c]);
    ss = fmaf(t, t, ss);
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.0f;
#pragma unroll
  for (int i = 0; i < THREADS / 32; i++) tot += red[i];
  const float rms = rsqrtf(tot / (float)hidden + eps);
#pragma unroll
  for (int i = 0; i < PER_THREAD; i++) {
    const int c = threadIdx.x + i * THREADS;
    if (c < hidden) {
      float o = (v[i] * rms) * Act<T>::to_f(w[c]);
      if (res) o += Act<T>::to_f(res[row * hidden + c]);
      y[row * hidden + c] = Act<T>::from_f(o);
    }
  }
  for (int c = threadIdx.x + PER_THREAD * THREADS; c < hidden; c += THREADS) {
    float o = (Act<T>::to_f(xr[c]) * rms) * Act<T>::to_f(w[c]);
    if (res) o += Act<T>::to_f(res[row * hidden + c]);
    y[row * hidden + c] = Act<T>::from_f(o);
  }
}

template <typename T> __device__ __forceinline__ void unpack8(const uint4& u, float (&v)[8]) {
  const T* h = reinterpret_cast<const T*>(&u);
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = Act<T>::to_f(h[i]);
}
// Eight 16-bit values, one 128-bit access.  From L2, coherently: a kernel that starts under the one before it (programmatic
// stream serialization) may find x still being written when it begins, and in place x is written by the kernel
// itself; the read-only path (and const __restrict__, which lets the compiler take it) is defined only for data that
// nobody writes while the kernel runs.  That holds for the norm weight and the tables: __ldg there.
template <typename T> __device__ __forceinline__ void load8v(const T* p, float (&v)[8]) {
  unpack8<T>(__ldcg(reinterpret_cast<const uint4*>(p)), v);
}
template <typename T> __device__ __forceinline__ void store8v(T* p, const float (&v)[8]) {
  uint4 u;
  T* h = reinterpret_cast<T*>(&u);
#pragma unroll
  for (int i = 0; i < 8; i++) h[i] = Act<T>::from_f(v[i]);
  *reinterpret_cast<uint4*>(p) = u;
}
static bool aligned16(const void* a, const void* b, const void* c = nullptr, const void* d = nullptr) {
  return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d) & 15u) == 0;
}

// A launch that may start under the previous kernel of the stream (both wait with griddepcontrol before they touch memory)
static cudaLaunchConfig_t overlapped(int grid, int threads, cudaStream_t st, cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = st;
  at->id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at->val.programmaticStreamSerializationAllowed = overlap_launches() ? 1 : 0;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// The same row for 16-bit types in 128-bit accesses: a row stays in registers between the two passes.
// Bound by HBM (three streams with a residual); with 2-byte accesses the loads in flight were an eighth
// of this and [1111, 4096] fp16 took 14 us where the bytes need 4.2.  Launched with programmatic stream
// serialization: the CTAs are in place when the previous kernel of the stream ends.
template <typename T, int THREADS, int PER>
__global__ void __launch_bounds__(THREADS) rmsnorm_vec_kernel(const T* x, const T* __restrict__ w, const T* res, T* y, int nvec, float eps) {
  __shared__ float red[THREADS / 32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const size_t row = (size_t)blockIdx.x * nvec * 8;
  float v[PER][8], ss = 0.0f;
  uint4 wv[PER], rv[PER];
#pragma unroll
  for (int i = 0; i < PER; i++) {
    const int c = threadIdx.x + i * THREADS;
    if (c < nvec) {
      load8v(x + row + c * 8, v[i]);
      wv[i] = __ldg(reinterpret_cast<const uint4*>(w) + c);
      if (res) rv[i] = __ldcg(reinterpret_cast<const uint4*>(res + row) + c);      // before any store: y may be res
#pragma unroll
      for (int e = 0; e < 8; e++) ss = fmaf(v[i][e], v[i][e], ss);
    }
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.0f;
#pragma unroll
  for (int i = 0; i < THREADS / 32; i++) tot += red[i];
  const float rms = rsqrtf(tot / (float)(nvec * 8) + eps);
#pragma unroll
  for (int i = 0; i < PER; i++) {
    const int c = threadIdx.x + i * THREADS;
    if (c < nvec) {
      float g[8], o[8];
      unpack8<T>(wv[i], g);
#pragma unroll
      for (int e = 0; e < 8; e++) o[e] = (v[i][e] * rms) * g[e];
      if (res) {
        unpack8<T>(rv[i], g);
#pragma unroll
        for (int e = 0; e < 8; e++) o[e] += g[e];
      }
      store8v(y + row + c * 8, o);
    }
  }
}

template <typename T>
static int launch_rmsnorm_vec(const void* x, const void* w, const void* res, void* y, int rows, int hidden, float eps, cudaStream_t st) {
  const int nvec = hidden / 8;
  cudaLaunchAttribute at;
  cudaLaunchConfig_t cfg = overlapped(rows, 0, st, &at);
#define MLXR_RMS(TH, PER) do { cfg.blockDim = dim3(TH); MLXR_CUDA_TRY(cudaLaunchKernelEx(&cfg, rmsnorm_vec_kernel<T, TH, PER>, (const T*)x, (const T*)w, (const T*)res, (T*)y, nvec, eps)); } while (0)
  if (nvec <= 128) MLXR_RMS(128, 1);
  else if (nvec <= 256) MLXR_RMS(256, 1);
  else if (nvec <= 512) MLXR_RMS(256, 2);
  else if (nvec <= 1024) MLXR_RMS(256, 4);
  else MLXR_RMS(512, 4);
#undef MLXR_RMS
  count_launch();
  return MLXR_OK;
}

int launch_rmsnorm(const void* x, const void* w, const void* res, void* y, int rows, int hidden,
                   float eps, int dtype, cudaStream_t st) {
  if (rows == 0 || hidden == 0) return MLXR_OK;
  // whole 128-bit vectors and a row that 512 threads hold in registers
  if (dtype != MLXR_F32 && hidden % 8 == 0 && hidden <= 16384 && aligned16(x, w, res, y))
    return dtype == MLXR_F16 ? launch_rmsnorm_vec<__half>(x, w, res, y, rows, hidden, eps, st)
                             : launch_rmsnorm_vec<__nv_bfloat16>(x, w, res, y, rows, hidden, eps, st);
  MLXR_DISPATCH_DTYPE(dtype, T, {
    if (hidden <= 1024)
      rmsnorm_kernel<T, 128, 8><<<rows, 128, 0, st>>>((const T*)x, (const T*)w, (const T*)res,
                                                      (T*)y, hidden, eps);
    else
      rmsnorm_kernel<T, 512, 16><<<rows, 512, 0, st>>>((const T*)x, (const T*)w, (const T*)res,
                                                       (T*)y, hidden, eps);
  });
  MLXR_LAUNCH_CHECK("rmsnorm_kernel");
  return MLXR_OK;
}

// ---- swish / swiglu --------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) swiglu_kernel(const T* g,
                                                     const T* u, T* o,
                                                     size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    float s = swish_f(Act<T>::to_f(g[i]));
    if (u) s *= Act<T>::to_f(u[i]);
    o[i] = Act<T>::from_f(s);
  }
}

// The same for 16-bit types, 128-bit accesses, resident CTAs: a thread has two vectors of each operand in work and the next
// two on their way.  Bound by HBM (three streams).  With the exact division, in a grid of 3889 short CTAs, it was bound by
// issue (73 %).  rmsnorm, rope_apply of q and of k, swiglu on 1111 tokens of 4096 x 14336: 55.4 us a pass, 51.1 with this and the
// rotation's 32-bit quotients.
template <typename T, bool UP>
__global__ void __launch_bounds__(256, 4) swiglu_vec_kernel(const T* g, const T* u, T* o, size_t nvec) {
  const size_t step = (size_t)gridDim.x * 256;
  size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  uint4 a[2], b[2];
  auto load = [&](size_t at, uint4 (&x)[2], uint4 (&y)[2]) {
#pragma unroll
    for (int k = 0; k < 2; k++)
      if (at + k * step < nvec) {
        x[k] = __ldcg(reinterpret_cast<const uint4*>(g) + at + k * step);
        if constexpr (UP) y[k] = __ldcg(reinterpret_cast<const uint4*>(u) + at + k * step);
      }
  };
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  load(i, a, b);
  for (; i < nvec; i += 2 * step) {
    uint4 na[2], nb[2];
    load(i + 2 * step, na, nb);
#pragma unroll
    for (int k = 0; k < 2; k++) {
      if (i + k * step >= nvec) break;
      float x[8], y[8];
      unpack8<T>(a[k], x);
      if constexpr (UP) unpack8<T>(b[k], y);
#pragma unroll
      for (int e = 0; e < 8; e++) x[e] = UP ? swish_h(x[e]) * y[e] : swish_h(x[e]);
      store8v(o + (i + k * step) * 8, x);
    }
#pragma unroll
    for (int k = 0; k < 2; k++) { a[k] = na[k]; if constexpr (UP) b[k] = nb[k]; }
  }
}

int launch_swiglu(const void* g, const void* u, void* o, size_t n, int dtype, cudaStream_t st) {
  if (n == 0) return MLXR_OK;
  // up to 2^18 elements one element per thread is done sooner than eight one after the other (4096: 2.0 us and 2.8, 2^18: 2.6
  // and 2.9, 2^21: 7.4 and 4.6)
  if (dtype != MLXR_F32 && n % 8 == 0 && n > 1 << 18 && aligned16(g, o, u)) {
    const size_t nvec = n / 8;
    const int vb = (int)std::min<size_t>((nvec + 511) / 512, 148 * 4);
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = overlapped(vb, 256, st, &at);
#define MLXR_SWIGLU(T) do { if (u) MLXR_CUDA_TRY(cudaLaunchKernelEx(&cfg, swiglu_vec_kernel<T, true>, (const T*)g, (const T*)u, (T*)o, nvec)); \
                            else MLXR_CUDA_TRY(cudaLaunchKernelEx(&cfg, swiglu_vec_kernel<T, false>, (const T*)g, (const T*)u, (T*)o, nvec)); } while (0)
    if (dtype == MLXR_F16) MLXR_SWIGLU(__half); else MLXR_SWIGLU(__nv_bfloat16);
#undef MLXR_SWIGLU
    count_launch();
    return MLXR_OK;
  }
  size_t blocks = (n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  MLXR_DISPATCH_DTYPE(dtype, T, {
    swiglu_kernel<T><<<(int)blocks, 256, 0, st>>>((const T*)g, (const T*)u, (T*)o, n);
  });
  MLXR_LAUNCH_CHECK("swiglu_kernel");
  return MLXR_OK;
}

// ---- widening cast (partial sums of a sharded linear on the generic path) ------------------
template <typename T>
__global__ void __launch_bounds__(256) cast_f32_kernel(const T* __restrict__ x, float* __restrict__ y, size_t n) {
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) y[i] = Act<T>::to_f(x[i]);
}

template <typename T>
__global__ void __launch_bounds__(256) cast_from_f32_kernel(const float* __restrict__ x, T* __restrict__ y, size_t n) {
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) y[i] = Act<T>::from_f(x[i]);
}

int launch_cast_from_f32(const float* x, void* y, size_t n, int dtype, cudaStream_t st) {
  if (n == 0) return MLXR_OK;
  size_t blocks = (n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  MLXR_DISPATCH_DTYPE(dtype, T, { cast_from_f32_kernel<T><<<(int)blocks, 256, 0, st>>>(x, (T*)y, n); });
  MLXR_LAUNCH_CHECK("cast_from_f32_kernel");
  return MLXR_OK;
}

int launch_cast_to_f32(const void* x, float* y, size_t n, int dtype, cudaStream_t st) {
  if (n == 0) return MLXR_OK;
  size_t blocks = (n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  MLXR_DISPATCH_DTYPE(dtype, T, { cast_f32_kernel<T><<<(int)blocks, 256, 0, st>>>((const T*)x, y, n); });
  MLXR_LAUNCH_CHECK("cast_f32_kernel");
  return MLXR_OK;
}

// ---- RoPE ------------------------------------------------------------------------------
// One thread per (token, head, pair): interleaved pairs (2p, 2p+1), binary16 tables, fp32
// math, one rounding at the store (rope_apply.metal:103-172).  A token whose position
// falls outside the table is left untouched and flagged in *status.
template <typename T>
__global__ void __launch_bounds__(256) rope_kernel(const T* x,
                                                   const __half* __restrict__ cos_t,
                                                   const __half* __restrict__ sin_t,
                                                   const int32_t* __restrict__ positions,
                                                   T* y, size_t tokens, int heads,
                                                   int pairs, int max_seq, int linear,
                                                   float scale, int offset, int* status) {
  const size_t total = tokens * heads * pairs;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const int p = (int)(i % pairs);
    const size_t th = i / pairs;  // token * heads + head
    const size_t tok = th / heads;
    const long long pos = (long long)positions[tok] + offset;
    if (pos < 0 || pos >= max_seq) {
      if (status) atomicExch_system(status, 1);
      continue;
    }
    const float c = __half2float(cos_t[(size_t)pos * pairs + p]);
    const float s = __half2float(sin_t[(size_t)pos * pairs + p]);
    const size_t e = th * (size_t)(2 * pairs) + 2 * p;
    const float xe = Act<T>::to_f(x[e]), xo = Act<T>::to_f(x[e + 1]);
    float ye = __fsub_rn(__fmul_rn(xe, c), __fmul_rn(xo, s));
    float yo = __fadd_rn(__fmul_rn(xo, c), __fmul_rn(xe, s));
    if (linear) { ye *= scale; yo *= scale; }
    y[e] = Act<T>::from_f(ye);
    y[e + 1] = Act<T>::from_f(yo);
  }
}

// Quotients of n < 2^31 by a divisor known to the host (Granlund and Montgomery, "Division by invariant integers using
// multiplication", 1994): a 64-bit division of the vector's number took more instructions than its rotation.
struct Divisor {
  uint32_t d, mul, shift;
  explicit Divisor(uint32_t d_) : d(d_), shift(0) {
    while ((1ull << shift) < d) shift++;
    mul = (uint32_t)((((1ull << 32) * ((1ull << shift) - d)) / d) + 1);
  }
  __device__ __forceinline__ uint32_t quot(uint32_t n) const { return (__umulhi(n, mul) + n) >> shift; }
};

// The same for 16-bit types and heads of a multiple of 8 elements: 128-bit accesses to x and y, 64-bit to the tables.  A thread
// rotates the same four pairs of HP heads of a token: the quotients, the position and the table values are found once for all of them, and
// HP loads of x are in flight (32 heads of 1111 tokens: a thread per four pairs of one head spent half its instructions on finding them).
//
// Two tensors that share the positions (q and k of a layer) can go in one launch: units from `total` on are z's,
// up to total_z.
//
// A checked call waits for the answer on the host.  The last CTA to finish writes it straight to pinned memory (1: done, 2: done, with
// a position outside the table), where the host sees it some 5 us before cudaStreamSynchronize would return; when it is there
// every CTA has done its last access, and all results are visible (each CTA's barrier and fence before it is counted, the last one's fence
// for the system before the answer).
struct RopeArgs {
  const __half *cos_t, *sin_t;
  const int32_t* positions;
  size_t total, total_z;
  Divisor per, per_z, per_head;          // units of a token of x, of z, of a group of heads
  int heads, heads_z;
  int max_seq, linear;
  float scale;
  int offset;
  int* status;                           // unchecked: flag for positions outside the table, or null
  unsigned* count;                       // checked: CTAs finished (+ 2^16 for each that met such a position); the last one clears it
  volatile int* answer;
};
template <typename T, int HP, bool WIDE>          // WIDE: 2^31 units and more
__global__ void __launch_bounds__(256) rope_vec_kernel(const T* x, T* y, T* z, const RopeArgs A) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  using Index = typename std::conditional<WIDE, size_t, uint32_t>::type;
  const Index total = (Index)A.total, all = (Index)(A.total + A.total_z);
  bool outside = false;
  for (size_t j0 = (size_t)blockIdx.x * 256 + threadIdx.x; j0 < all; j0 += (size_t)gridDim.x * 256) {
    const Index j = (Index)j0;
    const bool first = j < total;
    const Index i = first ? j : j - total;
    const Divisor& per = first ? A.per : A.per_z;
    const T* src = first ? x : z;
    T* dst = first ? y : z;
    const int heads = first ? A.heads : A.heads_z;
    Index tok;
    if constexpr (WIDE) tok = i / per.d; else tok = per.quot(i);
    uint32_t c = (uint32_t)(i - tok * per.d);
    const uint32_t h = A.per_head.quot(c), vh = A.per_head.d;
    c -= h * vh;
    const int have = min(HP, heads - (int)h * HP);
    const size_t v0 = ((size_t)tok * heads + h * HP) * vh + c;
    uint4 xv[HP];
#pragma unroll
    for (int k = 0; k < HP; k++) if (k < have) xv[k] = __ldcg(reinterpret_cast<const uint4*>(src) + v0 + k * vh);
    const long long pos = (long long)__ldcg(A.positions + tok) + A.offset;
    if (pos < 0 || pos >= A.max_seq) {
      outside = true;
      continue;
    }
    const uint2 cv = __ldg(reinterpret_cast<const uint2*>(A.cos_t) + (size_t)pos * vh + c);
    const uint2 sv = __ldg(reinterpret_cast<const uint2*>(A.sin_t) + (size_t)pos * vh + c);
    const __half *hc = reinterpret_cast<const __half*>(&cv), *hs = reinterpret_cast<const __half*>(&sv);
    float cs[4], sn[4];
#pragma unroll
    for (int p = 0; p < 4; p++) { cs[p] = __half2float(hc[p]); sn[p] = __half2float(hs[p]); }
#pragma unroll
    for (int k = 0; k < HP; k++) {
      if (k >= have) break;
      const T* hx = reinterpret_cast<const T*>(&xv[k]);
      float o[8];
#pragma unroll
      for (int p = 0; p < 4; p++) {
        const float xe = Act<T>::to_f(hx[2 * p]), xo = Act<T>::to_f(hx[2 * p + 1]);
        o[2 * p] = __fsub_rn(__fmul_rn(xe, cs[p]), __fmul_rn(xo, sn[p]));
        o[2 * p + 1] = __fadd_rn(__fmul_rn(xo, cs[p]), __fmul_rn(xe, sn[p]));
        if (A.linear) { o[2 * p] *= A.scale; o[2 * p + 1] *= A.scale; }
      }
      store8v(dst + (v0 + k * vh) * 8, o);
    }
  }
  if (!A.answer) {
    if (outside && A.status) atomicExch_system(A.status, 1);
    return;
  }
  const bool any = __syncthreads_or(outside);
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned mine = 1u + (any ? 1u << 16 : 0u), sum = atomicAdd(A.count, mine) + mine;
    if ((sum & 0xFFFFu) == gridDim.x) {
      *A.count = 0u;
      __threadfence_system();
      *A.answer = sum >> 16 ? 2 : 1;
    }
  }
}

// word: checked ? where the answer goes, with ctl a zeroed word of device memory : flag for positions outside the table
template <typename T>
static int launch_rope_vec(const void* x, const uint16_t* cos_t, const uint16_t* sin_t, const int32_t* positions, void* y, size_t tokens, int heads,
                           void* z, int heads_z, int head_dim, int max_seq, int linear, float scale, int offset, int* word, uint32_t* ctl, cudaStream_t st) {
  const int vh = head_dim / 8;
  const size_t vectors = tokens * ((size_t)heads + heads_z) * vh;
  // four heads a thread as long as that leaves three CTAs per SM, or two (8 heads of 1111 tokens: one)
  const int hp = vectors >= (size_t)148 * 3 * 256 * 4 ? 4 : vectors >= (size_t)148 * 3 * 256 * 2 ? 2 : 1;
  const int gx = (heads + hp - 1) / hp, gz = (heads_z + hp - 1) / hp;
  const RopeArgs A = {(const __half*)cos_t, (const __half*)sin_t, positions, tokens * gx * vh, tokens * gz * vh,
                      Divisor((uint32_t)gx * vh), Divisor((uint32_t)std::max(1, gz * vh)), Divisor((uint32_t)vh), heads, heads_z, max_seq, linear, scale, offset,
                      ctl ? nullptr : word, ctl, ctl ? word : nullptr};
  const size_t all = A.total + A.total_z;
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = overlapped((int)std::min<size_t>((all + 255) / 256, 148 * 8 * 4), 256, st, &at);
  auto launch = [&](auto kern) { return cudaLaunchKernelEx(&cfg, kern, (const T*)x, (T*)y, (T*)z, A); };
  if (all >> 31) MLXR_CUDA_TRY(launch(rope_vec_kernel<T, 4, true>));
  else MLXR_CUDA_TRY(launch(hp == 4 ? rope_vec_kernel<T, 4, false> : hp == 2 ? rope_vec_kernel<T, 2, false> : rope_vec_kernel<T, 1, false>));
  count_launch();
  return MLXR_OK;
}
static bool rope_vec_ok(const void* x, const void* y, const uint16_t* cos_t, const uint16_t* sin_t, int head_dim, int dtype) {
  return dtype != MLXR_F32 && head_dim % 8 == 0 && aligned16(x, y) && (((uintptr_t)cos_t | (uintptr_t)sin_t) & 7u) == 0;
}
bool rope_qk_supported(const void* q, const void* k, const uint16_t* cos_t, const uint16_t* sin_t, int head_dim, int dtype) {
  return rope_vec_ok(q, k, cos_t, sin_t, head_dim, dtype);
}
int launch_rope_qk(void* q, void* k, const uint16_t* cos_t, const uint16_t* sin_t, const int32_t* positions, size_t tokens, int q_heads, int kv_heads,
                   int head_dim, int max_seq, int offset, int dtype, int* status, cudaStream_t st) {
  return dtype == MLXR_F16 ? launch_rope_vec<__half>(q, cos_t, sin_t, positions, q, tokens, q_heads, k, kv_heads, head_dim, max_seq, 0, 1.0f, offset, status, nullptr, st)
                           : launch_rope_vec<__nv_bfloat16>(q, cos_t, sin_t, positions, q, tokens, q_heads, k, kv_heads, head_dim, max_seq, 0, 1.0f, offset, status, nullptr, st);
}

int launch_rope(const void* x, const uint16_t* cos_t, const uint16_t* sin_t,
                const int32_t* positions, void* y, size_t tokens, int heads, int head_dim,
                int max_seq, int mode, float scale, int offset, int dtype, int* status,
                uint32_t* ctl, bool* answers, cudaStream_t st) {
  const size_t total = tokens * heads * (head_dim / 2);
  if (answers) *answers = false;
  if (total == 0) return MLXR_OK;
  if (rope_vec_ok(x, y, cos_t, sin_t, head_dim, dtype)) {
    if (answers) *answers = true; else ctl = nullptr;
    return dtype == MLXR_F16 ? launch_rope_vec<__half>(x, cos_t, sin_t, positions, y, tokens, heads, nullptr, 0, head_dim, max_seq, mode == MLXR_ROPE_LINEAR, scale, offset, status, ctl, st)
                             : launch_rope_vec<__nv_bfloat16>(x, cos_t, sin_t, positions, y, tokens, heads, nullptr, 0, head_dim, max_seq, mode == MLXR_ROPE_LINEAR, scale, offset, status, ctl, st);
  }
  size_t blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  MLXR_DISPATCH_DTYPE(dtype, T, {
    rope_kernel<T><<<(int)blocks, 256, 0, st>>>(
        (const T*)x, (const __half*)cos_t, (const __half*)sin_t, positions, (T*)y, tokens, heads,
        head_dim / 2, max_seq, mode == MLXR_ROPE_LINEAR, scale, offset, status);
  });
  MLXR_LAUNCH_CHECK("rope_kernel");
  return MLXR_OK;
}

// ---- RoPE, split-half convention --------------------------------------------------------
// graph::RotaryEmbedding::forward (core/graph/layers.cpp:157-225): the head is split in two
// halves (x1 = first d/2 elements, x2 = the rest), positions are the contiguous range
// offset .. offset + seq, tables are float32 [max_seq, d/2]:
//   y1 = x1 * cos - x2 * sin,  y2 = x2 * cos + x1 * sin
// as four products and two sums, each rounded to float32 (the composition materialises every
// product as an array); one rounding to T at the store.  One thread per (token, head, p).
template <typename T>
__global__ void __launch_bounds__(256) rope_split_half_kernel(const T* __restrict__ x, const float* __restrict__ cos_t,
                                                              const float* __restrict__ sin_t, T* __restrict__ y,
                                                              size_t batch, int seq, int heads, int half, int offset) {
  const size_t total = batch * seq * heads * half;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int p = (int)(i % half);
    const size_t th = i / half;            // (batch * seq + t) * heads + head
    const int t = (int)((th / heads) % seq);
    const size_t tab = (size_t)(offset + t) * half + p;
    const float c = cos_t[tab], sn = sin_t[tab];
    const size_t e = th * (size_t)(2 * half) + p;
    const float x1 = Act<T>::to_f(x[e]), x2 = Act<T>::to_f(x[e + half]);
    y[e] = Act<T>::from_f(__fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, sn)));
    y[e + half] = Act<T>::from_f(__fadd_rn(__fmul_rn(x2, c), __fmul_rn(x1, sn)));
  }
}

int launch_rope_split_half(const void* x, const float* cos_t, const float* sin_t, void* y, size_t batch, int seq,
                           int heads, int head_dim, int offset, int dtype, cudaStream_t st) {
  const size_t total = batch * seq * heads * (head_dim / 2);
  if (total == 0) return MLXR_OK;
  size_t blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  MLXR_DISPATCH_DTYPE(dtype, T, {
    rope_split_half_kernel<T><<<(int)blocks, 256, 0, st>>>((const T*)x, cos_t, sin_t, (T*)y, batch, seq, heads,
                                                           head_dim / 2, offset);
  });
  MLXR_LAUNCH_CHECK("rope_split_half_kernel");
  return MLXR_OK;
}

}  // namespace mlxr
