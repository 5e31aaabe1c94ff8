// Host-side launchers of the CUDA kernels (one per .cu file) and shared constants.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>

namespace mlxr {

// Zero-initialised 32-bit words per workspace for counters and barriers.
constexpr int kSyncWords = 4096;
constexpr int kTileCounters = 16;      // the first of the words that count the parts of shared output tiles

int launch_dequantize(const void* w, void* out, int N, int K, int qt, int out_dtype, int flags,
                      cudaStream_t st);
int launch_repack_ggml_q4_0(const void* src, void* dst, size_t nblocks, cudaStream_t st);
int launch_qgemm_generic(const void* x, const void* w, const void* bias, void* y, int M, int N,
                         int K, int qt, int dtype, cudaStream_t st);
bool gemv_rows_supported(int qt, int M, int K, const void* x, const void* w);
int launch_gemv_rows(const void* x, const void* w, const void* bias, void* y, int M, int N, int K, int qt, int dtype,
                     cudaStream_t st);
int launch_linear_dense(const void* x, const void* w, const void* bias, void* y, int M, int N, int K,
                        int dtype, cudaStream_t st);
int launch_rmsnorm(const void* x, const void* w, const void* res, void* y, int rows, int hidden,
                   float eps, int dtype, cudaStream_t st);
// device status word of the (device, stream) workspace: kernels record time-outs there
int stream_status_word(cudaStream_t st, int** status);
int launch_cast_from_f32(const float* x, void* y, size_t n, int dtype, cudaStream_t st);
int launch_cast_to_f32(const void* x, float* y, size_t n, int dtype, cudaStream_t st);
int launch_swiglu(const void* g, const void* u, void* o, size_t n, int dtype, cudaStream_t st);
// answers (checked calls): set if the kernel will write 1 (done) or 2 (done, a position outside the table) to *status, pinned host memory, when it
// is done with all its accesses, counting its CTAs in ctl, a zeroed word of device memory; else, and without it, *status becomes 1 for such a position
int launch_rope(const void* x, const uint16_t* cos_t, const uint16_t* sin_t,
                const int32_t* positions, void* y, size_t tokens, int heads, int head_dim,
                int max_seq, int mode, float scale, int offset, int dtype, int* status,
                uint32_t* ctl, bool* answers, cudaStream_t st);

// rope_apply on q and k [tokens, heads, head_dim] in place, one launch; false if their layout needs launch_rope
bool rope_qk_supported(const void* q, const void* k, const uint16_t* cos_t, const uint16_t* sin_t, int head_dim, int dtype);
int launch_rope_qk(void* q, void* k, const uint16_t* cos_t, const uint16_t* sin_t, const int32_t* positions, size_t tokens, int q_heads, int kv_heads,
                   int head_dim, int max_seq, int offset, int dtype, int* status, cudaStream_t st);
int launch_rope_split_half(const void* x, const float* cos_t, const float* sin_t, void* y, size_t batch, int seq,
                           int heads, int head_dim, int offset, int dtype, cudaStream_t st);

// ---- exchange buffer of the tensor-parallel block (tp.cu, decode_kernel.cuh) -------------------
// One per rank, mapped by every peer:
// [flags: kTpMaxWorld x kTpFlagsPerRank uint32][pad to kTpFlagBytes][slots: 2 parities x kTpMaxWorld x kTpSlotElems float]
constexpr int kTpMaxWorld = 8;
constexpr int kTpFlagsPerRank = 1024;              // indexed by CTA (exchange kernel) or by output tile (fused decode)
constexpr size_t kTpSlotElems = 256 * 1024;        // = MLXR_TP_PEER_MAX_ELEMS
constexpr size_t kTpFlagBytes = 64 * 1024;
constexpr size_t kTpXchgBytes = kTpFlagBytes + 2 * kTpMaxWorld * kTpSlotElems * sizeof(float);
// What the decode kernel needs to push its partial sums to the peers and reduce: every rank's
// exchange buffer as mapped in this process, this rank, the world size, the sequence words
// ([0] sequence number, [1] CTAs finished) and the final output [M, hidden] of the activation dtype.
struct DecodeTp {
  char* peer[kTpMaxWorld];
  int rank, world;
  uint32_t* ctl;
  void* y;
};

// ---- persistent decode kernel (decode.cu) ---------------------------------------------------
// One linear (or up to three stacked along N, or gate/up interleaved) of a decode phase.
struct DecodeLinear {
  const void* w[3];
  int rows[3];
  int nmat;
  int interleave;          // gate/up in 8+8 row tiles with the SiLU(gate)*up epilogue
  int K;
  const void* x;           // [M, K]
  const void* gamma;       // RMSNorm weight or null
  float eps;
  // launch_gemv, 4-bit formats: the normalised activations are rounded to the activation type before they are
  // multiplied, as the composition of RMSNorm and a linear rounds them (Q8_0 and launch_decode always round)
  int round_n;
  void* y[3];
  const void* bias[3];
  int epi[3];              // 0 plain, 2 RoPE, 3 plain fp32 store (y is float*)
  const uint16_t* cos_t;
  const uint16_t* sin_t;
  const int32_t* positions;
  int head_dim, max_seq, pos_offset;
  // Hand-over between two chained phases (gate/up -> down) without a grid barrier: the first
  // phase's SiLU(gate)*up epilogue writes 8-byte words {payload, launch sequence number} to
  // y_tagged ([M][rows / per_word] words; per_word = 2 for 16-bit activations, 1 for float), the
  // second phase has x pointing at the same words and x_tagged = 1.
  void* y_tagged;
  int x_tagged;
};
// Bytes of the tagged hand-over buffer for h [M, inter].
inline size_t decode_tagged_bytes(int M, int inter, int dtype) { return (size_t)M * inter * (dtype == MLXR_F32 ? 8 : 4); }
// Limit of every device-side wait (mbarrier, hand-over words, peer flags), in nanoseconds.
void set_wait_limit_ns(unsigned long long ns);
unsigned long long wait_limit_ns();
// Environment probes for tuning exist only in builds with -DMLXR_TUNING.
#ifdef MLXR_TUNING
inline const char* tune_env(const char* name) { return getenv(name); }
#else
inline const char* tune_env(const char*) { return nullptr; }
#endif
constexpr size_t kDecodeScratchBytes = (size_t)8 << 20;  // split-K partial sums
void set_decode_trace(void* dev_ptr);
void* get_decode_trace();
void set_decode_launch_mode(int mode);
bool overlap_launches();                 // launches may start under the previous kernel of the stream (MLXR_DECODE_LAUNCH_OVERLAPPED)
bool decode_supported(int qt, int M, int K, const void* const* w, int nmat);
// tp (optional): the last phase must be a single plain linear with epi 3 (float partial sums); its
// sums then go straight into the peers' exchange buffers and the kernel ends with the reduction.
int launch_decode(const DecodeLinear* lin, int nphases, int M, int qt, int dtype, void* scratch,
                  size_t scratch_bytes, uint32_t* sync, uint32_t* bar_host, int* status, cudaStream_t st,
                  const DecodeTp* tp = nullptr);
// The tensor-parallel block in one launch when the decode kernel takes the shapes (else MLXR_ERR_UNSUPPORTED
// and nothing is launched): inter_local is this rank's share of the intermediate size.
int mlp_block_tp_fused(const void* x, const void* norm_weight, const void* w_gate, const void* w_up, const void* w_down,
                       int M, int hidden, int inter_local, int qt, float eps, int dtype, const DecodeTp* tp,
                       cudaStream_t st);

// ---- linears for one or two tokens (gemv.cu): Q4_K, Q4_0, and Q8_0 with 16-bit activations ------------------
// One launch per linear (or per stacked / interleaved group of linears); takes the DecodeLinear description
// (no tagged hand-over: chained linears are separate launches).  rows: weight rows in all.
bool gemv_supported(int qt, int M, int K, int rows, int dtype, const void* const* w, int nmat);
int launch_gemv(const DecodeLinear& L, int M, int qt, int dtype, int* status, cudaStream_t st);

// Q4_K, one and two tokens, small matrices (stream_gemv.cu): single or stacked linears
bool stream_gemv_supported(int qt, int M, int K, int rows, const void* const* w, int nmat);
int launch_stream_gemv(const DecodeLinear& L, int M, int dtype, int* status, cudaStream_t st);

// ---- up to eight tokens of 16-bit activations (gemv_tokens.cu): canonical Q4_K from one token on, Q8_0, Q4_K, Q4_0 from three ----
// rows: weight rows in all.  w[0 .. nmat): one matrix, gate and up (y[0] = SiLU(X gate^T) * (X up^T), rows[0] columns), or stacked
enum TokensForm { kTokensPlain = 0, kTokensGateUp = 1, kTokensStacked = 2 };
bool gemv_tokens_faster(int qt, int M, int K, int rows, int form, int dtype);       // the part of the rule that is about time
bool gemv_tokens_supported(int qt, int M, int K, int rows, int form, int dtype, const void* x, const void* const* w, int nmat);
int launch_gemv_tokens(const void* x, const void* const* w, const int* rows, int nmat, int form, const void* bias, void* const* y, int M, int K, int qt, int dtype,
                       int* status, cudaStream_t st);

// ---- small-batch tensor-core linear (smallm.cu): Q4_K, Q4_0, Q8_0, NF4, canonical Q4_K; 1 <= M <= 64, fp16 / bf16 ----
bool smallm_supported(int qt, int M, int N, int K, int dtype, const void* x, const void* w);
void smallm_partition(long long units, int ctas, int cta, long long unit, long long* begin, long long* end, int* owner);
// grid size, the most CTAs that share one output tile, and the bytes of fp32 partial sums needed;
// rows = weight rows streamed (N, or 2 N for the gate/up form)
int smallm_plan(int qt, bool stacked, int M, int rows, int K, int* grid, int* maxc, size_t* partial_bytes);
// nmat stacked matrices y[i] [M, rows[i]] = X w[i]^T (+ bias, one matrix only), or swiglu: w[0] = gate, w[1] = up
int launch_smallm(const void* x, const void* const* w, const int* rows, int nmat, bool swiglu, const void* bias, void* const* y, int M, int K, int qt, int dtype,
                  int* status, float* partials, uint32_t* counters, int grid, int maxc, cudaStream_t st);

// ---- the same form for more tokens (widem.cu): Q4_K, Q4_0, Q8_0, NF4, fp16 / bf16 ---------------------
struct WidePlan {
  int nt, ntt, ntiles;     // tokens per tile, token tiles, tiles in all
  int grid, whole;         // CTAs; 1: whole tiles per pair, 0: ranges of work units
  size_t partial_bytes;    // fp32 partial sums needed
  double cost_us;          // the plan's own estimate
};
bool widem_supported(int qt, int M, int N, int K, int dtype, const void* x, const void* w);
int widem_plan(int qt, int dtype, int M, int rows, int K, WidePlan* out);     // rows = weight rows streamed (N, or 2 N for the gate/up form)
int launch_widem(const void* x, const void* w, const void* w2, const void* bias, void* y, int M, int N, int K, int qt, int dtype,
                 int* status, float* partials, uint32_t* counters, const WidePlan& plan, cudaStream_t st);

// ---- many tokens (dense.cu): 16-bit weights once, then a dense GEMM; Q4_K, Q4_0, Q8_0, NF4, fp16 / bf16 ---
struct DensePlan {
  int nt, slice;           // weight rows per tile; rows of the 16-bit buffer filled at a time
  size_t bytes;            // scratch for the 16-bit weights
  double cost_us;
};
bool dense_supported(int qt, int M, int N, int K, int dtype, const void* x, const void* w);
int dense_plan(int M, int rows, int K, DensePlan* out);
int launch_dense(const void* x, const void* w, const void* w2, const void* bias, void* y, int M, int N, int K, int qt, int dtype,
                 int* status, void* buf, const DensePlan& plan, cudaStream_t st);

}  // namespace mlxr
