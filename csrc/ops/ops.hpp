// Host entry points of the model-operator kernels (sm_100a).  All launchers
// enqueue on the given stream and return the launch status.  The reference has
// no counterpart for these: its models run on stock PyTorch/MPS operators
// (examples/ddp_utils.py:41-147); they exist here because the headline
// benchmark is a training step, and on a B200 that step is bound by these
// operators, not by the collectives.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

namespace mccl {
namespace ops {

// Number of operator kernels launched so far (all launchers below count).
uint64_t launch_count();
void count_launch(int n = 1);

// ---- normalisation: y = (x - mean) * rstd * w + b  (LayerNorm, bias != null)
//                     y = x * rstd * w                (RMSNorm, bias == null)
// x, y: [rows, dim] bf16; w, b: fp32; mean / rstd: fp32 [rows] saved for backward (both may be null).
cudaError_t norm_fwd(const __nv_bfloat16* x, const float* w, const float* b, __nv_bfloat16* y, float* mean, float* rstd,
                     int rows, int dim, float eps, cudaStream_t stream);
// x = bf16(sum + bias + residual) and y = norm(x), for a product left in `parts` parts of fp32 [rows, dim], `stride` elements apart and added
// in order; bias may be null; dim up to 2048.
cudaError_t norm_sum_fwd(const float* sum, int parts, long long stride, const float* bias, const __nv_bfloat16* residual, __nv_bfloat16* x, const float* w, const float* b, __nv_bfloat16* y,
                         int rows, int dim, float eps, cudaStream_t stream);
// dx: [rows, dim] bf16; dw, db: fp32 [dim].  With scratch (fp32, 2 * colsum_slabs(rows) * dim
// elements) dw / db are overwritten by a two-stage, order-fixed reduction; with scratch == nullptr
// the slab sums are added to dw / db atomically in one pass.  dx_add (optional, [rows, dim] bf16) is a
// second gradient of x (a residual path) that is added to dx before the one rounding to bf16.
cudaError_t norm_bwd(const __nv_bfloat16* dy, const __nv_bfloat16* x, const float* w, const float* mean, const float* rstd,
                     __nv_bfloat16* dx, float* dw, float* db, float* scratch, int rows, int dim, bool layernorm,
                     cudaStream_t stream, const __nv_bfloat16* dx_add = nullptr, int parts = 3);
// The same backward in one pass: dw, db (LayerNorm) and, where given, the column sums of dx_add and of dx are ADDED into fp32
// [dim] buffers.  dim <= 1024, or 2048 for RMSNorm without column sums; cudaErrorNotSupported otherwise.
// With in_order each of the four (those given) is a block [norm_bwd_parts(rows, dim), dim] instead, written and not added into, for sum_parts.
cudaError_t norm_bwd_fused(const __nv_bfloat16* dy, const __nv_bfloat16* x, const float* w, const float* mean, const float* rstd,
                           __nv_bfloat16* dx, const __nv_bfloat16* dx_add, float* dw, float* db, float* sum_add, float* sum_dx, int rows,
                           int dim, bool layernorm, cudaStream_t stream, bool in_order = false);
int norm_bwd_parts(int rows, int dim);
// Sums whose parts a kernel left in rows: out[c] = in[0, c] + in[1, c] + ... in an order that depends on sizes alone.
struct PartSum {
  const float* in;   // [rows, cols]
  float* out;        // [cols]
  int rows, cols;
};
constexpr int kPartSums = 8;
struct PartSums {
  PartSum s[kPartSums];
  int first[kPartSums + 1];   // first group of 32 columns of each
  int count;
  cudaError_t set(const PartSum* sums, int n);
};
cudaError_t sum_parts(const PartSum* sums, int count, cudaStream_t stream);
// out[c] = sum over rows of in[r, c] (bias gradients).  scratch: colsum_slabs(rows) * dim floats,
// or nullptr to add into out atomically in one pass.
cudaError_t colsum_bf16(const __nv_bfloat16* in, float* out, float* scratch, int rows, int dim, cudaStream_t stream);
int colsum_slabs(int rows);

// ---- fused AdamW over flat fp32 buffers; step is a device scalar (float) so the
// launch can be replayed from a CUDA graph.  p16 (optional) receives bf16(p).  With zero_grad the gradient
// is cleared in the same pass (it has just been read), which replaces the memset at the start of the next step.
cudaError_t adamw_flat(float* p, float* g, float* m, float* v, __nv_bfloat16* p16, long long n, float lr, float beta1,
                       float beta2, float eps, float wd, const float* step, float grad_scale, cudaStream_t stream,
                       bool zero_grad = false, int ctas_per_sm = 8);

// ---- softmax cross entropy, forward and backward in one pass over the logits:
// loss_rows[t] = logsumexp(logits[t]) - logits[t, target[t]];
// logits[t] is overwritten by (softmax - onehot) * grad_scale.
cudaError_t cross_entropy_fwd_bwd(__nv_bfloat16* logits, const long long* targets, float* loss_rows, int rows, int vocab,
                                  float grad_scale, cudaStream_t stream);

// out = mean of n fp32 values, always added in the same order.
cudaError_t mean_f32(const float* in, float* out, long long n, cudaStream_t stream);

// ---- out[c, r] = in[r, c] for a bf16 matrix [rows, cols].
cudaError_t transpose_bf16(const __nv_bfloat16* in, __nv_bfloat16* out, int rows, int cols, cudaStream_t stream);
// fp32 → bf16 cast of n elements.
cudaError_t cast_f32_bf16(const float* in, __nv_bfloat16* out, long long n, cudaStream_t stream);
// out = bf16(alpha * (part 0 + part 1 + ...)) over n elements; the parts are `stride` elements apart; alpha: device scalar (null: one).
cudaError_t sum_slabs_bf16(const float* in, int parts, long long stride, __nv_bfloat16* out, long long n, const float* alpha, cudaStream_t stream);
// The same for `count` tensors, tensor i into out[dst_offset[i], ...); 16-byte aligned sources and places.
cudaError_t cast_many(const float* const* src, const long long* numel, const long long* dst_offset, int count, __nv_bfloat16* out,
                      cudaStream_t stream);
// GELU backward on a pre-activation: dz = dy * gelu'(z).
cudaError_t gelu_bwd(const __nv_bfloat16* dy, const __nv_bfloat16* z, __nv_bfloat16* dz, long long n, cudaStream_t stream);

// ---- token (+ learned position) embedding.  y[t, :] = bf16(tok[ids[t], :] + pos[t % seq, :]);
// tok / pos are fp32 [vocab, dim] / [>= seq, dim] (pos may be null); dim % 8 == 0.
cudaError_t embed_fwd(const long long* ids, const float* tok, const float* pos, __nv_bfloat16* y, int tokens, int seq, int dim,
                      int vocab, cudaStream_t stream);
// Adds dy[t, :] into dtok[ids[t], :] and dpos[t % seq, :] (fp32, atomically; dpos may be null).
cudaError_t embed_bwd(const long long* ids, const __nv_bfloat16* dy, float* dtok, float* dpos, int tokens, int seq, int dim,
                      int vocab, cudaStream_t stream, float scale = 1.f);

// ---- causal self-attention straight from the fused QKV projection.
// qkv: [B, S, 3, H, hd] bf16; o: [B, S, H, hd]; lse: [B, H, S] fp32 (log2 domain, saved for backward).
// Both ways: S <= 256 and hd <= 64 (a multiple of 8).
// cudaErrorNotSupported otherwise: the caller falls back.
bool attention_supported(int S, int hd);
cudaError_t attention_fwd(const __nv_bfloat16* qkv, __nv_bfloat16* o, float* lse, int B, int S, int H, int hd, float softmax_scale,
                          cudaStream_t stream);
// dqkv: [B, S, 3, H, hd] bf16, every element written.  colsum (optional, fp32 [3 * H * hd]): its column sums are added here, or with in_order
// written to a block [attention_bwd_parts(B, S), 3 * H * hd] for sum_parts.
cudaError_t attention_bwd(const __nv_bfloat16* qkv, const __nv_bfloat16* o, const __nv_bfloat16* d_o, const float* lse,
                          __nv_bfloat16* dqkv, float* colsum, int B, int S, int H, int hd, float softmax_scale, cudaStream_t stream,
                          bool in_order = false);
int attention_bwd_parts(int B, int S);

// ---- rotary embedding of the fused QKV projection's output (pairs of even and odd elements; cos / sin: fp32
// [>= seq, head_dim / 2]; token t has position t % seq).  qkv [tokens, 3, H, hd] -> qk [tokens, 2, H, hd].
cudaError_t rope_qk_fwd(const __nv_bfloat16* qkv, const float* cos_t, const float* sin_t, __nv_bfloat16* qk, long long tokens, int seq,
                        int heads, int head_dim, cudaStream_t stream);
// A gradient [batch, head, position, head_dim] with contiguous head_dim and these strides (elements, multiples of 8).
struct StridedGrad {
  const __nv_bfloat16* p;
  long long sb, sh, ss;
};
// d: gradients of the rotated q, the rotated k, and v -> dqkv [tokens, 3, H, hd], every element written.
cudaError_t rope_qkv_bwd(const StridedGrad (&d)[3], const float* cos_t, const float* sin_t, __nv_bfloat16* dqkv, long long tokens, int seq,
                         int heads, int head_dim, cudaStream_t stream);
// ---- SwiGLU on the fused projection [rows, 2 f] = [gate | up]: h = silu(gate) * up, and the gradient of [gate | up].
cudaError_t swiglu_fwd(const __nv_bfloat16* gu, __nv_bfloat16* h, long long rows, int f, cudaStream_t stream);
cudaError_t swiglu_bwd(const __nv_bfloat16* dh, const __nv_bfloat16* gu, __nv_bfloat16* dgu, long long rows, int f, cudaStream_t stream);

// ---- tcgen05 GEMM: D[M,N] = A[M,K] · B[N,K]^T (+ bias[N]) (GELU) ; A, B bf16 with K contiguous.
enum GemmEpilogue : int {
  EPI_NONE = 0,       // D = acc
  EPI_BIAS = 1,       // D = acc + bias[n]
  EPI_BIAS_GELU = 2,  // Z = acc + bias[n] (written to aux), D = gelu(Z)
  EPI_GELU = 3,       // Z = acc (written to aux), D = gelu(Z)
  EPI_BIAS_GELU_D = 4,  // Z = acc + bias[n], D = gelu(Z), aux = gelu'(Z): backward then only multiplies (see GemmArgs::mul)
  EPI_GELU_D = 5,       // the same without bias
};
struct GemmArgs {
  const __nv_bfloat16* a = nullptr;  // [M, K], row stride lda (elements); a_mn_major: stored [K, M]
  const __nv_bfloat16* b = nullptr;  // [N, K], row stride ldb;            b_mn_major: stored [K, N]
  bool a_mn_major = false;
  bool b_mn_major = false;
  void* d = nullptr;                 // [M, N] bf16 or fp32, row stride ldd
  __nv_bfloat16* aux = nullptr;      // [M, N] second output of GELU epilogues (may be null: not written)
  const float* bias = nullptr;       // [N]
  const __nv_bfloat16* residual = nullptr;  // [M, N] added after bias / activation, row stride ldd
  const __nv_bfloat16* mul = nullptr;       // [M, N]: D = acc * mul (e.g. the saved gelu'(z): the input gradient through a GELU), row stride ldd
  float* colsum = nullptr;                  // [N] fp32: column sums of D are added here (bf16 output without bias or residual, B MN-major)
  bool colsum_in_order = false;             // colsum is [ceil(M / 32), N] instead: the sums of 32 rows each, written, for sum_parts
  int m = 0, n = 0, k = 0;
  int lda = 0, ldb = 0, ldd = 0;
  bool d_fp32 = false;
  bool accumulate = false;           // D += result (fp32 output only)
  const float* alpha = nullptr;      // device scalar: the product is multiplied by it.  A weight gradient (fp32, both operands MN-major) or an input
                                     // gradient (bf16, MN-major B) without bias, activation, residual, multiplier or column sums
  int epilogue = EPI_NONE;
};
// Returns cudaErrorNotSupported for shapes the kernel does not cover
// (N % 8 != 0, unaligned pointers or row strides); the caller falls back.
cudaError_t gemm_bf16_tn(const GemmArgs& args, cudaStream_t stream);
// d[M, N] = silu(gate) * up of [gate | up] = A · B^T, B [2 N, K]; `aux` [M, 2 N] (may be null) takes [gate | up] itself.  N % 32 == 0.
// cudaErrorNotSupported also where a product and swiglu_fwd are the better choice.
cudaError_t gemm_swiglu(const GemmArgs& args, cudaStream_t stream);
// d[M, 2 N] = gradient of [gate | up] (`aux`, [M, 2 N]) for dh = A · B, B [K, N] (b_mn_major, rows ldb): swiglu_bwd on a product's way out.
cudaError_t gemm_swiglu_grad(const GemmArgs& args, cudaStream_t stream);
// Up to any number of weight gradients dW[N, K] = dY[tokens, N]^T · X[tokens, K] over the same tokens, worked through together
// (sixteen products per launch).  A product is a GemmArgs with both operands MN-major, fp32 output, no epilogue; all of them
// accumulate, or none.
// `sums` (up to kPartSums, of kernels before this one) are finished by the first launch beside its products, see sum_parts.
cudaError_t gemm_group(const GemmArgs* args, int count, cudaStream_t stream, const PartSum* sums = nullptr, int sum_count = 0);
// A product shared out over K: part i is left as fp32 sums [M, N] at i * `stride` elements of d, for a reader that adds the parts in order
// (norm_sum_fwd, sum_slabs_bf16).  Plain product only, d_fp32, ldd = N, A not MN-major.  d has room for count * stride elements.
struct Slabs {
  int count;          // parts, chosen by sizes and by how many SMs products may use
  long long stride;   // elements from one to the next (rows are rounded up to 32, and what is beyond M is written too)
  int tile, workers;  // the rest of the choice: a cap on the CTAs that moves between the two calls changes nothing
};
Slabs gemm_slabs(const GemmArgs& args);
cudaError_t gemm_to_slabs(const GemmArgs& args, const Slabs& slabs, cudaStream_t stream);
// Whether a bf16 product without epilogue is better computed this way: a long contraction whose tiles leave much of the GPU idle.
bool gemm_wants_slabs(const GemmArgs& args);
// Caps the number of CTAs (= SMs) plain GEMM launches occupy from now on; 0 restores one CTA per SM.  A
// data-parallel trainer lowers it during backward so that a few SMs stay free for the gradient collectives
// that run beside the GEMMs.  The value is read at launch time, so it is baked into a captured CUDA graph.
void set_gemm_cta_limit(int ctas);
// Which kernel plain products use: "pair" / "tile" (the default: tile chosen by size), "tile64", "tile128", "tile192",
// "pair256" (that tile), "persistent" (one CTA per SM); "" = default.
void set_gemm_kernel(const std::string& name);
int gemm_cta_limit();
// What set_gemm_kernel or MCCL_GEMM_KERNEL asks for: a tile (64 ... 256), 0 for one of the kernel's choosing, -1 for the persistent kernel.
int gemm_kernel_choice();
int gemm_sm_count();
// Why the last gemm_bf16_tn call on this thread returned cudaErrorNotSupported ("" otherwise).
const char* gemm_last_reason();
// Non-zero when a pipeline wait inside a GEMM kernel ran out (kernel returned early).
int gemm_error_flag();

}  // namespace ops
}  // namespace mccl
