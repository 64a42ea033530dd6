// A pre-LayerNorm GELU decoder layer as a sequence of launches, forward and backward (see bind_layers.cpp).
#pragma once

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <algorithm>
#include <cmath>

#include "../core/errors.hpp"
#include "../ops/ops.hpp"

namespace mccl {
namespace layers {

using bf16 = __nv_bfloat16;

inline void check(cudaError_t rc, const char* what) {
  MCCL_CHECK_T(rc == cudaSuccess, CudaError, "decoder layer: " << what << " failed: " << cudaGetErrorString(rc) << " " << ops::gemm_last_reason());
}
inline bf16* bf(const at::Tensor& t) { return reinterpret_cast<bf16*>(t.data_ptr()); }
inline void need(const at::Tensor& t, at::ScalarType dt, int64_t numel, const char* what) {
  MCCL_CHECK_TENSOR(t.defined() && t.is_cuda() && t.is_contiguous() && t.scalar_type() == dt && t.numel() == numel,
                    "decoder layer: " << what << ": a contiguous CUDA tensor of " << numel << " " << c10::toString(dt) << " elements expected");
}

inline bool all_contiguous(at::TensorList tensors) {
  for (const at::Tensor& t : tensors)
    if (!t.is_contiguous()) return false;
  return true;
}

// Order of a layer's parameters everywhere below.
enum Param { LN1_W, LN1_B, QKV_W, QKV_B, PROJ_W, PROJ_B, LN2_W, LN2_B, UP_W, UP_B, DOWN_W, DOWN_B, kParams };

struct Dims {
  int B, S, H, D, F;
  int tokens() const { return B * S; }
  int head_dim() const { return D / H; }
};

inline int64_t param_numel(const Dims& d, int p) {
  const int64_t D = d.D, F = d.F;
  switch (p) {
    case QKV_W: return 3 * D * D;
    case QKV_B: return 3 * D;
    case PROJ_W: return D * D;
    case UP_W:
    case DOWN_W: return D * F;
    case UP_B: return F;
    default: return D;
  }
}

struct Weights {
  const float *ln1_w, *ln1_b, *qkv_b, *proj_b, *ln2_w, *ln2_b, *up_b, *down_b;
  const bf16 *qkv, *proj, *up, *down;
};
inline Weights weights_of(const std::vector<at::Tensor>& p, const Dims& d) {
  MCCL_CHECK_TENSOR(p.size() == kParams, "decoder layer: " << static_cast<int>(kParams) << " parameters expected");
  for (int i = 0; i < kParams; ++i) {
    const bool matrix = i == QKV_W || i == PROJ_W || i == UP_W || i == DOWN_W;
    need(p[i], matrix ? at::kBFloat16 : at::kFloat, param_numel(d, i), "parameter");
  }
  auto f = [&](int i) { return p[i].data_ptr<float>(); };
  return {f(LN1_W), f(LN1_B), f(QKV_B), f(PROJ_B), f(LN2_W), f(LN2_B), f(UP_B), f(DOWN_B), bf(p[QKV_W]), bf(p[PROJ_W]), bf(p[UP_W]), bf(p[DOWN_W])};
}

// Activations of a layer that backward reads, in one allocation.
struct Slab {
  bf16 *h1, *qkv, *o, *y, *h2, *act, *gelu_grad;
  float *mean1, *rstd1, *mean2, *rstd2, *lse;
  static int64_t place(Slab* s, uint8_t* base, const Dims& d) {
    int64_t at = 0;
    const int64_t T = d.tokens();
    auto take = [&](auto*& p, int64_t elems) {
      p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + at);
      at += (elems * static_cast<int64_t>(sizeof(*p)) + 255) / 256 * 256;
    };
    take(s->h1, T * d.D);
    take(s->qkv, T * 3 * d.D);
    take(s->o, T * d.D);
    take(s->y, T * d.D);
    take(s->h2, T * d.D);
    take(s->act, T * d.F);
    take(s->gelu_grad, T * d.F);
    take(s->mean1, T);
    take(s->rstd1, T);
    take(s->mean2, T);
    take(s->rstd2, T);
    take(s->lse, T * d.H);
    return at;
  }
};

// y[M, N] = x[M, K] · w[N, K]^T + bias (+ residual), or GELU with its derivative in `aux` (null: not wanted)
inline void product(const bf16* x, const bf16* w, const float* bias, bf16* y, int M, int N, int K, const bf16* residual, bool gelu, bf16* aux,
             cudaStream_t stream, const char* what) {
  ops::GemmArgs g;
  g.a = x;
  g.b = w;
  g.d = y;
  g.aux = aux;
  g.bias = bias;
  g.residual = residual;
  g.m = M;
  g.n = N;
  g.k = K;
  g.lda = g.ldb = K;
  g.ldd = N;
  g.epilogue = gelu ? (aux ? ops::EPI_BIAS_GELU_D : ops::EPI_BIAS_GELU) : (bias ? ops::EPI_BIAS : ops::EPI_NONE);
  check(ops::gemm_bf16_tn(g, stream), what);
}
// h[M, N] = silu(gate) * up of [gate | up] = x[M, K] · w[2 N, K]^T, which goes to gu where given; not supported: product and swiglu_fwd
inline cudaError_t gated(const bf16* x, const bf16* w, bf16* h, bf16* gu, int M, int N, int K, cudaStream_t stream) {
  ops::GemmArgs g;
  g.a = x;
  g.b = w;
  g.d = h;
  g.aux = gu;
  g.m = M;
  g.n = g.ldd = N;
  g.k = g.lda = g.ldb = K;
  return ops::gemm_swiglu(g, stream);
}
// dx[M, K] = dy[M, N] · w[N, K] (times mul, with its column sums added to colsum, or in_order: left there in parts)
inline void input_gradient(const bf16* dy, const bf16* w, bf16* dx, int M, int N, int K, const bf16* mul, float* colsum, cudaStream_t stream,
                    const char* what, bool in_order = false) {
  ops::GemmArgs g;
  g.a = dy;
  g.b = w;
  g.b_mn_major = true;
  g.d = dx;
  g.mul = mul;
  g.colsum = colsum;
  g.colsum_in_order = in_order;
  g.m = M;
  g.n = K;
  g.k = N;
  g.lda = N;
  g.ldb = g.ldd = K;
  check(ops::gemm_bf16_tn(g, stream), what);
}
inline ops::GemmArgs weight_gradient(const bf16* dy, const bf16* x, float* dw, int tokens, int N, int K) {
  ops::GemmArgs g;
  g.a = dy;
  g.b = x;
  g.d = dw;
  g.a_mn_major = g.b_mn_major = g.d_fp32 = g.accumulate = true;
  g.m = N;
  g.n = K;
  g.k = tokens;
  g.lda = N;
  g.ldb = g.ldd = K;
  return g;
}

// What the weight gradients of a layer are made of.
struct Pending {
  const bf16 *dout, *dz, *dqkv, *dy;
  Slab s;
  float *down, *up, *qkv, *proj;
};
inline void weight_gradients(const std::vector<Pending>& layers, const Dims& d, cudaStream_t stream, const ops::PartSum* sums = nullptr, int sum_count = 0) {
  const int T = d.tokens(), D = d.D, F = d.F;
  std::vector<ops::GemmArgs> args;
  for (const Pending& p : layers) {
    args.push_back(weight_gradient(p.dout, p.s.act, p.down, T, D, F));
    args.push_back(weight_gradient(p.dz, p.s.h2, p.up, T, F, D));
    args.push_back(weight_gradient(p.dqkv, p.s.h1, p.qkv, T, 3 * D, D));
    args.push_back(weight_gradient(p.dy, p.s.o, p.proj, T, D, D));
  }
  check(ops::gemm_group(args.data(), static_cast<int>(args.size()), stream, sums, sum_count), "weight gradients");
}

// Whether the down projection of these sizes is better left in parts, which the norm behind it adds: a single row of tiles that fills a
// quarter of the GPU at most, with a contraction long enough to share out.
inline bool down_as_sums(const Dims& d) { return d.tokens() <= 128 && d.D <= 2048 && d.D % 8 == 0 && d.D / 64 * 4 <= ops::gemm_sm_count() && d.F >= 1024 && d.F >= d.D; }
// x[M, K] · w[N, K]^T, to be left in parts
inline ops::GemmArgs product_in_parts(const bf16* x, const bf16* w, float* parts, int M, int N, int K) {
  ops::GemmArgs g;
  g.a = x;
  g.b = w;
  g.d = parts;
  g.d_fp32 = true;
  g.m = M;
  g.n = g.ldd = N;
  g.k = g.lda = g.ldb = K;
  return g;
}
// Room for the parts of a layer's down projection: one, every layer's next norm has read it before it is written again.
struct Parts {
  float* at = nullptr;
  ops::Slabs slabs{};
};
// What the layer before left for this one's first norm to finish, in place of x.
struct Unfinished {
  Parts parts;
  const float* bias;
  const bf16* residual;
};
inline void finish(const Unfinished& u, bf16* x, const float* w, const float* b, bf16* y, int rows, int dim, float eps, cudaStream_t st, const char* what) {
  check(ops::norm_sum_fwd(u.parts.at, u.parts.slabs.count, u.parts.slabs.stride, u.bias, u.residual, x, w, b, y, rows, dim, eps, st), what);
}

// With `parts` the down projection is left there instead of in `out`; with `before` x is written here.
inline void layer_forward(bf16* x, bf16* out, const Weights& w, const Slab& s, const Dims& d, float eps, bool keep, cudaStream_t st, const Parts* parts = nullptr,
                          const Unfinished* before = nullptr) {
  const int T = d.tokens(), D = d.D, F = d.F;
  const float scale = 1.f / std::sqrt(static_cast<float>(d.head_dim()));
  if (before) finish(*before, x, w.ln1_w, w.ln1_b, s.h1, T, D, eps, st, "first norm");
  else check(ops::norm_fwd(x, w.ln1_w, w.ln1_b, s.h1, keep ? s.mean1 : nullptr, keep ? s.rstd1 : nullptr, T, D, eps, st), "first norm");
  product(s.h1, w.qkv, w.qkv_b, s.qkv, T, 3 * D, D, nullptr, false, nullptr, st, "qkv projection");
  check(ops::attention_fwd(s.qkv, s.o, s.lse, d.B, d.S, d.H, d.head_dim(), scale, st), "attention");
  product(s.o, w.proj, w.proj_b, s.y, T, D, D, x, false, nullptr, st, "output projection");
  check(ops::norm_fwd(s.y, w.ln2_w, w.ln2_b, s.h2, keep ? s.mean2 : nullptr, keep ? s.rstd2 : nullptr, T, D, eps, st), "second norm");
  product(s.h2, w.up, w.up_b, s.act, T, F, D, nullptr, true, keep ? s.gelu_grad : nullptr, st, "up projection");
  if (parts) check(ops::gemm_to_slabs(product_in_parts(s.act, w.down, parts->at, T, D, F), parts->slabs, st), "down projection");
  else product(s.act, w.down, w.down_b, out, T, D, F, s.y, false, nullptr, st, "down projection");
}

inline Dims dims_of(const at::Tensor& x, int64_t B, int64_t S, int64_t H, int64_t F) {
  MCCL_CHECK_TENSOR(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.is_contiguous() && x.dim() >= 2, "decoder layer: a contiguous bf16 CUDA activation expected");
  const int64_t D = x.size(-1);
  MCCL_CHECK_TENSOR(B > 0 && S > 0 && H > 0 && D % H == 0 && x.numel() == B * S * D && B * S < (1ll << 31), "decoder layer: bad sizes");
  return {static_cast<int>(B), static_cast<int>(S), static_cast<int>(H), static_cast<int>(D), static_cast<int>(F)};
}

// The vectors' gradients of a layer as the kernels that hold the tensors leave them with in_order: one row per contributor.
struct VectorParts {
  float* part[kParams] = {};
  int rows[kParams] = {};
  static int64_t place(VectorParts* v, float* base, const Dims& d) {
    const int T = d.tokens(), norm = ops::norm_bwd_parts(T, d.D), attention = ops::attention_bwd_parts(d.B, d.S);
    int64_t at = 0;
    for (int i : {LN1_W, LN1_B, QKV_B, PROJ_B, LN2_W, LN2_B, UP_B, DOWN_B}) {
      v->rows[i] = i == QKV_B ? attention : (i == UP_B ? (T + 31) / 32 : norm);
      v->part[i] = base + at;
      at += static_cast<int64_t>(v->rows[i]) * param_numel(d, i);
    }
    return at;
  }
};

// Backward of a layer.  g: gradient buffers of the 12 parameters, added into (in_order: the vectors' are written, as sums in an order that
// does not depend on scheduling).  Returns (dx, gradients between the kernels); with defer the matrices' gradients are left
// for weight_gradients(), which needs the second.
inline std::pair<at::Tensor, at::Tensor> layer_backward(const at::Tensor& dout, const at::Tensor& x, const Weights& w, const Slab& s, float* const (&g)[kParams],
                                                        const Dims& d, bool defer, bool in_order) {
  const int T = d.tokens(), D = d.D, F = d.F;
  const float scale = 1.f / std::sqrt(static_cast<float>(d.head_dim()));
  cudaStream_t st = at::cuda::getCurrentCUDAStream(x.get_device()).stream();
  // dz [T, F], dqkv [T, 3 D], and three of [T, D]
  const int64_t TD = static_cast<int64_t>(T) * D;
  const int64_t elems = TD * 6 + static_cast<int64_t>(T) * F;
  VectorParts parts;
  const int64_t room = in_order ? VectorParts::place(&parts, nullptr, d) : 0;   // fp32, behind the others
  at::Tensor tmp = at::empty({elems + 2 * room}, x.options());
  bf16 *dh = bf(tmp), *dy = dh + TD, *d_o = dy + TD, *dqkv = d_o + TD, *dz = dqkv + 3 * TD;
  at::Tensor dx = at::empty_like(x);
  float* v[kParams];   // where the kernels leave the vectors' gradients
  std::copy(std::begin(g), std::end(g), v);
  if (in_order) {
    VectorParts::place(&parts, reinterpret_cast<float*>(bf(tmp) + elems), d);
    for (int i = 0; i < kParams; ++i)
      if (parts.part[i]) v[i] = parts.part[i];
  }
  input_gradient(bf(dout), w.down, dz, T, D, F, s.gelu_grad, v[UP_B], st, "down projection backward", in_order);
  input_gradient(dz, w.up, dh, T, F, D, nullptr, nullptr, st, "up projection backward");
  check(ops::norm_bwd_fused(dh, s.y, w.ln2_w, s.mean2, s.rstd2, dy, bf(dout), v[LN2_W], v[LN2_B], v[DOWN_B], v[PROJ_B], T, D, true, st, in_order),
        "second norm backward");
  input_gradient(dy, w.proj, d_o, T, D, D, nullptr, nullptr, st, "output projection backward");
  check(ops::attention_bwd(s.qkv, s.o, d_o, s.lse, dqkv, v[QKV_B], d.B, d.S, d.H, d.head_dim(), scale, st, in_order), "attention backward");
  input_gradient(dqkv, w.qkv, dh, T, 3 * D, D, nullptr, nullptr, st, "qkv projection backward");
  check(ops::norm_bwd_fused(dh, bf(x), w.ln1_w, s.mean1, s.rstd1, bf(dx), dy, v[LN1_W], v[LN1_B], nullptr, nullptr, T, D, true, st, in_order),
        "first norm backward");
  ops::PartSum sums[kParams];
  int n = 0;
  for (int i = 0; i < kParams; ++i)
    if (parts.part[i]) sums[n++] = {parts.part[i], g[i], parts.rows[i], static_cast<int>(param_numel(d, i))};
  if (!defer) {
    const Pending p = {bf(dout), dz, dqkv, dy, s, g[DOWN_W], g[UP_W], g[QKV_W], g[PROJ_W]};
    weight_gradients({p}, d, st, sums, n);
  } else if (in_order) {
    check(ops::sum_parts(sums, n, st), "sums of the vectors' gradients");
  }
  return {dx, tmp};
}

}  // namespace layers
}  // namespace mccl
