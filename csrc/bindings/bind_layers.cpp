// A pre-LayerNorm GELU decoder layer as two calls, forward and backward, and a decoder's forward without gradients as one.
//
// Op by op from Python a layer was 12 autograd nodes and some 40 launches, each with its own binding call, allocations and
// stream lookup: 200 us of host time forward and 300 backward, more than the kernels take below a few thousand tokens.
// Here the launches of a layer follow each other from C++ over one slab of saved activations (one allocation), and
// what only a view of the whole layer allows is taken: bias gradients come out of the kernels that produce or read the
// tensors they sum (norm backward, attention backward, the GELU product), and the four weight gradients are one launch.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <cmath>

#include "../core/errors.hpp"
#include "../ops/ops.hpp"
#include "bind.hpp"

namespace py = pybind11;

namespace mccl {

namespace {

using bf16 = __nv_bfloat16;

void check(cudaError_t rc, const char* what) {
  MCCL_CHECK_T(rc == cudaSuccess, CudaError, "decoder layer: " << what << " failed: " << cudaGetErrorString(rc) << " " << ops::gemm_last_reason());
}
bf16* bf(const at::Tensor& t) { return reinterpret_cast<bf16*>(t.data_ptr()); }
void need(const at::Tensor& t, at::ScalarType dt, int64_t numel, const char* what) {
  MCCL_CHECK_TENSOR(t.defined() && t.is_cuda() && t.is_contiguous() && t.scalar_type() == dt && t.numel() == numel,
                    "decoder layer: " << what << ": a contiguous CUDA tensor of " << numel << " " << c10::toString(dt) << " elements expected");
}

// Order of a layer's parameters everywhere below.
enum Param { LN1_W, LN1_B, QKV_W, QKV_B, PROJ_W, PROJ_B, LN2_W, LN2_B, UP_W, UP_B, DOWN_W, DOWN_B, kParams };

struct Dims {
  int B, S, H, D, F;
  int tokens() const { return B * S; }
  int head_dim() const { return D / H; }
};

int64_t param_numel(const Dims& d, int p) {
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
Weights weights_of(const std::vector<at::Tensor>& p, const Dims& d) {
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
void product(const bf16* x, const bf16* w, const float* bias, bf16* y, int M, int N, int K, const bf16* residual, bool gelu, bf16* aux,
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
// dx[M, K] = dy[M, N] · w[N, K] (times mul, with its column sums added to colsum)
void input_gradient(const bf16* dy, const bf16* w, bf16* dx, int M, int N, int K, const bf16* mul, float* colsum, cudaStream_t stream,
                    const char* what) {
  ops::GemmArgs g;
  g.a = dy;
  g.b = w;
  g.b_mn_major = true;
  g.d = dx;
  g.mul = mul;
  g.colsum = colsum;
  g.m = M;
  g.n = K;
  g.k = N;
  g.lda = N;
  g.ldb = g.ldd = K;
  check(ops::gemm_bf16_tn(g, stream), what);
}
ops::GemmArgs weight_gradient(const bf16* dy, const bf16* x, float* dw, int tokens, int N, int K) {
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
void weight_gradients(const std::vector<Pending>& layers, const Dims& d, cudaStream_t stream) {
  const int T = d.tokens(), D = d.D, F = d.F;
  std::vector<ops::GemmArgs> args;
  for (const Pending& p : layers) {
    args.push_back(weight_gradient(p.dout, p.s.act, p.down, T, D, F));
    args.push_back(weight_gradient(p.dz, p.s.h2, p.up, T, F, D));
    args.push_back(weight_gradient(p.dqkv, p.s.h1, p.qkv, T, 3 * D, D));
    args.push_back(weight_gradient(p.dy, p.s.o, p.proj, T, D, D));
  }
  check(ops::gemm_group(args.data(), static_cast<int>(args.size()), stream), "weight gradients");
}

void layer_forward(const bf16* x, bf16* out, const Weights& w, const Slab& s, const Dims& d, float eps, bool keep, cudaStream_t st) {
  const int T = d.tokens(), D = d.D, F = d.F;
  const float scale = 1.f / std::sqrt(static_cast<float>(d.head_dim()));
  check(ops::norm_fwd(x, w.ln1_w, w.ln1_b, s.h1, keep ? s.mean1 : nullptr, keep ? s.rstd1 : nullptr, T, D, eps, st), "first norm");
  product(s.h1, w.qkv, w.qkv_b, s.qkv, T, 3 * D, D, nullptr, false, nullptr, st, "qkv projection");
  check(ops::attention_fwd(s.qkv, s.o, s.lse, d.B, d.S, d.H, d.head_dim(), scale, st), "attention");
  product(s.o, w.proj, w.proj_b, s.y, T, D, D, x, false, nullptr, st, "output projection");
  check(ops::norm_fwd(s.y, w.ln2_w, w.ln2_b, s.h2, keep ? s.mean2 : nullptr, keep ? s.rstd2 : nullptr, T, D, eps, st), "second norm");
  product(s.h2, w.up, w.up_b, s.act, T, F, D, nullptr, true, keep ? s.gelu_grad : nullptr, st, "up projection");
  product(s.act, w.down, w.down_b, out, T, D, F, s.y, false, nullptr, st, "down projection");
}

Dims dims_of(const at::Tensor& x, int64_t B, int64_t S, int64_t H, int64_t F) {
  MCCL_CHECK_TENSOR(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.is_contiguous() && x.dim() >= 2, "decoder layer: a contiguous bf16 CUDA activation expected");
  const int64_t D = x.size(-1);
  MCCL_CHECK_TENSOR(B > 0 && S > 0 && H > 0 && D % H == 0 && x.numel() == B * S * D && B * S < (1ll << 31), "decoder layer: bad sizes");
  return {static_cast<int>(B), static_cast<int>(S), static_cast<int>(H), static_cast<int>(D), static_cast<int>(F)};
}

}  // namespace

void bind_layers(py::module_& m) {
  // Whether decoder_layer_fwd / _bwd cover these sizes.
  m.def("decoder_layer_supported", [](int64_t seq, int64_t heads, int64_t dim, int64_t ff) {
    return heads > 0 && dim % heads == 0 && dim % 64 == 0 && ff % 64 == 0 && dim <= 1024 && seq < (1 << 30) && dim / heads < (1 << 30) &&
           ops::attention_supported(static_cast<int>(seq), static_cast<int>(dim / heads));
  });
  // x [B, S, D] -> (layer(x), slab of saved activations).  params: ln1 w, b; qkv w (bf16), b; proj w (bf16), b; ln2 w, b;
  // up w (bf16), b; down w (bf16), b; vectors fp32.
  m.def("decoder_layer_fwd", [](const at::Tensor& x, const std::vector<at::Tensor>& params, int64_t B, int64_t S, int64_t H, double eps) {
    const Dims d = dims_of(x, B, S, H, params.at(UP_B).numel());
    c10::cuda::CUDAGuard guard(x.device());
    const Weights w = weights_of(params, d);
    Slab s;
    at::Tensor slab = at::empty({Slab::place(&s, nullptr, d)}, x.options().dtype(at::kByte));
    Slab::place(&s, slab.data_ptr<uint8_t>(), d);
    at::Tensor out = at::empty_like(x);
    layer_forward(bf(x), bf(out), w, s, d, static_cast<float>(eps), true, at::cuda::getCurrentCUDAStream(x.get_device()).stream());
    return std::make_pair(out, slab);
  });
  // (gradient of x, gradients of the parameters, see decoder_layer_wgrads).  The gradients of the parameters are ADDED into `grads` (fp32, one per parameter, same order)
  // where given, else returned as views of one new buffer.  With defer, those of the four matrices are left for
  // decoder_layer_wgrads.
  m.def("decoder_layer_bwd", [](const at::Tensor& dout, const at::Tensor& x, const at::Tensor& slab, const std::vector<at::Tensor>& params,
                                std::vector<at::Tensor> grads, int64_t B, int64_t S, int64_t H, bool defer) {
    const Dims d = dims_of(x, B, S, H, params.at(UP_B).numel());
    c10::cuda::CUDAGuard guard(x.device());
    const Weights w = weights_of(params, d);
    need(dout, at::kBFloat16, x.numel(), "output gradient");
    if (grads.empty()) {
      int64_t total = 0, at[kParams];
      for (int i = 0; i < kParams; ++i) {
        at[i] = total;
        total += (param_numel(d, i) + 7) / 8 * 8;
      }
      const at::Tensor flat = at::zeros({total}, x.options().dtype(at::kFloat));
      for (int i = 0; i < kParams; ++i) grads.push_back(flat.as_strided(params[i].sizes(), params[i].strides(), at[i]));
    }
    MCCL_CHECK_TENSOR(grads.size() == kParams, "decoder layer: one gradient buffer per parameter expected");
    float* g[kParams];
    for (int i = 0; i < kParams; ++i) {
      need(grads[i], at::kFloat, param_numel(d, i), "gradient buffer");
      g[i] = grads[i].data_ptr<float>();
    }
    Slab s;
    MCCL_CHECK_TENSOR(slab.is_cuda() && slab.numel() == Slab::place(&s, nullptr, d), "decoder layer: not the slab of this forward");
    Slab::place(&s, slab.data_ptr<uint8_t>(), d);
    const int T = d.tokens(), D = d.D, F = d.F;
    const float scale = 1.f / std::sqrt(static_cast<float>(d.head_dim()));
    cudaStream_t st = at::cuda::getCurrentCUDAStream(x.get_device()).stream();
    // gradients between the kernels: dz [T, F], dqkv [T, 3 D], and three of [T, D]
    const int64_t TD = static_cast<int64_t>(T) * D;
    at::Tensor tmp = at::empty({TD * 6 + static_cast<int64_t>(T) * F}, x.options());
    bf16 *dh = bf(tmp), *dy = dh + TD, *d_o = dy + TD, *dqkv = d_o + TD, *dz = dqkv + 3 * TD;
    at::Tensor dx = at::empty_like(x);
    input_gradient(bf(dout), w.down, dz, T, D, F, s.gelu_grad, g[UP_B], st, "down projection backward");
    input_gradient(dz, w.up, dh, T, F, D, nullptr, nullptr, st, "up projection backward");
    check(ops::norm_bwd_fused(dh, s.y, w.ln2_w, s.mean2, s.rstd2, dy, bf(dout), g[LN2_W], g[LN2_B], g[DOWN_B], g[PROJ_B], T, D, true, st),
          "second norm backward");
    input_gradient(dy, w.proj, d_o, T, D, D, nullptr, nullptr, st, "output projection backward");
    check(ops::attention_bwd(s.qkv, s.o, d_o, s.lse, dqkv, g[QKV_B], d.B, d.S, d.H, d.head_dim(), scale, st), "attention backward");
    input_gradient(dqkv, w.qkv, dh, T, 3 * D, D, nullptr, nullptr, st, "qkv projection backward");
    check(ops::norm_bwd_fused(dh, bf(x), w.ln1_w, s.mean1, s.rstd1, bf(dx), dy, g[LN1_W], g[LN1_B], nullptr, nullptr, T, D, true, st),
          "first norm backward");
    if (!defer) {
      const Pending p = {bf(dout), dz, dqkv, dy, s, g[DOWN_W], g[UP_W], g[QKV_W], g[PROJ_W]};
      weight_gradients({p}, d, st);
    }
    return std::make_tuple(dx, grads, defer ? tmp : at::Tensor());
  });
  // The weight gradients of layers whose backward was called with defer: (output gradient, slab, the third result of
  // decoder_layer_bwd, gradient buffers) of each; the buffers are added into.
  m.def("decoder_layer_wgrads", [](const std::vector<std::tuple<at::Tensor, at::Tensor, at::Tensor, std::vector<at::Tensor>>>& layers, int64_t B,
                                   int64_t S, int64_t H) {
    if (layers.empty()) return;
    const at::Tensor& first = std::get<0>(layers[0]);
    const Dims d = dims_of(first, B, S, H, std::get<3>(layers[0]).at(UP_B).numel());
    c10::cuda::CUDAGuard guard(first.device());
    const int64_t TD = static_cast<int64_t>(d.tokens()) * d.D;
    std::vector<Pending> pending;
    for (const auto& [dout, slab, tmp, grads] : layers) {
      Pending p;
      need(dout, at::kBFloat16, TD, "output gradient");
      need(tmp, at::kBFloat16, TD * 6 + static_cast<int64_t>(d.tokens()) * d.F, "gradients between the kernels");
      MCCL_CHECK_TENSOR(slab.is_cuda() && slab.numel() == Slab::place(&p.s, nullptr, d) && grads.size() == kParams, "decoder layer: layers of one size expected");
      Slab::place(&p.s, slab.data_ptr<uint8_t>(), d);
      for (int i = 0; i < kParams; ++i) need(grads[i], at::kFloat, param_numel(d, i), "gradient buffer");
      p.dout = bf(dout);
      p.dy = bf(tmp) + TD;
      p.dqkv = bf(tmp) + 3 * TD;
      p.dz = bf(tmp) + 6 * TD;
      p.down = grads[DOWN_W].data_ptr<float>();
      p.up = grads[UP_W].data_ptr<float>();
      p.qkv = grads[QKV_W].data_ptr<float>();
      p.proj = grads[PROJ_W].data_ptr<float>();
      pending.push_back(p);
    }
    weight_gradients(pending, d, at::cuda::getCurrentCUDAStream(first.get_device()).stream());
  });
  // bf16 copies of fp32 tensors: views of one buffer, made by one launch (or few).
  m.def("cast_many", [](const std::vector<at::Tensor>& in) {
    std::vector<at::Tensor> out;
    if (in.empty()) return out;
    std::vector<const float*> src;
    std::vector<long long> numel, off;
    long long total = 0;
    for (const auto& t : in) {
      need(t, at::kFloat, t.numel(), "cast_many");
      src.push_back(t.data_ptr<float>());
      numel.push_back(t.numel());
      off.push_back(total);
      total += (t.numel() + 7) / 8 * 8;
    }
    c10::cuda::CUDAGuard guard(in[0].device());
    at::Tensor flat = at::empty({total}, in[0].options().dtype(at::kBFloat16));
    cudaError_t rc = ops::cast_many(src.data(), numel.data(), off.data(), static_cast<int>(in.size()), bf(flat),
                                    at::cuda::getCurrentCUDAStream(in[0].get_device()).stream());
    MCCL_CHECK_T(rc == cudaSuccess, CudaError, "cast_many failed: " << cudaGetErrorString(rc));
    for (size_t i = 0; i < in.size(); ++i) {
      out.push_back(at::alias(flat).as_strided(in[i].sizes(), in[i].strides(), off[i]));
    }
    return out;
  });
  // Logits [B, S, V] of a whole decoder, no gradients.  `layers`: per layer the 12 parameters above, or for the RMSNorm / RoPE /
  // SwiGLU family (cos / sin given) ln1 w, qkv w, proj w, ln2 w, gate_up w, down w.  Matrices are fp32 and cast here (one
  // launch for all), or bf16 copies the caller keeps up to date.
  m.def(
      "decoder_fwd",
      [](const at::Tensor& tokens, const at::Tensor& tok, const c10::optional<at::Tensor>& pos, std::vector<at::Tensor> layers,
         const at::Tensor& lnf_w, const c10::optional<at::Tensor>& lnf_b, at::Tensor head, int64_t H, double eps_in,
         const c10::optional<at::Tensor>& cos_t, const c10::optional<at::Tensor>& sin_t) {
        at::NoGradGuard no_grad;
        MCCL_CHECK_TENSOR(tokens.is_cuda() && tokens.dim() == 2 && tokens.scalar_type() == at::kLong, "decoder_fwd: int64 CUDA tokens [B, S] expected");
        c10::cuda::CUDAGuard guard(tokens.device());
        cudaStream_t st = at::cuda::getCurrentCUDAStream(tokens.get_device()).stream();
        const at::Tensor ids = tokens.contiguous();
        const bool rope = cos_t.has_value();
        const int per = rope ? 6 : static_cast<int>(kParams);
        MCCL_CHECK_TENSOR(layers.size() % per == 0, "decoder_fwd: " << per << " parameters per layer expected");
        const int L = static_cast<int>(layers.size() / per);
        const float eps = static_cast<float>(eps_in);
        Dims d;
        d.B = static_cast<int>(ids.size(0));
        d.S = static_cast<int>(ids.size(1));
        d.H = static_cast<int>(H);
        d.D = static_cast<int>(tok.size(1));
        d.F = L == 0 ? 0 : static_cast<int>(rope ? layers[5].size(1) : layers[DOWN_W].size(1));
        const int T = d.tokens(), D = d.D, F = d.F, V = static_cast<int>(head.size(0)), hd = D / d.H;
        // bf16 copies of what is fp32
        std::vector<const float*> src;
        std::vector<long long> numel, off;
        std::vector<std::pair<bool, size_t>> target;   // (head, index in `layers`)
        long long total = 0;
        auto want = [&](const at::Tensor& t, bool is_head, size_t index) {
          MCCL_CHECK_TENSOR(t.is_cuda() && t.is_contiguous(), "decoder_fwd: contiguous CUDA weights expected");
          if (t.scalar_type() == at::kBFloat16) return;
          need(t, at::kFloat, t.numel(), "weight");
          src.push_back(t.data_ptr<float>());
          numel.push_back(t.numel());
          off.push_back(total);
          target.emplace_back(is_head, index);
          total += (t.numel() + 7) / 8 * 8;
        };
        static const int kGeluMatrices[4] = {QKV_W, PROJ_W, UP_W, DOWN_W}, kRopeMatrices[4] = {1, 2, 4, 5};
        const int* matrices = rope ? kRopeMatrices : kGeluMatrices;
        for (int l = 0; l < L; ++l)
          for (int k = 0; k < 4; ++k) want(layers[l * per + matrices[k]], false, static_cast<size_t>(l * per + matrices[k]));
        want(head, true, 0);
        std::vector<const bf16*> w16(L * 4 + 1);
        for (int l = 0; l < L; ++l)
          for (int k = 0; k < 4; ++k) w16[l * 4 + k] = bf(layers[l * per + matrices[k]]);
        w16[L * 4] = bf(head);
        at::Tensor flat;
        const auto opt16 = tok.options().dtype(at::kBFloat16).requires_grad(false);
        if (total > 0) {
          flat = at::empty({total}, opt16);
          check(ops::cast_many(src.data(), numel.data(), off.data(), static_cast<int>(src.size()), bf(flat), st), "weight casts");
          for (size_t i = 0; i < target.size(); ++i) {
            size_t at = static_cast<size_t>(L) * 4;
            if (!target[i].first) {
              const size_t l = target[i].second / per, p = target[i].second % per;
              for (size_t k = 0; k < 4; ++k)
                if (static_cast<size_t>(matrices[k]) == p) at = l * 4 + k;
            }
            w16[at] = bf(flat) + off[i];
          }
        }
        need(tok, at::kFloat, tok.numel(), "token table");
        need(lnf_w, at::kFloat, D, "final norm");
        if (lnf_b.has_value()) need(*lnf_b, at::kFloat, D, "final norm");
        MCCL_CHECK_TENSOR(!pos.has_value() || (pos->is_cuda() && pos->is_contiguous() && pos->scalar_type() == at::kFloat && pos->size(0) >= d.S && pos->size(1) == D),
                          "decoder_fwd: position table too small");
        at::Tensor x = at::empty({T, D}, opt16), x2 = at::empty({T, D}, opt16);
        check(ops::embed_fwd(reinterpret_cast<const long long*>(ids.data_ptr<int64_t>()), tok.data_ptr<float>(), pos.has_value() ? pos->data_ptr<float>() : nullptr,
                             bf(x), T, d.S, D, static_cast<int>(tok.size(0)), st),
              "embedding");
        auto f32 = [&](int l, int p, int64_t n) {
          const at::Tensor& t = layers[l * per + p];
          need(t, at::kFloat, n, "parameter");
          return static_cast<const float*>(t.data_ptr<float>());
        };
        if (!rope) {
          Slab s;
          at::Tensor slab = at::empty({Slab::place(&s, nullptr, d)}, opt16.dtype(at::kByte));
          Slab::place(&s, slab.data_ptr<uint8_t>(), d);
          for (int l = 0; l < L; ++l) {
            const Weights w = {f32(l, LN1_W, D), f32(l, LN1_B, D), f32(l, QKV_B, 3 * D), f32(l, PROJ_B, D), f32(l, LN2_W, D), f32(l, LN2_B, D),
                               f32(l, UP_B, F), f32(l, DOWN_B, D), w16[l * 4], w16[l * 4 + 1], w16[l * 4 + 2], w16[l * 4 + 3]};
            layer_forward(bf(x), bf(x2), w, s, d, eps, false, st);
            std::swap(x, x2);
          }
        } else {
          need(*cos_t, at::kFloat, cos_t->numel(), "cos");
          need(*sin_t, at::kFloat, cos_t->numel(), "sin");
          MCCL_CHECK_TENSOR(cos_t->numel() >= static_cast<int64_t>(d.S) * hd / 2, "decoder_fwd: rotary tables too small");
          at::Tensor h = at::empty({T, D}, opt16), y = at::empty({T, D}, opt16), qkv = at::empty({d.B, d.S, 3, d.H, hd}, opt16);
          at::Tensor qk = at::empty({d.B, d.S, 2, d.H, hd}, opt16), gu = at::empty({T, 2 * static_cast<int64_t>(F)}, opt16), act = at::empty({T, F}, opt16);
          const at::Tensor q = qk.select(2, 0).transpose(1, 2), k = qk.select(2, 1).transpose(1, 2), v = qkv.select(2, 2).transpose(1, 2);
          for (int l = 0; l < L; ++l) {
            check(ops::norm_fwd(bf(x), f32(l, 0, D), nullptr, bf(h), nullptr, nullptr, T, D, eps, st), "first norm");
            product(bf(h), w16[l * 4], nullptr, bf(qkv), T, 3 * D, D, nullptr, false, nullptr, st, "qkv projection");
            check(ops::rope_qk_fwd(bf(qkv), cos_t->data_ptr<float>(), sin_t->data_ptr<float>(), bf(qk), T, d.S, d.H, hd, st), "rotary embedding");
            const at::Tensor o = at::scaled_dot_product_attention(q, k, v, {}, 0.0, true).transpose(1, 2).contiguous();
            product(bf(o), w16[l * 4 + 1], nullptr, bf(y), T, D, D, bf(x), false, nullptr, st, "output projection");
            check(ops::norm_fwd(bf(y), f32(l, 3, D), nullptr, bf(h), nullptr, nullptr, T, D, eps, st), "second norm");
            product(bf(h), w16[l * 4 + 2], nullptr, bf(gu), T, 2 * F, D, nullptr, false, nullptr, st, "gate and up projection");
            check(ops::swiglu_fwd(bf(gu), bf(act), T, F, st), "activation");
            product(bf(act), w16[l * 4 + 3], nullptr, bf(x2), T, D, F, bf(y), false, nullptr, st, "down projection");
            std::swap(x, x2);
          }
        }
        check(ops::norm_fwd(bf(x), lnf_w.data_ptr<float>(), lnf_b.has_value() ? lnf_b->data_ptr<float>() : nullptr, bf(x2), nullptr, nullptr, T, D, eps, st),
              "final norm");
        at::Tensor logits = at::empty({d.B, d.S, V}, opt16);
        product(bf(x2), w16[L * 4], nullptr, bf(logits), T, V, D, nullptr, false, nullptr, st, "head");
        return logits;
      },
      py::arg("tokens"), py::arg("tok"), py::arg("pos"), py::arg("layers"), py::arg("lnf_w"), py::arg("lnf_b"), py::arg("head"), py::arg("heads"),
      py::arg("eps"), py::arg("cos") = py::none(), py::arg("sin") = py::none());
}

}  // namespace mccl
