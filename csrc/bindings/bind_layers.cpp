// A pre-LayerNorm GELU decoder layer as two calls, forward and backward, and a decoder's forward without gradients as one.
//
// Op by op from Python a layer was 12 autograd nodes and some 40 launches, each with its own binding call, allocations and
// stream lookup: 200 us of host time forward and 300 backward, more than the kernels take below a few thousand tokens.
// Here the launches of a layer follow each other from C++ over one slab of saved activations (one allocation), and
// what only a view of the whole layer allows is taken: bias gradients come out of the kernels that produce or read the
// tensors they sum (norm backward, attention backward, the GELU product), and the four weight gradients are one launch.
#include "bind.hpp"
#include "decoder_layer.hpp"

namespace py = pybind11;

namespace mccl {

using namespace layers;

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
  // (gradient of x, gradients of the parameters, see decoder_layer_wgrads).  The gradients of the parameters are
  // ADDED into `grads` (fp32, one per parameter, same order) where given, else returned as views of one new buffer.  With defer, those of the four matrices are left for
  // decoder_layer_wgrads.
  m.def("decoder_layer_bwd", [](const at::Tensor& dout, const at::Tensor& x, const at::Tensor& slab, const std::vector<at::Tensor>& params,
                                std::vector<at::Tensor> grads, int64_t B, int64_t S, int64_t H, bool defer) {
    const Dims d = dims_of(x, B, S, H, params.at(UP_B).numel());
    c10::cuda::CUDAGuard guard(x.device());
    const Weights w = weights_of(params, d);
    need(dout, at::kBFloat16, x.numel(), "output gradient");
    const bool in_order = grads.empty();   // a trainer's buffers are added into as the sums arrive
    if (in_order) {
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
    const auto [dx, tmp] = layer_backward(dout, x, w, s, g, d, defer, in_order);
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
      need(tmp, at::kBFloat16, tmp.numel(), "gradients between the kernels");
      MCCL_CHECK_TENSOR(tmp.numel() >= TD * 6 + static_cast<int64_t>(d.tokens()) * d.F, "decoder layer: not the gradients of this backward");
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
  // launch for all), or bf16 copies the caller keeps up to date.  None when a parameter is laid out in another order: the operators
  // copy such a weight first.
  m.def(
      "decoder_fwd",
      [](const at::Tensor& tokens, const at::Tensor& tok, const c10::optional<at::Tensor>& pos, std::vector<at::Tensor> layers,
         const at::Tensor& lnf_w, const c10::optional<at::Tensor>& lnf_b, at::Tensor head, int64_t H, double eps_in,
         const c10::optional<at::Tensor>& cos_t, const c10::optional<at::Tensor>& sin_t) -> c10::optional<at::Tensor> {
        at::NoGradGuard no_grad;
        if (!all_contiguous(layers) || !all_contiguous({tok, lnf_w, head})) return c10::nullopt;
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
        // few tokens: the down projections in parts, which the norm behind each adds
        const bool as_sums = L > 0 && down_as_sums(d);
        at::Tensor room;
        Parts parts;
        if (as_sums) {
          parts.slabs = ops::gemm_slabs(product_in_parts(bf(x), w16[3], nullptr, T, D, F));
          room = at::empty({parts.slabs.count * parts.slabs.stride}, opt16.dtype(at::kFloat));
          parts.at = room.data_ptr<float>();
        }
        Unfinished before = {parts, nullptr, nullptr};
        at::Tensor kept;   // what `before` points into
        auto f32 = [&](int l, int p, int64_t n) {
          const at::Tensor& t = layers[l * per + p];
          need(t, at::kFloat, n, "parameter");
          return static_cast<const float*>(t.data_ptr<float>());
        };
        if (!rope) {
          Slab s;
          at::Tensor slab = at::empty({Slab::place(&s, nullptr, d)}, opt16.dtype(at::kByte));
          Slab::place(&s, slab.data_ptr<uint8_t>(), d);
          kept = slab;
          for (int l = 0; l < L; ++l) {
            const Weights w = {f32(l, LN1_W, D), f32(l, LN1_B, D), f32(l, QKV_B, 3 * D), f32(l, PROJ_B, D), f32(l, LN2_W, D), f32(l, LN2_B, D),
                               f32(l, UP_B, F), f32(l, DOWN_B, D), w16[l * 4], w16[l * 4 + 1], w16[l * 4 + 2], w16[l * 4 + 3]};
            layer_forward(bf(x), bf(x2), w, s, d, eps, false, st, as_sums ? &parts : nullptr, as_sums && l > 0 ? &before : nullptr);
            before = {parts, w.down_b, s.y};
            if (!as_sums) std::swap(x, x2);
          }
        } else {
          need(*cos_t, at::kFloat, cos_t->numel(), "cos");
          need(*sin_t, at::kFloat, cos_t->numel(), "sin");
          MCCL_CHECK_TENSOR(cos_t->numel() >= static_cast<int64_t>(d.S) * hd / 2, "decoder_fwd: rotary tables too small");
          at::Tensor h = at::empty({T, D}, opt16), y = at::empty({T, D}, opt16), qkv = at::empty({d.B, d.S, 3, d.H, hd}, opt16);
          at::Tensor qk = at::empty({d.B, d.S, 2, d.H, hd}, opt16), gu, act = at::empty({T, F}, opt16);
          kept = y;
          const at::Tensor q = qk.select(2, 0).transpose(1, 2), k = qk.select(2, 1).transpose(1, 2), v = qkv.select(2, 2).transpose(1, 2);
          for (int l = 0; l < L; ++l) {
            if (as_sums && l > 0) finish(before, bf(x), f32(l, 0, D), nullptr, bf(h), T, D, eps, st, "first norm");
            else check(ops::norm_fwd(bf(x), f32(l, 0, D), nullptr, bf(h), nullptr, nullptr, T, D, eps, st), "first norm");
            product(bf(h), w16[l * 4], nullptr, bf(qkv), T, 3 * D, D, nullptr, false, nullptr, st, "qkv projection");
            check(ops::rope_qk_fwd(bf(qkv), cos_t->data_ptr<float>(), sin_t->data_ptr<float>(), bf(qk), T, d.S, d.H, hd, st), "rotary embedding");
            const at::Tensor o = at::scaled_dot_product_attention(q, k, v, {}, 0.0, true).transpose(1, 2).contiguous();
            product(bf(o), w16[l * 4 + 1], nullptr, bf(y), T, D, D, bf(x), false, nullptr, st, "output projection");
            check(ops::norm_fwd(bf(y), f32(l, 3, D), nullptr, bf(h), nullptr, nullptr, T, D, eps, st), "second norm");
            const cudaError_t fused = gated(bf(h), w16[l * 4 + 2], bf(act), nullptr, T, F, D, st);
            if (fused != cudaSuccess) {
              if (fused != cudaErrorNotSupported) check(fused, "gate and up projection");
              if (!gu.defined()) gu = at::empty({T, 2 * static_cast<int64_t>(F)}, opt16);
              product(bf(h), w16[l * 4 + 2], nullptr, bf(gu), T, 2 * F, D, nullptr, false, nullptr, st, "gate and up projection");
              check(ops::swiglu_fwd(bf(gu), bf(act), T, F, st), "activation");
            }
            if (as_sums) {
              before = {parts, nullptr, bf(y)};
              check(ops::gemm_to_slabs(product_in_parts(bf(act), w16[l * 4 + 3], parts.at, T, D, F), parts.slabs, st), "down projection");
            } else {
              product(bf(act), w16[l * 4 + 3], nullptr, bf(x2), T, D, F, bf(y), false, nullptr, st, "down projection");
              std::swap(x, x2);
            }
          }
        }
        const float* final_b = lnf_b.has_value() ? lnf_b->data_ptr<float>() : nullptr;
        if (as_sums) finish(before, bf(x), lnf_w.data_ptr<float>(), final_b, bf(x2), T, D, eps, st, "final norm");
        else check(ops::norm_fwd(bf(x), lnf_w.data_ptr<float>(), final_b, bf(x2), nullptr, nullptr, T, D, eps, st), "final norm");
        at::Tensor logits = at::empty({d.B, d.S, V}, opt16);
        product(bf(x2), w16[L * 4], nullptr, bf(logits), T, V, D, nullptr, false, nullptr, st, "head");
        return logits;
      },
      py::arg("tokens"), py::arg("tok"), py::arg("pos"), py::arg("layers"), py::arg("lnf_w"), py::arg("lnf_b"), py::arg("head"), py::arg("heads"),
      py::arg("eps"), py::arg("cos") = py::none(), py::arg("sin") = py::none());
}

}  // namespace mccl
