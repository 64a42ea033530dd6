// The training loss of a GELU decoder for stock PyTorch loops: the same autograd graph as the Python modules build (one node
// per layer, so gradients become ready layer by layer), made of C++ nodes in one call.  From Python a node cost 60 us of
// host time each way, more than its kernels take below a few thousand tokens: a step of the 2-layer model on 192 tokens
// was 810 us of host work around 160 us of kernels.
//
// Used where every parameter wants a gradient and none goes straight into a trainer's buffer.
#include "bind.hpp"
#include "decoder_layer.hpp"

namespace py = pybind11;

namespace mccl {

using namespace layers;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

cudaStream_t stream_on(const at::Tensor& t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
// One buffer of zeros for several fp32 gradients: a memset, which costs the host 2 us where a fill operator costs 9.
at::Tensor zeros_f32(int64_t numel, const at::Tensor& like) {
  at::Tensor t = at::empty({numel}, like.options().dtype(at::kFloat).requires_grad(false));
  check(cudaMemsetAsync(t.data_ptr(), 0, static_cast<size_t>(numel) * 4, stream_on(like)), "gradient buffer");
  return t;
}
const long long* ids_of(const at::Tensor& t) { return reinterpret_cast<const long long*>(t.data_ptr<int64_t>()); }

// bf16(tok[ids] + pos[position])
struct EmbeddingNode : torch::autograd::Function<EmbeddingNode> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& ids, const at::Tensor& tok, const at::Tensor& pos) {
    const int T = static_cast<int>(ids.numel()), S = static_cast<int>(ids.size(1)), D = static_cast<int>(tok.size(1));
    at::Tensor y = at::empty({ids.size(0), ids.size(1), D}, tok.options().dtype(at::kBFloat16));
    check(ops::embed_fwd(ids_of(ids), tok.data_ptr<float>(), pos.data_ptr<float>(), bf(y), T, S, D, static_cast<int>(tok.size(0)), stream_on(tok)), "embedding");
    ctx->save_for_backward({ids, tok, pos});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &ids = saved[0], &tok = saved[1], &pos = saved[2], dy = grads[0].contiguous();
    c10::cuda::CUDAGuard guard(tok.device());
    const int64_t at_pos = (tok.numel() + 7) / 8 * 8;
    const at::Tensor buffer = zeros_f32(at_pos + pos.numel(), tok);
    at::Tensor dtok = buffer.as_strided(tok.sizes(), tok.strides(), 0), dpos = buffer.as_strided(pos.sizes(), pos.strides(), at_pos);
    check(ops::embed_bwd(ids_of(ids), bf(dy), dtok.data_ptr<float>(), dpos.data_ptr<float>(), static_cast<int>(ids.numel()), static_cast<int>(ids.size(1)),
                         static_cast<int>(tok.size(1)), static_cast<int>(tok.size(0)), stream_on(tok)),
          "embedding backward");
    return {at::Tensor(), dtok, dpos};
  }
};

// params: the 12 of a layer; the bf16 copies of its matrices are at `off` in `flat`.
struct LayerNode : torch::autograd::Function<LayerNode> {
  static Weights weights(at::TensorList p, const at::Tensor& flat, const int64_t* off) {
    auto f = [&](int i) { return static_cast<const float*>(p[i].data_ptr<float>()); };
    const bf16* w = bf(flat);
    return {f(LN1_W), f(LN1_B), f(QKV_B), f(PROJ_B), f(LN2_W), f(LN2_B), f(UP_B), f(DOWN_B), w + off[0], w + off[1], w + off[2], w + off[3]};
  }
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& x, at::TensorList params, const at::Tensor& flat, std::vector<int64_t> off, int64_t heads,
                            double eps) {
    const Dims d = dims_of(x, x.size(0), x.size(1), heads, params[UP_B].numel());
    Slab s;
    at::Tensor slab = at::empty({Slab::place(&s, nullptr, d)}, x.options().dtype(at::kByte));
    Slab::place(&s, slab.data_ptr<uint8_t>(), d);
    at::Tensor out = at::empty_like(x);
    layer_forward(bf(x), bf(out), weights(params, flat, off.data()), s, d, static_cast<float>(eps), true, stream_on(x));
    variable_list keep = {x, slab, flat};
    keep.insert(keep.end(), params.begin(), params.end());
    ctx->save_for_backward(std::move(keep));
    ctx->saved_data["off"] = off;
    ctx->saved_data["heads"] = heads;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &x = saved[0], &slab = saved[1], &flat = saved[2];
    const at::TensorList params = at::TensorList(saved).slice(3);
    const std::vector<int64_t> off = ctx->saved_data["off"].toIntVector();
    const Dims d = dims_of(x, x.size(0), x.size(1), ctx->saved_data["heads"].toInt(), params[UP_B].numel());
    c10::cuda::CUDAGuard guard(x.device());
    const at::Tensor dout = grads[0].contiguous();
    int64_t total = 0, at[kParams];
    for (int i = 0; i < kParams; ++i) {
      at[i] = total;
      total += (param_numel(d, i) + 7) / 8 * 8;
    }
    const at::Tensor buffer = zeros_f32(total, x);
    float* g[kParams];
    variable_list out(1 + kParams + 4);   // x, parameters, flat, off, heads, eps
    for (int i = 0; i < kParams; ++i) {
      g[i] = buffer.data_ptr<float>() + at[i];
      out[1 + i] = buffer.as_strided(params[i].sizes(), params[i].strides(), at[i]);
    }
    Slab s;
    Slab::place(&s, slab.data_ptr<uint8_t>(), d);
    out[0] = layer_backward(dout, x, weights(params, flat, off.data()), s, g, d, false, true).first;
    return out;
  }
};

struct NormNode : torch::autograd::Function<NormNode> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& w, const at::Tensor& b, double eps) {
    const int D = static_cast<int>(x.size(-1)), T = static_cast<int>(x.numel() / D);
    at::Tensor y = at::empty_like(x), stats = at::empty({2, T}, w.options());
    float* mean = stats.data_ptr<float>();
    check(ops::norm_fwd(bf(x), w.data_ptr<float>(), b.data_ptr<float>(), bf(y), mean, mean + T, T, D, static_cast<float>(eps), stream_on(x)), "final norm");
    ctx->save_for_backward({x, w, b, stats});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &x = saved[0], &w = saved[1], &stats = saved[3], dy = grads[0].contiguous();
    c10::cuda::CUDAGuard guard(x.device());
    const int D = static_cast<int>(x.size(-1)), T = static_cast<int>(x.numel() / D);
    const float* mean = stats.data_ptr<float>();
    const int64_t at_b = (D + 7) / 8 * 8;
    const int rows = ops::norm_bwd_parts(T, D);
    at::Tensor dx = at::empty_like(x), g = at::empty({2 * at_b + 2 * static_cast<int64_t>(rows) * D}, stats.options());   // the sums, and the parts they are made of
    float *dw = g.data_ptr<float>(), *pw = dw + 2 * at_b, *pb = pw + static_cast<int64_t>(rows) * D;
    check(ops::norm_bwd_fused(bf(dy), bf(x), w.data_ptr<float>(), mean, mean + T, bf(dx), nullptr, pw, pb, nullptr, nullptr, T, D, true, stream_on(x), true),
          "final norm backward");
    const ops::PartSum sums[2] = {{pw, dw, rows, D}, {pb, dw + at_b, rows, D}};
    check(ops::sum_parts(sums, 2, stream_on(x)), "final norm backward");
    return {dx, g.as_strided({D}, {1}, 0), g.as_strided({D}, {1}, at_b), at::Tensor()};
  }
};

// Mean cross entropy of h · head^T against targets; the gradient of the logits replaces them in the forward pass, for an
// upstream gradient of one.  Backward's two products multiply by the one that comes (a scaled loss, a sum of several).
struct CrossEntropyNode : torch::autograd::Function<CrossEntropyNode> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& h, const at::Tensor& head, const at::Tensor& flat, int64_t off, const at::Tensor& targets) {
    const int D = static_cast<int>(h.size(-1)), T = static_cast<int>(h.numel() / D), V = static_cast<int>(head.size(0));
    at::Tensor logits = at::empty({T, V}, h.options()), rows = at::empty({T}, head.options());
    product(bf(h), bf(flat) + off, nullptr, bf(logits), T, V, D, nullptr, false, nullptr, stream_on(h), "head");
    check(ops::cross_entropy_fwd_bwd(bf(logits), ids_of(targets), rows.data_ptr<float>(), T, V, 1.f / static_cast<float>(T), stream_on(h)), "cross entropy");
    ctx->save_for_backward({h, head, flat, logits});
    ctx->saved_data["off"] = off;
    at::Tensor loss = at::empty({}, rows.options());
    check(ops::mean_f32(rows.data_ptr<float>(), loss.data_ptr<float>(), T, stream_on(h)), "mean loss");
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &h = saved[0], &head = saved[1], &flat = saved[2], &dlogits = saved[3];
    c10::cuda::CUDAGuard guard(h.device());
    const at::Tensor upstream = grads[0].to(head.options());
    const int D = static_cast<int>(h.size(-1)), T = static_cast<int>(h.numel() / D), V = static_cast<int>(head.size(0));
    cudaStream_t st = stream_on(h);
    at::Tensor dh = at::empty_like(h);
    const bf16* w = bf(flat) + ctx->saved_data["off"].toInt();
    ops::GemmArgs g;
    g.a = bf(dlogits);
    g.b = w;
    g.b_mn_major = true;
    g.d = dh.data_ptr();
    g.m = T;
    g.n = g.ldb = g.ldd = D;
    g.k = g.lda = V;
    if (ops::gemm_wants_slabs(g)) {
      g.d_fp32 = true;
      const ops::Slabs slabs = ops::gemm_slabs(g);
      at::Tensor parts = at::empty({slabs.count * slabs.stride}, head.options());
      g.d = parts.data_ptr();
      check(ops::gemm_to_slabs(g, slabs, st), "head backward");
      check(ops::sum_slabs_bf16(parts.data_ptr<float>(), slabs.count, slabs.stride, bf(dh), static_cast<long long>(T) * D, upstream.data_ptr<float>(), st), "head backward");
    } else {
      g.alpha = upstream.data_ptr<float>();
      check(ops::gemm_bf16_tn(g, st), "head backward");
    }
    at::Tensor dw = at::empty({V, D}, head.options());
    ops::GemmArgs wg = weight_gradient(bf(dlogits), bf(h), dw.data_ptr<float>(), T, V, D);
    wg.accumulate = false;
    wg.alpha = upstream.data_ptr<float>();
    check(ops::gemm_bf16_tn(wg, st), "head weight gradient");
    return {dh, dw, at::Tensor(), at::Tensor(), at::Tensor()};
  }
};

}  // namespace

void bind_decoder_autograd(py::module_& m) {
  // Mean next-token loss of a GELU / LayerNorm decoder with learned positions.  layers: 12 fp32 parameters per layer in the order
  // of decoder_layer_fwd; head: the fp32 output table (tok itself where they are tied).  None when a parameter is laid out in another order.
  m.def(
      "decoder_loss",
      [](const at::Tensor& tokens, const at::Tensor& targets, const at::Tensor& tok, const at::Tensor& pos, const std::vector<at::Tensor>& layers,
         const at::Tensor& lnf_w, const at::Tensor& lnf_b, const at::Tensor& head, int64_t heads, double eps) -> c10::optional<at::Tensor> {
        if (!all_contiguous(layers) || !all_contiguous({tok, pos, lnf_w, lnf_b, head})) return c10::nullopt;
        MCCL_CHECK_TENSOR(tokens.is_cuda() && tokens.dim() == 2 && tokens.scalar_type() == at::kLong && targets.is_cuda() &&
                              targets.scalar_type() == at::kLong && targets.numel() == tokens.numel(),
                          "decoder_loss: int64 CUDA tokens [B, S] and as many targets expected");
        MCCL_CHECK_TENSOR(layers.size() % kParams == 0 && pos.dim() == 2 && pos.size(0) >= tokens.size(1) && pos.size(1) == tok.size(1),
                          "decoder_loss: bad parameters");
        c10::cuda::CUDAGuard guard(tokens.device());
        const int L = static_cast<int>(layers.size() / kParams);
        static const int kMatrices[4] = {QKV_W, PROJ_W, UP_W, DOWN_W};
        std::vector<const float*> src;
        std::vector<long long> numel, off;
        long long total = 0;
        auto want = [&](const at::Tensor& t) {
          need(t, at::kFloat, t.numel(), "weight");
          src.push_back(t.data_ptr<float>());
          numel.push_back(t.numel());
          off.push_back(total);
          total += (t.numel() + 7) / 8 * 8;
        };
        Dims d{};
        d.D = static_cast<int>(tok.size(1));
        d.F = L ? static_cast<int>(layers[UP_B].numel()) : 0;
        for (size_t i = 0; i < layers.size(); ++i) need(layers[i], at::kFloat, param_numel(d, static_cast<int>(i % kParams)), "parameter");
        for (int l = 0; l < L; ++l)
          for (int k : kMatrices) want(layers[l * kParams + k]);
        want(head);
        need(tok, at::kFloat, tok.numel(), "token table");
        need(pos, at::kFloat, pos.numel(), "position table");
        need(lnf_w, at::kFloat, d.D, "final norm");
        need(lnf_b, at::kFloat, d.D, "final norm");
        const at::Tensor flat = at::empty({total}, tok.options().dtype(at::kBFloat16).requires_grad(false));
        check(ops::cast_many(src.data(), numel.data(), off.data(), static_cast<int>(src.size()), bf(flat), stream_on(tok)), "weight casts");
        at::Tensor x = EmbeddingNode::apply(tokens.contiguous(), tok, pos);
        for (int l = 0; l < L; ++l) {
          const std::vector<int64_t> at = {off[4 * l], off[4 * l + 1], off[4 * l + 2], off[4 * l + 3]};
          x = LayerNode::apply(x, at::TensorList(layers).slice(l * kParams, kParams), flat, at, heads, eps);
        }
        x = NormNode::apply(x, lnf_w, lnf_b, eps);
        return CrossEntropyNode::apply(x, head, flat, static_cast<int64_t>(off[4 * L]), targets.contiguous());
      },
      py::call_guard<py::gil_scoped_release>());
}

}  // namespace mccl
