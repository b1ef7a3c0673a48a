// The layer-side operators (gate and beta activation, short convolution, gated RMS norm) with autograd on the native host path.
#include "host_common.h"

namespace cula_host {

namespace {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

bool grad_wanted(std::initializer_list<OptTensor> ts) {
    for (const OptTensor& t : ts)
        if (t.has_value() && has_tangent(*t)) return true;
    if (!at::GradMode::is_enabled()) return false;
    for (const OptTensor& t : ts)
        if (t.has_value() && t->defined() && t->requires_grad()) return true;
    return false;
}
OptTensor opt_of(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }
bool is_float(const Tensor& t) { return is_bf16(t) || is_f32(t); }

// ------------------------------------------------ gate activation ------------------------------------------------
Tensor gate_forward(const Tensor& g, const Tensor& a32, const OptTensor& b32, std::optional<double> lower_bound, at::ScalarType out_dtype) {
    c10::cuda::CUDAGuard guard(g.device());
    const int64_t H = g.size(-2), K = g.size(-1);
    Tensor y = device_empty(g.sizes(), g.options().dtype(out_dtype));
    check(lib.cula_kda_gate_fwd(ptr(g), is_f32(g), fptr(a32), fptr(b32), ptr(y), out_dtype == at::kFloat, g.numel() / (H * K), (int)H, (int)K,
                                lower_bound.has_value(), (float)lower_bound.value_or(0.0), stream_of(g)), "cula_kda_gate_fwd");
    return y;
}

struct Gate : torch::autograd::Function<Gate> {
    static Tensor forward(AutogradContext* ctx, const Tensor& g_in, const Tensor& A_log, const OptTensor& dt_bias, std::optional<double> lower_bound,
                          int64_t out_dtype) {
        const Tensor g = g_in.contiguous(), a32 = contiguous_f32(A_log);
        const OptTensor b32 = contiguous_f32(dt_bias);
        ctx->save_for_backward({g, a32, b32.value_or(Tensor())});
        ctx->saved_data["lb"] = lower_bound.has_value() ? c10::IValue(*lower_bound) : c10::IValue();
        ctx->set_materialize_grads(false);
        return gate_forward(g, a32, b32, lower_bound, (at::ScalarType)out_dtype);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
        auto s = ctx->get_saved_variables();
        const Tensor &g = s[0], &a32 = s[1];
        const OptTensor b32 = opt_of(s[2]);
        c10::cuda::CUDAGuard guard(g.device());
        const int64_t H = g.size(-2), K = g.size(-1);
        Tensor dy = grads[0].contiguous();
        if (!is_float(dy)) dy = dy.to(at::kFloat);
        const c10::IValue lb = ctx->saved_data["lb"];
        Tensor dg = device_empty(g.sizes(), g.options());
        // the two accumulated gradients share one cleared buffer
        const int64_t n_bias = b32.has_value() ? b32->numel() : 0;
        Tensor both = device_zeros({n_bias + a32.numel()}, a32.options(), stream_of(g));
        Tensor dA = part_of(both, n_bias, a32.sizes());
        Tensor dbias = b32.has_value() ? part_of(both, 0, b32->sizes()) : Tensor();
        check(lib.cula_kda_gate_bwd(ptr(g), is_f32(g), fptr(a32), fptr(b32), ptr(dy), is_f32(dy), ptr(dg), fptr(dA), fptr(dbias), g.numel() / (H * K),
                                    (int)H, (int)K, !lb.isNone(), lb.isNone() ? 0.f : (float)lb.toDouble(), stream_of(g)), "cula_kda_gate_bwd");
        return {dg, dA, dbias, Tensor(), Tensor()};
    }
};

Tensor kda_gate(const Tensor& g, const Tensor& A_log, const OptTensor& dt_bias, std::optional<double> lower_bound, bool out_fp32) {
    require(is_float(g), "g must be in bfloat16 or float32.");
    const int64_t H = g.size(-2), K = g.size(-1);
    require(A_log.numel() == H && (!dt_bias.has_value() || dt_bias->numel() == H * K), "A_log must be [H] and dt_bias [H * K].");
    assert_blackwell(g);
    const at::ScalarType dt = out_fp32 ? at::kFloat : at::kBFloat16;
    if (grad_wanted({g, A_log, dt_bias})) return Gate::apply(g, A_log, dt_bias, lower_bound, (int64_t)dt);
    at::NoGradGuard no_grad;
    return gate_forward(g.contiguous(), contiguous_f32(A_log), contiguous_f32(dt_bias), lower_bound, dt);
}

// ------------------------------------------------ beta activation ------------------------------------------------
Tensor beta_forward(const Tensor& x) {
    c10::cuda::CUDAGuard guard(x.device());
    Tensor y = device_empty(x.sizes(), x.options().dtype(at::kFloat));
    check(lib.cula_kda_beta_sigmoid_fwd(ptr(x), is_f32(x), fptr(y), x.numel(), stream_of(x)), "cula_kda_beta_sigmoid_fwd");
    return y;
}
struct Beta : torch::autograd::Function<Beta> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x_in) {
        const Tensor x = x_in.contiguous();
        ctx->save_for_backward({x});
        ctx->set_materialize_grads(false);
        return beta_forward(x);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        if (!grads[0].defined()) return {Tensor()};
        const Tensor x = ctx->get_saved_variables()[0], dy = contiguous_f32(grads[0]);
        c10::cuda::CUDAGuard guard(x.device());
        Tensor dx = device_empty(x.sizes(), x.options());
        check(lib.cula_kda_beta_sigmoid_bwd(ptr(x), is_f32(x), fptr(dy), ptr(dx), x.numel(), stream_of(x)), "cula_kda_beta_sigmoid_bwd");
        return {dx};
    }
};
Tensor beta_sigmoid(const Tensor& x) {
    require(is_float(x), "x must be in bfloat16 or float32.");
    assert_blackwell(x);
    if (grad_wanted({x})) return Beta::apply(x);
    at::NoGradGuard no_grad;
    return beta_forward(x.contiguous());
}

// ------------------------------------------------ short convolution ------------------------------------------------
std::pair<Tensor, Tensor> conv_forward(const Tensor& x, const Tensor& w32, const OptTensor& b32, const OptTensor& c32, bool want_final, bool silu,
                                       const Tables* tab) {
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t B = x.size(0), T = x.size(1), D = x.size(2), W = w32.size(-1);
    const int64_t n_seqs = tab ? tab->n_seqs : B, num_chunks = tab ? tab->num_chunks : B * ((T + CHUNK - 1) / CHUNK);
    Tensor y = device_empty(x.sizes(), x.options());
    if (tab && tab->total_tokens < T) y.narrow(1, tab->total_tokens, T - tab->total_tokens).zero_();     // rows past the packed tokens
    Tensor fin = want_final ? device_zeros({n_seqs, D, W}, w32.options(), stream_of(x)) : Tensor();
    check(lib.cula_kda_short_conv_fwd(ptr(x), fptr(w32), fptr(b32), fptr(c32), ptr(y), fptr(fin), tab ? iptr(tab->cu_seqlens) : nullptr,
                                      tab ? iptr(tab->chunk_indices) : nullptr, (int)num_chunks, (int)T, (int)D, (int)W, silu, stream_of(x)),
          "cula_kda_short_conv_fwd");
    return {y, fin};
}
struct Conv : torch::autograd::Function<Conv> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x_in, const Tensor& weight, const OptTensor& bias, const OptTensor& cache,
                                 bool want_final, bool silu, const Tables* tab) {
        const Tensor x = x_in.contiguous(), w32 = contiguous_f32(weight);
        const OptTensor b32 = contiguous_f32(bias), c32 = contiguous_f32(cache);
        ctx->save_for_backward({x, w32, b32.value_or(Tensor()), c32.value_or(Tensor())});
        ctx->saved_data["silu"] = silu;
        if (tab) {
            ctx->saved_data["tab"] = std::vector<Tensor>{tab->cu_seqlens, tab->chunk_indices};
            ctx->saved_data["tab_sizes"] = std::vector<int64_t>{tab->num_chunks, tab->total_tokens};
        }
        ctx->set_materialize_grads(false);
        auto r = conv_forward(x, w32, b32, c32, want_final, silu, tab);
        if (!want_final) return {r.first};
        ctx->mark_non_differentiable({r.second});
        return {r.first, r.second};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        variable_list none(7);
        if (!grads[0].defined()) return none;
        auto s = ctx->get_saved_variables();
        const Tensor &x = s[0], &w32 = s[1];
        const OptTensor b32 = opt_of(s[2]), c32 = opt_of(s[3]);
        c10::cuda::CUDAGuard guard(x.device());
        const int64_t B = x.size(0), T = x.size(1), D = x.size(2), W = w32.size(-1);
        Tensor dy = grads[0].contiguous();
        if (!is_bf16(dy)) dy = dy.to(at::kBFloat16);
        Tensor dx = device_empty(x.sizes(), x.options()), cu, ci;
        int64_t num_chunks = B * ((T + CHUNK - 1) / CHUNK);
        if (auto it = ctx->saved_data.find("tab"); it != ctx->saved_data.end()) {
            auto t = it->second.toTensorVector();
            auto n = ctx->saved_data["tab_sizes"].toIntVector();
            cu = t[0]; ci = t[1]; num_chunks = n[0];
            if (n[1] < T) dx.narrow(1, n[1], T - n[1]).zero_();
        }
        Tensor dw = device_zeros(w32.sizes(), w32.options(), stream_of(x));                // the two accumulated gradients
        Tensor db = b32.has_value() ? device_zeros(b32->sizes(), w32.options(), stream_of(x)) : Tensor();
        check(lib.cula_kda_short_conv_bwd(ptr(x), fptr(w32), fptr(b32), fptr(c32), ptr(dy), ptr(dx), fptr(dw), fptr(db), (int*)ptr(cu), (int*)ptr(ci),
                                          (int)num_chunks, (int)T, (int)D, (int)W, ctx->saved_data["silu"].toBool(), stream_of(x)),
              "cula_kda_short_conv_bwd");
        return {dx, dw, db, Tensor(), Tensor(), Tensor(), Tensor()};
    }
};
std::pair<Tensor, OptTensor> short_conv(const Tensor& x, const Tensor& weight_in, const OptTensor& bias, const OptTensor& cache, bool want_final,
                                        bool silu, const Tables* tab) {
    require(x.dim() == 3 && is_bf16(x), "x must be [B, T, D] in bfloat16.");
    const Tensor weight = weight_in.dim() == 3 ? weight_in.squeeze(1) : weight_in;
    const int64_t D = weight.size(0), W = weight.size(1);
    require(x.size(2) == D && D % 8 == 0 && 1 <= W && W <= 4, "weight must be [D, W] with W <= 4 and D a multiple of 8.");
    if (tab && x.size(0) != 1)
        throw pybind11::value_error("The batch size is expected to be 1 rather than " + std::to_string(x.size(0)) + " when using `cu_seqlens`.");
    const int64_t n_seqs = tab ? tab->n_seqs : x.size(0);
    if (cache.has_value()) require(cache->dim() == 3 && cache->size(0) == n_seqs && cache->size(1) == D && cache->size(2) == W, "initial_state must be [N, D, W].");
    assert_blackwell(x);
    if (grad_wanted({x, weight, bias})) {
        auto out = Conv::apply(x, weight, bias, cache, want_final, silu, tab);
        return {out[0], out.size() > 1 ? OptTensor(out[1]) : OptTensor()};
    }
    at::NoGradGuard no_grad;
    auto r = conv_forward(x.contiguous(), contiguous_f32(weight), contiguous_f32(bias), contiguous_f32(cache), want_final, silu, tab);
    return {r.first, opt_of(r.second)};
}

// ------------------------------------------------ gated RMS norm ------------------------------------------------
std::pair<Tensor, Tensor> norm_forward(const Tensor& x, const Tensor& g, const Tensor& w32, bool swish, double eps) {
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t D = x.size(-1), R = x.numel() / D;
    Tensor y = device_empty(x.sizes(), x.options()), rstd = device_empty({R}, w32.options());
    check(lib.cula_kda_rms_norm_gated_fwd(ptr(x), ptr(g), fptr(w32), ptr(y), fptr(rstd), R, (int)D, swish, (float)eps, stream_of(x)),
          "cula_kda_rms_norm_gated_fwd");
    return {y, rstd};
}
struct Norm : torch::autograd::Function<Norm> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x_in, const Tensor& g_in, const Tensor& weight, bool swish, double eps) {
        const Tensor x = x_in.contiguous(), g = g_in.contiguous(), w32 = contiguous_f32(weight);
        auto r = norm_forward(x, g, w32, swish, eps);
        ctx->save_for_backward({x, g, w32});
        ctx->saved_data["rstd"] = r.second;
        ctx->saved_data["swish"] = swish;
        ctx->set_materialize_grads(false);
        return r.first;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        if (!grads[0].defined()) return variable_list(5);
        auto s = ctx->get_saved_variables();
        const Tensor &x = s[0], &g = s[1], &w32 = s[2];
        c10::cuda::CUDAGuard guard(x.device());
        const int64_t D = x.size(-1), R = x.numel() / D;
        Tensor dy = grads[0].contiguous();
        if (!is_bf16(dy)) dy = dy.to(at::kBFloat16);
        Tensor dx = device_empty(x.sizes(), x.options()), dg = device_empty(g.sizes(), g.options()), dw = device_zeros(w32.sizes(), w32.options(), stream_of(x));
        check(lib.cula_kda_rms_norm_gated_bwd(ptr(x), ptr(g), fptr(w32), fptr(ctx->saved_data["rstd"].toTensor()), ptr(dy), ptr(dx), ptr(dg), fptr(dw), R,
                                              (int)D, ctx->saved_data["swish"].toBool(), stream_of(x)), "cula_kda_rms_norm_gated_bwd");
        return {dx, dg, dw, Tensor(), Tensor()};
    }
};
Tensor rms_norm_gated(const Tensor& x, const Tensor& g, const Tensor& weight, bool swish, double eps) {
    require(x.sizes() == g.sizes() && is_bf16(x) && is_bf16(g), "x and g must be bfloat16 tensors of one shape.");
    const int64_t D = x.size(-1);
    require((D == 128 || D == 256 || D == 512 || D == 1024) && weight.numel() == D, "the normalised dim must be 128/256/512/1024.");
    assert_blackwell(x);
    if (grad_wanted({x, g, weight})) return Norm::apply(x, g, weight, swish, eps);
    at::NoGradGuard no_grad;
    return norm_forward(x.contiguous(), g.contiguous(), contiguous_f32(weight), swish, eps).first;
}

}  // namespace

void bind_layer_ops(pybind11::module_& m) {
    m.def("kda_gate", &kda_gate);
    m.def("beta_sigmoid", &beta_sigmoid);
    m.def("short_conv", &short_conv);
    m.def("rms_norm_gated", &rms_norm_gated);
}

}  // namespace cula_host
