// Host side of the mixer and block glue in C++: the autograd nodes of the glue kernels, and the mixer's sequence of
// projections and glue around the operator.  A layer's forward and reverse pass is some sixty launches; in Python their
// checks, ctypes blocks, autograd.Function and view objects cost 1.1 ms a layer forward + reverse and 0.3 ms for the
// seven launches of a cached token, several times the device time of short sequences.
#include "sd_host.h"

#include <algorithm>

#include <c10/core/Event.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>

namespace {

Tensor bf16_contiguous(const Tensor& t) { return t.to(at::kBFloat16).contiguous(); }
Tensor f32_contiguous(const Tensor& t) { return t.detach().to(at::kFloat).contiguous(); }

void require_bf16_cuda(const char* name, const Tensor& t) {
    if (!t.is_cuda() || t.scalar_type() != at::kBFloat16)
        throw py::type_error(std::string(name) + " must be a BF16 CUDA tensor");
}

bool records_gradients(std::initializer_list<const Tensor*> tensors) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : tensors)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

// FP32 copies of parameters that the inference kernels read in FP32, made again when a parameter has changed.  A copy is
// made on the stream of the call that misses it: the first call on another stream waits for it there and keeps its
// memory from being used again too early.  While a graph is captured nothing is kept (a conversion then belongs to the graph) and nothing
// is waited for (a capture begins behind a synchronisation).
struct Fp32Copies {
    struct Entry {
        const void* ptr = nullptr;
        int64_t version = -1;
        Tensor copy;
        std::vector<c10::Stream> ordered;   // streams whose work follows the conversion
        std::shared_ptr<c10::Event> made;
    };
    std::vector<Entry> entries;
    static bool capturing() {
        return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
    }
    Tensor get(size_t slot, const Tensor& t) {
        if (t.scalar_type() == at::kFloat && t.is_contiguous()) return t.detach();
        if (entries.size() <= slot) entries.resize(slot + 1);
        Entry& e = entries[slot];
        const bool cuda = t.is_cuda();
        if (e.ptr != t.data_ptr() || e.version != (int64_t)t._version()) {
            if (cuda && capturing()) return f32_contiguous(t);
            e.copy = f32_contiguous(t);
            e.ptr = t.data_ptr();
            e.version = (int64_t)t._version();
            e.ordered.clear();
            if (cuda) {
                e.ordered.push_back(c10::cuda::getCurrentCUDAStream(t.device().index()));
                e.made = std::make_shared<c10::Event>(c10::DeviceType::CUDA);
                e.made->record(e.ordered.front());
            }
        } else if (cuda) {
            const c10::Stream now = c10::cuda::getCurrentCUDAStream(t.device().index());
            if (std::find(e.ordered.begin(), e.ordered.end(), now) == e.ordered.end() && !capturing()) {
                e.made->block(now);
                e.copy.record_stream(now);
                if (e.ordered.size() < 16) e.ordered.push_back(now);   // past that a call waits each time
            }
        }
        return e.copy;
    }
};

// ---- depthwise causal conv (4 taps) + SiLU ------------------------------------------------------------------
Tensor conv_forward(const Tensor& x, const Tensor& w32, const Tensor& init, Tensor fin, const Tensor& valid,
                    const Tensor& reset) {
    const c10::cuda::CUDAGuard guard(x.device());
    Tensor y = bf16_like(x, x.sizes());
    sd_conv4_forward_args a{};
    a.B = (int32_t)x.size(0); a.T = (int32_t)x.size(1); a.D = (int32_t)x.size(2);
    a.x = x.data_ptr(); a.x_stride_b = x.stride(0); a.x_stride_t = x.stride(1);
    a.weight = f32(w32);
    a.initial_state = raw(init); a.y = y.data_ptr(); a.final_state = raw(fin);
    a.valid_mask = bytes(valid); a.reset_mask = bytes(reset);
    check(sd_conv4_silu_forward(&a, stream_of(x)));
    return y;
}

struct ConvFunction : torch::autograd::Function<ConvFunction> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const OptTensor& init_in,
                                 bool want_state, const OptTensor& valid, const OptTensor& reset) {
        const Tensor w32 = f32_contiguous(weight);
        const Tensor init = init_in.has_value() ? bf16_contiguous(init_in->detach()) : Tensor();
        Tensor fin = want_state ? bf16_like(x, {x.size(0), x.size(2), 3}) : Tensor();
        const Tensor y = conv_forward(x, w32, init, fin, given(valid), given(reset));
        ctx->save_for_backward({x, w32, init, given(valid), given(reset)});
        ctx->saved_data["dtype"] = (int64_t)weight.scalar_type();
        ctx->set_materialize_grads(false);
        if (!want_state) return {y};
        ctx->mark_non_differentiable({fin});
        return {y, fin};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        const Tensor &x = sv[0], &w32 = sv[1], &init = sv[2];
        const auto dtype = (at::ScalarType)ctx->saved_data["dtype"].toInt();
        const int64_t B = x.size(0), T = x.size(1), D = x.size(2);
        const c10::cuda::CUDAGuard guard(x.device());
        if (!grads[0].defined())
            return {at::zeros_like(x), at::zeros({D, 4}, x.options().dtype(dtype)), Tensor(), Tensor(), Tensor(), Tensor()};
        const Tensor dy = bf16_contiguous(grads[0]);
        Tensor dx = bf16_like(x, x.sizes()), dw = f32_like(x, {D, 4});
        Tensor dinit = init.defined() ? bf16_like(x, {B, D, 3}) : Tensor();
        const Tensor scratch = workspace(x, sd_conv4_backward_scratch_bytes((int32_t)B, (int32_t)T, (int32_t)D));
        sd_conv4_backward_args a{};
        a.B = (int32_t)B; a.T = (int32_t)T; a.D = (int32_t)D;
        a.x = x.data_ptr(); a.x_stride_b = x.stride(0); a.x_stride_t = x.stride(1);
        a.weight = f32(w32); a.initial_state = raw(init);
        a.dy = dy.data_ptr(); a.dx = dx.data_ptr(); a.dweight = f32(dw); a.dinitial_state = raw(dinit);
        a.scratch = scratch.data_ptr(); a.scratch_bytes = (size_t)scratch.numel();
        a.valid_mask = bytes(sv[3]); a.reset_mask = bytes(sv[4]);
        check(sd_conv4_silu_backward(&a, stream_of(x)));
        return {dx, dw.to(dtype), dinit, Tensor(), Tensor(), Tensor()};
    }
};

OptTensor conv_mask(const char* name, const OptTensor& mask, const Tensor& x) {
    if (!mask.has_value()) return std::nullopt;
    if (mask->scalar_type() != at::kBool || !is_shape(*mask, {x.size(0), x.size(1)}))
        throw py::value_error(std::string(name) + " must be bool [B,T]");
    value_error(mask->device() != x.device(), "masks must share the activation device");
    return mask->contiguous();
}

// (y, final state or undefined)
std::pair<Tensor, Tensor> conv(const Tensor& x, const Tensor& weight, const OptTensor& init, bool want_state,
                               const OptTensor& valid_in, const OptTensor& reset_in, bool inplace_state) {
    require_bf16_cuda("x", x);
    value_error(x.dim() != 3 || x.stride(-1) != 1, "x must be [B,T,D] with unit channel stride");
    value_error(!is_shape(weight, {x.size(2), 4}), "conv weight must have shape [D,4]");
    value_error(init.has_value() && !is_shape(*init, {x.size(0), x.size(2), 3}), "conv initial state must have shape [B,D,3]");
    const OptTensor valid = conv_mask("valid_mask", valid_in, x), reset = conv_mask("reset_mask", reset_in, x);
    if (x.size(1) == 0) {
        Tensor fin;
        if (want_state) fin = init.has_value() ? init->to(at::kBFloat16) : at::zeros({x.size(0), x.size(2), 3}, x.options());
        return {at::zeros(x.sizes(), x.options()), fin};
    }
    const Tensor init_t = given(init);
    if (!records_gradients({&x, &weight, &init_t})) {
        // a cache that owns its state may have a single-token step update it in place: a thread reads the three
        // entries of its channels before it writes them
        const bool inplace = inplace_state && want_state && init.has_value() && x.size(1) == 1 &&
                             !at::GradMode::is_enabled() && !valid.has_value() && !reset.has_value() &&
                             init->scalar_type() == at::kBFloat16 && init->is_contiguous();
        const Tensor state = init.has_value() ? bf16_contiguous(init->detach()) : Tensor();
        Tensor fin = inplace ? state : want_state ? bf16_like(x, {x.size(0), x.size(2), 3}) : Tensor();
        return {conv_forward(x.detach(), f32_contiguous(weight), state, fin, given(valid), given(reset)), fin};
    }
    const variable_list out = ConvFunction::apply(x, weight, init, want_state, valid, reset);
    return {out[0], want_state ? out[1] : Tensor()};
}

py::tuple conv4_silu(const Tensor& x, const Tensor& weight, const OptTensor& init, bool want_state,
                     const OptTensor& valid, const OptTensor& reset, bool inplace_state) {
    const auto [y, fin] = conv(x, weight, init, want_state, valid, reset, inplace_state);
    if (!fin.defined()) return py::make_tuple(y, py::none());
    return py::make_tuple(y, fin);
}

// ---- decay gate ---------------------------------------------------------------------------------------------
Tensor gate_forward(const Tensor& raw_in, const Tensor& A, const Tensor& b) {
    const c10::cuda::CUDAGuard guard(raw_in.device());
    const int64_t H = raw_in.size(-2), r = raw_in.size(-1);
    Tensor out = f32_like(raw_in, raw_in.sizes());
    sd_kda_gate_args a{};
    a.rows = raw_in.numel() / (H * r); a.H = (int32_t)H; a.r = (int32_t)r;
    a.raw = raw_in.data_ptr(); a.log_rate = f32(A); a.bias = f32(b); a.log_decay = f32(out);
    check(sd_kda_gate_forward(&a, stream_of(raw_in)));
    return out;
}

struct GateFunction : torch::autograd::Function<GateFunction> {
    static Tensor forward(AutogradContext* ctx, const Tensor& raw_in, const Tensor& log_rate, const Tensor& bias) {
        const Tensor x = raw_in.contiguous(), A = f32_contiguous(log_rate), b = f32_contiguous(bias);
        ctx->save_for_backward({x, A, b});
        ctx->saved_data["rate_shape"] = log_rate.sizes().vec();
        ctx->saved_data["bias_shape"] = bias.sizes().vec();
        ctx->saved_data["rate_dtype"] = (int64_t)log_rate.scalar_type();
        ctx->saved_data["bias_dtype"] = (int64_t)bias.scalar_type();
        return gate_forward(x, A, b);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        const Tensor& x = sv[0];
        const int64_t H = x.size(-2), r = x.size(-1), rows = x.numel() / (H * r);
        const c10::cuda::CUDAGuard guard(x.device());
        const Tensor dout = grads[0].to(at::kFloat).contiguous();
        Tensor dx = at::empty_like(x), dA = f32_like(x, {H}), db = f32_like(x, {H, r});
        const Tensor scratch = workspace(x, sd_kda_gate_backward_scratch_bytes(rows, (int32_t)H, (int32_t)r));
        sd_kda_gate_args a{};
        a.rows = rows; a.H = (int32_t)H; a.r = (int32_t)r;
        a.raw = x.data_ptr(); a.log_rate = f32(sv[1]); a.bias = f32(sv[2]); a.dlog_decay = f32(dout);
        a.draw = dx.data_ptr(); a.dlog_rate = f32(dA); a.dbias = f32(db);
        a.scratch = scratch.data_ptr(); a.scratch_bytes = (size_t)scratch.numel();
        check(sd_kda_gate_backward(&a, stream_of(x)));
        return {dx, dA.reshape(ctx->saved_data["rate_shape"].toIntVector()).to((at::ScalarType)ctx->saved_data["rate_dtype"].toInt()),
                db.reshape(ctx->saved_data["bias_shape"].toIntVector()).to((at::ScalarType)ctx->saved_data["bias_dtype"].toInt())};
    }
};

Tensor kda_decay_gate(const Tensor& raw_in, const Tensor& log_rate, const Tensor& bias) {
    require_bf16_cuda("raw", raw_in);
    const int64_t H = raw_in.size(-2), r = raw_in.size(-1);
    value_error(log_rate.numel() != H || bias.numel() != H * r, "log_rate must have H entries and bias H*r entries");
    if (!records_gradients({&raw_in, &log_rate, &bias}))
        return gate_forward(raw_in.detach().contiguous(), f32_contiguous(log_rate), f32_contiguous(bias));
    return GateFunction::apply(raw_in, log_rate, bias);
}

// ---- sigmoid-gated RMSNorm, alone and in front of a projection ----------------------------------------------
Tensor norm_gate_forward(const Tensor& x, const Tensor& gate, const Tensor& w, double eps) {
    const c10::cuda::CUDAGuard guard(x.device());
    Tensor y = bf16_like(x, x.sizes());
    sd_norm_gate_args a{};
    a.V = (int32_t)x.size(-1); a.rows = x.numel() / a.V; a.eps = (float)eps;
    a.x = x.data_ptr(); a.gate = gate.data_ptr(); a.weight = f32(w); a.y = y.data_ptr();
    check(sd_norm_gate_forward(&a, stream_of(x)));
    return y;
}

// (dx, dgate, dweight FP32)
std::array<Tensor, 3> norm_gate_backward(const Tensor& x, const Tensor& gate, const Tensor& w, double eps, const Tensor& dy) {
    Tensor dx = at::empty_like(x), dg = at::empty_like(gate), dw = f32_like(x, {x.size(-1)});
    sd_norm_gate_args a{};
    a.V = (int32_t)x.size(-1); a.rows = x.numel() / a.V; a.eps = (float)eps;
    const Tensor scratch = workspace(x, sd_norm_gate_backward_scratch_bytes(a.rows, a.V));
    a.x = x.data_ptr(); a.gate = gate.data_ptr(); a.weight = f32(w); a.dy = dy.data_ptr();
    a.dx = dx.data_ptr(); a.dgate = dg.data_ptr(); a.dweight = f32(dw);
    a.scratch = scratch.data_ptr(); a.scratch_bytes = (size_t)scratch.numel();
    check(sd_norm_gate_backward(&a, stream_of(x)));
    return {dx, dg, dw};
}

struct NormGateFunction : torch::autograd::Function<NormGateFunction> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x_in, const Tensor& gate_in, const Tensor& weight, double eps) {
        const Tensor x = x_in.contiguous(), gate = gate_in.contiguous(), w = f32_contiguous(weight);
        ctx->save_for_backward({x, gate, w});
        ctx->saved_data["eps"] = eps;
        ctx->saved_data["dtype"] = (int64_t)weight.scalar_type();
        return norm_gate_forward(x, gate, w, eps);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        const c10::cuda::CUDAGuard guard(sv[0].device());
        const auto [dx, dg, dw] =
            norm_gate_backward(sv[0], sv[1], sv[2], ctx->saved_data["eps"].toDouble(), bf16_contiguous(grads[0]));
        return {dx, dg, dw.to((at::ScalarType)ctx->saved_data["dtype"].toInt()), Tensor()};
    }
};

// Gated RMSNorm in front of a projection.  The normalised panel is not kept for the reverse pass: it is produced again
// from x and gate there (one more pass of the norm kernel instead of a saved [..., H*D] BF16 tensor per layer).
// causallsso/ops/norm_gate.py:46-159
Tensor norm_linear_forward(const Tensor& x, const Tensor& gate, const Tensor& w, const Tensor& packed, const Tensor& bias, double eps) {
    return at::linear(norm_gate_forward(x, gate, w, eps).flatten(-2), packed,
                      bias.defined() ? OptTensor(bias.detach().to(at::kBFloat16)) : OptTensor());
}
// (dx, dgate, dweight of the norm FP32, dweight of the projection BF16, dbias FP32 or undefined)
std::array<Tensor, 5> norm_linear_backward(const Tensor& x, const Tensor& gate, const Tensor& w, const Tensor& packed, bool bias,
                                           double eps, const Tensor& dout_in) {
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor dout = dout_in.to(at::kBFloat16).reshape({-1, dout_in.size(-1)});
    Tensor dlinear;
    {
        const Tensor y = norm_gate_forward(x, gate, w, eps);   // regenerated, not saved
        dlinear = at::mm(dout.t(), y.view({dout.size(0), -1}));
    }
    const auto [dx, dg, dw] = norm_gate_backward(x, gate, w, eps, at::mm(dout, packed).view(x.sizes()));
    return {dx, dg, dw, dlinear, bias ? dout.to(at::kFloat).sum(0) : Tensor()};
}

struct NormGateLinearFunction : torch::autograd::Function<NormGateLinearFunction> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x_in, const Tensor& gate_in, const Tensor& norm_weight,
                          const Tensor& weight, const OptTensor& bias, double eps) {
        const Tensor x = x_in.contiguous(), gate = gate_in.contiguous(), w = f32_contiguous(norm_weight);
        const Tensor packed = weight.detach().to(at::kBFloat16);
        ctx->save_for_backward({x, gate, w, packed});
        ctx->saved_data["eps"] = eps;
        ctx->saved_data["norm_dtype"] = (int64_t)norm_weight.scalar_type();
        ctx->saved_data["weight_dtype"] = (int64_t)weight.scalar_type();
        ctx->saved_data["bias_dtype"] = bias.has_value() ? (int64_t)bias->scalar_type() : (int64_t)-1;
        ctx->set_materialize_grads(false);
        return norm_linear_forward(x, gate, w, packed, given(bias), eps);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
        const variable_list sv = ctx->get_saved_variables();
        const int64_t bias_dtype = ctx->saved_data["bias_dtype"].toInt();
        auto [dx, dg, dw, dlinear, dbias] = norm_linear_backward(sv[0], sv[1], sv[2], sv[3], bias_dtype >= 0,
                                                                 ctx->saved_data["eps"].toDouble(), grads[0]);
        if (dbias.defined()) dbias = dbias.to((at::ScalarType)bias_dtype);
        return {dx, dg, dw.to((at::ScalarType)ctx->saved_data["norm_dtype"].toInt()),
                dlinear.to((at::ScalarType)ctx->saved_data["weight_dtype"].toInt()), dbias, Tensor()};
    }
};

void norm_gate_checks(const Tensor& x, const Tensor& gate, const Tensor& weight) {
    require_bf16_cuda("x", x);
    require_bf16_cuda("gate", gate);
    value_error(x.sizes() != gate.sizes() || x.dim() < 2, "x and gate must have the same [...,H,D] shape");
    value_error(!is_shape(weight, {x.size(-1)}), "weight must have shape [D]");
}

Tensor rms_norm_gated(const Tensor& x, const Tensor& gate, const Tensor& weight, double eps) {
    norm_gate_checks(x, gate, weight);
    if (!records_gradients({&x, &gate, &weight}))
        return norm_gate_forward(x.detach().contiguous(), gate.detach().contiguous(), f32_contiguous(weight), eps);
    return NormGateFunction::apply(x, gate, weight, eps);
}

Tensor rms_norm_gated_linear(const Tensor& x, const Tensor& gate, const Tensor& norm_weight, const Tensor& weight,
                             const OptTensor& bias, double eps) {
    norm_gate_checks(x, gate, norm_weight);
    value_error(weight.dim() != 2 || weight.size(1) != x.size(-2) * x.size(-1), "the linear layer must take the flattened [H*D] rows");
    const Tensor b = given(bias);
    if (!records_gradients({&x, &gate, &norm_weight, &weight, &b}))
        return norm_linear_forward(x.detach().contiguous(), gate.detach().contiguous(), f32_contiguous(norm_weight),
                                   weight.detach().to(at::kBFloat16), b, eps);
    return NormGateLinearFunction::apply(x, gate, norm_weight, weight, bias, eps);
}

// The two halves above for the node of rms_norm_gated_linear (mixer_ops.py), whose saved tensors callers can list.
Tensor norm_linear_raw(const Tensor& x, const Tensor& gate, const Tensor& norm_weight, const Tensor& weight, const OptTensor& bias,
                       double eps) {
    norm_gate_checks(x, gate, norm_weight);
    value_error(weight.dim() != 2 || weight.size(1) != x.size(-2) * x.size(-1), "the linear layer must take the flattened [H*D] rows");
    return norm_linear_forward(x, gate, norm_weight, weight, given(bias), eps);
}
std::vector<OptTensor> norm_linear_raw_backward(const Tensor& x, const Tensor& gate, const Tensor& w, const Tensor& weight, bool bias,
                                                double eps, const Tensor& dout) {
    std::vector<OptTensor> out;
    for (const Tensor& t : norm_linear_backward(x, gate, w, weight, bias, eps, dout)) out.push_back(optional(t));
    return out;
}

// ---- residual add + RMSNorm ---------------------------------------------------------------------------------
bool addnorm_reverse_ok(int64_t width) { return width > 0 && width % 256 == 0 && width <= 2048; }

// (sum or undefined when delta is, normed)
std::pair<Tensor, Tensor> addnorm_forward(const Tensor& x, const Tensor& delta, const Tensor& w, double eps) {
    const c10::cuda::CUDAGuard guard(x.device());
    Tensor normed = at::empty_like(x), total = delta.defined() ? at::empty_like(x) : Tensor();
    sd_add_rmsnorm_args a{};
    a.D = (int32_t)x.size(-1); a.rows = x.numel() / a.D; a.eps = (float)eps;
    a.x = x.data_ptr(); a.delta = raw(delta); a.weight = f32(w); a.sum = raw(total); a.normed = normed.data_ptr();
    check(sd_add_rmsnorm(&a, stream_of(x)));
    return {total, normed};
}

// (x + delta, RMSNorm(x + delta) * weight) with one reverse kernel: the cotangents of both outputs become the single
// gradient that x and delta share, plus the weight gradient.  Only the sum is saved.  Without delta the sum is x itself
// and only the norm is returned.
struct AddNormFunction : torch::autograd::Function<AddNormFunction> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x_in, const OptTensor& delta_in, const Tensor& weight,
                                 double eps) {
        const Tensor x = x_in.contiguous(), delta = delta_in.has_value() ? delta_in->contiguous() : Tensor();
        const Tensor w = f32_contiguous(weight);
        const auto [total, normed] = addnorm_forward(x, delta, w, eps);
        ctx->save_for_backward({delta.defined() ? total : x, w});
        ctx->saved_data["eps"] = eps;
        ctx->saved_data["delta"] = delta.defined();
        ctx->saved_data["dtype"] = (int64_t)weight.scalar_type();
        ctx->set_materialize_grads(false);
        if (!delta.defined()) return {normed};
        return {total, normed};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        const Tensor &total = sv[0], &w = sv[1];
        const bool has_delta = ctx->saved_data["delta"].toBool();
        const Tensor dtotal = has_delta ? grads[0] : Tensor(), dnormed = grads.back();
        if (!dnormed.defined()) return {dtotal, has_delta ? dtotal : Tensor(), Tensor(), Tensor()};
        const c10::cuda::CUDAGuard guard(total.device());
        const Tensor dn = bf16_contiguous(dnormed), dt = dtotal.defined() ? bf16_contiguous(dtotal) : Tensor();
        Tensor dx = at::empty_like(total), dw = f32_like(total, {total.size(-1)});
        sd_add_rmsnorm_backward_args a{};
        a.D = (int32_t)total.size(-1); a.rows = total.numel() / a.D; a.eps = (float)ctx->saved_data["eps"].toDouble();
        const Tensor scratch = workspace(total, sd_add_rmsnorm_backward_scratch_bytes(a.rows, a.D));
        a.sum = total.data_ptr(); a.weight = f32(w); a.dsum = raw(dt); a.dnormed = dn.data_ptr(); a.dx = dx.data_ptr();
        a.dweight = f32(dw); a.scratch = scratch.data_ptr(); a.scratch_bytes = (size_t)scratch.numel();
        check(sd_add_rmsnorm_backward(&a, stream_of(total)));
        return {dx, has_delta ? dx : Tensor(), dw.to((at::ScalarType)ctx->saved_data["dtype"].toInt()), Tensor()};
    }
};

py::tuple add_rmsnorm(const Tensor& x, const OptTensor& delta_in, const Tensor& weight, double eps) {
    require_bf16_cuda("x", x);
    const Tensor delta = given(delta_in);
    if (delta.defined()) {
        require_bf16_cuda("delta", delta);
        value_error(x.sizes() != delta.sizes(), "x and delta must share a shape [...,D]");
    }
    value_error(!is_shape(weight, {x.size(-1)}), "weight must be [D]");
    const bool reverse_ok = addnorm_reverse_ok(x.size(-1));
    if (records_gradients({&x, &weight, &delta})) {
        value_error(!reverse_ok, "the reverse pass takes rows of 256, 512, ..., 2048 channels");
        const variable_list out = AddNormFunction::apply(x, delta_in, weight, eps);
        return delta.defined() ? py::make_tuple(out[0], out[1]) : py::make_tuple(x, out[0]);
    }
    value_error(weight.scalar_type() != at::kFloat, "weight must be FP32 [D]");
    value_error(!delta.defined() && !reverse_ok, "the norm alone takes rows of 256, 512, ..., 2048 channels");
    const auto [total, normed] = addnorm_forward(x.detach().contiguous(), delta.defined() ? delta.detach().contiguous() : delta,
                                                 weight.detach().contiguous(), eps);
    return py::make_tuple(delta.defined() ? total : x, normed);
}

// ---- gated MLP ----------------------------------------------------------------------------------------------
Tensor swiglu_forward(const Tensor& gv) {
    const c10::cuda::CUDAGuard guard(gv.device());
    std::vector<int64_t> shape = gv.sizes().vec();
    shape.back() /= 2;
    Tensor out = bf16_like(gv, shape);
    sd_swiglu_args a{};
    a.I = (int32_t)shape.back(); a.rows = out.numel() / a.I; a.gate_value = gv.data_ptr(); a.out = out.data_ptr();
    check(sd_swiglu(&a, stream_of(gv)));
    return out;
}

struct SwigluFunction : torch::autograd::Function<SwigluFunction> {
    static Tensor forward(AutogradContext* ctx, const Tensor& gate_value) {
        const Tensor gv = gate_value.contiguous();
        ctx->save_for_backward({gv});
        return swiglu_forward(gv);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const Tensor gv = ctx->get_saved_variables()[0];
        const c10::cuda::CUDAGuard guard(gv.device());
        const Tensor dout = bf16_contiguous(grads[0]);
        Tensor dgv = at::empty_like(gv);
        sd_swiglu_args a{};
        a.I = (int32_t)(gv.size(-1) / 2); a.rows = gv.numel() / (2 * a.I);
        a.gate_value = gv.data_ptr(); a.dout = dout.data_ptr(); a.dgate_value = dgv.data_ptr();
        check(sd_swiglu_backward(&a, stream_of(gv)));
        return {dgv};
    }
};

Tensor swiglu(const Tensor& gate_value) {
    require_bf16_cuda("gate_value", gate_value);
    value_error(gate_value.size(-1) % 2 != 0, "the last axis must hold gate and value halves");
    if (records_gradients({&gate_value})) return SwigluFunction::apply(gate_value);
    return swiglu_forward(gate_value.detach().contiguous());
}

constexpr int64_t GEMV_MAX_ROWS = 4;
bool aligned16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }

// The projection of a cached single-token step in k_token_linear, or undefined when the call is not one it takes.
Tensor small_projection(const Tensor& x, const Tensor& weight, const Tensor& bias, bool with_swiglu) {
    if (!x.is_cuda() || x.scalar_type() != at::kBFloat16 || weight.scalar_type() != at::kBFloat16 || weight.dim() != 2) return {};
    const int64_t K = x.size(-1), N = weight.size(0);
    const int64_t rows = K > 0 ? x.numel() / K : 0;
    if (rows < 1 || rows > GEMV_MAX_ROWS || x.stride(-1) != 1 || records_gradients({&x, &weight})) return {};
    if (weight.size(1) != K || !weight.is_contiguous() || weight.device() != x.device() || K % 8 != 0 ||
        (bias.defined() && (bias.scalar_type() != at::kBFloat16 || !bias.is_contiguous())))
        return {};
    const Tensor x2 = x.reshape({rows, K});   // a view for the layouts a decode step produces
    const int64_t stride = rows > 1 ? x2.stride(0) : K;
    if (stride % 8 != 0 || !aligned16(x2) || !aligned16(weight) || (with_swiglu && N % 2 != 0)) return {};
    const c10::cuda::CUDAGuard guard(x.device());
    std::vector<int64_t> shape = x.sizes().vec();
    shape.back() = with_swiglu ? N / 2 : N;
    Tensor out = bf16_like(x, shape);
    sd_gemv_args a{};
    a.M = (int32_t)rows; a.N = (int32_t)N; a.K = (int32_t)K; a.swiglu = with_swiglu ? 1 : 0;
    a.x = x2.data_ptr(); a.x_stride = stride; a.weight = weight.data_ptr(); a.bias = raw(bias);
    a.y = out.data_ptr(); a.y_stride = shape.back();
    check(sd_gemv(&a, stream_of(x)));
    return out;
}

std::optional<Tensor> small_linear(const Tensor& x, const Tensor& weight, const OptTensor& bias, bool with_swiglu) {
    return optional(small_projection(x, weight, given(bias), with_swiglu));
}

// x W^T (+ b) in the activation's type: the small kernel for a few rows, else the library product
Tensor projection(const Tensor& x, const Tensor& weight_in, const OptTensor& bias_in) {
    const Tensor weight = weight_in.to(x.scalar_type()), bias = bias_in.has_value() ? bias_in->to(x.scalar_type()) : Tensor();
    const Tensor small = small_projection(x, weight, bias, false);
    if (small.defined()) return small;
    if (!bias.defined()) return at::linear(x, weight);
    // one GEMM with the bias in its epilogue: on a strided slice of the projection row at::linear would run the product
    // and a separate element-wise add
    std::vector<int64_t> shape = x.sizes().vec();
    shape.back() = weight.size(0);
    return at::addmm(bias, x.reshape({-1, x.size(-1)}), weight.t()).view(shape);
}

Tensor gated_mlp(const Tensor& x, const Tensor& up, const OptTensor& up_bias, const Tensor& down, const OptTensor& down_bias) {
    // a cached single-token step: projection + activation in one launch, then the second projection
    Tensor act = small_projection(x, up, given(up_bias), true);
    if (!act.defined()) act = swiglu(at::linear(x, up, up_bias));   // activation and product in one kernel
    const Tensor out = small_projection(act, down, given(down_bias), false);
    return out.defined() ? out : at::linear(act, down, down_bias);
}

// ---- slices of the fused projection row ---------------------------------------------------------------------
// One BF16 row-shaped tensor holding `pieces` side by side (undefined: zeros), or undefined when the layout is not one
// the kernel takes.
Tensor pack(const variable_list& pieces, at::IntArrayRef widths, at::IntArrayRef row_shape, at::TensorOptions options) {
    const int64_t P = row_shape.back();
    if (!options.device().is_cuda() || widths.size() > SD_PACK_MAX_PIECES || P % 8 != 0) return {};
    sd_pack_rows_args a{};
    variable_list held(pieces.size());
    for (size_t k = 0; k < widths.size(); ++k) {
        if (widths[k] % 8 != 0 || (pieces[k].defined() && pieces[k].scalar_type() != at::kBFloat16)) return {};
        if (pieces[k].defined()) held[k] = pieces[k].contiguous();
        a.piece[k].src = raw(held[k]);
        a.piece[k].width = (int32_t)widths[k];
    }
    const c10::cuda::CUDAGuard guard(options.device());
    Tensor out = at::empty(row_shape, options.dtype(at::kBFloat16));
    a.rows = out.numel() / P; a.pieces = (int32_t)widths.size(); a.row_width = (int32_t)P; a.dst = out.data_ptr();
    check(sd_pack_rows(&a, stream_of(out)));
    return out;
}

std::optional<Tensor> pack_rows(const std::vector<OptTensor>& pieces, const std::vector<int64_t>& widths,
                                const std::vector<int64_t>& row_shape, const at::Device& device) {
    variable_list list;
    for (const OptTensor& p : pieces) list.push_back(given(p));
    return optional(pack(list, widths, row_shape, at::TensorOptions().device(device)));
}

// Slices of the fused projection row as views (no copy), with a reverse pass that writes every slice gradient once into
// one row-shaped buffer.  Plain slicing would make autograd allocate and add one zero-filled full row per slice (ten
// rows of 7488 columns per token for the mixer).
variable_list row_slices(const Tensor& row, at::IntArrayRef sizes) {
    variable_list pieces;
    int64_t start = 0;
    for (const int64_t size : sizes) {
        pieces.push_back(row.narrow(-1, start, size));
        start += size;
    }
    return pieces;
}

struct SplitRowFunction : torch::autograd::Function<SplitRowFunction> {
    static variable_list forward(AutogradContext* ctx, const Tensor& row, std::vector<int64_t> sizes) {
        ctx->saved_data["sizes"] = sizes;
        ctx->saved_data["shape"] = row.sizes().vec();
        ctx->saved_data["dtype"] = (int64_t)row.scalar_type();
        ctx->saved_data["device"] = row.device();
        ctx->set_materialize_grads(false);
        return row_slices(row, sizes);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const std::vector<int64_t> sizes = ctx->saved_data["sizes"].toIntVector(), shape = ctx->saved_data["shape"].toIntVector();
        const auto options = at::TensorOptions().device(ctx->saved_data["device"].toDevice())
                                 .dtype((at::ScalarType)ctx->saved_data["dtype"].toInt());
        bool any = false;
        for (const Tensor& g : grads) any = any || g.defined();
        if (!any) return {Tensor(), Tensor()};
        if (options.dtype() == at::kBFloat16) {
            const Tensor packed = pack(grads, sizes, shape, options);   // one kernel for the whole row
            if (packed.defined()) return {packed, Tensor()};
        }
        Tensor drow = at::empty(shape, options);
        int64_t start = 0;
        for (size_t k = 0; k < sizes.size(); ++k) {
            Tensor target = drow.narrow(-1, start, sizes[k]);
            if (grads[k].defined()) target.copy_(grads[k]); else target.zero_();
            start += sizes[k];
        }
        if (start < shape.back()) drow.narrow(-1, start, shape.back() - start).zero_();   // padding of the projection
        return {drow, Tensor()};
    }
};

// ---- the mixer around the operator --------------------------------------------------------------------------
struct MixerShape {
    int64_t heads, width, value_width;
    // q | k | v stay one slice when they go through the conv, which reads it in place
    std::vector<int64_t> sizes(bool conv) const {
        const int64_t hr = heads * width, hv = heads * value_width;
        if (conv) return {2 * hr + hv, hr, hr, hr, hv, heads, value_width, value_width};
        return {hr, hr, hv, hr, hr, hr, hv, heads, value_width, value_width};
    }
};

// From the hidden rows to the operator's operands: fused projection, conv4 + SiLU, decay gate, geometry rate, output
// gate.  Returns (u, h, q, keys, values, log_decay, erase_raw, write_raw, geometry_write, output_gate, conv state |
// None).  causallsso/model.py:321-394
py::tuple mixer_front(const Tensor& x, int64_t heads, int64_t width, int64_t value_width, const Tensor& in_weight,
                      const OptTensor& in_bias, const OptTensor& conv_weight, const OptTensor& conv_state,
                      const OptTensor& valid, const OptTensor& reset, bool want_state, bool inplace_state,
                      const Tensor& decay_weight, const Tensor& gate_weight, const OptTensor& gate_bias,
                      const Tensor& log_rate, const Tensor& decay_bias, const Tensor& geometry_bias, bool geometry_enabled,
                      bool decay_enabled) {
    const MixerShape shape{heads, width, value_width};
    const bool with_conv = conv_weight.has_value();
    const std::vector<int64_t> sizes = shape.sizes(with_conv);
    const Tensor row = projection(x, in_weight, in_bias);   // [B,T,P], slices stay views
    const variable_list piece = records_gradients({&row}) ? SplitRowFunction::apply(row, sizes) : row_slices(row, sizes);
    const auto view = [&](const Tensor& t, int64_t w) { return t.unflatten(-1, {heads, w}); };
    Tensor q, k, v, fin;
    size_t at = 1;
    if (with_conv) {
        const auto [qkv, state] = conv(piece[0], *conv_weight, conv_state, want_state, valid, reset, inplace_state);
        fin = state;
        const variable_list parts = qkv.split_with_sizes({heads * width, heads * width, heads * value_width}, -1);
        q = parts[0]; k = parts[1]; v = parts[2];
    } else {
        q = at::silu(piece[0]); k = at::silu(piece[1]); v = at::silu(piece[2]);
        at = 3;
    }
    const Tensor decay_raw = view(projection(piece[at + 5], decay_weight, std::nullopt), width);
    const Tensor output_gate = view(projection(piece[at + 6], gate_weight, gate_bias), value_width);
    Tensor log_decay = kda_decay_gate(decay_raw, log_rate, decay_bias);
    Tensor geometry = at::sigmoid(piece[at + 4].to(at::kFloat) + geometry_bias.to(at::kFloat).view({1, 1, heads}));
    if (!geometry_enabled) geometry = at::zeros_like(geometry);
    if (!decay_enabled) log_decay = at::zeros_like(log_decay);
    return py::make_tuple(view(piece[at], width), view(piece[at + 1], width), view(q, width), view(k, width).unsqueeze(-2),
                          view(v, value_width).unsqueeze(-2), log_decay, view(piece[at + 2], width).unsqueeze(-2),
                          view(piece[at + 3], value_width).unsqueeze(-2), geometry, output_gate,
                          fin.defined() ? py::cast(fin) : py::none());
}

// Where the slices of the projection row stand, and the operator's operands on that row and on the conv's output.
struct RowPlan {
    int64_t B, T, H, r, V, P;   // P: columns of the row
    int64_t conv() const { return 2 * H * r + H * V; }           // q | k | v, then u, h, erase, write
    int64_t geometry() const { return conv() + 3 * H * r + H * V; }
    int64_t decay_hidden() const { return geometry() + H; }
    int64_t gate_hidden() const { return decay_hidden() + V; }
    int64_t used() const { return gate_hidden() + V; }
    sd_shape shape() const { return sd_shape{(int32_t)B, (int32_t)T, (int32_t)H, (int32_t)r, (int32_t)V}; }
    template <class Args>
    void fill(Args& a, const void* row, const void* qkv, const void* log_decay, const void* rate) const {
        a.shape = shape();
        const auto on_row = [&](int64_t col, int64_t w) { return sd_operand{static_cast<const char*>(row) + 2 * col, T * P, P, w}; };
        const int64_t D = conv();
        const auto on_conv = [&](int64_t col, int64_t w) { return sd_operand{static_cast<const char*>(qkv) + 2 * col, T * D, D, w}; };
        a.u = on_row(D, r); a.h = on_row(D + H * r, r);
        a.erase_raw = on_row(D + 2 * H * r, r); a.write_raw = on_row(D + 3 * H * r, V);
        a.q = on_conv(0, r); a.keys = on_conv(H * r, r); a.values = on_conv(2 * H * r, V);
        a.log_decay = sd_operand{log_decay, T * H * r, H * r, r};
        a.gamma = sd_operand{rate, T * H, H, 1};
    }
};

// The whole layer as one autograd node: what its separate nodes do, on the same kernels.  One node because the separate
// ones cost the host 1.2 ms a training call, more than the device needs below some four thousand tokens, and because
// the reverse pass knows where every gradient belongs: the operator's kernels write dq, dk, dv straight into the conv's
// cotangent rows and du, dh, d erase, d write into the projection row's gradient, the conv and the two small products
// write their columns of it, and no kernel gathers them (130 us of 3250 at 8 x 2048 tokens of width 1024).
struct MixerFunction : torch::autograd::Function<MixerFunction> {
    static RowPlan plan(const Tensor& x, int64_t H, int64_t r, int64_t V, const Tensor& in_weight) {
        return RowPlan{x.size(0), x.size(1), H, r, V, in_weight.size(0)};
    }

    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& in_weight, const OptTensor& in_bias,
                          const Tensor& conv_weight, const Tensor& decay_weight, const Tensor& gate_weight, const OptTensor& gate_bias,
                          const Tensor& log_rate, const Tensor& decay_bias, const Tensor& geometry_bias, const Tensor& norm_weight,
                          const Tensor& out_weight, const OptTensor& out_bias, const OptTensor& valid, const OptTensor& reset,
                          int64_t heads, int64_t width, int64_t value_width, double eps) {
        const c10::cuda::CUDAGuard guard(x.device());
        const RowPlan m = plan(x, heads, width, value_width, in_weight);
        const int64_t H = m.H, r = m.r, V = m.V, P = m.P, R = m.B * m.T, Dc = m.conv();
        void* stream = stream_of(x);
        const Tensor x2 = x.view({R, x.size(2)});
        const auto product = [](const Tensor& a, const Tensor& w, const OptTensor& b) {
            return b.has_value() ? at::addmm(*b, a, w.t()) : at::mm(a, w.t());
        };
        const Tensor row = product(x2, in_weight, in_bias);
        const Tensor w32 = f32_contiguous(conv_weight), A32 = f32_contiguous(log_rate), b32 = f32_contiguous(decay_bias);
        const Tensor n32 = f32_contiguous(norm_weight);
        const Tensor qkv = bf16_like(x, {R, Dc});
        sd_conv4_forward_args c{};
        c.B = (int32_t)m.B; c.T = (int32_t)m.T; c.D = (int32_t)Dc;
        c.x = row.data_ptr(); c.x_stride_b = m.T * P; c.x_stride_t = P;
        c.weight = f32(w32); c.y = qkv.data_ptr();
        c.valid_mask = bytes(given(valid)); c.reset_mask = bytes(given(reset));
        check(sd_conv4_silu_forward(&c, stream));
        const Tensor decay_raw = product(row.narrow(1, m.decay_hidden(), V), decay_weight, std::nullopt);
        const Tensor gate = product(row.narrow(1, m.gate_hidden(), V), gate_weight, gate_bias).view({R * H, V});
        const Tensor log_decay = gate_forward(decay_raw.view({R, H, r}), A32, b32);
        const Tensor rate = at::add(row.narrow(1, m.geometry(), H), geometry_bias.to(at::kFloat)).sigmoid_();
        const sd_shape sh = m.shape();
        const Tensor y = bf16_like(x, {R * H, V}), saved = workspace(x, sd_saved_bytes(&sh));
        {
            const Tensor scratch = workspace(x, sd_forward_scratch_bytes(&sh));
            sd_forward_args a{};
            m.fill(a, row.data_ptr(), qkv.data_ptr(), log_decay.data_ptr(), rate.data_ptr());
            a.y = y.data_ptr();
            a.saved = saved.data_ptr(); a.saved_bytes = (size_t)saved.numel();
            a.scratch = scratch.data_ptr(); a.scratch_bytes = (size_t)scratch.numel();
            a.valid_mask = c.valid_mask; a.reset_mask = c.reset_mask;
            check(sd_forward(&a, stream));
        }
        const Tensor out = product(norm_gate_forward(y, gate, n32, eps).view({R, H * V}), out_weight, out_bias);
        ctx->set_materialize_grads(false);
        ctx->save_for_backward({x, in_weight, decay_weight, gate_weight, out_weight, row, qkv, decay_raw, gate, log_decay, rate, y, saved,
                                w32, A32, b32, n32, given(valid), given(reset)});
        auto& data = ctx->saved_data;
        data["heads"] = heads; data["width"] = width; data["value_width"] = value_width; data["eps"] = eps;
        data["in_bias"] = in_bias.has_value(); data["gate_bias"] = gate_bias.has_value(); data["out_bias"] = out_bias.has_value();
        data["x"] = x.requires_grad();
        const auto remember = [&](const char* name, const Tensor& t) { data[name] = (int64_t)t.scalar_type(); };
        remember("conv", conv_weight); remember("rate", log_rate); remember("decay", decay_bias);
        remember("geometry", geometry_bias); remember("norm", norm_weight);
        data["rate_shape"] = log_rate.sizes().vec(); data["decay_shape"] = decay_bias.sizes().vec();
        return out.view({m.B, m.T, out_weight.size(0)});
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        variable_list result(19);
        if (!grads[0].defined()) return result;
        // first-order gradients only, also under create_graph=True: the kernels have no second derivative, and products
        // into columns of a tensor are refused while gradients are recorded
        const at::NoGradGuard no_grad;
        const variable_list sv = ctx->get_saved_variables();
        auto& data = ctx->saved_data;
        const Tensor &x = sv[0], &in_weight = sv[1], &decay_weight = sv[2], &gate_weight = sv[3], &out_weight = sv[4], &row = sv[5];
        const Tensor &qkv = sv[6], &decay_raw = sv[7], &gate = sv[8], &log_decay = sv[9], &rate = sv[10], &y = sv[11], &saved = sv[12];
        const Tensor &w32 = sv[13], &A32 = sv[14], &b32 = sv[15], &n32 = sv[16], &valid = sv[17], &reset = sv[18];
        const c10::cuda::CUDAGuard guard(x.device());
        const double eps = data["eps"].toDouble();
        const RowPlan m = plan(x, data["heads"].toInt(), data["width"].toInt(), data["value_width"].toInt(), in_weight);
        const int64_t H = m.H, r = m.r, V = m.V, P = m.P, R = m.B * m.T, Dc = m.conv();
        void* stream = stream_of(x);
        const auto as = [&](const char* name, const Tensor& t) { return t.to((at::ScalarType)data[name].toInt()); };
        // output projection and gated norm
        const Tensor dout = grads[0].to(at::kBFloat16).reshape({R, out_weight.size(0)});
        result[11] = at::mm(dout.t(), norm_gate_forward(y, gate, n32, eps).view({R, H * V}));   // the norm is produced again
        if (data["out_bias"].toBool()) result[12] = dout.to(at::kFloat).sum(0).to(at::kBFloat16);
        const auto [dy, dgate3, dnorm] = norm_gate_backward(y, gate, n32, eps, at::mm(dout, out_weight).view({R * H, V}));
        result[10] = as("norm", dnorm);
        // the projection row's gradient, written piece by piece
        Tensor drow = bf16_like(x, {R, P});
        const Tensor dqkv = bf16_like(x, {R, Dc});
        const auto at_col = [&](const Tensor& t, int64_t col) { return static_cast<char*>(t.data_ptr()) + 2 * col; };
        const Tensor dgate = dgate3.view({R, H * V});
        Tensor piece = drow.narrow(1, m.gate_hidden(), V);
        at::mm_out(piece, dgate, gate_weight);
        result[5] = at::mm(dgate.t(), row.narrow(1, m.gate_hidden(), V));
        if (data["gate_bias"].toBool()) result[6] = dgate.sum(0);
        Tensor dld = f32_like(x, {R, H * r}), drate = f32_like(x, {R, H});
        const sd_shape sh = m.shape();
        {
            const Tensor scratch = workspace(x, sd_backward_scratch_bytes(&sh));
            sd_backward_args a{};
            m.fill(a, row.data_ptr(), qkv.data_ptr(), log_decay.data_ptr(), rate.data_ptr());
            a.dy = sd_operand{dy.data_ptr(), m.T * H * V, H * V, V};
            a.saved = saved.data_ptr(); a.saved_bytes = (size_t)saved.numel();
            a.scratch = scratch.data_ptr(); a.scratch_bytes = (size_t)scratch.numel();
            a.dq = at_col(dqkv, 0); a.dkeys = at_col(dqkv, H * r); a.dvalues = at_col(dqkv, 2 * H * r);
            a.du = at_col(drow, Dc); a.dh = at_col(drow, Dc + H * r);
            a.derase_raw = at_col(drow, Dc + 2 * H * r); a.dwrite_raw = at_col(drow, Dc + 3 * H * r);
            a.dlog_decay = f32(dld); a.dgamma = f32(drate);
            a.valid_mask = bytes(valid); a.reset_mask = bytes(reset);
            check(sd_backward_pitched(&a, Dc, P, stream));
        }
        {   // decay gate and its small product
            Tensor draw = at::empty_like(decay_raw), dA = f32_like(x, {H}), db = f32_like(x, {H * r});
            const Tensor scratch = workspace(x, sd_kda_gate_backward_scratch_bytes(R, (int32_t)H, (int32_t)r));
            sd_kda_gate_args k{};
            k.rows = R; k.H = (int32_t)H; k.r = (int32_t)r;
            k.raw = decay_raw.data_ptr(); k.log_rate = f32(A32); k.bias = f32(b32); k.dlog_decay = f32(dld);
            k.draw = draw.data_ptr(); k.dlog_rate = f32(dA); k.dbias = f32(db);
            k.scratch = scratch.data_ptr(); k.scratch_bytes = (size_t)scratch.numel();
            check(sd_kda_gate_backward(&k, stream));
            result[7] = as("rate", dA).view(data["rate_shape"].toIntVector());
            result[8] = as("decay", db).view(data["decay_shape"].toIntVector());
            piece = drow.narrow(1, m.decay_hidden(), V);
            at::mm_out(piece, draw, decay_weight);
            result[4] = at::mm(draw.t(), row.narrow(1, m.decay_hidden(), V));
        }
        const Tensor dgeometry = at::sigmoid_backward(drate, rate);
        drow.narrow(1, m.geometry(), H).copy_(dgeometry);
        result[9] = as("geometry", dgeometry.sum(0));
        if (m.used() < P) drow.narrow(1, m.used(), P - m.used()).zero_();
        {   // conv
            const Tensor dw = f32_like(x, {Dc, 4});
            const Tensor scratch = workspace(x, sd_conv4_backward_scratch_bytes((int32_t)m.B, (int32_t)m.T, (int32_t)Dc));
            sd_conv4_backward_args c{};
            c.B = (int32_t)m.B; c.T = (int32_t)m.T; c.D = (int32_t)Dc;
            c.x = row.data_ptr(); c.x_stride_b = m.T * P; c.x_stride_t = P;
            c.weight = f32(w32); c.dy = dqkv.data_ptr(); c.dx = drow.data_ptr(); c.dweight = f32(dw);
            c.scratch = scratch.data_ptr(); c.scratch_bytes = (size_t)scratch.numel();
            c.valid_mask = bytes(valid); c.reset_mask = bytes(reset);
            check(sd_conv4_silu_backward_pitched(&c, P, stream));
            result[3] = as("conv", dw);
        }
        // input projection
        result[1] = at::mm(drow.t(), x.view({R, x.size(2)}));
        if (data["in_bias"].toBool()) result[2] = drow.sum(0);
        if (data["x"].toBool()) result[0] = at::mm(drow, in_weight).view(x.sizes());
        return result;
    }
};

// The layer on [B,T,D] with gradients recorded, from empty states, or None when this is not a call the node takes.
OptTensor mixer_train(const Tensor& x, int64_t heads, int64_t width, int64_t value_width, const Tensor& in_weight, const OptTensor& in_bias,
                      const Tensor& conv_weight, const Tensor& decay_weight, const Tensor& gate_weight, const OptTensor& gate_bias,
                      const Tensor& log_rate, const Tensor& decay_bias, const Tensor& geometry_bias, const Tensor& norm_weight, double eps,
                      const Tensor& out_weight, const OptTensor& out_bias, const OptTensor& valid, const OptTensor& reset) {
    if (!at::GradMode::is_enabled() || !x.is_cuda() || x.scalar_type() != at::kBFloat16 || x.dim() != 3 || !x.is_contiguous() || x.numel() == 0)
        return std::nullopt;
    const RowPlan m{x.size(0), x.size(1), heads, width, value_width, in_weight.size(0)};
    const auto dense = [&](const Tensor& t) { return t.is_contiguous() && t.scalar_type() == at::kBFloat16 && t.device() == x.device() && t.requires_grad(); };
    for (const Tensor* t : {&in_weight, &decay_weight, &gate_weight, &out_weight})
        if (!dense(*t) || !aligned16(*t)) return std::nullopt;
    for (const OptTensor* t : {&in_bias, &gate_bias, &out_bias})
        if (t->has_value() && !dense(**t)) return std::nullopt;
    for (const Tensor* t : {&conv_weight, &log_rate, &decay_bias, &geometry_bias, &norm_weight})
        if (t->device() != x.device() || !t->requires_grad()) return std::nullopt;
    const int64_t H = heads, r = width, V = value_width;
    if (r % 8 != 0 || V % 8 != 0 || r > 128 || V > 128 || m.P % 8 != 0 || m.P < m.used() || in_weight.size(1) != x.size(2) ||
        !is_shape(decay_weight, {H * r, V}) || !is_shape(gate_weight, {H * V, V}) || out_weight.dim() != 2 || out_weight.size(1) != H * V ||
        !is_shape(conv_weight, {m.conv(), 4}) || log_rate.numel() != H || decay_bias.numel() != H * r || geometry_bias.numel() != H ||
        !is_shape(norm_weight, {V}))
        return std::nullopt;
    const OptTensor v = conv_mask("valid_mask", valid, x), z = conv_mask("reset_mask", reset, x);
    return MixerFunction::apply(x, in_weight, in_bias, conv_weight, decay_weight, gate_weight, gate_bias, log_rate, decay_bias,
                                geometry_bias, norm_weight, out_weight, out_bias, v, z, heads, width, value_width, eps);
}

// One cached token between the fused projection row and the output projection, in one launch: conv4 + SiLU of the
// q | k | v slice against the conv window [B,D,3] (advanced in place), decay gate, geometry rate, the recurrent step on
// the FP32 states (updated in place), gated norm.  The rows are views of the projection row; parameters are FP32.
struct DecodeToken {
    Tensor u, h, erase, write, qkv, conv_weight, conv_state, decay_raw, log_rate, decay_bias, geometry_raw, geometry_bias;
    Tensor predictor, memory, output_gate, norm_weight;
    Tensor decay_hidden, decay_weight, gate_hidden, gate_weight, gate_bias;   // the fused gate projections, or undefined
    double eps;
};

Tensor decode_launch(const DecodeToken& t) {
    const int64_t B = t.u.size(0), H = t.u.size(2), r = t.u.size(3), V = t.write.size(-1), D = 2 * H * r + H * V;
    value_error(t.u.size(1) != 1, "mixer_decode_step takes exactly one token");
    const bool fused = t.decay_weight.defined();
    for (const auto& [name, x] : {std::pair<const char*, const Tensor&>{"u", t.u}, {"h", t.h}, {"erase_raw", t.erase},
                                  {"write_raw", t.write}, {"qkv", t.qkv}, {"geometry_raw", t.geometry_raw}, {"conv_state", t.conv_state}})
        require_bf16_cuda(name, x);
    if (!fused) require_bf16_cuda("decay_raw", t.decay_raw);
    for (const auto& [name, x] : {std::pair<const char*, const Tensor&>{"conv_weight", t.conv_weight}, {"log_rate", t.log_rate},
                                  {"decay_bias", t.decay_bias}, {"geometry_bias", t.geometry_bias},
                                  {"predictor", t.predictor}, {"memory", t.memory}})
        if (x.scalar_type() != at::kFloat || !x.is_contiguous()) throw py::type_error(std::string(name) + " must be contiguous FP32");
    value_error(!is_shape(t.qkv, {B, 1, D}) || !is_shape(t.conv_state, {B, D, 3}) || !t.conv_state.is_contiguous(),
                "qkv must be [B,1,D] and conv_state contiguous [B,D,3] with D = 2*H*r + H*V");
    value_error(t.qkv.stride(-1) != 1 || t.geometry_raw.stride(-1) != 1 || (t.decay_raw.defined() && t.decay_raw.stride(-1) != 1),
                "row operands require unit innermost stride");
    const c10::cuda::CUDAGuard guard(t.u.device());
    Tensor y = bf16_like(t.u, {B, 1, H, V});
    sd_mixer_decode_args a{};
    a.shape = sd_shape{(int32_t)B, 1, (int32_t)H, (int32_t)r, (int32_t)V};
    a.u = operand(t.u); a.h = operand(t.h); a.erase_raw = operand(t.erase); a.write_raw = operand(t.write);
    a.qkv = t.qkv.data_ptr(); a.qkv_stride_b = t.qkv.stride(0);
    a.conv_weight = f32(t.conv_weight); a.conv_state = t.conv_state.data_ptr();
    const Tensor decay = t.decay_raw.defined() ? t.decay_raw.contiguous().view({B, H * r}) : Tensor();
    if (decay.defined()) {
        a.decay_raw = decay.data_ptr();
        a.decay_stride_b = decay.stride(0);
    }
    a.log_rate = f32(t.log_rate); a.decay_bias = f32(t.decay_bias);
    a.geometry_raw = t.geometry_raw.data_ptr(); a.geometry_stride_b = t.geometry_raw.stride(0);
    a.geometry_bias = f32(t.geometry_bias);
    a.C = f32(t.predictor); a.S = f32(t.memory); a.y = y.data_ptr();
    if (fused) {
        const int64_t G = t.decay_hidden.size(-1);
        for (const auto& [name, x] : {std::pair<const char*, const Tensor&>{"decay_hidden", t.decay_hidden}, {"decay_proj.weight", t.decay_weight},
                                      {"gate_hidden", t.gate_hidden}, {"output_gate_proj.weight", t.gate_weight}})
            require_bf16_cuda(name, x);
        value_error(!is_shape(t.decay_weight, {H * r, G}) || !is_shape(t.gate_weight, {H * V, G}) || !t.decay_weight.is_contiguous() ||
                        !t.gate_weight.is_contiguous() || G % 8 != 0 || G > 128 || !t.norm_weight.defined(),
                    "fused gate projections: weights [H*r,G] / [H*V,G] contiguous, G a multiple of 8, at most 128, and the fused norm");
        a.gate_rank = (int32_t)G;
        a.decay_hidden = t.decay_hidden.data_ptr(); a.decay_hidden_stride_b = t.decay_hidden.stride(0);
        a.gate_hidden = t.gate_hidden.data_ptr(); a.gate_hidden_stride_b = t.gate_hidden.stride(0);
        a.decay_proj_weight = t.decay_weight.data_ptr(); a.gate_proj_weight = t.gate_weight.data_ptr();
        a.gate_proj_bias = raw(t.gate_bias);
    }
    if (t.norm_weight.defined()) {
        value_error(!fused && (!t.output_gate.defined() || t.output_gate.scalar_type() != at::kBFloat16 || !t.output_gate.is_contiguous()),
                    "the fused norm needs a contiguous BF16 output_gate [B,1,H,V]");
        type_error(t.norm_weight.scalar_type() != at::kFloat || !is_shape(t.norm_weight, {V}), "norm_weight must be FP32 [V]");
        a.norm_weight = f32(t.norm_weight); a.norm_eps = (float)t.eps;
        if (t.output_gate.defined()) {
            a.output_gate = t.output_gate.data_ptr();
            a.output_gate_stride_b = H * V;
        }
    }
    check(sd_mixer_decode_step(&a, stream_of(t.u)));
    return y;
}

// The whole mixer for one cached token without gradients: fused projection, decode launch (conv window and operator
// states advanced in place), output projection.
Tensor mixer_decode(Fp32Copies& copies, const Tensor& x, int64_t heads, int64_t width, int64_t value_width, const Tensor& in_weight,
                    const OptTensor& in_bias, const Tensor& conv_weight, const Tensor& conv_state, const Tensor& decay_weight,
                    const Tensor& gate_weight, const OptTensor& gate_bias, const Tensor& log_rate, const Tensor& decay_bias,
                    const Tensor& geometry_bias, const Tensor& predictor, const Tensor& memory, const Tensor& norm_weight, double eps,
                    const Tensor& out_weight, const OptTensor& out_bias) {
    const MixerShape shape{heads, width, value_width};
    const int64_t B = x.size(0);
    const Tensor row = projection(x, in_weight, in_bias);
    const variable_list piece = row_slices(row, shape.sizes(true));
    const auto view = [&](const Tensor& t, int64_t w) { return t.unflatten(-1, {heads, w}); };
    DecodeToken t;
    t.u = view(piece[1], width); t.h = view(piece[2], width);
    t.erase = view(piece[3], width); t.write = view(piece[4], value_width);
    t.qkv = piece[0];
    t.conv_weight = copies.get(0, conv_weight); t.conv_state = conv_state;
    t.log_rate = copies.get(1, log_rate); t.decay_bias = copies.get(2, decay_bias);
    t.geometry_raw = piece[5]; t.geometry_bias = copies.get(3, geometry_bias);
    t.predictor = predictor; t.memory = memory;
    t.norm_weight = copies.get(4, norm_weight); t.eps = eps;
    const Tensor gb = given(gate_bias);
    if (decay_weight.scalar_type() == at::kBFloat16 && gate_weight.scalar_type() == at::kBFloat16 && decay_weight.is_contiguous() &&
        gate_weight.is_contiguous() && (!gb.defined() || gb.scalar_type() == at::kBFloat16) && decay_weight.size(1) % 16 == 0 &&
        decay_weight.size(1) <= 128 && aligned16(decay_weight) && aligned16(gate_weight)) {
        // the two small projections in front of the gates run inside the kernel too
        t.decay_hidden = piece[6]; t.decay_weight = decay_weight;
        t.gate_hidden = piece[7]; t.gate_weight = gate_weight; t.gate_bias = gb;
    } else {
        t.decay_raw = view(projection(piece[6], decay_weight, std::nullopt), width);
        t.output_gate = view(projection(piece[7], gate_weight, gate_bias), value_width);
    }
    return projection(decode_launch(t).view({B, 1, heads * value_width}), out_weight, out_bias);
}

// ---- a cached token through the whole stack ------------------------------------------------------------------
// The blocks and the final norm of a model for one cached token without gradients, as one call: five chained launches a
// layer on pointers into one workspace (seven past sixteen rows, where the norms are launches of their own).  The
// parameters are held as the module's own tensors; what is watched says when the module has changed under it (see
// token_stack.py).
struct TokenLayer {
    Tensor mixer_norm, mlp_norm;
    Tensor in_weight, in_bias, conv_weight, decay_weight, gate_weight, gate_bias, log_rate, decay_bias, geometry_bias;
    Tensor out_norm, out_weight, out_bias, up_weight, down_weight;
    double mixer_eps, mlp_eps, out_eps;
    int64_t heads, width, value_width;
    Fp32Copies copies;
};

struct TokenStack {
    std::vector<TokenLayer> layers;
    Tensor norm;
    double norm_eps = 0;
    Fp32Copies copies;
    std::vector<std::tuple<py::dict, py::object, py::object>> same;   // dict[key] is value
    std::vector<std::pair<py::dict, py::object>> absent;              // key not in dict
    std::vector<py::dict> empty;                                      // hooks

    bool unchanged() const {
        for (const auto& [d, k, v] : same)
            if (PyDict_GetItemWithError(d.ptr(), k.ptr()) != v.ptr()) return false;
        for (const auto& [d, k] : absent)
            if (PyDict_Contains(d.ptr(), k.ptr()) != 0) return false;
        for (const auto& d : empty)
            if (PyDict_Size(d.ptr()) != 0) return false;
        return true;
    }

    void add_layer(const Tensor& mixer_norm, double mixer_eps, const Tensor& mlp_norm, double mlp_eps, int64_t heads, int64_t width,
                   int64_t value_width, const Tensor& in_weight, const OptTensor& in_bias, const Tensor& conv_weight,
                   const Tensor& decay_weight, const Tensor& gate_weight, const OptTensor& gate_bias, const Tensor& log_rate,
                   const Tensor& decay_bias, const Tensor& geometry_bias, const Tensor& out_norm, double out_eps,
                   const Tensor& out_weight, const OptTensor& out_bias, const Tensor& up_weight, const Tensor& down_weight) {
        layers.push_back(TokenLayer{mixer_norm, mlp_norm, in_weight, given(in_bias), conv_weight, decay_weight, gate_weight,
                                    given(gate_bias), log_rate, decay_bias, geometry_bias, out_norm, out_weight, given(out_bias),
                                    up_weight, down_weight, mixer_eps, mlp_eps, out_eps, heads, width, value_width, {}});
    }

    struct LayerFp32 { Tensor mixer_norm, conv, log_rate, decay_bias, geometry_bias, out_norm, mlp_norm; };
    std::vector<LayerFp32> layer_copies() {
        std::vector<LayerFp32> out;
        out.reserve(layers.size());
        for (TokenLayer& l : layers)
            out.push_back(LayerFp32{l.copies.get(0, l.mixer_norm), l.copies.get(1, l.conv_weight), l.copies.get(2, l.log_rate),
                                    l.copies.get(3, l.decay_bias), l.copies.get(4, l.geometry_bias), l.copies.get(5, l.out_norm),
                                    l.copies.get(6, l.mlp_norm)});
        return out;
    }

    static bool bf16_dense(const Tensor& t, const Tensor& like) {
        return t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.device() == like.device() && aligned16(t);
    }
    static bool weights_ok(const TokenLayer& l, const Tensor& x) {
        const int64_t D = x.size(-1), H = l.heads, r = l.width, V = l.value_width;
        for (const Tensor* t : {&l.in_weight, &l.decay_weight, &l.gate_weight, &l.out_weight, &l.up_weight, &l.down_weight})
            if (!bf16_dense(*t, x)) return false;
        for (const Tensor* t : {&l.in_bias, &l.gate_bias, &l.out_bias})
            if (t->defined() && !bf16_dense(*t, x)) return false;
        const int64_t inner = l.up_weight.size(0) / 2;
        return l.in_weight.size(1) == D && l.in_weight.size(0) % 8 == 0 && is_shape(l.out_weight, {D, H * V}) && l.up_weight.size(1) == D &&
               is_shape(l.down_weight, {D, inner}) && l.up_weight.size(0) % 16 == 0 && (H * V) % 8 == 0 && (H * r) % 8 == 0 &&
               is_shape(l.decay_weight, {H * r, V}) && is_shape(l.gate_weight, {H * V, V}) && V % 16 == 0 && V <= 128 && r <= 128 &&
               l.conv_weight.size(0) == 2 * H * r + H * V;
    }
    static bool layer_ok(const TokenLayer& l, const Tensor& x) {
        return weights_ok(l, x) && fits_smem(x.size(0), l.up_weight.size(0) / 2) && fits_smem(x.size(0), l.heads * l.value_width);
    }
    static bool fits_smem(int64_t rows, int64_t width) { return rows * (width + 96) * 2 <= 200 * 1024; }

    // hidden [B,1,D] and the cache's per-layer dicts -> the normalised hidden rows [B,1,D], or with `head` [vocabulary, D]
    // the logits; None when this is not a call the launches take (nothing has been touched then)
    std::optional<Tensor> step(const Tensor& x, const py::list& states, const OptTensor& head) {
        const int64_t B = x.size(0), D = x.size(2);
        if (!x.is_cuda() || x.scalar_type() != at::kBFloat16 || !x.is_contiguous() || x.size(1) != 1 || B < 1 || B > SD_TOKEN_MAX_ROWS ||
            D % 8 != 0 || D > 2048 || !aligned16(x) || !fits_smem(B, D) || states.size() != layers.size() ||
            (head.has_value() && (!bf16_dense(*head, x) || head->size(1) != D)))
            return std::nullopt;
        struct State { Tensor C, S, conv; };
        std::vector<State> state;
        state.reserve(layers.size());
        // interned once and never released: a static Python object must not outlive the interpreter
        static PyObject* const recurrent_key = PyUnicode_InternFromString("recurrent_state");
        static PyObject* const conv_key = PyUnicode_InternFromString("conv_state");
        size_t row_max = 0, y_max = 0, act_max = 0;
        for (size_t i = 0; i < layers.size(); ++i) {
            const TokenLayer& l = layers[i];
            const py::object entry = states[i];
            if (!layer_ok(l, x) || !PyDict_Check(entry.ptr())) return std::nullopt;
            PyObject* pair = PyDict_GetItemWithError(entry.ptr(), recurrent_key);
            PyObject* conv_obj = PyDict_GetItemWithError(entry.ptr(), conv_key);
            if (pair == nullptr || conv_obj == nullptr || !PyTuple_Check(pair) || PyTuple_GET_SIZE(pair) != 2) return std::nullopt;
            PyObject *c = PyTuple_GET_ITEM(pair, 0), *s = PyTuple_GET_ITEM(pair, 1);
            if (!THPVariable_Check(c) || !THPVariable_Check(s) || !THPVariable_Check(conv_obj)) return std::nullopt;
            State st{THPVariable_Unpack(c), THPVariable_Unpack(s), THPVariable_Unpack(conv_obj)};
            const int64_t H = l.heads, r = l.width, V = l.value_width;
            if (!is_shape(st.C, {B, H, r, r}) || !is_shape(st.S, {B, H, r, V}) || !is_shape(st.conv, {B, 2 * H * r + H * V, 3})) return std::nullopt;
            for (const Tensor* t : {&st.C, &st.S, &st.conv})
                if (!t->is_contiguous() || t->device() != x.device() || t->scalar_type() != (t == &st.conv ? at::kBFloat16 : at::kFloat))
                    return std::nullopt;
            state.push_back(std::move(st));
            row_max = std::max(row_max, (size_t)l.in_weight.size(0));
            y_max = std::max(y_max, (size_t)(H * V));
            act_max = std::max(act_max, (size_t)(l.up_weight.size(0) / 2));
        }
        const bool fuse_norm = B <= 16;
        if (!fuse_norm && (D % 256 != 0)) return std::nullopt;   // the norm alone takes whole groups of 256 channels
        const c10::cuda::CUDAGuard guard(x.device());
        void* stream = stream_of(x);
        // All FP32 copies are taken here, ahead of the first launch: one that is missing or out of date is a conversion
        // kernel, and a chained launch reads its parameters while the kernel directly before it still runs.
        const std::vector<LayerFp32> params = layer_copies();
        const Tensor last_norm = copies.get(0, norm);
        const auto piece = [&](size_t width) { return (width * (size_t)B * 2 + 255) & ~size_t(255); };
        const size_t row_b = piece(row_max), y_b = piece(y_max), act_b = piece(act_max), d_b = piece((size_t)D);
        const Tensor work = workspace(x, row_b + y_b + act_b + 5 * d_b);
        char* base = static_cast<char*>(work.data_ptr());
        char *row = base, *y = row + row_b, *act = y + y_b, *mixed = act + act_b, *mlp = mixed + d_b, *normed = mlp + d_b;
        char* sums[2] = {normed + d_b, normed + 2 * d_b};
        int next = 0;
        const void* residual = x.data_ptr();
        const void* delta = nullptr;
        bool chained = false;   // nothing of this call is in flight: the first launch follows the stream in full
        const auto linear = [&](const void* in, int64_t K, const Tensor& weight, const void* bias, void* out, bool with_swiglu,
                                const float* norm_w, double eps) {
            if (B > 16 && !with_swiglu && weight.size(0) >= 16 * 148) {
                // wide products of more than 16 rows: the library's tiles read a row of x once for many columns
                // (32 rows x 32000 x 1024: 14 us against 32)
                const auto options = x.options();
                const Tensor in_t = at::from_blob(const_cast<void*>(in), {B, K}, options);
                Tensor out_t = at::from_blob(out, {B, weight.size(0)}, options);
                if (bias != nullptr)
                    at::addmm_out(out_t, at::from_blob(const_cast<void*>(bias), {weight.size(0)}, options), in_t, weight.t());
                else
                    at::mm_out(out_t, in_t, weight.t());
                chained = false;
                return;
            }
            sd_token_linear_args a{};
            a.M = (int32_t)B; a.N = (int32_t)weight.size(0); a.K = (int32_t)K; a.swiglu = with_swiglu;
            a.x = in; a.x_stride = K; a.weight = weight.data_ptr(); a.bias = bias;
            a.y = out; a.y_stride = with_swiglu ? weight.size(0) / 2 : weight.size(0);
            a.chained = chained;
            chained = true;
            if (norm_w != nullptr) {
                a.norm_weight = norm_w; a.norm_eps = (float)eps; a.delta = delta;
                if (delta != nullptr) a.sum = sums[next];
            }
            check(sd_token_linear(&a, stream));
        };
        const auto advance = [&] {   // the sum that a norm has just stored is the residual stream from here on
            if (delta == nullptr) return;
            residual = sums[next];
            next ^= 1;
        };
        const auto norm_rows = [&](const float* norm_w, double eps, void* out) {
            sd_add_rmsnorm_args a{};
            a.rows = B; a.D = (int32_t)D; a.eps = (float)eps;
            a.x = residual; a.delta = delta; a.weight = norm_w; a.sum = delta != nullptr ? sums[next] : nullptr; a.normed = out;
            // without delta: the first launch, in the kernel for many rows, which follows the stream in full
            check(chained && delta != nullptr ? sd_add_rmsnorm_chained(&a, stream) : sd_add_rmsnorm(&a, stream));
            chained = delta != nullptr;
            advance();
        };
        // projection of the normalised residual stream
        const auto norm_linear = [&](const float* norm_w, double eps, const Tensor& weight, const void* bias, void* out, bool with_swiglu) {
            if (fuse_norm) {
                linear(residual, D, weight, bias, out, with_swiglu, norm_w, eps);
                advance();
            } else {
                norm_rows(norm_w, eps, normed);
                linear(normed, D, weight, bias, out, with_swiglu, nullptr, 0);
            }
        };
        for (size_t i = 0; i < layers.size(); ++i) {
            const TokenLayer& l = layers[i];
            const LayerFp32& w = params[i];
            State& st = state[i];
            const int64_t H = l.heads, r = l.width, V = l.value_width, P = l.in_weight.size(0);
            norm_linear(f32(w.mixer_norm), l.mixer_eps, l.in_weight, raw(l.in_bias), row, false);
            sd_mixer_decode_args a{};
            a.shape = sd_shape{(int32_t)B, 1, (int32_t)H, (int32_t)r, (int32_t)V};
            const auto at_col = [&](int64_t c) { return row + 2 * c; };
            const int64_t qkv = 2 * H * r + H * V, geom = qkv + 3 * H * r + H * V;
            a.u = sd_operand{at_col(qkv), P, P, r};
            a.h = sd_operand{at_col(qkv + H * r), P, P, r};
            a.erase_raw = sd_operand{at_col(qkv + 2 * H * r), P, P, r};
            a.write_raw = sd_operand{at_col(qkv + 3 * H * r), P, P, V};
            a.qkv = row; a.qkv_stride_b = P;
            a.conv_weight = f32(w.conv); a.conv_state = st.conv.data_ptr();
            a.log_rate = f32(w.log_rate); a.decay_bias = f32(w.decay_bias);
            a.geometry_raw = at_col(geom); a.geometry_stride_b = P; a.geometry_bias = f32(w.geometry_bias);
            a.C = f32(st.C); a.S = f32(st.S); a.y = y;
            a.norm_weight = f32(w.out_norm); a.norm_eps = (float)l.out_eps;
            a.gate_rank = (int32_t)V;
            a.decay_hidden = at_col(geom + H); a.decay_hidden_stride_b = P;
            a.gate_hidden = at_col(geom + H + V); a.gate_hidden_stride_b = P;
            a.decay_proj_weight = l.decay_weight.data_ptr(); a.gate_proj_weight = l.gate_weight.data_ptr();
            a.gate_proj_bias = raw(l.gate_bias);
            check(sd_mixer_decode_step_chained(&a, stream));
            linear(y, H * V, l.out_weight, raw(l.out_bias), mixed, false, nullptr, 0);
            delta = mixed;
            norm_linear(f32(w.mlp_norm), l.mlp_eps, l.up_weight, nullptr, act, true);
            linear(act, l.up_weight.size(0) / 2, l.down_weight, nullptr, mlp, false, nullptr, 0);
            delta = mlp;
        }
        Tensor out = bf16_like(x, {B, 1, head.has_value() ? head->size(0) : D});
        if (head.has_value())
            norm_linear(f32(last_norm), norm_eps, *head, nullptr, out.data_ptr(), false);
        else
            norm_rows(f32(last_norm), norm_eps, out.data_ptr());
        return out;
    }

    // A prompt [B,T,D] through the stack without gradients, from empty states: the launches of the module path, in its
    // order, on pointers into one workspace.  Module calls, views and small tensors cost the host about 270 us a layer,
    // which is more than the device needs below some two thousand tokens.  Returns the normalised hidden rows and, per
    // layer, (C, S, conv window) when they are wanted; None when this is not a call it takes.
    py::object prompt(const Tensor& x, bool want_states) {
        if (!x.is_cuda() || x.scalar_type() != at::kBFloat16 || !x.is_contiguous() || x.dim() != 3 || x.size(0) < 1 || x.size(1) < 2)
            return py::none();
        const int64_t B = x.size(0), T = x.size(1), D = x.size(2), R = B * T;
        if (R <= SD_TOKEN_MAX_ROWS || !addnorm_reverse_ok(D) || !aligned16(x)) return py::none();
        struct Plan { size_t saved, scratch; };
        std::vector<Plan> plan;
        const auto up256 = [](size_t n) { return (n + 255) & ~size_t(255); };
        const auto bf16_rows = [&](int64_t width) { return up256((size_t)R * (size_t)width * 2); };
        // the mixer's buffers and the MLP's are never alive together
        size_t area = 0;
        for (const TokenLayer& l : layers) {
            if (!weights_ok(l, x)) return py::none();
            const int64_t H = l.heads, r = l.width, V = l.value_width;
            const sd_shape sh{(int32_t)B, (int32_t)T, (int32_t)H, (int32_t)r, (int32_t)V};
            const Plan pl{up256(sd_inference_bytes(&sh)), up256(sd_forward_scratch_bytes(&sh))};
            const size_t mixer = bf16_rows(l.in_weight.size(0)) + bf16_rows(2 * H * r + H * V) + 3 * bf16_rows(H * r) + bf16_rows(2 * H) +
                                 3 * bf16_rows(H * V) + pl.saved + pl.scratch;
            area = std::max({area, mixer, bf16_rows(l.up_weight.size(0)) + bf16_rows(l.up_weight.size(0) / 2)});
            plan.push_back(pl);
        }
        const c10::cuda::CUDAGuard guard(x.device());
        void* stream = stream_of(x);
        const std::vector<LayerFp32> params = layer_copies();
        const size_t d_b = bf16_rows(D);
        const Tensor work = workspace(x, area + 5 * d_b);
        char* const base = static_cast<char*>(work.data_ptr());
        char *mixed = base + area, *mlp = mixed + d_b, *normed = mlp + d_b;
        char* sums[2] = {normed + d_b, normed + 2 * d_b};
        const auto bf16 = x.options(), fp32 = x.options().dtype(at::kFloat);
        const auto matrix = [&](const void* p, int64_t cols, int64_t pitch) {
            return at::from_blob(const_cast<void*>(p), {R, cols}, {pitch, 1}, bf16);
        };
        const auto linear = [&](const void* in, int64_t pitch, const Tensor& weight, const Tensor& bias, void* out) {
            Tensor out_t = matrix(out, weight.size(0), weight.size(0));
            if (bias.defined())
                at::addmm_out(out_t, bias, matrix(in, weight.size(1), pitch), weight.t());
            else
                at::mm_out(out_t, matrix(in, weight.size(1), pitch), weight.t());
        };
        int next = 0;
        const void* residual = x.data_ptr();
        const void* delta = nullptr;
        const auto norm_rows = [&](const Tensor& w, double eps, void* out) {
            sd_add_rmsnorm_args a{};
            a.rows = R; a.D = (int32_t)D; a.eps = (float)eps;
            a.x = residual; a.delta = delta; a.weight = f32(w); a.sum = delta != nullptr ? sums[next] : nullptr; a.normed = out;
            check(sd_add_rmsnorm(&a, stream));
            if (delta == nullptr) return;
            residual = sums[next];
            next ^= 1;
        };
        py::list states;
        for (size_t i = 0; i < layers.size(); ++i) {
            const TokenLayer& l = layers[i];
            const LayerFp32& w32 = params[i];
            const int64_t H = l.heads, r = l.width, V = l.value_width, P = l.in_weight.size(0), Dc = 2 * H * r + H * V;
            const RowPlan rows{B, T, H, r, V, P};
            char* at = base;
            const auto take = [&](size_t bytes) { char* p = at; at += bytes; return p; };
            char *row = take(bf16_rows(P)), *qkv = take(bf16_rows(Dc)), *decay_raw = take(bf16_rows(H * r));
            char *log_decay = take(2 * bf16_rows(H * r)), *geometry = take(bf16_rows(2 * H)), *gate = take(bf16_rows(H * V));
            char *y = take(bf16_rows(H * V)), *y_normed = take(bf16_rows(H * V)), *saved = take(plan[i].saved), *scratch = take(plan[i].scratch);
            norm_rows(w32.mixer_norm, l.mixer_eps, normed);
            linear(normed, D, l.in_weight, l.in_bias, row);
            Tensor C, S, window;
            if (want_states) {
                C = f32_like(x, {B, H, r, r});
                S = f32_like(x, {B, H, r, V});
                window = bf16_like(x, {B, Dc, 3});
            }
            sd_conv4_forward_args c{};
            c.B = (int32_t)B; c.T = (int32_t)T; c.D = (int32_t)Dc;
            c.x = row; c.x_stride_b = T * P; c.x_stride_t = P;
            c.weight = f32(w32.conv); c.y = qkv; c.final_state = raw(window);
            check(sd_conv4_silu_forward(&c, stream));
            const auto at_col = [&](int64_t col) { return row + 2 * col; };
            linear(at_col(rows.decay_hidden()), P, l.decay_weight, Tensor(), decay_raw);
            linear(at_col(rows.gate_hidden()), P, l.gate_weight, l.gate_bias, gate);
            sd_kda_gate_args k{};
            k.rows = R; k.H = (int32_t)H; k.r = (int32_t)r;
            k.raw = decay_raw; k.log_rate = f32(w32.log_rate); k.bias = f32(w32.decay_bias);
            k.log_decay = reinterpret_cast<float*>(log_decay);
            check(sd_kda_gate_forward(&k, stream));
            Tensor rate = at::from_blob(geometry, {R, H}, fp32);
            at::add_out(rate, matrix(at_col(rows.geometry()), H, P), w32.geometry_bias);
            at::sigmoid_(rate);
            sd_forward_args a{};
            rows.fill(a, row, qkv, log_decay, geometry);
            a.y = y; a.C_T = f32(C); a.S_T = f32(S);
            a.saved = saved; a.saved_bytes = plan[i].saved; a.scratch = scratch; a.scratch_bytes = plan[i].scratch;
            check(sd_forward_inference(&a, stream));
            sd_norm_gate_args g{};
            g.V = (int32_t)V; g.rows = R * H; g.eps = (float)l.out_eps;
            g.x = y; g.gate = gate; g.weight = f32(w32.out_norm); g.y = y_normed;
            check(sd_norm_gate_forward(&g, stream));
            linear(y_normed, H * V, l.out_weight, l.out_bias, mixed);
            delta = mixed;
            norm_rows(w32.mlp_norm, l.mlp_eps, normed);
            const int64_t inner = l.up_weight.size(0) / 2;
            char *up = base, *act = base + bf16_rows(2 * inner);
            linear(normed, D, l.up_weight, Tensor(), up);
            sd_swiglu_args w{};
            w.I = (int32_t)inner; w.rows = R; w.gate_value = up; w.out = act;
            check(sd_swiglu(&w, stream));
            linear(act, inner, l.down_weight, Tensor(), mlp);
            delta = mlp;
            if (want_states) states.append(py::make_tuple(C, S, window));
        }
        Tensor out = bf16_like(x, x.sizes());
        norm_rows(copies.get(0, norm), norm_eps, out.data_ptr());
        return py::make_tuple(out, states);
    }
};

}  // namespace

void register_glue(py::module_& m) {
    // holds nothing that a copy or a pickle of its module has to carry
    py::class_<Fp32Copies>(m, "Fp32Copies")
        .def(py::init<>())
        .def("get", &Fp32Copies::get)
        .def("__deepcopy__", [](const Fp32Copies&, py::dict) { return Fp32Copies(); })
        .def(py::pickle([](const Fp32Copies&) { return py::tuple(); }, [](py::tuple) { return Fp32Copies(); }));
    py::class_<TokenStack>(m, "TokenStack")
        .def(py::init([](const Tensor& norm, double eps) {
            TokenStack t;
            t.norm = norm;
            t.norm_eps = eps;
            return t;
        }))
        .def("add_layer", &TokenStack::add_layer)
        .def("watch_same", [](TokenStack& t, py::dict d, py::object k, py::object v) { t.same.emplace_back(d, k, v); })
        .def("watch_absent", [](TokenStack& t, py::dict d, py::object k) { t.absent.emplace_back(d, k); })
        .def("watch_empty", [](TokenStack& t, py::dict d) { t.empty.push_back(d); })
        .def("unchanged", &TokenStack::unchanged)
        .def("step", &TokenStack::step)
        .def("prompt", &TokenStack::prompt);
    m.def("conv4_silu", &conv4_silu);
    m.def("kda_decay_gate", &kda_decay_gate);
    m.def("rms_norm_gated", &rms_norm_gated);
    m.def("rms_norm_gated_linear", &rms_norm_gated_linear);
    m.def("norm_linear_forward", &norm_linear_raw);
    m.def("norm_linear_backward", &norm_linear_raw_backward);
    m.def("add_rmsnorm", &add_rmsnorm);
    m.def("swiglu", &swiglu);
    m.def("small_linear", &small_linear);
    m.def("gated_mlp", &gated_mlp);
    m.def("pack_rows", &pack_rows);
    m.def("mixer_front", &mixer_front);
    m.def("mixer_train", &mixer_train);
    m.def("mixer_decode", &mixer_decode);
}
