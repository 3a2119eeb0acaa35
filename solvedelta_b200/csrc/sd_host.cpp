// Host side of the operator's entry points in C++: argument checks, output and workspace tensors, argument blocks and
// the autograd node.  The kernels behind it are reached through the C ABI (include/solvedelta_b200.h) only.
//
// Why it is native: at T = 1 the kernel takes 7 us, and the same steps in Python (checks, nine ctypes operands, tensor
// allocation, torch.autograd.Function) took 59 us a call forward-only and 300 us with the reverse pass, so short calls
// were bound by the interpreter.
#include "sd_host.h"

namespace {

// The nine operands, k / v / gate logits without their edit axis, gamma as [B,T,H].
struct Operands {
    Tensor u, h, q, k, v, ld, er, wr, gam;
    sd_shape shape() const {
        return sd_shape{(int32_t)u.size(0), (int32_t)u.size(1), (int32_t)u.size(2), (int32_t)u.size(3), (int32_t)v.size(3)};
    }
    template <class Args>
    void fill(Args& a) const {
        a.shape = shape();
        a.u = operand(u); a.h = operand(h); a.q = operand(q);
        a.keys = operand(k); a.values = operand(v);
        a.erase_raw = operand(er); a.write_raw = operand(wr);
        a.log_decay = operand(ld); a.gamma = operand(gam);
    }
};

struct ForwardResult {
    Tensor y, C_T, S_T, saved;
};

// `states`: whether the final states are wanted; `keep`: whether the reverse pass's panels are.
ForwardResult forward_launch(const Operands& x, const Tensor& C0, const Tensor& S0, const Tensor& valid,
                             const Tensor& reset, bool states, bool keep) {
    const sd_shape s = x.shape();
    ForwardResult out;
    out.y = bf16_like(x.u, {s.B, s.T, s.H, s.V});
    if (states) {
        out.C_T = f32_like(x.u, {s.B, s.H, s.r, s.r});
        out.S_T = f32_like(x.u, {s.B, s.H, s.r, s.V});
    }
    out.saved = workspace(x.u, keep ? sd_saved_bytes(&s) : sd_inference_bytes(&s));
    const Tensor scratch = workspace(x.u, sd_forward_scratch_bytes(&s));
    sd_forward_args a{};
    x.fill(a);
    a.C0 = f32(C0); a.S0 = f32(S0);
    a.y = out.y.data_ptr(); a.C_T = f32(out.C_T); a.S_T = f32(out.S_T);
    a.saved = out.saved.data_ptr(); a.saved_bytes = (size_t)out.saved.numel();
    a.scratch = scratch.data_ptr(); a.scratch_bytes = (size_t)scratch.numel();
    a.valid_mask = bytes(valid); a.reset_mask = bytes(reset);
    check(keep ? sd_forward(&a, stream_of(x.u)) : sd_forward_inference(&a, stream_of(x.u)));
    return out;
}

struct OperatorFunction : torch::autograd::Function<OperatorFunction> {
    static variable_list forward(AutogradContext* ctx, const Tensor& u, const Tensor& h, const Tensor& q,
                                 const Tensor& k, const Tensor& v, const Tensor& ld, const Tensor& er, const Tensor& wr,
                                 const Tensor& gam, const OptTensor& C0_in, const OptTensor& S0_in,
                                 const OptTensor& valid_in, const OptTensor& reset_in) {
        const c10::cuda::CUDAGuard guard(u.device());
        const Tensor C0 = given(C0_in), S0 = given(S0_in), valid = given(valid_in), reset = given(reset_in);
        // k, v and the gate logits come and go with their edit axis: dropping it out here would record a view node each
        const Operands x{u, h, q, k.squeeze(-2), v.squeeze(-2), ld, er.squeeze(-2), wr.squeeze(-2), gam};
        const ForwardResult r = forward_launch(x, C0.defined() ? C0.contiguous() : C0,
                                               S0.defined() ? S0.contiguous() : S0, valid, reset, true, true);
        ctx->set_materialize_grads(false);
        ctx->saved_data["C0"] = C0.defined();
        ctx->saved_data["S0"] = S0.defined();
        ctx->save_for_backward({u, h, q, k, v, ld, er, wr, gam, r.saved, valid, reset});
        return {r.y, r.C_T, r.S_T};
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        const Operands x{sv[0], sv[1], sv[2], sv[3].squeeze(-2), sv[4].squeeze(-2), sv[5], sv[6].squeeze(-2), sv[7].squeeze(-2), sv[8]};
        const Tensor &saved = sv[9], &valid = sv[10], &reset = sv[11];
        const sd_shape s = x.shape();
        const c10::cuda::CUDAGuard guard(x.u.device());
        Tensor dy = grads[0], dC = grads[1], dS = grads[2];
        if (!dy.defined())
            dy = at::zeros({s.B, s.T, s.H, s.V}, x.u.options());
        else if (dy.scalar_type() != at::kBFloat16 || dy.stride(-1) != 1)
            dy = dy.to(at::kBFloat16).contiguous();
        if (dC.defined()) dC = dC.to(at::kFloat).contiguous();
        if (dS.defined()) dS = dS.to(at::kFloat).contiguous();
        const int64_t B = s.B, T = s.T, H = s.H, r = s.r, V = s.V;
        Tensor du = bf16_like(x.u, {B, T, H, r}), dh = bf16_like(x.u, {B, T, H, r}), dq = bf16_like(x.u, {B, T, H, r});
        Tensor dk = bf16_like(x.u, {B, T, H, 1, r}), dv = bf16_like(x.u, {B, T, H, 1, V}), der = bf16_like(x.u, {B, T, H, 1, r});
        Tensor dwr = bf16_like(x.u, {B, T, H, 1, V}), dld = f32_like(x.u, {B, T, H, r}), dgam = f32_like(x.u, {B, T, H});
        const bool want_C = ctx->saved_data["C0"].toBool(), want_S = ctx->saved_data["S0"].toBool();
        Tensor dC0 = want_C ? f32_like(x.u, {B, H, r, r}) : Tensor(), dS0 = want_S ? f32_like(x.u, {B, H, r, V}) : Tensor();
        const Tensor scratch = workspace(x.u, sd_backward_scratch_bytes(&s));
        sd_backward_args a{};
        x.fill(a);
        a.dy = operand(dy);
        a.dC_T = f32(dC); a.dS_T = f32(dS);
        a.saved = saved.data_ptr(); a.saved_bytes = (size_t)saved.numel();
        a.scratch = scratch.data_ptr(); a.scratch_bytes = (size_t)scratch.numel();
        a.du = du.data_ptr(); a.dh = dh.data_ptr(); a.dq = dq.data_ptr();
        a.dkeys = dk.data_ptr(); a.dvalues = dv.data_ptr();
        a.derase_raw = der.data_ptr(); a.dwrite_raw = dwr.data_ptr();
        a.dlog_decay = f32(dld); a.dgamma = f32(dgam);
        a.dC0 = f32(dC0); a.dS0 = f32(dS0);
        a.valid_mask = bytes(valid); a.reset_mask = bytes(reset);
        check(sd_backward(&a, stream_of(x.u)));
        return {du, dh, dq, dk, dv, dld, der, dwr, dgam, dC0, dS0, Tensor(), Tensor()};
    }
};

// bool [B,T] -> the same bytes, contiguous
OptTensor mask_bytes(const OptTensor& m) { return m.has_value() ? OptTensor(m->contiguous()) : OptTensor(); }

// The dense path from raw gate logits (causallsso/ops/residual_frame/operator.py:154-304): the checks in upstream's
// order and with its exception types (operator.py:169-196,247-262), the T = 1 branch, the chunked path.
// Returns (y, C | None, S | None).
py::tuple residual_frame(const Tensor& u, const Tensor& h, const Tensor& q, const Tensor& keys, const Tensor& values,
                         const Tensor& ld_in, const Tensor& erase, const Tensor& write, const Tensor& geometry,
                         const OptTensor& C0_in, const OptTensor& S0_in, bool want_state, const OptTensor& valid_in,
                         const OptTensor& reset_in, bool inplace) {
    value_error(u.dim() != 4, "u must have shape [B,T,H,r]");
    const int64_t B = u.size(0), T = u.size(1), H = u.size(2), r = u.size(3);
    value_error(!is_shape(h, u.sizes()) || !is_shape(q, u.sizes()), "h and q must match u");
    value_error(!is_shape(keys, {B, T, H, 1, r}), "Residual-Frame SolveDelta requires keys [B,T,H,1,r]");
    value_error(values.dim() != 5 || !is_shape(values, {B, T, H, 1, values.size(4)}), "values must have shape [B,T,H,1,d_v]");
    const int64_t V = values.size(4);
    value_error(!is_shape(ld_in, {B, T, H, r}), "associative_log_decay must have shape [B,T,H,r]");
    value_error(!is_shape(erase, keys.sizes()) || !is_shape(write, values.sizes()),
                "erase_raw/write_raw shapes must match keys/values");
    const bool per_token = is_shape(geometry, {B, T, H});
    value_error(!per_token && !is_shape(geometry, {H}) && !is_shape(geometry, {1, H}),
                "geometry_write must have shape [H], [1,H], or [B,T,H]");
    type_error(!u.is_cuda() || u.scalar_type() != at::kBFloat16,
               "the production Residual-Frame path requires BF16 CUDA operands");
    for (const Tensor* t : {&h, &q, &keys, &values, &erase, &write})
        type_error(t->scalar_type() != at::kBFloat16, "all public vector operands must be BF16");
    type_error(ld_in.scalar_type() != at::kFloat, "associative_log_decay must be FP32");
    type_error(geometry.scalar_type() != at::kFloat, "geometry_write must be FP32");
    value_error(r > 128 || V > 128, "the B200 kernels support head widths up to 128");
    for (const Tensor* t : {&u, &h, &q, &keys, &values, &erase, &write})
        value_error(t->stride(-1) != 1, "native vector operands require unit innermost stride");
    const Tensor C0 = given(C0_in), S0 = given(S0_in);
    if (C0.defined() || S0.defined()) {
        value_error(!C0.defined() || !S0.defined() || !is_shape(C0, {B, H, r, r}) || !is_shape(S0, {B, H, r, V}),
                    "initial_state shapes do not match the input geometry");
        type_error(C0.scalar_type() != at::kFloat || S0.scalar_type() != at::kFloat,
                   "all continuation states must be FP32");
    }
    Operands x;
    x.ld = ld_in.stride(-1) != 1 ? ld_in.contiguous() : ld_in;
    x.gam = per_token ? geometry : geometry.reshape({1, 1, H}).expand({B, T, H});
    const bool empty = T == 0, masked = valid_in.has_value() || reset_in.has_value();
    if (empty) {
        const Tensor y = at::zeros({B, 0, H, V}, values.options());
        if (!want_state) return py::make_tuple(y, py::none(), py::none());
        if (C0.defined()) return py::make_tuple(y, C0, S0);
        return py::make_tuple(y, at::zeros({B, H, r, r}, ld_in.options()), at::zeros({B, H, r, V}, ld_in.options()));
    }
    Tensor y, C_T, S_T;
    if (!at::GradMode::is_enabled()) {
        // inference: no autograd node, and at T = 1 the single-token recurrent step
        // (causallsso/ops/residual_frame/operator.py:198-216)
        const c10::cuda::CUDAGuard guard(u.device());
        x.u = u; x.h = h; x.q = q;
        x.k = keys.squeeze(-2); x.v = values.squeeze(-2);
        x.er = erase.squeeze(-2); x.wr = write.squeeze(-2);
        const Tensor Cin = C0.defined() ? C0.contiguous() : C0, Sin = S0.defined() ? S0.contiguous() : S0;
        if (T == 1 && !masked) {
            // the updated states are new tensors, as upstream returns them, unless the caller's cache owns its state
            const bool keep = inplace && C0.defined() && C0.is_contiguous() && S0.is_contiguous();
            y = bf16_like(u, {B, 1, H, V});
            C_T = keep ? Cin : f32_like(u, {B, H, r, r});
            S_T = keep ? Sin : f32_like(u, {B, H, r, V});
            sd_decode_args a{};
            x.fill(a);
            a.C = f32(C_T); a.S = f32(S_T); a.y = y.data_ptr();
            check(sd_decode_step_from(&a, f32(Cin), f32(Sin), stream_of(u)));
        } else {
            const ForwardResult f = forward_launch(x, Cin, Sin, given(mask_bytes(valid_in)), given(mask_bytes(reset_in)), want_state, false);
            y = f.y; C_T = f.C_T; S_T = f.S_T;
        }
    } else {
        const variable_list out = OperatorFunction::apply(u, h, q, keys, values, x.ld, erase, write, x.gam, C0_in, S0_in,
                                                          mask_bytes(valid_in), mask_bytes(reset_in));
        y = out[0]; C_T = out[1]; S_T = out[2];
    }
    if (!want_state) return py::make_tuple(y, py::none(), py::none());
    return py::make_tuple(y, C_T, S_T);
}

// The additional checks of the public dense entry (causallsso/ops/operator.py:27-41), then the path above.
py::tuple dense(const Tensor& u, const Tensor& h, const Tensor& q, const Tensor& keys, const Tensor& values,
                const Tensor& ld, const Tensor& erase, const Tensor& write, const Tensor& geometry, const OptTensor& C0,
                const OptTensor& S0, bool want_state, bool inplace) {
    type_error(!u.is_cuda() || u.scalar_type() != at::kBFloat16, "solvedelta_native requires BF16 CUDA activations");
    value_error(keys.dim() != 5 || keys.size(-2) != 1, "the current production path requires num_edits=1");
    value_error(!is_shape(erase, keys.sizes()) || erase.scalar_type() != at::kBFloat16,
                "erase_raw must be BF16 with the same shape as keys");
    value_error(!is_shape(write, values.sizes()) || write.scalar_type() != at::kBFloat16,
                "write_raw must be BF16 with the same shape as values");
    for (const Tensor* t : {&u, &h, &q, &keys, &values, &erase, &write})
        value_error(t->stride(-1) != 1, "native vector operands require unit innermost stride");
    return residual_frame(u, h, q, keys, values, ld, erase, write, geometry, C0, S0, want_state, std::nullopt,
                          std::nullopt, inplace);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("dense", &dense);
    m.def("residual_frame", &residual_frame);
    register_glue(m);
}
