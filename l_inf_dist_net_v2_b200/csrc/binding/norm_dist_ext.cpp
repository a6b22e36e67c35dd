// pybind11 / PyTorch binding of the C ABI (include/ldn_b200.h): the compiled counterpart of the reference's
// extension module (core/cuda/norm_dist.cpp:40-204).  Twelve functions with the reference's names, argument
// order and in-place semantics; every tensor must be a contiguous CUDA tensor (norm_dist.cpp:8-10), shapes are
// read from the tensors as the reference does (norm_dist.cpp:44,73,127).  Differences: launches go to the
// current stream of the tensors' device (with a device guard) and a non-zero status raises.
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <cmath>

#include "ldn_b200.h"

namespace {

using torch::Tensor;

const float* fptr(const Tensor& t, const char* name) {
    TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
    TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
    return t.data_ptr<float>();  // raises for a wrong dtype, like the reference
}
float* fptr_mut(Tensor& t, const char* name) { return const_cast<float*>(fptr(t, name)); }
int* iptr(const Tensor& t, const char* name) {
    TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
    TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
    return t.data_ptr<int>();
}
float* opt_fptr(c10::optional<Tensor>& t, const char* name) { return t.has_value() ? fptr_mut(*t, name) : nullptr; }

ldn_stream_t stream() { return reinterpret_cast<ldn_stream_t>(at::cuda::getCurrentCUDAStream().stream()); }

void check(int status, const char* what) {
    TORCH_CHECK(status == 0, what, " failed with status ", status, ": ", ldn_status_string(status));
}

void norm_dist_forward(Tensor& input, Tensor& weight, Tensor& output, int G, float p) {
    const float *x = fptr(input, "input"), *w = fptr(weight, "weight");
    float* y = fptr_mut(output, "output");
    const c10::cuda::CUDAGuard guard(input.device());
    check(ldn_norm_dist_forward(x, w, input.size(0), output.size(1), input.size(1), G, input.size(2), y, p, stream()),
          "norm_dist_forward");
}

void norm_dist_forward_with_max(Tensor& input, Tensor& weight, Tensor& max_output, Tensor& output, int G, float p) {
    const float *x = fptr(input, "input"), *w = fptr(weight, "weight"), *m = fptr(max_output, "max_output");
    float* y = fptr_mut(output, "output");
    const c10::cuda::CUDAGuard guard(input.device());
    check(ldn_norm_dist_forward_with_max(x, w, m, input.size(0), output.size(1), input.size(1), G, input.size(2), y, p,
                                         stream()),
          "norm_dist_forward_with_max");
}

void norm_dist_backward_input(Tensor& grad_output, Tensor& input, Tensor& weight, Tensor& output, Tensor& grad_input,
                              int G, float p) {
    const float *g = fptr(grad_output, "grad_output"), *x = fptr(input, "input"), *w = fptr(weight, "weight"),
                *y = fptr(output, "output");
    float* gx = fptr_mut(grad_input, "grad_input");
    const c10::cuda::CUDAGuard guard(input.device());
    check(ldn_norm_dist_backward_input(g, x, w, y, grad_output.size(0), output.size(1), input.size(1), G, input.size(2),
                                       gx, p, stream()),
          "norm_dist_backward_input");
}

// grad_input may be None when the caller does not need it (an extension of the reference interface)
void norm_dist_backward_input_weight(Tensor& grad_output, Tensor& input, Tensor& weight, Tensor& output,
                                     c10::optional<Tensor> grad_input, Tensor& grad_weight, int G, float p) {
    const float *g = fptr(grad_output, "grad_output"), *x = fptr(input, "input"), *w = fptr(weight, "weight"),
                *y = fptr(output, "output");
    float* gx = opt_fptr(grad_input, "grad_input");
    float* gw = fptr_mut(grad_weight, "grad_weight");
    const c10::cuda::CUDAGuard guard(input.device());
    check(ldn_norm_dist_backward_input_weight(g, x, w, y, grad_output.size(0), output.size(1), input.size(1), G,
                                              input.size(2), gx, gw, p, stream()),
          "norm_dist_backward_input_weight");
}

void inf_dist_forward(Tensor& input, Tensor& weight, Tensor& output, Tensor& pos, int G) {
    const float *x = fptr(input, "input"), *w = fptr(weight, "weight");
    float* y = fptr_mut(output, "output");
    int* ps = iptr(pos, "pos");
    const c10::cuda::CUDAGuard guard(input.device());
    check(ldn_inf_dist_forward(x, w, input.size(0), output.size(1), input.size(1), G, input.size(2), y, ps, stream()),
          "inf_dist_forward");
}

void inf_dist_forward_nograd(Tensor& input, Tensor& weight, Tensor& output, int G) {
    const float *x = fptr(input, "input"), *w = fptr(weight, "weight");
    float* y = fptr_mut(output, "output");
    const c10::cuda::CUDAGuard guard(input.device());
    check(ldn_inf_dist_forward_nograd(x, w, input.size(0), output.size(1), input.size(1), G, input.size(2), y, stream()),
          "inf_dist_forward_nograd");
}

void inf_dist_backward_input(Tensor& grad_output, Tensor& pos, Tensor& grad_input, int G) {
    const float* g = fptr(grad_output, "grad_output");
    const int* ps = iptr(pos, "pos");
    float* gx = fptr_mut(grad_input, "grad_input");
    const c10::cuda::CUDAGuard guard(grad_output.device());
    check(ldn_inf_dist_backward_input(g, ps, grad_output.size(0), grad_output.size(1), grad_input.size(1), G,
                                      grad_input.size(2), gx, stream()),
          "inf_dist_backward_input");
}

void inf_dist_backward_input_weight(Tensor& grad_output, Tensor& pos, c10::optional<Tensor> grad_input,
                                    Tensor& grad_weight, int G) {
    const float* g = fptr(grad_output, "grad_output");
    const int* ps = iptr(pos, "pos");
    float* gx = opt_fptr(grad_input, "grad_input");
    float* gw = fptr_mut(grad_weight, "grad_weight");
    const c10::cuda::CUDAGuard guard(grad_output.device());
    check(ldn_inf_dist_backward_input_weight(g, ps, grad_output.size(0), grad_output.size(1), grad_weight.size(1) * G, G,
                                             grad_output.size(2), gx, gw, stream()),
          "inf_dist_backward_input_weight");
}

void bound_inf_dist_forward(Tensor& inputL, Tensor& inputU, Tensor& weight, Tensor& outputL, Tensor& outputU,
                            Tensor& posL, Tensor& posU, int G) {
    const float *xl = fptr(inputL, "inputL"), *xu = fptr(inputU, "inputU"), *w = fptr(weight, "weight");
    float *yl = fptr_mut(outputL, "outputL"), *yu = fptr_mut(outputU, "outputU");
    int *pl = iptr(posL, "posL"), *pu = iptr(posU, "posU");
    const c10::cuda::CUDAGuard guard(inputL.device());
    check(ldn_bound_inf_dist_forward(xl, xu, w, inputL.size(0), outputL.size(1), inputL.size(1), G, inputL.size(2), yl, yu,
                                     pl, pu, stream()),
          "bound_inf_dist_forward");
}

void bound_inf_dist_forward_nograd(Tensor& inputL, Tensor& inputU, Tensor& weight, Tensor& outputL, Tensor& outputU,
                                   int G) {
    const float *xl = fptr(inputL, "inputL"), *xu = fptr(inputU, "inputU"), *w = fptr(weight, "weight");
    float *yl = fptr_mut(outputL, "outputL"), *yu = fptr_mut(outputU, "outputU");
    const c10::cuda::CUDAGuard guard(inputL.device());
    check(ldn_bound_inf_dist_forward_nograd(xl, xu, w, inputL.size(0), outputL.size(1), inputL.size(1), G, inputL.size(2),
                                            yl, yu, stream()),
          "bound_inf_dist_forward_nograd");
}

void bound_inf_dist_backward_input(Tensor& grad_outputL, Tensor& grad_outputU, Tensor& posL, Tensor& posU,
                                   Tensor& grad_inputL, Tensor& grad_inputU, int G) {
    const float *gl = fptr(grad_outputL, "grad_outputL"), *gu = fptr(grad_outputU, "grad_outputU");
    const int *pl = iptr(posL, "posL"), *pu = iptr(posU, "posU");
    float *gxl = fptr_mut(grad_inputL, "grad_inputL"), *gxu = fptr_mut(grad_inputU, "grad_inputU");
    const c10::cuda::CUDAGuard guard(grad_outputL.device());
    check(ldn_bound_inf_dist_backward_input(gl, gu, pl, pu, grad_outputL.size(0), grad_outputL.size(1), grad_inputL.size(1),
                                            G, grad_inputL.size(2), gxl, gxu, stream()),
          "bound_inf_dist_backward_input");
}

void bound_inf_dist_backward_input_weight(Tensor& grad_outputL, Tensor& grad_outputU, Tensor& posL, Tensor& posU,
                                          Tensor& grad_inputL, Tensor& grad_inputU, Tensor& grad_weight, int G) {
    const float *gl = fptr(grad_outputL, "grad_outputL"), *gu = fptr(grad_outputU, "grad_outputU");
    const int *pl = iptr(posL, "posL"), *pu = iptr(posU, "posU");
    float *gxl = fptr_mut(grad_inputL, "grad_inputL"), *gxu = fptr_mut(grad_inputU, "grad_inputU");
    float* gw = fptr_mut(grad_weight, "grad_weight");
    const c10::cuda::CUDAGuard guard(grad_outputL.device());
    check(ldn_bound_inf_dist_backward_input_weight(gl, gu, pl, pu, grad_outputL.size(0), grad_outputL.size(1),
                                                   grad_weight.size(1) * G, G, grad_outputL.size(2), gxl, gxu, gw,
                                                   stream()),
          "bound_inf_dist_backward_input_weight");
}

// not part of the reference's extension module: patches as columns and the adjoint (ldn_unfold / ldn_fold)
void unfold(Tensor& x, Tensor& cols, std::pair<int, int> kernel, int stride, int padding, int dilation) {
    const float* a = fptr(x, "x");
    float* c = fptr_mut(cols, "cols");
    const c10::cuda::CUDAGuard guard(x.device());
    check(ldn_unfold(a, x.size(0), x.size(1), x.size(2), x.size(3), kernel.first, kernel.second, stride, padding, dilation,
                     c, stream()),
          "unfold");
}
void fold(Tensor& cols, Tensor& x, std::pair<int, int> kernel, int stride, int padding, int dilation) {
    const float* c = fptr(cols, "cols");
    float* a = fptr_mut(x, "x");
    const c10::cuda::CUDAGuard guard(x.device());
    check(ldn_fold(c, x.size(0), x.size(1), x.size(2), x.size(3), kernel.first, kernel.second, stride, padding, dilation, a,
                   stream()),
          "fold");
}

// ---- the operators as autograd functions ---------------------------------------------------------------------------
//
// The Python autograd functions (norm_dist.py, modules.py) restated in C++: the same steps in the same order.  A forward and
// backward pass of a Python autograd function costs 55 us on the host before it does anything (the engine's thread takes
// the interpreter lock and runs the Python backward), more than the kernels of a small layer; here it is 25 us.  The
// entry points return None for whatever the Python functions should see instead (other devices, types and layouts, shapes
// that do not fit, tensors that carry a forward-mode tangent or intercept operators): those raise or handle it.
//
// The linear maps (mean shift, unfold) replace torch operators that can be differentiated and transformed in any way, so
// where a gradient is itself to be differentiated, or is not plain memory, their backward steps are those operators.

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// whether the tracer or a dispatch mode looks at the operators as they are called
bool observed() { return torch::jit::tracer::isTracing() || c10::impl::dispatch_mode_enabled(); }
bool plain(const Tensor& t, int64_t dim) {
    return t.is_cuda() && t.scalar_type() == at::kFloat && t.layout() == at::kStrided && t.dim() == dim && t.is_contiguous() &&
           t.numel() > 0 && t.has_storage() && !t._fw_grad(0).defined() && !t.unsafeGetTensorImpl()->is_python_dispatch();
}
bool fits(const Tensor& x, const Tensor& w, int64_t G) {
    return plain(x, 3) && plain(w, 2) && x.device() == w.device() && G > 0 && G <= w.size(0) && w.size(1) * G == x.size(1);
}
Tensor output_of(const Tensor& x, const Tensor& w) { return at::empty({x.size(0), w.size(0), x.size(2)}, x.options()); }

struct NormDistFn : public torch::autograd::Function<NormDistFn> {
    static Tensor forward(AutogradContext* ctx, Tensor x, Tensor w, int64_t G, double p, bool need_grad) {
        Tensor y = output_of(x, w);
        ctx->saved_data["G"] = G;
        ctx->saved_data["p"] = p;
        const int g = static_cast<int>(G);
        if (std::isinf(p)) {
            if (!need_grad) {
                inf_dist_forward_nograd(x, w, y, g);
            } else {
                Tensor pos = at::empty(y.sizes(), y.options().dtype(at::kInt));
                inf_dist_forward(x, w, y, pos, g);
                ctx->save_for_backward({x, w, pos});
            }
        } else {
            norm_dist_forward(x, w, y, g, static_cast<float>(p));
            ctx->save_for_backward({x, w, y});
        }
        return y;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        Tensor go = grads[0].contiguous();
        const int g = static_cast<int>(ctx->saved_data["G"].toInt());
        const double p = ctx->saved_data["p"].toDouble();
        const bool need_x = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(1);
        variable_list saved = ctx->get_saved_variables();
        Tensor &x = saved[0], &w = saved[1], &third = saved[2];
        Tensor gx, gw;
        c10::optional<Tensor> maybe_gx;
        if (need_x) maybe_gx = gx = at::empty_like(x);
        if (need_w) {
            gw = at::empty_like(w);
            if (std::isinf(p)) inf_dist_backward_input_weight(go, third, maybe_gx, gw, g);
            else norm_dist_backward_input_weight(go, x, w, third, maybe_gx, gw, g, static_cast<float>(p));
        } else if (need_x) {
            if (std::isinf(p)) inf_dist_backward_input(go, third, gx, g);
            else norm_dist_backward_input(go, x, w, third, gx, g, static_cast<float>(p));
        }
        return {gx, gw, Tensor(), Tensor(), Tensor()};
    }
};

struct BoundInfDistFn : public torch::autograd::Function<BoundInfDistFn> {
    static variable_list forward(AutogradContext* ctx, Tensor xl, Tensor xu, Tensor w, int64_t G, bool need_grad) {
        Tensor yl = output_of(xl, w), yu = at::empty_like(yl);
        ctx->saved_data["G"] = G;
        const int g = static_cast<int>(G);
        if (!need_grad) {
            bound_inf_dist_forward_nograd(xl, xu, w, yl, yu, g);
        } else {
            Tensor pl = at::empty(yl.sizes(), yl.options().dtype(at::kInt)), pu = at::empty_like(pl);
            bound_inf_dist_forward(xl, xu, w, yl, yu, pl, pu, g);
            ctx->save_for_backward({xl, xu, w, pl, pu});
        }
        return {yl, yu};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        Tensor gl = grads[0].contiguous(), gu = grads[1].contiguous();
        const int g = static_cast<int>(ctx->saved_data["G"].toInt());
        variable_list saved = ctx->get_saved_variables();
        Tensor &xl = saved[0], &xu = saved[1], &w = saved[2], &pl = saved[3], &pu = saved[4];
        const bool need_l = ctx->needs_input_grad(0), need_u = ctx->needs_input_grad(1), need_w = ctx->needs_input_grad(2);
        Tensor gxl, gxu, gw;
        if (need_w || (need_l && need_u)) {
            gxl = at::empty_like(xl);
            gxu = at::empty_like(xu);
            if (need_w) {
                gw = at::empty_like(w);
                bound_inf_dist_backward_input_weight(gl, gu, pl, pu, gxl, gxu, gw, g);
            } else {
                bound_inf_dist_backward_input(gl, gu, pl, pu, gxl, gxu, g);
            }
        } else {
            gxl = at::zeros_like(xl);
            gxu = at::zeros_like(xu);
        }
        return {need_l ? gxl : Tensor(), need_u ? gxu : Tensor(), gw, Tensor(), Tensor()};
    }
};

// x - mean over the batch and the positions; running_mean may be undefined
void subtract_mean(const Tensor& x, const Tensor& running_mean, double momentum, Tensor& out) {
    const float* a = fptr(x, "x");
    float* rm = running_mean.defined() ? const_cast<float*>(fptr(running_mean, "running_mean")) : nullptr;
    float* y = fptr_mut(out, "out");
    const c10::cuda::CUDAGuard guard(x.device());
    const int B = x.size(0), C = x.size(1), HW = x.size(2);
    const float m = static_cast<float>(momentum);
    if (HW == 1) check(ldn_mean_shift_rows(a, B, C, rm, m, y, nullptr, stream()), "mean_shift_rows");
    else check(ldn_mean_shift_planes(a, B, C, HW, rm, m, y, stream()), "mean_shift_planes");
}

// whether a kernel of this package may compute a linear map's gradient from this one
bool plain_gradient(const Tensor& grad, int64_t dim) {
    return plain(grad, dim) && !observed() && !(at::GradMode::is_enabled() && grad.requires_grad());
}

struct MeanShiftFn : public torch::autograd::Function<MeanShiftFn> {
    static Tensor forward(AutogradContext*, Tensor x, Tensor running_mean, double momentum) {
        Tensor out = at::empty_like(x);
        subtract_mean(x, running_mean, momentum, out);
        return out;
    }
    static variable_list backward(AutogradContext*, variable_list grads) {
        Tensor go = grads[0].contiguous();
        if (!plain_gradient(go, 3)) return {go - go.mean(at::IntArrayRef({0, 2}), true), Tensor(), Tensor()};
        Tensor gx = at::empty_like(go);
        subtract_mean(go, Tensor(), 0.0, gx);
        return {gx, Tensor(), Tensor()};
    }
};

struct UnfoldFn : public torch::autograd::Function<UnfoldFn> {
    static Tensor forward(AutogradContext* ctx, Tensor x, int64_t positions, int64_t kh, int64_t kw, int64_t stride,
                          int64_t padding, int64_t dilation) {
        ctx->saved_data["image"] = x.sizes().vec();
        ctx->saved_data["geometry"] = std::vector<int64_t>{kh, kw, stride, padding, dilation};
        Tensor cols = at::empty({x.size(0), x.size(1) * kh * kw, positions}, x.options());
        unfold(x, cols, {static_cast<int>(kh), static_cast<int>(kw)}, static_cast<int>(stride), static_cast<int>(padding),
               static_cast<int>(dilation));
        return cols;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        Tensor go = grads[0].contiguous(), gx;
        const std::vector<int64_t> n = ctx->saved_data["geometry"].toIntVector();
        const std::vector<int64_t> image = ctx->saved_data["image"].toIntVector();
        if (plain_gradient(go, 3)) {
            gx = at::empty(image, go.options());
            fold(go, gx, {static_cast<int>(n[0]), static_cast<int>(n[1])}, static_cast<int>(n[2]), static_cast<int>(n[3]),
                 static_cast<int>(n[4]));
        } else {
            gx = at::col2im(go, {image[2], image[3]}, {n[0], n[1]}, {n[4], n[4]}, {n[3], n[3]}, {n[2], n[2]});
        }
        return {gx, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

// Margins behind the last layer (models.py) and the hinge loss (losses.py).  Both replace torch operators that can be
// differentiated in any way; where a gradient is itself to be differentiated or is not plain memory, their backward steps are
// those operators.
const long long* lptr(const Tensor& t) { return reinterpret_cast<const long long*>(t.data_ptr<int64_t>()); }

struct MarginsFn : public torch::autograd::Function<MarginsFn> {
    static variable_list forward(AutogradContext* ctx, Tensor dist, Tensor targets, double eps) {
        ctx->set_materialize_grads(false);
        ctx->saved_data["eps"] = eps;
        ctx->save_for_backward({targets});
        Tensor of_target = at::gather(dist, 1, targets.view({-1, 1}));  // (it checks the targets)
        Tensor logits = at::empty_like(dist), margin = at::empty_like(dist);
        const c10::cuda::CUDAGuard guard(dist.device());
        check(ldn_margins(fptr(dist, "dist"), fptr(of_target, "dist"), lptr(targets), dist.size(0), dist.size(1),
                          static_cast<float>(eps), 1.0f / static_cast<float>(2 * eps), fptr_mut(logits, "logits"),
                          fptr_mut(margin, "margin"), stream()),
              "margins");
        return {logits, margin};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        if (!grads[0].defined() && !grads[1].defined()) return {Tensor(), Tensor(), Tensor()};
        const double eps = ctx->saved_data["eps"].toDouble();
        const Tensor targets = ctx->get_saved_variables()[0];
        const Tensor gl = grads[0].defined() ? grads[0].contiguous() : Tensor();
        const Tensor gm = grads[1].defined() ? grads[1].contiguous() : Tensor();
        if ((gl.defined() && !plain_gradient(gl, 2)) || (gm.defined() && !plain_gradient(gm, 2))) {
            Tensor g;
            if (gm.defined()) {
                const Tensor col = targets.view({-1, 1}), m = (gm / (2 * eps)).scatter(1, col, 0);
                g = (-m).scatter_add(1, col, m.sum(1, true));
            }
            if (gl.defined()) g = g.defined() ? g - gl : -gl;
            return {g, Tensor(), Tensor()};
        }
        Tensor g = at::empty_like(gl.defined() ? gl : gm);
        const c10::cuda::CUDAGuard guard(g.device());
        check(ldn_margins_backward(gl.defined() ? fptr(gl, "grad") : nullptr, gm.defined() ? fptr(gm, "grad") : nullptr,
                                   lptr(targets), g.size(0), g.size(1), 1.0f / static_cast<float>(2 * eps), fptr_mut(g, "grad"),
                                   stream()),
              "margins_backward");
        return {g, Tensor(), Tensor()};
    }
};

struct HingeFn : public torch::autograd::Function<HingeFn> {
    static Tensor forward(AutogradContext* ctx, Tensor margin, double mix) {
        ctx->saved_data["mix"] = mix;
        Tensor loss = at::empty({}, margin.options()), first = at::empty({margin.size(0)}, margin.options().dtype(at::kInt));
        const c10::cuda::CUDAGuard guard(margin.device());
        check(ldn_hinge(fptr(margin, "margin"), margin.size(0), margin.size(1), mix, fptr_mut(loss, "loss"), iptr(first, "first"),
                        stream()),
              "hinge");
        ctx->save_for_backward({margin, first});
        return loss;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const double mix = ctx->saved_data["mix"].toDouble();
        variable_list saved = ctx->get_saved_variables();
        const Tensor &margin = saved[0], &g = grads[0];
        if (!plain_gradient(g, 0)) {
            const Tensor part = at::full_like(margin, mix / margin.numel())
                                    .scatter_add(1, saved[1].to(at::kLong).view({-1, 1}),
                                                 at::full({margin.size(0), 1}, (1 - mix) / margin.size(0), margin.options()));
            return {at::where(margin.detach() >= 0, g * part, at::zeros({}, margin.options())), Tensor()};
        }
        Tensor grad = at::empty_like(margin);
        const c10::cuda::CUDAGuard guard(margin.device());
        check(ldn_hinge_backward(fptr(g, "grad"), fptr(margin, "margin"), iptr(saved[1], "first"), margin.size(0), margin.size(1),
                                 mix, fptr_mut(grad, "grad"), stream()),
              "hinge_backward");
        return {grad, Tensor()};
    }
};

constexpr int64_t kMostLogits = 1 << 20;  // (beyond, the operators are as fast, and one cluster is not enough for the loss)
// A row is a warp's at most, and all rows one cluster's: on the device 16384 x 10 take 23 us forward (operators 25), 65536 x 10 74
// (35).  Launched one by one, forward and backward, the operators take 185 us whatever the size, these kernels 58 up to here.
constexpr int64_t kMostHingeClasses = 1024, kMostHingeRows = 32768;

c10::optional<std::tuple<Tensor, Tensor>> margins(const Tensor& dist, const Tensor& targets, double eps) {
    if (!plain(dist, 2) || dist.numel() > kMostLogits || !targets.is_cuda() || targets.scalar_type() != at::kLong ||
        targets.layout() != at::kStrided || targets.dim() != 1 || !targets.is_contiguous() || targets.size(0) != dist.size(0) ||
        targets.device() != dist.device() || !targets.has_storage() || targets.unsafeGetTensorImpl()->is_python_dispatch() ||
        !(eps > 0) || !std::isnormal(static_cast<float>(2 * eps)) || observed())
        return c10::nullopt;
    variable_list out = MarginsFn::apply(dist, targets, eps);
    return std::make_tuple(out[0], out[1]);
}

c10::optional<Tensor> hinge(const Tensor& margin, double mix) {
    if (!plain(margin, 2) || margin.numel() > kMostLogits || margin.size(1) > kMostHingeClasses || margin.size(0) > kMostHingeRows ||
        !std::isfinite(mix) || observed())
        return c10::nullopt;
    return HingeFn::apply(margin, mix);
}

c10::optional<Tensor> norm_dist(const Tensor& x, const Tensor& w, double p, int64_t G) {
    if (!fits(x, w, G) || !(p > 0.0) || observed()) return c10::nullopt;
    const bool need_grad = at::GradMode::is_enabled() && (x.requires_grad() || w.requires_grad());
    return NormDistFn::apply(x, w, G, p, need_grad);
}

c10::optional<std::tuple<Tensor, Tensor>> bound_inf_dist(const Tensor& xl, const Tensor& xu, const Tensor& w, int64_t G) {
    if (!fits(xl, w, G) || !fits(xu, w, G) || xl.sizes() != xu.sizes() || observed()) return c10::nullopt;
    const bool need_grad = at::GradMode::is_enabled() && (xl.requires_grad() || xu.requires_grad() || w.requires_grad());
    variable_list y = BoundInfDistFn::apply(xl, xu, w, G, need_grad);
    return std::make_tuple(y[0], y[1]);
}

c10::optional<Tensor> mean_shift(const Tensor& x, const Tensor& running_mean, double momentum) {
    if (!plain(x, 3) || !plain(running_mean, 1) || x.device() != running_mean.device() || running_mean.requires_grad() ||
        running_mean.size(0) != x.size(1) || observed())
        return c10::nullopt;
    return MeanShiftFn::apply(x, running_mean, momentum);
}

c10::optional<Tensor> unfold_columns(const Tensor& x, int64_t positions, std::pair<int64_t, int64_t> kernel, int64_t stride,
                                     int64_t padding, int64_t dilation) {
    if (!plain(x, 4) || observed()) return c10::nullopt;
    return UnfoldFn::apply(x, positions, kernel.first, kernel.second, stride, padding, dilation);
}

// eval-mode layers (not part of the reference's extension module): (y - sub[o]) + add[o] applied in the store
void inf_dist_forward_nograd_shifted(Tensor& input, Tensor& weight, Tensor& output, c10::optional<Tensor> sub,
                                     c10::optional<Tensor> add, int G) {
    const float *x = fptr(input, "input"), *w = fptr(weight, "weight");
    float* y = fptr_mut(output, "output");
    const float *s = opt_fptr(sub, "sub"), *a = opt_fptr(add, "add");
    const c10::cuda::CUDAGuard guard(input.device());
    check(ldn_inf_dist_forward_nograd_shifted(x, w, input.size(0), output.size(1), input.size(1), G, input.size(2), y, s, a,
                                              stream()),
          "inf_dist_forward_nograd_shifted");
}

void bound_inf_dist_forward_nograd_shifted(Tensor& inputL, Tensor& inputU, Tensor& weight, Tensor& outputL, Tensor& outputU,
                                           c10::optional<Tensor> sub, c10::optional<Tensor> add, int G) {
    const float *xl = fptr(inputL, "inputL"), *xu = fptr(inputU, "inputU"), *w = fptr(weight, "weight");
    float *yl = fptr_mut(outputL, "outputL"), *yu = fptr_mut(outputU, "outputU");
    const float *s = opt_fptr(sub, "sub"), *a = opt_fptr(add, "add");
    const c10::cuda::CUDAGuard guard(inputL.device());
    check(ldn_bound_inf_dist_forward_nograd_shifted(xl, xu, w, inputL.size(0), outputL.size(1), inputL.size(1), G,
                                                    inputL.size(2), yl, yu, s, a, stream()),
          "bound_inf_dist_forward_nograd_shifted");
}

void check_status() { check(ldn_check_status(stream()), "device status check"); }

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("norm_dist_forward", &norm_dist_forward);
    m.def("norm_dist_forward_with_max", &norm_dist_forward_with_max);
    m.def("norm_dist_backward_input", &norm_dist_backward_input);
    m.def("norm_dist_backward_input_weight", &norm_dist_backward_input_weight);
    m.def("inf_dist_forward", &inf_dist_forward);
    m.def("inf_dist_forward_nograd", &inf_dist_forward_nograd);
    m.def("inf_dist_backward_input", &inf_dist_backward_input);
    m.def("inf_dist_backward_input_weight", &inf_dist_backward_input_weight);
    m.def("bound_inf_dist_forward", &bound_inf_dist_forward);
    m.def("bound_inf_dist_forward_nograd", &bound_inf_dist_forward_nograd);
    m.def("bound_inf_dist_backward_input", &bound_inf_dist_backward_input);
    m.def("bound_inf_dist_backward_input_weight", &bound_inf_dist_backward_input_weight);
    m.def("unfold", &unfold);
    m.def("fold", &fold);
    m.def("norm_dist", &norm_dist);
    m.def("bound_inf_dist", &bound_inf_dist);
    m.def("mean_shift", &mean_shift);
    m.def("unfold_columns", &unfold_columns);
    m.def("margins", &margins);
    m.def("hinge", &hinge);
    m.def("inf_dist_forward_nograd_shifted", &inf_dist_forward_nograd_shifted);
    m.def("bound_inf_dist_forward_nograd_shifted", &bound_inf_dist_forward_nograd_shifted);
    m.def("check_status", &check_status);
}
