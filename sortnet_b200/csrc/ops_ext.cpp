// Native form of the operator layer (ops.py): argument checks, output allocation, the library call and the autograd node of
// norm_dist, norm_dist_dropout, sort_neuron and bound_inf_dist in C++.  The Python classes of ops.py do the same
// steps at about four times the host time (a small layer's forward, backward and bounds: 310 us per pass against
// kernels of 30 us); they stay for what needs Python: gradient sinks, the profile, index-list validation.
// Also the layer table, the mask lists and the calls of a whole-net pass (a training pass of six layers on small images issued in 650 us
// through ctypes, 490 us here, against 360 us of kernels), and what a convolution does around its distance (patches, mean shift and
// bias over positions: a forward and backward of two convolutions issued in 740 us by Python functions, 503 here).
//
// The library is reached through function pointers (init), so this module links against PyTorch only.

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/extension.h>

#include <cmath>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/sortnet_b200.h"

namespace {

using at::Tensor;
using c10::optional;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Api {
    decltype(&snb_inf_dist_forward_ws) inf_forward;
    decltype(&snb_inf_dist_forward_sorted_ws) inf_forward_sorted;
    decltype(&snb_inf_dist_forward_sorted_workspace_bytes) inf_sorted_bytes;
    decltype(&snb_inf_dist_forward_nograd_ws) inf_forward_nograd;
    decltype(&snb_inf_dist_backward_input) inf_backward_x;
    decltype(&snb_inf_dist_backward_input_weight) inf_backward_xw;
    decltype(&snb_norm_dist_forward_ws) lp_forward;
    decltype(&snb_norm_dist_backward_ws) lp_backward;
    decltype(&snb_norm_dist_scratch_bytes) lp_bytes;
    decltype(&snb_bound_inf_dist_forward_nograd_ws) bound_forward_nograd;
    decltype(&snb_bound_inf_dist_forward_ws) bound_forward;
    decltype(&snb_bound_inf_dist_backward_input) bound_backward_x;
    decltype(&snb_bound_inf_dist_backward_input_weight) bound_backward_xw;
    decltype(&snb_sort_neuron_forward_nograd_ws) sort_forward_nograd;
    decltype(&snb_sort_neuron_forward_ws) sort_forward;
    decltype(&snb_sort_neuron_backward_input) sort_backward_x;
    decltype(&snb_sort_neuron_backward_input_weight) sort_backward_xw;
    decltype(&snb_bound_sort_neuron_forward_ws) bound_sort_forward;
    decltype(&snb_prune_scratch_bytes) scratch_bytes;
    decltype(&snb_prune_pays) pays;
    decltype(&snb_sample_mask_batch) sample_masks;
    decltype(&snb_mlp_applies) mlp_applies;
    decltype(&snb_mlp_saved_bytes) mlp_saved_bytes;
    decltype(&snb_mlp_scratch_bytes) mlp_scratch_bytes;
    decltype(&snb_mlp_backward_scratch_bytes) mlp_backward_bytes;
    decltype(&snb_mlp_train_forward) mlp_forward;
    decltype(&snb_mlp_train_backward) mlp_backward;
    decltype(&snb_unfold) unfold;
    decltype(&snb_fold) fold;
    decltype(&snb_plane_shift) plane_shift;
    decltype(&snb_plane_sum) plane_sum;
    decltype(&snb_plane_add) plane_add;
    decltype(&snb_status_string) status_string;
    decltype(&snb_last_cuda_error) last_cuda_error;
} api;
// A status code of the library: arrives in Python as the exception class that _lib.check raises.
struct LibraryError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
PyObject* library_error = PyExc_RuntimeError;

void init(const std::string& path, py::object error_class) {
    library_error = error_class.release().ptr();             // kept for the life of the process
    void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    TORCH_CHECK(h, "cannot load ", path, ": ", dlerror());
    auto get = [&](auto& f, const char* name) {
        f = reinterpret_cast<std::decay_t<decltype(f)>>(dlsym(h, name));
        TORCH_CHECK(f, path, " has no ", name);
    };
    get(api.inf_forward, "snb_inf_dist_forward_ws");
    get(api.inf_forward_sorted, "snb_inf_dist_forward_sorted_ws");
    get(api.inf_sorted_bytes, "snb_inf_dist_forward_sorted_workspace_bytes");
    get(api.inf_forward_nograd, "snb_inf_dist_forward_nograd_ws");
    get(api.inf_backward_x, "snb_inf_dist_backward_input");
    get(api.inf_backward_xw, "snb_inf_dist_backward_input_weight");
    get(api.lp_forward, "snb_norm_dist_forward_ws");
    get(api.lp_backward, "snb_norm_dist_backward_ws");
    get(api.lp_bytes, "snb_norm_dist_scratch_bytes");
    get(api.bound_forward_nograd, "snb_bound_inf_dist_forward_nograd_ws");
    get(api.bound_forward, "snb_bound_inf_dist_forward_ws");
    get(api.bound_backward_x, "snb_bound_inf_dist_backward_input");
    get(api.bound_backward_xw, "snb_bound_inf_dist_backward_input_weight");
    get(api.sort_forward_nograd, "snb_sort_neuron_forward_nograd_ws");
    get(api.sort_forward, "snb_sort_neuron_forward_ws");
    get(api.sort_backward_x, "snb_sort_neuron_backward_input");
    get(api.sort_backward_xw, "snb_sort_neuron_backward_input_weight");
    get(api.bound_sort_forward, "snb_bound_sort_neuron_forward_ws");
    get(api.scratch_bytes, "snb_prune_scratch_bytes");
    get(api.pays, "snb_prune_pays");
    get(api.sample_masks, "snb_sample_mask_batch");
    get(api.mlp_applies, "snb_mlp_applies");
    get(api.mlp_saved_bytes, "snb_mlp_saved_bytes");
    get(api.mlp_scratch_bytes, "snb_mlp_scratch_bytes");
    get(api.mlp_backward_bytes, "snb_mlp_backward_scratch_bytes");
    get(api.mlp_forward, "snb_mlp_train_forward");
    get(api.mlp_backward, "snb_mlp_train_backward");
    get(api.unfold, "snb_unfold");
    get(api.fold, "snb_fold");
    get(api.plane_shift, "snb_plane_shift");
    get(api.plane_sum, "snb_plane_sum");
    get(api.plane_add, "snb_plane_add");
    get(api.status_string, "snb_status_string");
    get(api.last_cuda_error, "snb_last_cuda_error");
}

void check(const Tensor& t, const char* name, at::ScalarType type = at::kFloat) {
    TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
    TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
    TORCH_CHECK(t.scalar_type() == type, name, " must have dtype ", type, ", got ", t.scalar_type());
}
void check_input(const Tensor& x, const Tensor& w, const char* name = "input") {
    check(x, name);
    check(w, "weight");
    // further axes of size 1 are fine
    TORCH_CHECK(x.dim() >= 3 && x.numel() == x.size(0) * x.size(1) * x.size(2) && w.dim() >= 2 && w.numel() == w.size(0) * w.size(1), name,
                " must have shape [B, C, HW] and weight [CO, CI / groups]");
    TORCH_CHECK(x.device() == w.device(), "all tensors must be on the same device");
}
void check_list(const optional<Tensor>& t, const char* name, int64_t B, int64_t G, int64_t width, const Tensor& x) {
    if (!t.has_value()) return;
    check(*t, name, at::kInt);
    TORCH_CHECK(t->dim() == 3 && t->size(0) == (B + 31) / 32 && t->size(1) == G && t->size(2) * G == width, name,
                " must have shape [", (B + 31) / 32, ", ", G, ", ", width / std::max<int64_t>(G, 1), "], got ", t->sizes());
    TORCH_CHECK(t->device() == x.device(), "all tensors must be on the same device");
}
const int* list_ptr(const optional<Tensor>& t) { return t.has_value() ? t->data_ptr<int>() : nullptr; }

void done(int rc, const char* what) {
    if (rc) {
        std::string why = api.status_string(rc);
        if (rc == SNB_STATUS_CUDA) why += std::string(": ") + api.last_cuda_error();
        throw LibraryError(std::string(what) + " failed: " + why + " (status " + std::to_string(rc) + ")");
    }
}

// Scratch of a forward call from PyTorch's caching allocator (stream-ordered).
struct Area {
    Tensor t;
    void* ptr = nullptr;
    size_t bytes = 0;
    Area(const Tensor& like, int tensors, int K, int words, int64_t B, int64_t CO, int64_t CI, int64_t W_CO, int64_t W_CI, bool lists,
         bool flat, size_t at_least = 0) {
        bytes = flat && api.pays(tensors, K, words, B, CO, W_CI) ? api.scratch_bytes(tensors, K, words, B, CO, CI, W_CO, W_CI, lists) : 0;
        bytes = std::max(bytes, at_least);
        if (bytes) {
            t = at::empty({(int64_t)bytes}, like.options().dtype(at::kByte));
            ptr = t.data_ptr();
        }
    }
};

struct Call {
    c10::cuda::OptionalCUDAGuard guard;
    cudaStream_t stream;
    explicit Call(const Tensor& t) : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()) {}
};

// ---- distance --------------------------------------------------------------------------------------
struct DistOut {
    Tensor y, pos;
};
DistOut dist_forward(const Tensor& x, const Tensor& w, const optional<Tensor>& ci, const optional<Tensor>& co, int64_t G, double p,
                     bool record, bool ascending) {
    check_input(x, w);
    const int64_t B = x.size(0), CI = x.size(1), HW = x.size(2);
    const int64_t CO = co.has_value() ? co->size(-1) * G : w.size(0);
    check_list(ci, "w_index_ci", B, G, CI, x);
    check_list(co, "w_index_co", B, G, CO, x);
    Call call(x);
    DistOut out;
    out.y = at::empty({B, CO, HW}, x.options());
    const bool flat = G == 1 && HW == 1;
    const int64_t W_CO = w.size(0), W_CI = w.size(1);
    if (std::isinf(p)) {
        if (!record) {
            Area ws(x, 1, 1, 0, B, CO, CI, CO, CI, false, flat);
            done(api.inf_forward_nograd(x.data_ptr<float>(), w.data_ptr<float>(), B, CO, CI, G, HW, out.y.data_ptr<float>(), ws.ptr,
                                        ws.bytes, call.stream), "inf_dist_forward_nograd");
            return out;
        }
        out.pos = at::empty({B, CO, HW}, x.options().dtype(at::kInt));
        const bool sorted = ascending && flat && (ci.has_value() || co.has_value());
        Area ws(x, 1, 1, 1, B, CO, CI, W_CO, W_CI, ci.has_value(), flat,
                !flat ? 0 : sorted ? api.inf_sorted_bytes(B, CO, W_CI) : sizeof(int64_t) * (size_t)(B * CO));
        auto f = sorted ? api.inf_forward_sorted : api.inf_forward;
        done(f(x.data_ptr<float>(), w.data_ptr<float>(), B, CO, CI, G, HW, out.y.data_ptr<float>(), out.pos.data_ptr<int>(),
               list_ptr(ci), list_ptr(co), W_CO, W_CI * G, ws.ptr, ws.bytes, call.stream), "inf_dist_forward");
        return out;
    }
    Area ws(x, 1, 1, 0, B, CO, CI, W_CO, W_CI, false, false, flat ? api.lp_bytes(0, B, CO, CI, W_CO, W_CI, (float)p, ci.has_value()) : 0);
    done(api.lp_forward(x.data_ptr<float>(), w.data_ptr<float>(), B, CO, CI, G, HW, out.y.data_ptr<float>(), (float)p, list_ptr(ci),
                        list_ptr(co), W_CO, W_CI * G, ws.ptr, ws.bytes, call.stream), "norm_dist_forward");
    return out;
}

struct DistFn : public torch::autograd::Function<DistFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const optional<Tensor>& ci, const optional<Tensor>& co,
                          int64_t G, double p, bool ascending) {
        DistOut out = dist_forward(x, w, ci, co, G, p, true, ascending);
        ctx->saved_data["p"] = p;
        ctx->saved_data["G"] = G;
        if (ci.has_value()) ctx->saved_data["ci"] = *ci;
        if (co.has_value()) ctx->saved_data["co"] = *co;
        ctx->save_for_backward({x, w, std::isinf(p) ? out.pos : out.y});
        return out.y;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &x = saved[0], &w = saved[1], &third = saved[2];
        const double p = ctx->saved_data["p"].toDouble();
        const int64_t G = ctx->saved_data["G"].toInt();
        optional<Tensor> ci, co;
        if (ctx->saved_data.count("ci")) ci = ctx->saved_data["ci"].toTensor();
        if (ctx->saved_data.count("co")) co = ctx->saved_data["co"].toTensor();
        const bool need_x = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(1);
        variable_list out(7);
        if (!need_x && !need_w) return out;
        Call call(x);
        const Tensor g = grads[0].contiguous();
        check(g, "grad_output");
        const int64_t B = g.size(0), CO = g.size(1), HW = g.size(2), CI = x.size(1);
        Tensor gx = at::empty_like(x), gw = need_w ? at::empty_like(w) : Tensor();
        const float* gp = g.data_ptr<float>();
        if (std::isinf(p)) {
            if (need_w)
                done(api.inf_backward_xw(gp, third.data_ptr<int>(), B, CO, CI, G, HW, gx.data_ptr<float>(), gw.data_ptr<float>(),
                                         list_ptr(ci), list_ptr(co), w.size(0), w.size(1) * G, call.stream),
                     "inf_dist_backward_input_weight");
            else
                done(api.inf_backward_x(gp, third.data_ptr<int>(), B, CO, CI, G, HW, gx.data_ptr<float>(), call.stream),
                     "inf_dist_backward_input");
        } else {
            const int64_t W_CO = w.size(0), W_CI = w.size(1);
            Area ws(x, 1, 1, 0, B, CO, CI, W_CO, W_CI, false, false,
                    G == 1 && HW == 1 ? api.lp_bytes(1, B, CO, CI, W_CO, W_CI, (float)p, ci.has_value()) : 0);
            done(api.lp_backward(gp, x.data_ptr<float>(), w.data_ptr<float>(), third.data_ptr<float>(), B, CO, CI, G, HW,
                                 gx.data_ptr<float>(), need_w ? gw.data_ptr<float>() : nullptr, (float)p, list_ptr(ci), list_ptr(co),
                                 W_CO, W_CI * G, ws.ptr, ws.bytes, call.stream),
                 need_w ? "norm_dist_backward_input_weight" : "norm_dist_backward_input");
        }
        if (need_x) out[0] = gx;
        out[1] = gw;
        return out;
    }
};

// record: some operand wants a gradient (always true for the masked operator, as in the Python form)
Tensor dist(const Tensor& x, const Tensor& w, const optional<Tensor>& ci, const optional<Tensor>& co, int64_t G, double p, bool record,
            bool ascending) {
    if (!std::isinf(p)) TORCH_CHECK(p > 0, "p must be positive");
    const bool graph = at::GradMode::is_enabled() && (x.requires_grad() || w.requires_grad());
    if (!graph) return dist_forward(x, w, ci, co, G, p, record, ascending).y;
    return DistFn::apply(x, w, ci, co, G, p, ascending);
}

// ---- sort neuron -----------------------------------------------------------------------------------
Tensor sort_forward(const Tensor& x, const Tensor& w, int64_t G, double q, int64_t K, Tensor* pos) {
    check_input(x, w);
    const int64_t B = x.size(0), CI = x.size(1), HW = x.size(2), CO = w.size(0);
    TORCH_CHECK(w.size(1) * G == CI, "shape mismatch");
    Call call(x);
    Tensor y = at::empty({B, CO, HW}, x.options());
    Area ws(x, 1, K, pos != nullptr, B, CO, CI, CO, CI, false, G == 1 && HW == 1);
    if (pos) {
        *pos = at::empty({K, B, CO, HW}, x.options().dtype(at::kInt));
        done(api.sort_forward(x.data_ptr<float>(), w.data_ptr<float>(), B, CO, CI, G, HW, y.data_ptr<float>(), pos->data_ptr<int>(),
                              (float)q, K, ws.ptr, ws.bytes, call.stream), "sort_neuron_forward");
    } else {
        done(api.sort_forward_nograd(x.data_ptr<float>(), w.data_ptr<float>(), B, CO, CI, G, HW, y.data_ptr<float>(), (float)q, K,
                                     ws.ptr, ws.bytes, call.stream), "sort_neuron_forward_nograd");
    }
    return y;
}

struct SortFn : public torch::autograd::Function<SortFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, int64_t G, double q, int64_t K) {
        Tensor pos, y = sort_forward(x, w, G, q, K, &pos);
        ctx->saved_data["G"] = G;
        ctx->saved_data["q"] = q;
        ctx->saved_data["K"] = K;
        ctx->save_for_backward({x, w, pos});
        return y;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &x = saved[0], &w = saved[1], &pos = saved[2];
        const int64_t G = ctx->saved_data["G"].toInt(), K = ctx->saved_data["K"].toInt();
        const float q = (float)ctx->saved_data["q"].toDouble();
        const bool need_x = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(1);
        variable_list out(5);
        if (!need_x && !need_w) return out;
        Call call(x);
        const Tensor g = grads[0].contiguous();
        check(g, "grad_output");
        const int64_t B = g.size(0), CO = g.size(1), HW = g.size(2), CI = x.size(1);
        Tensor gx = at::empty_like(x), gw = need_w ? at::empty_like(w) : Tensor();
        if (need_w)
            done(api.sort_backward_xw(g.data_ptr<float>(), pos.data_ptr<int>(), B, CO, CI, G, HW, gx.data_ptr<float>(),
                                      gw.data_ptr<float>(), q, K, call.stream), "sort_neuron_backward_input_weight");
        else
            done(api.sort_backward_x(g.data_ptr<float>(), pos.data_ptr<int>(), B, CO, CI, G, HW, gx.data_ptr<float>(), q, K,
                                     call.stream), "sort_neuron_backward_input");
        if (need_x) out[0] = gx;
        out[1] = gw;
        return out;
    }
};

Tensor sort_neuron(const Tensor& x, const Tensor& w, int64_t G, double q, int64_t K) {
    if (at::GradMode::is_enabled() && (x.requires_grad() || w.requires_grad())) return SortFn::apply(x, w, G, q, K);
    return sort_forward(x, w, G, q, K, nullptr);
}

// ---- interval bounds -------------------------------------------------------------------------------
std::tuple<Tensor, Tensor> bound_forward(const Tensor& xl, const Tensor& xu, const Tensor& w, int64_t G, Tensor* words) {
    check_input(xl, w, "inputL");
    check_input(xu, w, "inputU");
    const int64_t B = xl.size(0), CI = xl.size(1), HW = xl.size(2), CO = w.size(0);
    TORCH_CHECK(xl.sizes() == xu.sizes() && w.size(1) * G == CI, "shape mismatch");
    Call call(xl);
    Tensor yl = at::empty({B, CO, HW}, xl.options()), yu = at::empty({B, CO, HW}, xl.options());
    Area ws(xl, 2, 1, words != nullptr, B, CO, CI, CO, CI, false, G == 1 && HW == 1);
    if (words) {
        *words = at::empty({2, B, CO, HW}, xl.options().dtype(at::kInt));
        int* lw = words->data_ptr<int>();
        done(api.bound_forward(xl.data_ptr<float>(), xu.data_ptr<float>(), w.data_ptr<float>(), B, CO, CI, G, HW, yl.data_ptr<float>(),
                               yu.data_ptr<float>(), lw, lw + B * CO * HW, ws.ptr, ws.bytes, call.stream), "bound_inf_dist_forward");
    } else {
        done(api.bound_forward_nograd(xl.data_ptr<float>(), xu.data_ptr<float>(), w.data_ptr<float>(), B, CO, CI, G, HW,
                                      yl.data_ptr<float>(), yu.data_ptr<float>(), ws.ptr, ws.bytes, call.stream),
             "bound_inf_dist_forward_nograd");
    }
    return {yl, yu};
}

struct BoundFn : public torch::autograd::Function<BoundFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& xl, const Tensor& xu, const Tensor& w, int64_t G) {
        Tensor words;
        auto [yl, yu] = bound_forward(xl, xu, w, G, &words);
        ctx->saved_data["G"] = G;
        ctx->save_for_backward({xl, xu, w, words});
        return {yl, yu};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &xl = saved[0], &w = saved[2], &words = saved[3];
        const int64_t G = ctx->saved_data["G"].toInt();
        const bool need_l = ctx->needs_input_grad(0), need_u = ctx->needs_input_grad(1), need_w = ctx->needs_input_grad(2);
        variable_list out(4);
        Call call(xl);
        const int64_t B = words.size(1), CO = words.size(2), HW = words.size(3), CI = xl.size(1);
        Tensor g[2];
        for (int k = 0; k < 2; k++) {
            g[k] = grads[k].defined() ? grads[k].contiguous() : at::zeros({B, CO, HW}, xl.options());
            check(g[k], "grad_output");
        }
        const bool run = need_w || (need_l && need_u);      // one end of the box alone gets zeros, as in the Python form
        Tensor gl = run ? at::empty_like(xl) : at::zeros_like(xl), gu = run ? at::empty_like(xl) : at::zeros_like(xl);
        Tensor gw = need_w ? at::empty_like(w) : Tensor();
        const int* lw = words.data_ptr<int>();
        const float *pl = g[0].data_ptr<float>(), *pu = g[1].data_ptr<float>();
        if (need_w)
            done(api.bound_backward_xw(pl, pu, lw, lw + B * CO * HW, B, CO, CI, G, HW, gl.data_ptr<float>(), gu.data_ptr<float>(),
                                       gw.data_ptr<float>(), call.stream), "bound_inf_dist_backward_input_weight");
        else if (run)
            done(api.bound_backward_x(pl, pu, lw, lw + B * CO * HW, B, CO, CI, G, HW, gl.data_ptr<float>(), gu.data_ptr<float>(),
                                      call.stream), "bound_inf_dist_backward_input");
        if (need_l) out[0] = gl;
        if (need_u) out[1] = gu;
        out[2] = gw;
        return out;
    }
};

std::tuple<Tensor, Tensor> bound_inf_dist(const Tensor& xl, const Tensor& xu, const Tensor& w, int64_t G) {
    if (at::GradMode::is_enabled() && (xl.requires_grad() || xu.requires_grad() || w.requires_grad())) {
        auto y = BoundFn::apply(xl, xu, w, G);
        return {y[0], y[1]};
    }
    return bound_forward(xl, xu, w, G, nullptr);
}

std::tuple<Tensor, Tensor> bound_sort_neuron(const Tensor& xl, const Tensor& xu, const Tensor& w, int64_t G, double q, int64_t K) {
    check_input(xl, w, "inputL");
    check_input(xu, w, "inputU");
    const int64_t B = xl.size(0), CI = xl.size(1), HW = xl.size(2), CO = w.size(0);
    TORCH_CHECK(xl.sizes() == xu.sizes() && w.size(1) * G == CI, "shape mismatch");
    Call call(xl);
    Tensor yl = at::empty({B, CO, HW}, xl.options()), yu = at::empty({B, CO, HW}, xl.options());
    Area ws(xl, 2, K, 0, B, CO, CI, CO, CI, false, G == 1 && HW == 1);
    done(api.bound_sort_forward(xl.data_ptr<float>(), xu.data_ptr<float>(), w.data_ptr<float>(), B, CO, CI, G, HW, yl.data_ptr<float>(),
                                yu.data_ptr<float>(), (float)q, K, ws.ptr, ws.bytes, call.stream), "bound_sort_neuron_forward");
    return {yl, yu};
}

// ---- around the operators of a convolution -----------------------------------------------------------
struct UnfoldFn : public torch::autograd::Function<UnfoldFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& given, int64_t kh, int64_t kw, int64_t stride, int64_t pad, int64_t dil) {
        const Tensor x = given.contiguous();
        check(x, "x");
        TORCH_CHECK(x.dim() == 4, "x must have shape [B, C, H, W]");
        const int64_t B = x.size(0), C = x.size(1), H = x.size(2), W = x.size(3);
        auto places = [&](int64_t n, int64_t k) {            // rounded down, as Python divides
            const int64_t room = n + 2 * pad - dil * (k - 1) - 1;
            TORCH_CHECK(stride > 0, "stride must be positive");
            return std::max<int64_t>(room < 0 ? 0 : room / stride + 1, 0);
        };
        Call call(x);
        Tensor out = at::empty({B, C * kh * kw, places(H, kh) * places(W, kw)}, x.options());
        done(api.unfold(x.data_ptr<float>(), B, C, H, W, kh, kw, stride, pad, dil, out.data_ptr<float>(), call.stream), "unfold");
        ctx->saved_data["args"] = std::vector<int64_t>{B, C, H, W, kh, kw, stride, pad, dil};
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        variable_list out(6);
        if (!grads[0].defined() || !ctx->needs_input_grad(0)) return out;
        const auto a = ctx->saved_data["args"].toIntVector();
        const Tensor g = grads[0].contiguous();
        check(g, "g");
        Call call(g);
        out[0] = at::empty({a[0], a[1], a[2], a[3]}, g.options());
        done(api.fold(g.data_ptr<float>(), a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], out[0].data_ptr<float>(), call.stream),
             "fold");
        return out;
    }
};

// x [B, G kept, HW] with lists [S, G, kept]: (groups, kept channels per group).
std::pair<int, int> check_plane(const Tensor& x, const optional<Tensor>& index, int64_t channels) {
    check(x, "x");
    TORCH_CHECK(x.dim() == 3, "x must have shape [B, C, HW]");
    if (!index.has_value()) {
        TORCH_CHECK(x.size(1) == channels, "x must have all channels when there is no index");
        return {1, (int)channels};
    }
    check(*index, "index", at::kInt);
    TORCH_CHECK(index->dim() == 3 && index->device() == x.device() && index->size(0) == (x.size(0) + 31) / 32 &&
                    index->size(1) * index->size(2) == x.size(1), "index must have shape [sub-batches, groups, C / groups]");
    return {(int)index->size(1), (int)index->size(2)};
}
Tensor plane_shift(const Tensor& x, const optional<Tensor>& index, const Tensor& mean, const optional<Tensor>& running_mean, double momentum) {
    const auto [G, kept] = check_plane(x, index, mean.numel());
    Call call(x);
    Tensor y = at::empty_like(x);
    done(api.plane_shift(x.data_ptr<float>(), list_ptr(index), x.size(0), G, kept, x.size(2), mean.numel(), mean.data_ptr<float>(),
                         running_mean.has_value() ? running_mean->data_ptr<float>() : nullptr, (float)momentum, y.data_ptr<float>(),
                         call.stream), "plane_shift");
    return y;
}
struct PlaneShiftFn : public torch::autograd::Function<PlaneShiftFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& given, const optional<Tensor>& index, const Tensor& running_mean,
                                 double momentum) {
        const Tensor x = given.contiguous();
        check(running_mean, "running_mean");
        TORCH_CHECK(running_mean.device() == x.device(), "all tensors must be on the same device");
        Tensor mean = at::empty_like(running_mean), y = plane_shift(x, index, mean, running_mean, momentum);
        if (index.has_value()) ctx->saved_data["index"] = *index;
        ctx->saved_data["channels"] = running_mean.numel();
        ctx->mark_non_differentiable({mean});
        return {y, mean};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        variable_list out(4);
        if (!grads[0].defined() || !ctx->needs_input_grad(0)) return out;
        optional<Tensor> index;
        if (ctx->saved_data.count("index")) index = ctx->saved_data["index"].toTensor();
        const Tensor g = grads[0].contiguous();
        Tensor mean = at::empty({ctx->saved_data["channels"].toInt()}, g.options());
        out[0] = plane_shift(g, index, mean, c10::nullopt, 0.0);
        return out;
    }
};

struct PlaneSumFn;
struct PlaneAddFn : public torch::autograd::Function<PlaneAddFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& given, const Tensor& values, const optional<Tensor>& index) {
        const Tensor x = given.contiguous(), v = values.contiguous();
        check(v, "v");
        TORCH_CHECK(v.device() == x.device(), "all tensors must be on the same device");
        const auto [G, kept] = check_plane(x, index, v.numel());
        Call call(x);
        Tensor y = at::empty_like(x);
        done(api.plane_add(x.data_ptr<float>(), list_ptr(index), x.size(0), G, kept, x.size(2), v.numel(), v.data_ptr<float>(),
                           y.data_ptr<float>(), call.stream), "plane_add");
        if (index.has_value()) ctx->saved_data["index"] = *index;
        ctx->saved_data["channels"] = v.numel();
        return y;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads);
};
// The transpose of adding v: sums per channel.
struct PlaneSumFn : public torch::autograd::Function<PlaneSumFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& given, const optional<Tensor>& index, int64_t channels) {
        const Tensor x = given.contiguous();
        const auto [G, kept] = check_plane(x, index, channels);
        Call call(x);
        Tensor sum = at::empty({channels}, x.options());
        done(api.plane_sum(x.data_ptr<float>(), list_ptr(index), x.size(0), G, kept, x.size(2), channels, sum.data_ptr<float>(), call.stream),
             "plane_sum");
        if (index.has_value()) ctx->saved_data["index"] = *index;
        ctx->saved_data["shape"] = x.sizes().vec();
        return sum;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        variable_list out(3);
        if (!grads[0].defined()) return out;
        optional<Tensor> index;
        if (ctx->saved_data.count("index")) index = ctx->saved_data["index"].toTensor();
        out[0] = PlaneAddFn::apply(at::zeros(ctx->saved_data["shape"].toIntVector(), grads[0].options()), grads[0], index);
        return out;
    }
};
variable_list PlaneAddFn::backward(AutogradContext* ctx, variable_list grads) {
    variable_list out(3);
    if (!grads[0].defined()) return out;
    optional<Tensor> index;
    if (ctx->saved_data.count("index")) index = ctx->saved_data["index"].toTensor();
    if (ctx->needs_input_grad(0)) out[0] = grads[0];
    if (ctx->needs_input_grad(1)) out[1] = PlaneSumFn::apply(grads[0], index, ctx->saved_data["channels"].toInt());
    return out;
}

Tensor unfold(const Tensor& x, int64_t kh, int64_t kw, int64_t stride, int64_t pad, int64_t dil) {
    return UnfoldFn::apply(x, kh, kw, stride, pad, dil);
}
std::tuple<Tensor, Tensor> mean_shift(const Tensor& x, const optional<Tensor>& index, const Tensor& running_mean, double momentum) {
    auto out = PlaneShiftFn::apply(x, index, running_mean, momentum);
    return {out[0], out[1]};
}
Tensor add_per_channel(const Tensor& x, const Tensor& v, const optional<Tensor>& index) { return PlaneAddFn::apply(x, v, index); }

// ---- whole nets ------------------------------------------------------------------------------------
// The layer table of one call, with the tensors it points to.  Row: (weight, bias, running mean, momentum, kept list [S, 1, count],
// K, q) per layer.
using Row = std::tuple<Tensor, optional<Tensor>, optional<Tensor>, double, optional<Tensor>, int64_t, double>;
class MlpTable {
  public:
    explicit MlpTable(std::vector<Row> given) : rows_(std::move(given)) {
        auto at = [](const optional<Tensor>& t) { return t.has_value() ? t->data_ptr() : nullptr; };
        for (const auto& [w, bias, mean, momentum, kept, K, q] : rows_) {
            snb_mlp_layer l{};
            l.w = static_cast<const float*>(w.data_ptr());
            l.bias = static_cast<const float*>(at(bias));
            l.running_mean = static_cast<float*>(at(mean));
            l.kept_list = static_cast<const int*>(at(kept));
            l.in = (int)w.size(-1), l.out = (int)w.size(0), l.kept = kept.has_value() ? (int)kept->size(-1) : 0;
            l.K = (int)K, l.momentum = (float)momentum, l.q = (float)q;
            layers_.push_back(l);
        }
    }
    int64_t address() const { return (int64_t)layers_.data(); }
    bool applies(int64_t B) const { return api.mlp_applies(layers_.data(), depth(), (int)B) != 0; }
    // Whether every tensor is what the kernels read through its pointer: fp32 (int32 lists), contiguous, on the device of x [B, in],
    // of the shapes of a chain of layers.
    bool takes(const Tensor& x) const {
        if (x.dim() != 2) return false;
        const int64_t subs = (x.size(0) + 31) / 32;
        int64_t width = x.size(1);
        auto plain = [&](const Tensor& t, at::ScalarType type) { return t.device() == x.device() && t.scalar_type() == type && t.is_contiguous(); };
        for (const auto& [w, bias, mean, momentum, kept, K, q] : rows_) {
            if (w.dim() != 2 || w.size(1) != width || !plain(w, at::kFloat)) return false;
            width = w.size(0);
            for (const auto* t : {&bias, &mean})
                if (t->has_value() && ((*t)->dim() != 1 || (*t)->size(0) != width || !plain(**t, at::kFloat))) return false;
            if (kept.has_value() && (kept->dim() != 3 || kept->size(0) != subs || kept->size(1) != 1 || !plain(*kept, at::kInt))) return false;
        }
        return true;
    }
    // (loss, what the backward needs); x and targets as the caller has checked them
    std::tuple<Tensor, Tensor> train_forward(const Tensor& x, const Tensor& targets, double eps, double clip, double lam, double scale) const {
        const int B = (int)x.size(0);
        Call call(x);
        auto bytes = x.options().dtype(at::kByte);
        Tensor saved = at::empty({(int64_t)api.mlp_saved_bytes(layers_.data(), depth(), B)}, bytes);
        Tensor scratch = at::empty({(int64_t)api.mlp_scratch_bytes(layers_.data(), depth(), B, 1, 1)}, bytes);
        Tensor loss = at::empty({}, x.options());
        done(api.mlp_forward(layers_.data(), depth(), x.data_ptr<float>(), B, reinterpret_cast<const long long*>(targets.data_ptr<int64_t>()),
                             (float)eps, (float)clip, (float)lam, (float)scale, saved.data_ptr(), scratch.data_ptr(),
                             loss.data_ptr<float>(), nullptr, call.stream), "mlp_train_forward");
        return {loss, saved};
    }
    // grad_w: one tensor or None per layer
    void train_backward(int64_t B, const Tensor& grad_loss, const Tensor& saved, const std::vector<optional<Tensor>>& grad_w,
                        const optional<Tensor>& grad_bias, const optional<Tensor>& grad_x) const {
        auto at_of = [](const optional<Tensor>& t) { return t.has_value() ? t->data_ptr<float>() : nullptr; };
        Call call(saved);
        Tensor scratch = at::empty({(int64_t)api.mlp_backward_bytes(layers_.data(), depth(), (int)B)}, saved.options());
        std::vector<float*> gw;
        for (const auto& t : grad_w) gw.push_back(at_of(t));
        TORCH_CHECK((int)gw.size() == depth(), "one gradient (or None) per layer");
        done(api.mlp_backward(layers_.data(), depth(), (int)B, grad_loss.data_ptr<float>(), saved.data_ptr(), scratch.data_ptr(), gw.data(),
                              at_of(grad_bias), at_of(grad_x), nullptr, call.stream), "mlp_train_backward");
    }

  private:
    int depth() const { return (int)layers_.size(); }
    std::vector<Row> rows_;
    std::vector<snb_mlp_layer> layers_;
};

// Kept-channel lists [subs, 1, count] of several layers in one launch: count = how many of a layer's uniform numbers (on the host, one
// after the other in `uniform`) lie below its keep rate.
std::vector<Tensor> draw_lists(const Tensor& uniform, const Tensor& seeds, const std::vector<int64_t>& channels, const std::vector<double>& keep,
                               int64_t subs, const c10::Device& device) {
    TORCH_CHECK(uniform.device().is_cpu() && uniform.scalar_type() == at::kFloat && uniform.is_contiguous() && seeds.device().is_cpu() &&
                    seeds.scalar_type() == at::kLong && seeds.is_contiguous() && seeds.numel() == (int64_t)channels.size() &&
                    keep.size() == channels.size(), "draw_lists: host numbers expected");
    const float* u = uniform.data_ptr<float>();
    const float* end = u + uniform.numel();
    const auto options = at::TensorOptions().dtype(at::kInt).device(device);
    c10::cuda::OptionalCUDAGuard guard;
    if (device.has_index()) guard.set_device(device);
    std::vector<Tensor> out;
    std::vector<int*> at;
    std::vector<int> width, count;
    std::vector<unsigned long long> seed;
    for (size_t k = 0; k < channels.size(); k++) {
        TORCH_CHECK(channels[k] > 0 && channels[k] <= end - u, "draw_lists: too few numbers");
        const float rate = (float)keep[k];
        int64_t n = 0;
        for (const float* stop = u + channels[k]; u < stop; u++) n += *u < rate;
        n = std::min(std::max<int64_t>(n, 1), channels[k]);
        out.push_back(at::empty({subs, 1, n}, options));
        at.push_back(out.back().data_ptr<int>());
        width.push_back((int)channels[k]), count.push_back((int)n);
        seed.push_back((unsigned long long)seeds.data_ptr<int64_t>()[k]);
    }
    done(api.sample_masks((int)out.size(), at.data(), width.data(), count.data(), seed.data(), (int)subs,
                          c10::cuda::getCurrentCUDAStream(out[0].device().index()).stream()), "sample_mask_batch");
    return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const LibraryError& e) {
            PyErr_SetString(library_error, e.what());
        }
    });
    m.def("init", &init);
    m.def("dist", &dist);
    m.def("sort_neuron", &sort_neuron);
    m.def("bound_inf_dist", &bound_inf_dist);
    m.def("bound_sort_neuron", &bound_sort_neuron);
    m.def("unfold", &unfold);
    m.def("mean_shift", &mean_shift);
    m.def("add_per_channel", &add_per_channel);
    // A call that issues a whole pass takes long, and as long as the device does once the launch queue is full: other Python
    // threads run meanwhile.  None of the three touches a Python object.
    using Unlocked = py::call_guard<py::gil_scoped_release>;
    m.def("draw_lists", &draw_lists, Unlocked());
    py::class_<MlpTable>(m, "MlpTable")
        .def(py::init<std::vector<Row>>())
        .def("address", &MlpTable::address)
        .def("applies", &MlpTable::applies)
        .def("takes", &MlpTable::takes)
        .def("train_forward", &MlpTable::train_forward, Unlocked())
        .def("train_backward", &MlpTable::train_backward, Unlocked());
}
