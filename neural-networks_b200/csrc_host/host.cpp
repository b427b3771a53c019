// The host path between the Python layer API and the kernels, in C++: output allocation, argument checks and launches of the library's
// ops, and the library GEMMs of a projection in the same call.
//
// A training step of a small model is a few hundred launches of some microseconds each; from Python every one of them cost 15 to 25 us
// (tensor allocations, pointer checks and a ctypes call with up to 25 arguments, then each GEMM's own wrapper), so the device waited for
// the host. Here an op is one call of 2 to 5 us and a projection's forward or backward one call with its GEMMs inside.
#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <pybind11/stl.h>

#include <cmath>

#include "../../include/xlstm_b200.h"

namespace py = pybind11;
using at::Tensor;
typedef std::optional<Tensor> OptT;

static PyObject *g_check = nullptr, *g_error = nullptr;  // _lib.check(rc, what), _lib.XlstmError

[[noreturn]] static void refuse(const char* msg) {
    PyErr_SetString(g_error, msg);
    throw py::error_already_set();
}
static void check(int rc, const char* what) {
    if (rc == XLSTM_OK) return;
    PyObject* r = PyObject_CallFunction(g_check, "is", rc, what);
    Py_XDECREF(r);
    throw py::error_already_set();
}
static void* ptr(const Tensor& t) {
    if (!t.is_cuda()) refuse("xlstm_b200 ops take CUDA tensors only (there is no CPU path)");
    if (!t.is_contiguous()) refuse("xlstm_b200 ops take contiguous tensors");
    return t.data_ptr();
}
static void* ptr(const OptT& t) { return t ? ptr(*t) : nullptr; }
static float* fptr(const Tensor& t) { return (float*)ptr(t); }
static float* fptr(const OptT& t) { return (float*)ptr(t); }
static int dt(const Tensor& t) {
    if (t.scalar_type() == at::kFloat) return XLSTM_F32;
    if (t.scalar_type() == at::kBFloat16) return XLSTM_BF16;
    refuse("xlstm_b200 ops take fp32 or bf16 tensors");
}
static void* stream() {
    if (c10::cuda::device_count() == 0) refuse("no CUDA device: xlstm_b200 has no CPU path");
    return (void*)c10::cuda::getCurrentCUDAStream().stream();
}
static Tensor fresh(at::IntArrayRef size, at::ScalarType t, const Tensor& like) { return at::empty(size, like.options().dtype(t).requires_grad(false)); }
static at::ScalarType type_of(bool bf16) { return bf16 ? at::kBFloat16 : at::kFloat; }
static Tensor scratch(size_t bytes, const Tensor& like) { return fresh({(int64_t)(bytes ? bytes : 1)}, at::kByte, like); }
// Dispatch straight to the backend kernels: nothing here is recorded for autograd.
struct Below {
    at::AutoDispatchBelowADInplaceOrView g;
};

// ---- ops -------------------------------------------------------------------------------------------------------------------------
static py::tuple mlstm_fw(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& ig, const Tensor& fg, uintptr_t shape, const OptT& cC,
                          const OptT& cn, const OptT& cm, bool save, bool want) {
    Below guard;
    const auto* s = (const xlstm_mlstm_shape*)shape;
    const int64_t bh = (int64_t)s->B * s->H, n = (int64_t)s->B * s->T;
    Tensor y = fresh({n, (int64_t)s->H * s->dhv}, type_of(s->dtype == XLSTM_BF16), q);
    Tensor vec = fresh({3, bh, s->T}, at::kFloat, q);  // m, psi, q.n
    float* pv = (float*)vec.data_ptr();
    OptT saved, oC, on, om;
    if (save) saved = scratch(xlstm_mlstm_saved_bytes(s), q);
    if (want) {
        oC = fresh({bh, s->dhv, s->dqk}, at::kFloat, q);
        on = fresh({bh, s->dqk}, at::kFloat, q);
        om = fresh({bh}, at::kFloat, q);
    }
    const size_t wsb = xlstm_mlstm_fw_workspace_bytes(s);
    Tensor ws = scratch(wsb, q);
    check(xlstm_mlstm_fw(stream(), s, ptr(q), ptr(k), ptr(v), fptr(ig), fptr(fg), fptr(cC), fptr(cn), fptr(cm), ptr(y), pv, pv + bh * s->T,
                         pv + 2 * bh * s->T, ptr(saved), fptr(oC), fptr(on), fptr(om), ptr(ws), wsb), "mlstm_fused_fw");
    return py::make_tuple(y, vec.select(0, 0), vec.select(0, 1), vec.select(0, 2), saved, oC, on, om);
}

static py::tuple mlstm_bw(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& ig, const Tensor& fg, uintptr_t shape, const OptT& cC,
                          const OptT& cn, const OptT& cm, const Tensor& y, const Tensor& m, const Tensor& psi, const Tensor& qn, const OptT& saved,
                          const Tensor& dy, const OptT& dC, const OptT& dn, bool want) {
    Below guard;
    const auto* s = (const xlstm_mlstm_shape*)shape;
    const int64_t bh = (int64_t)s->B * s->H, n = (int64_t)s->B * s->T;
    const auto gt = type_of(s->gdtype == XLSTM_BF16);
    Tensor dq = fresh({n, (int64_t)s->H * s->dqk}, gt, q), dk = fresh({n, (int64_t)s->H * s->dqk}, gt, q), dv = fresh({n, (int64_t)s->H * s->dhv}, gt, q);
    Tensor dig = fresh({n, s->H}, at::kFloat, q), dfg = fresh({n, s->H}, at::kFloat, q);
    OptT oC, on;
    if (want) {
        oC = fresh({bh, s->dhv, s->dqk}, at::kFloat, q);
        on = fresh({bh, s->dqk}, at::kFloat, q);
    }
    const size_t wsb = xlstm_mlstm_bw_workspace_bytes(s, saved.has_value());
    Tensor ws = scratch(wsb, q);
    check(xlstm_mlstm_bw(stream(), s, ptr(q), ptr(k), ptr(v), fptr(ig), fptr(fg), fptr(cC), fptr(cn), fptr(cm), ptr(y), fptr(m), fptr(psi), fptr(qn),
                         ptr(saved), ptr(dy), fptr(dC), fptr(dn), ptr(dq), ptr(dk), ptr(dv), fptr(dig), fptr(dfg), fptr(oC), fptr(on), ptr(ws), wsb),
          "mlstm_fused_bw");
    return py::make_tuple(dq, dk, dv, dig, dfg, oC, on);
}

static void rms_fw_into(const Tensor& x, const Tensor& gamma, int group, const Tensor& out, const Tensor& inv, const OptT& xhat, float eps) {
    check(xlstm_rmsnorm_fw(stream(), ptr(x), dt(x), fptr(gamma), ptr(out), dt(out), fptr(inv), fptr(xhat), (int)x.size(0), (int)x.size(1), group, eps),
          "rms_norm_forward_into");
}
static py::tuple rms_fw(const Tensor& x, const Tensor& gamma, int group, bool bf16) {
    Below guard;
    if (group <= 0) refuse("rms_norm_forward: the group must be positive");
    Tensor y = fresh(x.sizes(), type_of(bf16), x), inv = fresh({x.size(0) * (x.size(1) / group)}, at::kFloat, x);
    rms_fw_into(x, gamma, group, y, inv, std::nullopt, 1e-6f);
    return py::make_tuple(y, inv);
}
static void rms_bw_into(const Tensor& dy, const Tensor& x, const Tensor& inv, const Tensor& gamma, int group, const Tensor& dx, const Tensor& dgamma,
                        const OptT& residual) {
    Below guard;
    const int rows = (int)dy.size(0), f = (int)dy.size(1);
    const size_t wsb = xlstm_rmsnorm_bw_workspace_bytes(rows, f);
    Tensor ws = scratch(wsb, dy);
    check(xlstm_rmsnorm_bw(stream(), fptr(dy), ptr(x), dt(x), fptr(inv), fptr(gamma), fptr(residual), ptr(dx), dt(dx), fptr(dgamma), rows, f, group, ptr(ws), wsb),
          "rms_norm_backward_into");
}
static Tensor rms_bw(const Tensor& dy, const Tensor& x, const Tensor& inv, const Tensor& gamma, int group, const Tensor& dgamma, const OptT& residual, bool bf16) {
    Below guard;
    Tensor dx = fresh(dy.sizes(), type_of(bf16), dy);
    rms_bw_into(dy, x, inv, gamma, group, dx, dgamma, residual);
    return dx;
}

static Tensor colsum_narrow(const Tensor& x, const Tensor& acc, float scale, bool narrow) {
    Below guard;
    const int rows = (int)x.size(0), cols = (int)x.size(1);
    OptT out;
    if (narrow && (x.scalar_type() != at::kBFloat16 || scale != 1.f)) out = fresh({rows, cols}, at::kBFloat16, x);
    const size_t wsb = xlstm_colsum_workspace_bytes(rows, cols);
    Tensor ws = scratch(wsb, x);
    check(xlstm_colsum_narrow(stream(), ptr(x), dt(x), rows, cols, scale, ptr(out), fptr(acc), ptr(ws), wsb), "colsum_narrow");
    return out ? *out : x;
}

static Tensor bias_rows(const Tensor& bias, int64_t rows, const OptT& residual) {
    Below guard;
    Tensor out = fresh({rows, bias.numel()}, at::kFloat, bias);
    check(xlstm_bias_rows(stream(), fptr(residual), fptr(bias), fptr(out), (int)rows, (int)bias.numel()), "bias_rows");
    return out;
}

static void cross_entropy(const Tensor& z, const Tensor& t, const Tensor& d, const Tensor& loss, const OptT& mask, float inv, float cap) {
    Below guard;
    const int rows = (int)z.size(0), c = (int)z.size(1);
    const size_t wsb = xlstm_ce_workspace_bytes(rows);
    Tensor ws = scratch(wsb, z);
    const uint32_t *tp = (const uint32_t*)ptr(t), *mp = (const uint32_t*)ptr(mask);
    if (cap > 0.f) check(xlstm_softcap_ce_fw_bw(stream(), fptr(z), tp, mp, fptr(d), fptr(loss), rows, c, inv, cap, ptr(ws), wsb), "softcap_cross_entropy");
    else check(xlstm_ce_fw_bw(stream(), fptr(z), tp, mp, fptr(d), fptr(loss), rows, c, inv, ptr(ws), wsb), "softmax_cross_entropy");
}

static Tensor swiglu_fw(const Tensor& g, const Tensor& v, bool bf16, const OptT& bg, const OptT& bv) {
    Below guard;
    Tensor out = fresh(g.sizes(), type_of(bf16), g);
    check(xlstm_swiglu_fw(stream(), ptr(g), ptr(v), dt(g), fptr(bg), fptr(bv), (int)g.size(-1), ptr(out), dt(out), (size_t)g.numel()), "swiglu_forward");
    return out;
}
static py::tuple swiglu_bw(const Tensor& d, const Tensor& g, const Tensor& v, bool bf16, const OptT& bg, const OptT& bv) {
    Below guard;
    Tensor dg = fresh(g.sizes(), type_of(bf16), g), dv = fresh(g.sizes(), type_of(bf16), g);
    check(xlstm_swiglu_bw(stream(), ptr(d), dt(d), ptr(g), ptr(v), dt(g), fptr(bg), fptr(bv), (int)g.size(-1), ptr(dg), ptr(dv), dt(dg), (size_t)g.numel()),
          "swiglu_backward");
    return py::make_tuple(dg, dv);
}
static Tensor ogate_fw(const Tensor& o, const Tensor& y, bool bf16, const OptT& bias) {
    Below guard;
    Tensor hc = fresh(o.sizes(), type_of(bf16), o);
    check(xlstm_ogate_fw(stream(), fptr(o), fptr(y), fptr(bias), (int)o.size(-1), ptr(hc), dt(hc), (size_t)o.numel()), "ogate_forward");
    return hc;
}
static py::tuple ogate_bw(const Tensor& d, const Tensor& o, const Tensor& y, bool bf16) {
    Below guard;
    Tensor dp = fresh(o.sizes(), type_of(bf16), o), dy = fresh(o.sizes(), at::kFloat, o);
    check(xlstm_ogate_bw(stream(), fptr(d), fptr(o), fptr(y), ptr(dp), dt(dp), fptr(dy), (size_t)o.numel()), "ogate_backward");
    return py::make_tuple(dp, dy);
}
static void embedding_scatter_add(const Tensor& table_g, const Tensor& ids, const Tensor& d) {
    Below guard;
    auto sorted = at::sort(ids.reshape(-1), /*stable=*/std::optional<bool>(true), 0, false);
    Tensor sid = std::get<0>(sorted).to(at::kInt), pos = std::get<1>(sorted).to(at::kInt);
    check(xlstm_embedding_scatter_add(stream(), fptr(d), (const int*)ptr(sid), (const int*)ptr(pos), fptr(table_g), (int)ids.numel(), (int)d.size(1)),
          "embedding_scatter_add");
}

// ---- projections: Y = X W + b --------------------------------------------------------------------------------------------------------
// mode 0: fp32 result with the bias; 1: the product alone, fp32; 2: residual + the product + bias (the seed is one pass, the product
// accumulates into it); 3: scale * (x W + b) rounded once to bf16, with the bias as narrow_biases leaves it; 4: the product alone as bf16.
static bool power_of_two(double s) {
    int e;
    return std::frexp(s, &e) == 0.5;
}
// The biases of a cell's narrowed projections in the operand type, from the fp32 ones at every forward call: a program may have written them
// since the last. With a factor on the bias too, the library spreads it over the whole output first and reads that back (32768 x 2048:
// 176 us); a power of two goes into the bias here, which changes no bit.
static std::vector<Tensor> narrow_biases(const std::vector<Tensor>& b, const std::vector<double>& scale) {
    Below guard;
    if (b.size() > 8 || b.size() != scale.size()) refuse("narrow_biases: at most eight, a scale each");
    const float* x[8];
    void* out[8];
    int n[8];
    float s[8];
    std::vector<Tensor> r;
    for (size_t i = 0; i < b.size(); ++i) {
        r.push_back(fresh(b[i].sizes(), at::kBFloat16, b[i]));
        x[i] = fptr(b[i]); out[i] = ptr(r[i]); n[i] = (int)b[i].numel();
        s[i] = power_of_two(scale[i]) ? (float)scale[i] : 1.f;
    }
    check(xlstm_narrow_vectors(stream(), x, out, n, s, (int)b.size()), "narrow_biases");
    return r;
}
static Tensor linear_fw(const Tensor& x, const Tensor& w, const Tensor& b, const OptT& narrowed, int mode, const OptT& residual, double scale) {
    Below guard;
    const bool bf = w.scalar_type() == at::kBFloat16;
    if (mode == 4) return at::mm(x, w);
    if (mode == 3) {
        const Tensor nb = narrowed ? *narrowed : narrow_biases({b}, {scale})[0];
        return at::addmm(nb, x, w, power_of_two(scale) ? 1.0 : scale, scale);
    }
    if (mode == 2) {
        Tensor out = bias_rows(b, residual->size(0), residual);
        if (bf) return at::addmm_out(out, out, x, w, at::kFloat);
        return out.addmm_(x, w);
    }
    if (mode == 0 && !bf) return at::addmm(b, x, w);
    Tensor y = bf ? at::mm(x, w, at::kFloat) : at::mm(x, w);
    return mode == 0 ? y.add_(b) : y;
}

// Multiply-adds up to which the fp32 weight-gradient kernel of this library measured faster than the library GEMM and the column sum (us, rows
// x k x n): 2048 x 128 x 128 12.5 against 31.5, 8192 x 256 x 256 54 against 76, 4096 x 256 x 1024 the same, 8192 x 512 x 512 174 against 127.
static constexpr int64_t kOwnGradWork = 1000000000;

// Accumulates dW and db; returns dx (added into `accum` when given), or none without `need_dx`.
static OptT linear_bw(const Tensor& dy_, const Tensor& x, const Tensor& w, const Tensor& wg, const Tensor& bg, bool need_dx, const OptT& accum,
                      double scale, bool narrow_dx) {
    Below guard;
    if (w.scalar_type() == at::kBFloat16) {
        // bias gradient and the narrowing of dy for both products in one pass over dy; a dy that arrives in bf16 is only summed, and
        // the scale rides in the products' alpha
        const bool was = dy_.scalar_type() == at::kBFloat16;
        const Tensor dy = colsum_narrow(dy_, bg, (float)scale, !was);
        const double alpha = was ? scale : 1.0;
        Tensor g = wg;
        at::addmm_out(g, g, x.t(), dy, at::kFloat, 1, alpha);
        if (!need_dx) return std::nullopt;
        const Tensor wt = w.t();
        if (!accum) {
            Tensor dx = narrow_dx ? at::mm(dy, wt) : at::mm(dy, wt, at::kFloat);
            return alpha == 1.0 ? dx : dx.mul_(alpha);
        }
        Tensor a = *accum;
        at::addmm_out(a, a, dy, wt, at::kFloat, 1, alpha);
        return a;
    }
    // fp32: the scale rides in the products' alpha as well. The kernels take rows that lie one behind the other; gradients of any other
    // strides (a transposed or expanded one), and none at all, go through the library.
    const int64_t rows = x.size(0), k = x.size(1), n = dy_.size(1);
    const bool plain = rows > 0 && dy_.is_contiguous();
    if (plain && x.is_contiguous() && rows * k * n <= kOwnGradWork) {
        const size_t wsb = xlstm_linear_grad_f32_workspace_bytes((int)rows, (int)k, (int)n);
        Tensor ws = scratch(wsb, x);
        check(xlstm_linear_grad_f32(stream(), fptr(x), fptr(dy_), fptr(wg), fptr(bg), (int)rows, (int)k, (int)n, (float)scale, ptr(ws), wsb), "linear_grad");
    } else {
        if (plain) {
            colsum_narrow(dy_, bg, (float)scale, false);
        } else {
            Tensor b = bg;
            b.add_(dy_.sum(0), scale);
        }
        Tensor g = wg;
        g.addmm_(x.t(), dy_, 1, scale);
    }
    if (!need_dx) return std::nullopt;
    const Tensor wt = w.t();
    if (!accum) {
        Tensor dx = at::mm(dy_, wt);
        return scale == 1.0 ? dx : dx.mul_(scale);
    }
    Tensor a = *accum;
    return a.addmm_(dy_, wt, 1, scale);
}

// One AdamW pass over (param, grad, m, v, decayed, bf16 shadow or None) tuples.
static void adamw(const py::list& items, double wd, double lr, double b1, double b2, double eps, double bc1, double bc2, bool zero_grad) {
    std::vector<xlstm_adamw_desc> d(items.size());
    auto at = [](const py::tuple& t, int i) -> const Tensor& {
        PyObject* o = PyTuple_GET_ITEM(t.ptr(), i);
        if (!THPVariable_Check(o)) refuse("adamw: parameter, gradient and moments must be tensors");
        return THPVariable_Unpack(o);
    };
    for (size_t i = 0; i < d.size(); ++i) {
        const py::tuple t = items[i];
        const Tensor& p = at(t, 0);
        d[i].p = fptr(p); d[i].g = fptr(at(t, 1)); d[i].m = fptr(at(t, 2)); d[i].v = fptr(at(t, 3));
        d[i].p_bf16 = PyTuple_GET_ITEM(t.ptr(), 5) == Py_None ? nullptr : ptr(at(t, 5));
        d[i].len = (uint64_t)p.numel();
        d[i].wd = PyObject_IsTrue(PyTuple_GET_ITEM(t.ptr(), 4)) ? (float)wd : 0.f;
        d[i]._pad = 0.f;
    }
    check(xlstm_adamw_multi(stream(), d.data(), (int)d.size(), (float)lr, (float)b1, (float)b2, (float)eps, (float)bc1, (float)bc2, zero_grad), "adamw_multi");
}

static uintptr_t raw_stream() { return (uintptr_t)stream(); }

void bind_plans(py::module_& m);  // plan.cpp

PYBIND11_MODULE(_host, m) {
    bind_plans(m);
    m.def("init", [](py::object check_fn, py::object error) {
        g_check = check_fn.release().ptr();
        g_error = error.release().ptr();
    });
    m.def("stream", &raw_stream);
    m.def("mlstm_fw", &mlstm_fw);
    m.def("mlstm_bw", &mlstm_bw);
    m.def("rms_fw_into", &rms_fw_into);
    m.def("rms_bw_into", &rms_bw_into);
    m.def("rms_fw", &rms_fw);
    m.def("rms_bw", &rms_bw);
    m.def("colsum_narrow", &colsum_narrow);
    m.def("bias_rows", &bias_rows);
    m.def("cross_entropy", &cross_entropy);
    m.def("swiglu_fw", &swiglu_fw);
    m.def("swiglu_bw", &swiglu_bw);
    m.def("ogate_fw", &ogate_fw);
    m.def("ogate_bw", &ogate_bw);
    m.def("embedding_scatter_add", &embedding_scatter_add);
    m.def("narrow_biases", &narrow_biases);
    m.def("linear_fw", &linear_fw);
    m.def("linear_bw", &linear_bw);
    m.def("adamw", &adamw);
}
