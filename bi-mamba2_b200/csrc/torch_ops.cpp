// The operator's host path in native code: argument checks, output and scratch allocation, the library calls and the
// autograd node of bimamba_chunk_scan_combined, for eager calls on CUDA tensors.
//
// What bounds a small problem is the host: a forward + backward pass enqueues 17 launches, and building the argument
// structures, allocating a dozen tensors and crossing into the library from Python took 200 us of the 300 us such a
// pass cost.  Here the per-pass quantities live in one allocation, scratch comes straight from the caching allocator,
// and nothing returns to the interpreter between the checks and the last launch.
//
// Everything this file does not take (torch.compile, tensor subclasses and modes, functorch, CPU tensors, arguments
// that fail a check) it hands back by returning None: the Python path then runs, or raises its precise error.
#include <ATen/ATen.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>

#include <optional>
#include <stdexcept>
#include <string>

#include "../../include/bissd.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

struct BissdError : std::runtime_error {                         // ssd._cabi.BissdError in Python
    using std::runtime_error::runtime_error;
};

void check(int rc) {
    if (rc == BISSD_OK) return;
    const char *cuda = bissd_last_cuda_error();
    std::string msg = "libbissd error " + std::to_string(rc) + ": " + bissd_strerror(rc);
    if (cuda && cuda[0]) msg += std::string(" [") + cuda + "]";
    throw BissdError(msg);
}

// Tests and debugging: a synchronising read of the device status word after every pass.
void check_device_status(bool on, const void *ws, void *stream) {
    if (!on) return;
    int st = 0;
    check(bissd_read_status(ws, stream, &st));
    if (st != 0)
        throw BissdError("libbissd device status " + std::to_string(st) + ": a device-side wait ran out; results are invalid");
}

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return BISSD_F32;
        case at::kBFloat16: return BISSD_BF16;
        case at::kHalf: return BISSD_F16;
        default: return -1;
    }
}

// Plain dense CUDA storage on `dev` that this path may take the address of.
bool plain(const Tensor &t, c10::Device dev) {
    const auto ks = t.key_set();
    return t.device() == dev && t.layout() == at::kStrided && !ks.has(c10::DispatchKey::Python) &&
           !ks.has(c10::DispatchKey::FuncTorchBatched) && !ks.has(c10::DispatchKey::FuncTorchGradWrapper) &&
           !ks.has(c10::DispatchKey::Functionalize) && !t.is_conj() && !t.is_neg() && !t._is_zerotensor();
}
bool plain(const OptTensor &t, c10::Device dev) { return !t || !t->defined() || plain(*t, dev); }
bool given(const OptTensor &t) { return t && t->defined(); }
Tensor value(const OptTensor &t) { return given(t) ? *t : Tensor(); }

// As the library reads it in place: unit inner stride and, for 16-bit tensors, 16-byte aligned rows; else a copy.
Tensor inner_contig(const Tensor &t) {
    if (!t.defined()) return t;
    const auto st = t.strides();
    bool ok = st.back() == 1;
    if (ok && t.element_size() == 2) {
        ok = reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
        for (size_t i = 0; i + 1 < st.size(); ++i) ok = ok && st[i] % 8 == 0;
    }
    return ok ? t : t.contiguous();
}
Tensor f32c(const Tensor &t) {
    if (!t.defined() || (t.scalar_type() == at::kFloat && t.is_contiguous())) return t;
    return t.to(at::kFloat).contiguous();
}
void *ptr(const Tensor &t) { return t.defined() ? const_cast<void *>(t.const_data_ptr()) : nullptr; }
bissd_tensor tensor4(const Tensor &t) {
    if (!t.defined()) return bissd_tensor{nullptr, 0, 0, 0};
    return bissd_tensor{ptr(t), t.stride(0), t.stride(1), t.stride(2)};
}
size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

struct ScanConfig {
    int64_t chunk = 0;
    bool softplus = false;
    double dt_min = 0, dt_max = 0;
    bool check_status = false;
};

// What the forward pass leaves for the backward pass, carved out of one allocation.
struct Saved {
    size_t dt_out, cs_f, cs_b, states_f, states_b, total;
    Saved(const bissd_problem &p, size_t esize) {
        const size_t nc = (p.seqlen + p.chunk_size - 1) / p.chunk_size;
        const size_t hq = align256((size_t)p.batch * p.nheads * nc * p.chunk_size * 4);
        const size_t st = align256((size_t)p.batch * nc * p.nheads * p.headdim * p.dstate * esize);
        dt_out = 0; cs_f = hq; cs_b = 2 * hq; states_f = 3 * hq; states_b = 3 * hq + st; total = 3 * hq + 2 * st;
    }
};

bissd_problem problem_of(const Tensor &x, const Tensor &dt, const Tensor &B, const Tensor &D, const Tensor &z,
                         const Tensor &dt_bias, const ScanConfig &cfg) {
    bissd_problem p{};
    p.batch = (int)x.size(0); p.seqlen = (int)x.size(1); p.nheads = (int)x.size(2); p.headdim = (int)x.size(3);
    p.ngroups = (int)B.size(2); p.dstate = (int)B.size(3); p.chunk_size = (int)cfg.chunk;
    p.x_dtype = dtype_code(x.scalar_type()); p.dt_dtype = dtype_code(dt.scalar_type());
    p.has_D = D.defined(); p.D_has_hdim = D.defined() && D.dim() == 2; p.has_z = z.defined();
    p.has_dt_bias = dt_bias.defined(); p.dt_softplus = cfg.softplus;
    p.dt_min = (float)cfg.dt_min; p.dt_max = (float)cfg.dt_max;
    return p;
}

struct ScanOut {
    Tensor out, out_x, saved, fin_f, fin_b;                      // fin_*: only when asked for
};

// One forward pass.  `keep`: the saved quantities outlive the call (a backward pass will read them), else they share
// the scratch allocation.
ScanOut scan_forward(const Tensor &x_, const Tensor &dt, const Tensor &A, const Tensor &B_, const Tensor &C_, const Tensor &D,
                     const Tensor &z_, const Tensor &dt_bias, const Tensor &init_f, const Tensor &init_b,
                     const ScanConfig &cfg, bool finals, bool keep) {
    const Tensor x = inner_contig(x_), B = inner_contig(B_), C = inner_contig(C_), z = inner_contig(z_);
    const Tensor A32 = f32c(A), D32 = f32c(D), bias32 = f32c(dt_bias), if32 = f32c(init_f), ib32 = f32c(init_b);
    const bissd_problem p = problem_of(x, dt, B, D, z, dt_bias, cfg);
    size_t ws_bytes = 0;
    check(bissd_workspace_bytes(&p, &ws_bytes, nullptr));
    const auto stream = c10::cuda::getCurrentCUDAStream(x.device().index());
    ScanOut r;
    r.out = at::empty(x.sizes(), x.options());
    if (z.defined()) r.out_x = at::empty(x.sizes(), x.options());
    const Saved at_(p, x.element_size());
    const size_t own = keep ? 0 : align256(at_.total);
    c10::DataPtr ws = c10::cuda::CUDACachingAllocator::get()->allocate(ws_bytes + own);
    char *ws_ptr = static_cast<char *>(ws.get());
    char *sv;
    if (keep) {
        r.saved = at::empty({(int64_t)at_.total}, x.options().dtype(at::kByte));
        sv = static_cast<char *>(r.saved.mutable_data_ptr());
    } else {
        sv = ws_ptr + align256(ws_bytes);
    }
    if (finals) {
        const Tensor fin = at::empty({2, x.size(0), x.size(2), x.size(3), B.size(3)}, x.options().dtype(at::kFloat));
        r.fin_f = fin.select(0, 0);
        r.fin_b = fin.select(0, 1);
    }
    bissd_fwd_args a{};
    a.p = p;
    a.x = tensor4(x); a.B = tensor4(B); a.C = tensor4(C); a.z = tensor4(z); a.dt = tensor4(dt);
    a.A = static_cast<const float *>(ptr(A32)); a.D = static_cast<const float *>(ptr(D32));
    a.dt_bias = static_cast<const float *>(ptr(bias32));
    a.out = tensor4(r.out); a.out_x = tensor4(r.out_x);
    a.dt_out = reinterpret_cast<float *>(sv + at_.dt_out); a.cs_f = reinterpret_cast<float *>(sv + at_.cs_f);
    a.cs_b = reinterpret_cast<float *>(sv + at_.cs_b);
    a.states_f = sv + at_.states_f; a.states_b = sv + at_.states_b;
    a.final_f = static_cast<float *>(ptr(r.fin_f)); a.final_b = static_cast<float *>(ptr(r.fin_b));
    a.init_f = static_cast<const float *>(ptr(if32)); a.init_b = static_cast<const float *>(ptr(ib32));
    a.phases = BISSD_PHASE_ALL;
    check(bissd_forward(&a, ws_ptr, ws_bytes, stream.stream()));
    check_device_status(cfg.check_status, ws_ptr, stream.stream());
    return r;
}

struct ScanGrads {
    Tensor dx, ddt, dA, dB, dC, dD, dz, ddt_bias, dinit_f, dinit_b;
};

ScanGrads scan_backward(const Tensor &dout_, const Tensor &x_, const Tensor &dt, const Tensor &A, const Tensor &B_,
                        const Tensor &C_, const Tensor &D, const Tensor &z_, const Tensor &dt_bias, const Tensor &out_x,
                        const Tensor &saved, const Tensor &dfin_f, const Tensor &dfin_b, bool want_dinit,
                        const ScanConfig &cfg) {
    const Tensor x = inner_contig(x_), B = inner_contig(B_), C = inner_contig(C_), z = inner_contig(z_), dout = inner_contig(dout_);
    const Tensor A32 = f32c(A), D32 = f32c(D), bias32 = f32c(dt_bias), ff32 = f32c(dfin_f), fb32 = f32c(dfin_b);
    const bissd_problem p = problem_of(x, dt, B, D, z, dt_bias, cfg);
    size_t ws_bytes = 0;
    check(bissd_workspace_bytes(&p, nullptr, &ws_bytes));
    const auto stream = c10::cuda::getCurrentCUDAStream(x.device().index());
    ScanGrads g;
    g.dx = at::empty(x.sizes(), x.options());
    if (z.defined()) g.dz = at::empty(x.sizes(), x.options());
    g.dB = at::empty(B.sizes(), B.options());
    g.dC = at::empty(C.sizes(), C.options());
    g.ddt = at::empty(dt.sizes(), dt.options());
    const auto f32 = x.options().dtype(at::kFloat);
    g.dA = at::empty({A.size(0)}, f32);
    if (dt_bias.defined()) g.ddt_bias = at::empty({A.size(0)}, f32);
    if (D.defined()) g.dD = at::empty(D.sizes(), f32);
    if (want_dinit) {
        const Tensor di = at::empty({2, x.size(0), x.size(2), x.size(3), B.size(3)}, f32);
        g.dinit_f = di.select(0, 0);
        g.dinit_b = di.select(0, 1);
    }
    const Saved at_(p, x.element_size());
    char *sv = static_cast<char *>(ptr(saved));
    c10::DataPtr ws = c10::cuda::CUDACachingAllocator::get()->allocate(ws_bytes);
    auto F = [](const Tensor &t) { return static_cast<float *>(ptr(t)); };
    bissd_bwd_args a{};
    a.p = p;
    a.x = tensor4(x); a.B = tensor4(B); a.C = tensor4(C); a.z = tensor4(z); a.dout = tensor4(dout);
    a.out_x = tensor4(out_x); a.dt = tensor4(dt);
    a.A = F(A32); a.D = F(D32); a.dt_bias = F(bias32);
    a.dt_out = reinterpret_cast<float *>(sv + at_.dt_out); a.cs_f = reinterpret_cast<float *>(sv + at_.cs_f);
    a.cs_b = reinterpret_cast<float *>(sv + at_.cs_b);
    a.states_f = sv + at_.states_f; a.states_b = sv + at_.states_b;
    a.dx = ptr(g.dx); a.dz = ptr(g.dz); a.dB = ptr(g.dB); a.dC = ptr(g.dC); a.ddt = ptr(g.ddt);
    a.dA = F(g.dA); a.dD = F(g.dD); a.ddt_bias = F(g.ddt_bias);
    a.dfinal_f = F(ff32); a.dfinal_b = F(fb32); a.dinit_f = F(g.dinit_f); a.dinit_b = F(g.dinit_b);
    a.phases = BISSD_PHASE_ALL;
    check(bissd_backward(&a, ws.get(), ws_bytes, stream.stream()));
    check_device_status(cfg.check_status, ws.get(), stream.stream());
    return g;
}

Tensor to_dtype_of(const Tensor &g, const Tensor &like) {
    return !g.defined() || g.scalar_type() == like.scalar_type() ? g : g.to(like.scalar_type());
}

// Autograd node of the eager operator.
struct ScanFn : public torch::autograd::Function<ScanFn> {
    static variable_list forward(AutogradContext *ctx, const Tensor &x, const Tensor &dt, const Tensor &A, const Tensor &B,
                                 const Tensor &C, const OptTensor &oD, const OptTensor &oz, const OptTensor &obias,
                                 const OptTensor &oif, const OptTensor &oib, int64_t chunk, bool softplus, double dt_min,
                                 double dt_max, bool finals, bool check_status) {
        const Tensor D = value(oD), z = value(oz), dt_bias = value(obias), init_f = value(oif), init_b = value(oib);
        const ScanConfig cfg{chunk, softplus, dt_min, dt_max, check_status};
        ScanOut r = scan_forward(x, dt, A, B, C, D, z, dt_bias, init_f, init_b, cfg, finals, true);
        ctx->save_for_backward({x, dt, A, B, C, D, z, dt_bias, r.out_x, r.saved});
        auto &s = ctx->saved_data;
        s["chunk"] = chunk; s["softplus"] = softplus; s["dt_min"] = dt_min; s["dt_max"] = dt_max;
        s["check_status"] = check_status;
        s["init"] = (int64_t)((init_f.defined() ? 1 : 0) | (init_b.defined() ? 2 : 0));
        ctx->set_materialize_grads(false);
        if (finals) return {r.out, r.fin_f, r.fin_b};
        return {r.out};
    }
    static variable_list backward(AutogradContext *ctx, variable_list go) {
        const variable_list v = ctx->get_saved_variables();
        const Tensor &x = v[0], &dt = v[1], &A = v[2], &B = v[3], &C = v[4], &D = v[5], &z = v[6], &dt_bias = v[7];
        auto &s = ctx->saved_data;
        const ScanConfig cfg{s["chunk"].toInt(), s["softplus"].toBool(), s["dt_min"].toDouble(), s["dt_max"].toDouble(),
                             s["check_status"].toBool()};
        const int64_t init = s["init"].toInt();
        const c10::cuda::CUDAGuard guard(x.device());
        at::AutoDispatchBelowADInplaceOrView below;              // nothing in here records a graph
        const Tensor dout = go[0].defined() ? go[0] : at::zeros(x.sizes(), x.options());
        const Tensor none;
        const ScanGrads g = scan_backward(dout, x, dt, A, B, C, D, z, dt_bias, v[8], v[9], go.size() > 1 ? go[1] : none,
                                          go.size() > 2 ? go[2] : none, init != 0, cfg);
        return {g.dx, g.ddt, to_dtype_of(g.dA, A), g.dB, g.dC, D.defined() ? to_dtype_of(g.dD, D) : none, g.dz,
                dt_bias.defined() ? to_dtype_of(g.ddt_bias, dt_bias) : none, (init & 1) ? g.dinit_f : none,
                (init & 2) ? g.dinit_b : none, none, none, none, none, none, none};
    }
};

// bimamba_chunk_scan_combined for plain CUDA tensors: the output, (output, final_f, final_b), or None where the
// arguments are for the Python path (see the head of this file).
py::object chunk_scan(const Tensor &x, const Tensor &dt, const Tensor &A, const Tensor &B, const Tensor &C, int64_t chunk,
                      const OptTensor &D, const OptTensor &z, const OptTensor &dt_bias, bool softplus, double dt_min,
                      double dt_max, bool finals, const OptTensor &init_f, const OptTensor &init_b, bool check_status) {
    if (!x.is_cuda() || x.dim() != 4 || B.dim() != 4 || dt.dim() != 3 || A.dim() != 1 || chunk < 32 || chunk > 256)
        return py::none();
    const auto dev = x.device();
    if (c10::impl::TorchDispatchModeTLS::any_modes_set()) return py::none();
    for (const Tensor *t : {&x, &dt, &A, &B, &C})
        if (!plain(*t, dev)) return py::none();
    for (const OptTensor *t : {&D, &z, &dt_bias, &init_f, &init_b})
        if (!plain(*t, dev)) return py::none();
    const int64_t b = x.size(0), L = x.size(1), H = x.size(2), P = x.size(3), G = B.size(2), N = B.size(3);
    if (x.numel() == 0 || B.numel() == 0 || H % G != 0 || B.size(0) != b || B.size(1) != L || C.sizes() != B.sizes() ||
        dt.size(0) != b || dt.size(1) != L || dt.size(2) != H || A.size(0) != H)
        return py::none();
    const auto st = x.scalar_type();
    if (dtype_code(st) < 0 || dtype_code(dt.scalar_type()) < 0 || B.scalar_type() != st || C.scalar_type() != st)
        return py::none();
    if (given(z) && (z->sizes() != x.sizes() || z->scalar_type() != st)) return py::none();
    if (given(D) && !(D->size(0) == H && (D->dim() == 1 || (D->dim() == 2 && D->size(1) == P)))) return py::none();
    if (given(dt_bias) && (dt_bias->dim() != 1 || dt_bias->size(0) != H)) return py::none();
    for (const OptTensor *t : {&init_f, &init_b})
        if (given(*t) && (*t)->numel() != b * H * P * N) return py::none();
    const Tensor none;
    auto opt = [&](const OptTensor &t) -> const Tensor & { return given(t) ? *t : none; };
    const c10::cuda::CUDAGuard guard(dev);
    bool grad = false;
    if (at::GradMode::is_enabled())
        for (const Tensor *t : {&x, &dt, &A, &B, &C, &opt(D), &opt(z), &opt(dt_bias), &opt(init_f), &opt(init_b)})
            grad = grad || (t->defined() && t->requires_grad());
    variable_list r;
    {
        py::gil_scoped_release nogil;
        if (grad) {
            r = ScanFn::apply(x, dt, A, B, C, D, z, dt_bias, init_f, init_b, chunk, softplus, dt_min,
                              dt_max, finals, check_status);
        } else {
            at::AutoDispatchBelowADInplaceOrView below;
            ScanOut o = scan_forward(x, dt, A, B, C, opt(D), opt(z), opt(dt_bias), opt(init_f), opt(init_b),
                                     ScanConfig{chunk, softplus, dt_min, dt_max, check_status}, finals, false);
            r = finals ? variable_list{o.out, o.fin_f, o.fin_b} : variable_list{o.out};
        }
    }
    if (finals) return py::make_tuple(r[0], r[1], r[2]);
    return py::cast(r[0]);
}

}  // namespace

PYBIND11_MODULE(_bissd_torch, m) {
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const BissdError &e) {
            PyErr_SetString(py::module_::import("ssd._cabi").attr("BissdError").ptr(), e.what());
        }
    });
    m.def("chunk_scan", &chunk_scan);
}
