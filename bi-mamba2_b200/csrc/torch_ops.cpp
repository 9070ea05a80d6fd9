// The operator's host path in native code: argument checks, output and scratch allocation, the library calls and the
// autograd node of bimamba_chunk_scan_combined, for eager calls on CUDA tensors.
//
// What bounds a small problem is the host: a forward + backward pass enqueues 13 launches (8 in fp32), and building the argument
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

// `call` with the least scratch its sizes need (and `extra` bytes behind it), and once more with all there may be if that
// turns out to be too little.
template <class F>
void with_workspace(const bissd_problem &p, bool forward, size_t extra, bool check_status, void *stream, F call) {
    int rc = BISSD_ERR_WORKSPACE;
    for (const auto size_of : {bissd_workspace_bytes_least, bissd_workspace_bytes}) {
        size_t bytes = 0;
        check(size_of(&p, forward ? &bytes : nullptr, forward ? nullptr : &bytes));
        const c10::DataPtr ws = c10::cuda::CUDACachingAllocator::get()->allocate(bytes + extra);
        rc = call(static_cast<char *>(ws.get()), bytes);
        if (rc == BISSD_OK) check_device_status(check_status, ws.get(), stream);
        if (rc != BISSD_ERR_WORKSPACE) break;
    }
    check(rc);
}

struct ScanOut {
    Tensor out, out_x, saved, fin_f, fin_b;                      // fin_*: only when asked for
};

// One forward pass.  `keep`: the saved quantities outlive the call (a backward pass will read them), else they share
// the scratch allocation.  With BISSD_PHASE_LOCAL alone only those are computed.
ScanOut scan_forward(const Tensor &x_, const Tensor &dt, const Tensor &A, const Tensor &B_, const Tensor &C_, const Tensor &D,
                     const Tensor &z_, const Tensor &dt_bias, const Tensor &init_f, const Tensor &init_b,
                     const ScanConfig &cfg, bool finals, bool keep, int phases = BISSD_PHASE_ALL) {
    const Tensor x = inner_contig(x_), B = inner_contig(B_), C = inner_contig(C_), z = inner_contig(z_);
    const Tensor A32 = f32c(A), D32 = f32c(D), bias32 = f32c(dt_bias), if32 = f32c(init_f), ib32 = f32c(init_b);
    const bissd_problem p = problem_of(x, dt, B, D, z, dt_bias, cfg);
    const auto stream = c10::cuda::getCurrentCUDAStream(x.device().index());
    ScanOut r;
    if (phases & BISSD_PHASE_FINISH) {
        r.out = at::empty(x.sizes(), x.options());
        if (z.defined()) r.out_x = at::empty(x.sizes(), x.options());
    }
    const Saved at_(p, x.element_size());
    if (keep) r.saved = at::empty({(int64_t)at_.total}, x.options().dtype(at::kByte));
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
    a.final_f = static_cast<float *>(ptr(r.fin_f)); a.final_b = static_cast<float *>(ptr(r.fin_b));
    a.init_f = static_cast<const float *>(ptr(if32)); a.init_b = static_cast<const float *>(ptr(ib32));
    a.phases = phases;
    const size_t own = keep ? 0 : align256(at_.total);
    with_workspace(p, true, own, cfg.check_status, stream.stream(), [&](char *ws, size_t bytes) {
        char *sv = keep ? static_cast<char *>(r.saved.mutable_data_ptr()) : ws + align256(bytes);
        a.dt_out = reinterpret_cast<float *>(sv + at_.dt_out); a.cs_f = reinterpret_cast<float *>(sv + at_.cs_f);
        a.cs_b = reinterpret_cast<float *>(sv + at_.cs_b);
        a.states_f = sv + at_.states_f; a.states_b = sv + at_.states_b;
        return bissd_forward(&a, ws, bytes, stream.stream());
    });
    return r;
}

struct ScanGrads {
    Tensor dx, ddt, dA, dB, dC, dD, dz, ddt_bias, dinit_f, dinit_b;
};

// One backward pass.  Of `g`, dx, dB, dC and ddt are written where they are given (any strides with 16-byte aligned
// rows); what is not given is allocated here.
void scan_backward(ScanGrads &g, const Tensor &dout_, const Tensor &x_, const Tensor &dt, const Tensor &A, const Tensor &B_,
                        const Tensor &C_, const Tensor &D, const Tensor &z_, const Tensor &dt_bias, const Tensor &out_x,
                        const Tensor &saved, const Tensor &dfin_f, const Tensor &dfin_b, bool want_dinit,
                        const ScanConfig &cfg) {
    const Tensor x = inner_contig(x_), B = inner_contig(B_), C = inner_contig(C_), z = inner_contig(z_), dout = inner_contig(dout_);
    const Tensor A32 = f32c(A), D32 = f32c(D), bias32 = f32c(dt_bias), ff32 = f32c(dfin_f), fb32 = f32c(dfin_b);
    const bissd_problem p = problem_of(x, dt, B, D, z, dt_bias, cfg);
    const auto stream = c10::cuda::getCurrentCUDAStream(x.device().index());
    if (!g.dx.defined()) g.dx = at::empty(x.sizes(), x.options());
    if (z.defined()) g.dz = at::empty(x.sizes(), x.options());
    if (!g.dB.defined()) g.dB = at::empty(B.sizes(), B.options());
    if (!g.dC.defined()) g.dC = at::empty(C.sizes(), C.options());
    if (!g.ddt.defined()) g.ddt = at::empty(dt.sizes(), dt.options());
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
    bissd_grad_strides gs;
    auto strides = [](int64_t *to, const Tensor &t) { for (int i = 0; i < 3; ++i) to[i] = t.stride(i); };
    strides(gs.dx, g.dx); strides(gs.dB, g.dB); strides(gs.dC, g.dC); strides(gs.ddt, g.ddt);
    with_workspace(p, false, 0, cfg.check_status, stream.stream(),
                   [&](char *ws, size_t bytes) { return bissd_backward_into(&a, &gs, ws, bytes, stream.stream()); });
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
        at::AutoDispatchBelowADInplaceOrView below;
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
        ScanGrads g;
        scan_backward(g, dout, x, dt, A, B, C, D, z, dt_bias, v[8], v[9], go.size() > 1 ? go[1] : none,
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

// ---- the layer after its input projection -----------------------------------------------------------------------
// split of zxbcdt -> depthwise conv1d + SiLU -> scan -> gated RMSNorm [-> output projection], as one autograd node.  It
// reads z, xBC and dt inside zxbcdt and writes their gradients inside dzxbcdt; the scan writes dx, dB and dC straight
// into the convolution's output gradient.  Against the separate operators that removes the copies, the concatenations
// and the small parameter kernels between them (0.9 of 7.0 ms at b16 L4096 d_model 1024) and most of the host time.
// `recompute`: keep zxbcdt, the scan's output and rstd only, and redo the rest in the backward pass.
struct LayerConfig {
    ScanConfig scan;
    int64_t headdim = 0, ngroups = 1, group = 0;
    bool a_log = false, norm_before_gate = true, recompute = false;
    double eps = 1e-5;
};
struct LayerDims {
    int64_t b, L, W, H, P, G, N, dim, channels;
};
struct LayerViews {
    Tensor z, xbc, dt;
};
struct XBC {
    Tensor x, B, C;
};

LayerViews split_in(const Tensor &zxbcdt, const LayerDims &d) {
    return {zxbcdt.narrow(2, 0, d.dim), zxbcdt.narrow(2, d.dim, d.channels), zxbcdt.narrow(2, d.dim + d.channels, d.H)};
}
XBC split_xbc(const Tensor &t, const LayerDims &d) {
    const int64_t sb = t.stride(0), sl = t.stride(1), o = t.storage_offset();
    return {t.as_strided({d.b, d.L, d.H, d.P}, {sb, sl, d.P, 1}, o),
            t.as_strided({d.b, d.L, d.G, d.N}, {sb, sl, d.N, 1}, o + d.dim),
            t.as_strided({d.b, d.L, d.G, d.N}, {sb, sl, d.N, 1}, o + d.dim + d.G * d.N)};
}

bissd_conv_args conv_args(const Tensor &x, const Tensor &w, const Tensor &bias, const Tensor &o) {
    bissd_conv_args a{};
    a.batch = (int)x.size(0); a.seqlen = (int)x.size(1); a.channels = (int)x.size(2); a.width = (int)w.size(-1);
    a.x_dtype = dtype_code(x.scalar_type()); a.w_dtype = dtype_code(w.scalar_type());
    a.x_stride_batch = x.stride(0); a.x_stride_row = x.stride(1);
    a.out_stride_batch = o.stride(0); a.out_stride_row = o.stride(1);
    a.x = ptr(x); a.weight = ptr(w); a.bias = ptr(bias);
    return a;
}
Tensor conv_forward(const Tensor &x, const Tensor &w, const Tensor &bias, void *stream) {
    Tensor out = at::empty(x.sizes(), x.options());
    bissd_conv_args a = conv_args(x, w, bias, out);
    a.out = ptr(out);
    check(bissd_dwconv_silu_forward(&a, stream));
    return out;
}
void conv_backward(const Tensor &x, const Tensor &w, const Tensor &bias, const Tensor &dout, const Tensor &dx,
                   const Tensor &dw, const Tensor &db, void *stream) {
    bissd_conv_args a = conv_args(x, w, bias, dout);
    a.dout = ptr(dout); a.dx = ptr(dx); a.dweight = ptr(dw); a.dbias = ptr(db);
    size_t need = 0;
    check(bissd_dwconv_silu_workspace_bytes(&a, &need));
    c10::DataPtr ws = c10::cuda::CUDACachingAllocator::get()->allocate(need);
    check(bissd_dwconv_silu_backward(&a, ws.get(), need, stream));
}

bissd_norm_args norm_args(const Tensor &x, const Tensor &z, const Tensor &w, const Tensor &rstd, const LayerConfig &cfg) {
    bissd_norm_args a{};
    a.hidden = (int)x.size(2); a.rows = x.size(0) * x.size(1); a.group_size = (int)cfg.group;
    a.x_dtype = dtype_code(x.scalar_type()); a.w_dtype = dtype_code(w.scalar_type());
    a.norm_before_gate = cfg.norm_before_gate; a.eps = (float)cfg.eps;
    a.stride_x = x.stride(1); a.stride_z = z.stride(1); a.stride_out = x.size(2);
    a.x = ptr(x); a.z = ptr(z); a.weight = ptr(w); a.rstd = static_cast<float *>(ptr(rstd));
    return a;
}
Tensor norm_forward(const Tensor &x, const Tensor &z, const Tensor &w, const Tensor &rstd, const LayerConfig &cfg, void *stream) {
    Tensor out = at::empty(x.sizes(), x.options());
    bissd_norm_args a = norm_args(x, z, w, rstd, cfg);
    a.out = ptr(out);
    check(bissd_rmsnorm_gated_forward(&a, stream));
    return out;
}
void norm_backward(const Tensor &x, const Tensor &z, const Tensor &w, const Tensor &rstd, const LayerConfig &cfg,
                   const Tensor &dout, const Tensor &dx, const Tensor &dz, const Tensor &dw, void *stream) {
    bissd_norm_args a = norm_args(x, z, w, rstd, cfg);
    a.dout = ptr(dout); a.dx = ptr(dx); a.dz = ptr(dz); a.dweight = ptr(dw);
    size_t need = 0;
    check(bissd_rmsnorm_gated_workspace_bytes(&a, &need));
    c10::DataPtr ws = c10::cuda::CUDACachingAllocator::get()->allocate(need);
    check(bissd_rmsnorm_gated_backward(&a, ws.get(), need, stream));
}

struct LayerParams {                                             // fp32 values the scan reads; one allocation
    Tensor A, D, bias;
};
bissd_layer_params layer_params_args(const Tensor &A, const Tensor &D, const Tensor &dt_bias, const LayerParams &p, bool a_log) {
    bissd_layer_params a{};
    a.nheads = (int)A.numel(); a.d_elems = (int)D.numel(); a.a_log = a_log;
    a.a_dtype = dtype_code(A.scalar_type()); a.d_dtype = dtype_code(D.scalar_type()); a.b_dtype = dtype_code(dt_bias.scalar_type());
    a.A = ptr(A); a.D = ptr(D); a.dt_bias = ptr(dt_bias);
    auto F = [](const Tensor &t) { return static_cast<float *>(ptr(t)); };
    a.A32 = F(p.A); a.D32 = F(p.D); a.dt_bias32 = F(p.bias);
    return a;
}
LayerParams carve_params(const Tensor &buf, const Tensor &A, const Tensor &D) {
    const int64_t h = A.numel();
    return {buf.narrow(0, 0, h), buf.narrow(0, 2 * h, D.numel()).view(D.sizes()), buf.narrow(0, h, h)};
}

struct LayerSaved {
    Tensor xbc_conv, scan_out, rstd, params, saved;
};

// zxbcdt -> the norm's output; what the backward pass reads goes to `keep` when it is given.
Tensor layer_forward(const Tensor &zxbcdt, const Tensor &conv_w, const Tensor &conv_b, const Tensor &dt_bias, const Tensor &A,
                     const Tensor &D, const Tensor &norm_w, const LayerConfig &cfg, const LayerDims &d, LayerSaved *keep) {
    void *stream = c10::cuda::getCurrentCUDAStream(zxbcdt.device().index()).stream();
    const LayerViews v = split_in(zxbcdt, d);
    const auto f32 = zxbcdt.options().dtype(at::kFloat);
    const Tensor buf = at::empty({2 * d.H + D.numel()}, f32);
    const LayerParams p = carve_params(buf, A, D);
    const bissd_layer_params pa = layer_params_args(A, D, dt_bias, p, cfg.a_log);
    check(bissd_layer_params_in(&pa, stream));
    const Tensor xbc = conv_forward(v.xbc, conv_w, conv_b, stream);
    const XBC s = split_xbc(xbc, d);
    const Tensor none;
    const ScanOut r = scan_forward(s.x, v.dt, p.A, s.B, s.C, p.D, none, p.bias, none, none, cfg.scan, false,
                                   keep && !cfg.recompute);
    const Tensor scan_out = r.out.view({d.b, d.L, d.dim});
    const Tensor rstd = at::empty({d.b * d.L, d.dim / cfg.group}, f32);
    const Tensor y = norm_forward(scan_out, v.z, norm_w, rstd, cfg, stream);
    if (keep) {
        keep->scan_out = scan_out; keep->rstd = rstd; keep->params = buf;
        if (!cfg.recompute) { keep->xbc_conv = xbc; keep->saved = r.saved; }
    }
    return y;
}

struct LayerFn : public torch::autograd::Function<LayerFn> {
    static variable_list forward(AutogradContext *ctx, const Tensor &zxbcdt, const Tensor &conv_w, const OptTensor &conv_b,
                                 const Tensor &dt_bias, const Tensor &A, const Tensor &D, const Tensor &norm_w,
                                 const OptTensor &out_w, const OptTensor &out_b, LayerConfig cfg, LayerDims d) {
        at::AutoDispatchBelowADInplaceOrView below;
        LayerSaved k;
        const Tensor cb = value(conv_b), ow = value(out_w), ob = value(out_b);
        Tensor y = layer_forward(zxbcdt, conv_w, cb, dt_bias, A, D, norm_w, cfg, d, &k);
        ctx->save_for_backward({zxbcdt, conv_w, cb, dt_bias, A, D, norm_w, ow, ob, k.xbc_conv, k.scan_out, k.rstd, k.params, k.saved});
        auto &s = ctx->saved_data;
        s["i"] = std::vector<int64_t>{cfg.scan.chunk, cfg.headdim, cfg.ngroups, cfg.group, cfg.a_log, cfg.norm_before_gate,
                                      cfg.recompute, cfg.scan.check_status, d.b, d.L, d.W, d.H, d.P, d.G, d.N, d.dim, d.channels};
        s["d"] = std::vector<double>{cfg.scan.dt_min, cfg.scan.dt_max, cfg.eps};
        return {ow.defined() ? at::linear(y, ow, out_b) : y};
    }
    static variable_list backward(AutogradContext *ctx, variable_list go) {
        const variable_list v = ctx->get_saved_variables();
        const Tensor &zxbcdt = v[0], &conv_w = v[1], &conv_b = v[2], &dt_bias = v[3], &A = v[4], &D = v[5], &norm_w = v[6],
                     &out_w = v[7], &out_b = v[8], &scan_out = v[10], &rstd = v[11], &params = v[12];
        const auto i = ctx->saved_data["i"].toIntVector();
        const auto f = ctx->saved_data["d"].toDoubleVector();
        LayerConfig cfg;
        cfg.scan = ScanConfig{i[0], true, f[0], f[1], i[7] != 0};
        cfg.headdim = i[1]; cfg.ngroups = i[2]; cfg.group = i[3]; cfg.a_log = i[4]; cfg.norm_before_gate = i[5];
        cfg.recompute = i[6]; cfg.eps = f[2];
        const LayerDims d{i[8], i[9], i[10], i[11], i[12], i[13], i[14], i[15], i[16]};
        const c10::cuda::CUDAGuard guard(zxbcdt.device());
        at::AutoDispatchBelowADInplaceOrView below;
        void *stream = c10::cuda::getCurrentCUDAStream(zxbcdt.device().index()).stream();
        const Tensor none;
        Tensor xbc = v[9], saved = v[13];
        const LayerViews in = split_in(zxbcdt, d);
        if (cfg.recompute) xbc = conv_forward(in.xbc, conv_w, conv_b, stream);
        const XBC s = split_xbc(xbc, d);
        const LayerParams p = carve_params(params, A, D);
        if (cfg.recompute)
            saved = scan_forward(s.x, in.dt, p.A, s.B, s.C, p.D, none, p.bias, none, none, cfg.scan, false, true,
                                 BISSD_PHASE_LOCAL).saved;
        Tensor dy = go[0].contiguous(), dout_w, dout_b;
        if (out_w.defined()) {
            const Tensor dres = dy.view({d.b * d.L, out_w.size(0)});
            dy = at::mm(dres, out_w).view({d.b, d.L, d.dim});
            const Tensor y = norm_forward(scan_out, in.z, norm_w, at::empty_like(rstd), cfg, stream);
            dout_w = at::mm(dres.t(), y.view({d.b * d.L, d.dim}));
            if (out_b.defined()) dout_b = dres.sum(0);
        }
        const Tensor dz_all = at::empty(zxbcdt.sizes(), zxbcdt.options());
        const LayerViews g = split_in(dz_all, d);
        const Tensor dscan = at::empty({d.b, d.L, d.dim}, zxbcdt.options());
        const Tensor dnorm_w = at::empty(norm_w.sizes(), norm_w.options());
        norm_backward(scan_out, in.z, norm_w, rstd, cfg, dy, dscan, g.z, dnorm_w, stream);
        const Tensor dxbc = at::empty({d.b, d.L, d.channels}, zxbcdt.options());
        const XBC gs = split_xbc(dxbc, d);
        ScanGrads sg;
        sg.dx = gs.x; sg.dB = gs.B; sg.dC = gs.C; sg.ddt = g.dt;
        scan_backward(sg, dscan.view({d.b, d.L, d.H, d.P}), s.x, in.dt, p.A, s.B, s.C, p.D, none, p.bias, none, saved, none, none,
                      false, cfg.scan);
        const Tensor dconv_w = at::empty(conv_w.sizes(), conv_w.options());
        const Tensor dconv_b = conv_b.defined() ? at::empty(conv_b.sizes(), conv_b.options()) : none;
        conv_backward(in.xbc, conv_w, conv_b, dxbc, g.xbc, dconv_w, dconv_b, stream);
        const Tensor dA = at::empty(A.sizes(), A.options()), dD = at::empty(D.sizes(), D.options()),
                     dbias = at::empty(dt_bias.sizes(), dt_bias.options());
        bissd_layer_params pa = layer_params_args(A, D, dt_bias, p, cfg.a_log);
        auto F = [](const Tensor &t) { return static_cast<const float *>(ptr(t)); };
        pa.dA32 = F(sg.dA); pa.dD32 = F(sg.dD); pa.ddt_bias32 = F(sg.ddt_bias);
        pa.dA = ptr(dA); pa.dD = ptr(dD); pa.ddt_bias = ptr(dbias);
        check(bissd_layer_params_out(&pa, stream));
        return {dz_all, dconv_w, dconv_b, dbias, dA, dD, dnorm_w, dout_w, dout_b, none, none};
    }
};

// The layer's node for plain CUDA tensors whose slices of zxbcdt the kernels read in place; None otherwise.
py::object layer(const Tensor &zxbcdt, const Tensor &conv_w, const OptTensor &conv_b, const Tensor &dt_bias, const Tensor &A,
                 bool a_log, const Tensor &D, int64_t chunk, double dt_min, double dt_max, const Tensor &norm_w, double eps,
                 int64_t group, bool norm_before_gate, int64_t headdim, int64_t ngroups, bool recompute, const OptTensor &out_w,
                 const OptTensor &out_b, bool check_status) {
    if (!zxbcdt.is_cuda() || zxbcdt.dim() != 3 || zxbcdt.numel() == 0 || !zxbcdt.is_contiguous() || chunk < 32 || chunk > 256 ||
        c10::impl::TorchDispatchModeTLS::any_modes_set())
        return py::none();
    const auto dev = zxbcdt.device();
    const auto st = zxbcdt.scalar_type();
    for (const Tensor *t : {&zxbcdt, &conv_w, &dt_bias, &A, &D, &norm_w})
        if (!plain(*t, dev) || !t->is_contiguous() || dtype_code(t->scalar_type()) < 0) return py::none();
    for (const OptTensor *t : {&conv_b, &out_w, &out_b})
        if (!plain(*t, dev) || (given(*t) && !(*t)->is_contiguous())) return py::none();
    LayerDims d{};
    d.b = zxbcdt.size(0); d.L = zxbcdt.size(1); d.W = zxbcdt.size(2);
    d.H = A.numel(); d.P = headdim; d.G = ngroups; d.dim = d.H * d.P;
    d.channels = conv_w.size(0);
    if (d.P <= 0 || d.G <= 0 || d.H % d.G || (d.channels - d.dim) <= 0 || (d.channels - d.dim) % (2 * d.G)) return py::none();
    d.N = (d.channels - d.dim) / (2 * d.G);
    const int64_t width = conv_w.size(-1);
    if (d.W != d.dim + d.channels + d.H || conv_w.numel() != d.channels * width || width % 2 == 0 || width > 7 || d.channels % 8 ||
        dt_bias.numel() != d.H || (D.numel() != d.H && D.numel() != d.dim) || D.dim() != (D.numel() == d.H ? 1 : 2) ||
        norm_w.numel() != d.dim)
        return py::none();
    auto weight_ok = [&](at::ScalarType t) { return t == st || t == at::kFloat; };
    if (!weight_ok(conv_w.scalar_type()) || !weight_ok(norm_w.scalar_type()) ||
        (given(conv_b) && (conv_b->scalar_type() != conv_w.scalar_type() || conv_b->numel() != d.channels)))
        return py::none();
    if (group <= 0 || group % 256 || d.dim % group || d.dim > 4096) return py::none();
    if (given(out_w) && (out_w->dim() != 2 || out_w->size(1) != d.dim || out_w->scalar_type() != st)) return py::none();
    if (given(out_b) && (!given(out_w) || out_b->scalar_type() != st)) return py::none();
    // z and xBC are read, and their gradients written, inside zxbcdt's rows
    if (d.W % 8 || d.dim % 8 || reinterpret_cast<uintptr_t>(zxbcdt.const_data_ptr()) % 16 || d.P % 8 || d.N % 8) return py::none();
    LayerConfig cfg;
    cfg.scan = ScanConfig{chunk, true, dt_min, dt_max, check_status};
    cfg.headdim = headdim; cfg.ngroups = ngroups; cfg.group = group; cfg.a_log = a_log; cfg.norm_before_gate = norm_before_gate;
    cfg.recompute = recompute; cfg.eps = eps;
    const c10::cuda::CUDAGuard guard(dev);
    bool grad = false;
    if (at::GradMode::is_enabled()) {
        for (const Tensor *t : {&zxbcdt, &conv_w, &dt_bias, &A, &D, &norm_w}) grad = grad || t->requires_grad();
        for (const OptTensor *t : {&conv_b, &out_w, &out_b}) grad = grad || (given(*t) && (*t)->requires_grad());
    }
    Tensor r;
    {
        py::gil_scoped_release nogil;
        if (grad) {
            r = LayerFn::apply(zxbcdt, conv_w, conv_b, dt_bias, A, D, norm_w, out_w, out_b, cfg, d)[0];
        } else {
            at::AutoDispatchBelowADInplaceOrView below;
            r = layer_forward(zxbcdt, conv_w, value(conv_b), dt_bias, A, D, norm_w, cfg, d, nullptr);
            if (given(out_w)) r = at::linear(r, *out_w, out_b);
        }
    }
    return py::cast(r);
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
    m.def("layer", &layer);
}
