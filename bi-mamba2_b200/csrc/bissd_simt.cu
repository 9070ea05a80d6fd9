// Launch code of the CUDA-core family (simt_products.cuh).
#include <type_traits>

#include "layouts.cuh"
#include "simt_products.cuh"

namespace bissd {

// Four-element access: pointers and strides that keep every row piece aligned to the four elements.
static bool quad(const void *p, size_t esize, long long a, long long b, long long c, int inner) {
    return !p || (reinterpret_cast<uintptr_t>(p) % (4 * esize) == 0 && a % 4 == 0 && b % 4 == 0 && c % 4 == 0 && inner % 4 == 0);
}
template <class V> static bool quad(const V &v, size_t esize, int inner) { return quad(v.ptr, esize, v.sb, v.sl, v.sh, inner); }

static int base_flags(const Dims &d) {
    return (d.Q % 4 == 0 ? simt::VEC_Q : 0) | (d.N % 4 == 0 ? simt::VEC_N : 0) | (d.P % 4 == 0 ? simt::VEC_P : 0);
}

// 16-bit inputs get here only with shapes the tensor cores refuse: they use 64-wide tiles throughout.
template <class T> static int tile_width(int n) { return std::is_same<T, float>::value ? simt::width_for(n) : 64; }
template <class T, class F> static int by_width(int width, F f) {
    if constexpr (std::is_same<T, float>::value) {
        if (width == 16) return f(std::integral_constant<int, 16>());
        if (width == 32) return f(std::integral_constant<int, 32>());
    }
    return f(std::integral_constant<int, 64>());
}

template <class T, bool GRAD>
static int launch_states(const Dims &d, const simt::StateArgs &sa, const View &Cm, const View &Bm, float *CB, int vec, bool states,
                         bool with_cb, int *header, cudaStream_t s) {
    const int tw = tile_width<T>(d.P), nt = ceil_div(d.Q, simt::TILE);
    const int first = states ? d.b * d.nc * d.H * ceil_div(2 * d.N, simt::TILE) * ceil_div(d.P, tw) : 0;
    const int cb = with_cb ? d.b * d.nc * d.G * nt * nt : 0;
    if (first + cb == 0) return BISSD_OK;
    return by_width<T>(tw, [&](auto width) -> int {
        BISSD_LAUNCH(GRAD ? "dstates_cb" : "chunk_state_cb", launch_pdl(simt::states_and_cb<T, GRAD, decltype(width)::value>, first + cb,
            simt::TB, sizeof(simt::Panels), s, d, sa, Cm, Bm, CB, vec, first, header));
        return BISSD_OK;
    });
}

template <class T> static int forward_t(const bissd_fwd_args &a, const Dims &d, char *ws, cudaStream_t s) {
    const FwdWs w = fwd_layout(d);
    float *loc = reinterpret_cast<float *>(ws + w.loc), *CB = reinterpret_cast<float *>(ws + w.cb);
    const View x = view_of(a.x), Bm = view_of(a.B), Cm = view_of(a.C), z = view_of(a.z);
    const MutView out = mview_of(a.out), out_x = mview_of(a.out_x);
    const bool local = a.phases & BISSD_PHASE_LOCAL, finish = a.phases & BISSD_PHASE_FINISH;
    int vec = base_flags(d);
    if (quad(x, sizeof(T), d.P) && quad(z, sizeof(T), d.P) && quad(out, sizeof(T), d.P) && quad(out_x, sizeof(T), d.P)) vec |= simt::VEC_X;
    if (quad(Bm, sizeof(T), d.N) && quad(Cm, sizeof(T), d.N)) vec |= simt::VEC_BC;
    simt::StateArgs sa{};
    sa.X = x; sa.Y = Bm;
    sa.dt = a.dt.ptr; sa.dt_dtype = a.p.dt_dtype; sa.dsb = a.dt.stride_batch; sa.dsl = a.dt.stride_seq; sa.dsh = a.dt.stride_head;
    sa.A = a.A; sa.dt_bias = a.dt_bias; sa.dt_out = a.dt_out; sa.cs_f = a.cs_f; sa.cs_b = a.cs_b; sa.out = loc;
    int rc = launch_states<T, false>(d, sa, Cm, Bm, CB, vec, local, finish, local ? reinterpret_cast<int *>(ws) : nullptr, s);
    if (rc != BISSD_OK) return rc;
    // the recurrence runs in both phases: from zero (or init_*) in LOCAL, again with init_* in FINISH
    if (local || a.init_f || a.init_b) {
        if (pass_by4(d)) {
            BISSD_LAUNCH("state_passing_fwd", launch_pdl(pass_ahead(d) ? simt::state_passing_fwd4<T, 8> : simt::state_passing_fwd4<T, 1>, pass_grid(d), pass_threads(d), 0, s,
                d, loc, a.cs_f, a.cs_b, a.init_f, a.init_b, a.states_f, a.states_b, a.final_f, a.final_b));
        } else {
            BISSD_LAUNCH("state_passing_fwd", simt::state_passing_fwd<T><<<dim3(d.b * d.H, ceil_div(d.P * d.N, simt::TB), 2), simt::TB, 0, s>>>(
                d, loc, a.cs_f, a.cs_b, a.init_f, a.init_b, a.states_f, a.states_b, a.final_f, a.final_b));
        }
    }
    if (finish) {
        const int tw = tile_width<T>(d.P);
        simt::ScanArgs sc{x, Cm, z, a.D, a.dt_out, a.cs_f, a.cs_b, CB, a.states_f, a.states_b, out, out_x};
        const int blocks = d.b * d.nc * d.H * ceil_div(d.Q, simt::TILE) * ceil_div(d.P, tw);
        return by_width<T>(tw, [&](auto width) -> int {
            BISSD_LAUNCH("chunk_scan", launch_pdl(simt::chunk_scan<T, decltype(width)::value>, blocks, simt::TB, sizeof(simt::Panels), s, d, sc, vec));
            return BISSD_OK;
        });
    }
    return BISSD_OK;
}

template <class T> static int backward_t(const bissd_bwd_args &a, const GradViews &gr, const Dims &d, char *ws, cudaStream_t s) {
    const BwdWs w = bwd_layout(d, false);
    auto F = [&](size_t off) { return reinterpret_cast<float *>(ws + off); };
    const View x = view_of(a.x), Bm = view_of(a.B), Cm = view_of(a.C), z = view_of(a.z), dout = view_of(a.dout), out_x = view_of(a.out_x);
    const bool local = a.phases & BISSD_PHASE_LOCAL, finish = a.phases & BISSD_PHASE_FINISH;
    int vec = base_flags(d);
    bool vx = true, vbc = true;
    for (const View &v : {x, z, dout, out_x}) vx = vx && quad(v, sizeof(T), d.P);
    for (const View &v : {Bm, Cm}) vbc = vbc && quad(v, sizeof(T), d.N);
    if (vx && quad(gr.dx, sizeof(T), d.P)) vec |= simt::VEC_X;
    if (vbc && quad(gr.dB, sizeof(T), d.N) && quad(gr.dC, sizeof(T), d.N)) vec |= simt::VEC_BC;
    if (!quad(a.dz, sizeof(T), 0, 0, 0, d.P)) vec &= ~simt::VEC_P;
    simt::StateArgs sa{};
    sa.X = dout; sa.Y = Cm; sa.z = z;
    sa.cs_f = const_cast<float *>(a.cs_f); sa.cs_b = const_cast<float *>(a.cs_b); sa.out = F(w.gloc);
    int rc = launch_states<T, true>(d, sa, Cm, Bm, F(w.cb), vec, local, finish, local ? reinterpret_cast<int *>(ws) : nullptr, s);
    if (rc != BISSD_OK) return rc;
    if (local || a.dfinal_f || a.dfinal_b) {
        if (pass_by4(d)) {
            BISSD_LAUNCH("state_passing_bwd", launch_pdl(pass_ahead(d) ? simt::state_passing_bwd4<T, 8, 0> : simt::state_passing_bwd4<T, 1, 0>, pass_grid(d), pass_threads(d), 0, s,
                d, F(w.gloc), a.states_f, a.states_b, a.cs_f, a.cs_b, a.dfinal_f, a.dfinal_b, F(w.E), nullptr, F(w.dTpart), a.dinit_f, a.dinit_b));
        } else {
            BISSD_LAUNCH("state_passing_bwd", simt::state_passing_bwd<T><<<dim3(d.b * d.H, ceil_div(d.P * d.N, simt::TB), 2), simt::TB, 0, s>>>(
                d, F(w.gloc), a.states_f, a.states_b, a.cs_f, a.cs_b, a.dfinal_f, a.dfinal_b, F(w.E), nullptr, F(w.dTpart), a.dinit_f, a.dinit_b));
        }
    }
    if (!finish) return BISSD_OK;
    simt::BwdArgs ba{};
    ba.x = x; ba.Bm = Bm; ba.Cm = Cm; ba.z = z; ba.dout = dout; ba.out_x = out_x;
    ba.D = a.D; ba.dt_out = a.dt_out; ba.cs_f = a.cs_f; ba.cs_b = a.cs_b; ba.CB = F(w.cb); ba.E = F(w.E);
    ba.states_f = a.states_f; ba.states_b = a.states_b;
    ba.dx = gr.dx; ba.dB = gr.dB; ba.dC = gr.dC; ba.dz = a.dz;
    ba.ddt_out = F(w.ddt_out); ba.dDpart = F(w.dDpart); ba.dB_part = F(w.dB_part); ba.dC_part = F(w.dC_part);
    ba.nf = F(w.nf); ba.nb = F(w.nb); ba.pf = F(w.pf); ba.pb = F(w.pb); ba.dCB = F(w.dCB); ba.u = F(w.u4);
    ba.hsplit = w.hsplit; ba.parts = simt_parts(d);
    const int nt = w.nlt, bch = d.b * d.nc * d.H, bcg = d.b * d.nc * d.G;
    const int dcb = bcg * w.hsplit * nt * nt, dx = bch * nt, dbc = bch * nt * 2;
    const int twp = tile_width<T>(d.P), twn = tile_width<T>(d.N);
    rc = by_width<T>(twp, [&](auto wp) {
        return by_width<T>(twn, [&](auto wn) -> int {
            BISSD_LAUNCH("dcb_dx_dbc", launch_pdl(simt::backward2<T, decltype(wp)::value, decltype(wn)::value>, dcb + dx + dbc, simt::TB,
                sizeof(simt::Panels), s, d, ba, vec, dcb, dx));
            return BISSD_OK;
        });
    });
    if (rc != BISSD_OK) return rc;
    simt::CumsumBwd cs{};
    cs.dt = a.dt.ptr; cs.dt_dtype = a.p.dt_dtype; cs.dsb = a.dt.stride_batch; cs.dsl = a.dt.stride_seq; cs.dsh = a.dt.stride_head;
    cs.A = a.A; cs.dt_bias = a.dt_bias; cs.dt_out = a.dt_out; cs.ddt_out = F(w.ddt_out);
    cs.nf = F(w.nf); cs.nb = F(w.nb); cs.pf = F(w.pf); cs.pb = F(w.pb); cs.u4 = F(w.u4); cs.u4_tiles = 2 * nt;
    cs.dTpart = F(w.dTpart); cs.nblk = w.nslots; cs.nsplit = 1; cs.ddt = gr.ddt; cs.dApart = F(w.dApart); cs.dbiaspart = F(w.dbiaspart);
    const int bmm = bcg * 2 * nt * ceil_div(d.N, twn);
    rc = by_width<T>(twn, [&](auto width) -> int {
        BISSD_LAUNCH("bmm_bwd_cumsum_bwd", launch_pdl(simt::backward3<T, decltype(width)::value>, bmm + bch, simt::TB, sizeof(simt::Panels), s,
            d, ba, cs, vec, bmm));
        return BISSD_OK;
    });
    if (rc != BISSD_OK) return rc;
    BISSD_LAUNCH("final_reduce", launch_pdl(simt::final_reduce<1024>, d.H, 1024, 0, s, d, F(w.dApart), F(w.dbiaspart),
        d.has_D ? F(w.dDpart) : nullptr, nt, 0, a.dA, d.has_bias ? a.ddt_bias : nullptr, d.has_D ? a.dD : nullptr));
    return BISSD_OK;
}

int simt_forward(const bissd_fwd_args &a, const Dims &d, char *ws, cudaStream_t s) {
    switch (a.p.x_dtype) {
        case BISSD_F32: return forward_t<float>(a, d, ws, s);
        case BISSD_BF16: return forward_t<__nv_bfloat16>(a, d, ws, s);
        default: return forward_t<__half>(a, d, ws, s);
    }
}
int simt_backward(const bissd_bwd_args &a, const GradViews &gr, const Dims &d, char *ws, cudaStream_t s) {
    switch (a.p.x_dtype) {
        case BISSD_F32: return backward_t<float>(a, gr, d, ws, s);
        case BISSD_BF16: return backward_t<__nv_bfloat16>(a, gr, d, ws, s);
        default: return backward_t<__half>(a, gr, d, ws, s);
    }
}

}  // namespace bissd
