// C ABI of libbissd (declared in include/bissd.h): argument validation, workspace layout, kernel sequencing.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include "common.cuh"
#include "host.cuh"
#include "layouts.cuh"
#include "side_stream.h"
#include "simt_kernels.cuh"
#include "tc_intra.cuh"
#include "tc_intra_sums.cuh"
#include "tc_intra_grp.cuh"
#include "tc_kernels.cuh"
#include "tc_dbc_tma.cuh"
#include "tc_dcb_tma.cuh"
#include "tc_bmm_tma.cuh"
#include "tc_cumsum.cuh"
#include "tc_dx_tma.cuh"
#include "tc_scan_tma.cuh"
#include "tc_scan_ws.cuh"
#include "tc_selftest.cuh"
#include "tc_state_tma.cuh"
#include "tc_walk_tma.cuh"

namespace bissd {

// ---- state declared in host.cuh ----------------------------------------------------------------------------
thread_local char g_cuda_err[256] = "";
std::mutex g_trace_mu;
std::vector<TraceRec> g_trace;
std::atomic<int> g_trace_on{0};
std::atomic<unsigned long long> g_launches{0};

// A second stream for the group-walking backward kernels: prev_terms_grp, which nothing before cumsum_bwd reads, forks from
// the caller's stream after the dx kernel and shares the GPU with the fused dCB / decay-gradient kernel; dbc_accum_grp goes
// with it where it writes partial results, or follows that kernel where it finishes dB and dC itself, then beside
// cumsum_bwd and final_reduce.  Each of these leaves a seventh of the SMs idle when it runs alone.  Stream order as the
// caller sees it is unchanged, also under stream capture (the side stream joins the capture through the events) and when a
// launch fails (side_stream.h).  BISSD_NO_SIDE=1 keeps everything on the caller's stream.
static bool side_allowed() {
    static const bool off = [] { const char *e = getenv("BISSD_NO_SIDE"); return e && e[0] == '1'; }();
    return !off && !g_trace_on.load(std::memory_order_relaxed);  // traced runs time every kernel alone, in line
}

// C and B as (dstate, group, seqlen, batch) tensors read in boxes of 64 state columns x 128 rows
template <class Args> static bool make_cb_maps(const Args &a, const Dims &d, CUtensorMap *mC, CUtensorMap *mB) {
    const unsigned long long dims[4] = {(unsigned long long)d.N, (unsigned long long)d.G, (unsigned long long)d.L, (unsigned long long)d.b};
    const unsigned long long sC[3] = {(unsigned long long)a.C.stride_head * 2, (unsigned long long)a.C.stride_seq * 2, (unsigned long long)a.C.stride_batch * 2};
    const unsigned long long sB[3] = {(unsigned long long)a.B.stride_head * 2, (unsigned long long)a.B.stride_seq * 2, (unsigned long long)a.B.stride_batch * 2};
    const unsigned box[4] = {64, 1, 128, 1};
    return tc::make_map4(mC, a.p.x_dtype, a.C.ptr, dims, sC, box) && tc::make_map4(mB, a.p.x_dtype, a.B.ptr, dims, sB, box);
}

// A 16-bit [Q x Q] tile per (batch, chunk, group) in boxes of 64 columns x 128 rows
static bool make_tile_map(const Dims &d, const void *ptr, CUtensorMap *m) {
    return tc::make_map2(m, BISSD_BF16, ptr, d.Q, (unsigned long long)d.b * d.nc * d.G * d.Q, 64, 128);
}

static int make_dims(const bissd_problem &p, Dims *d) {
    if (p.batch <= 0 || p.seqlen <= 0 || p.nheads <= 0 || p.headdim <= 0 || p.ngroups <= 0 || p.dstate <= 0)
        return BISSD_ERR_SHAPE;
    if (p.nheads % p.ngroups != 0) return BISSD_ERR_SHAPE;
    // the reference requires chunk_size >= 32 (src/ssd/bi/ssd_combined.py:306); 256 is this library's ceiling
    if (p.chunk_size < 32 || p.chunk_size > 256) return BISSD_ERR_SHAPE;
    if (p.x_dtype < BISSD_F32 || p.x_dtype > BISSD_F16 || p.dt_dtype < BISSD_F32 || p.dt_dtype > BISSD_F16)
        return BISSD_ERR_DTYPE;
    d->b = p.batch; d->L = p.seqlen; d->H = p.nheads; d->P = p.headdim; d->G = p.ngroups; d->N = p.dstate;
    d->Q = p.chunk_size; d->nc = ceil_div(p.seqlen, p.chunk_size); d->R = p.nheads / p.ngroups;
    d->has_D = p.has_D; d->D_hdim = p.D_has_hdim; d->has_z = p.has_z; d->has_bias = p.has_dt_bias;
    d->softplus = p.dt_softplus; d->dt_min = p.dt_min; d->dt_max = p.dt_max;
    return BISSD_OK;
}

// ---- which kernel family ---------------------------------------------------------------------------------
static bool tc_shape_ok(const bissd_problem &p) {
    return (p.x_dtype == BISSD_BF16 || p.x_dtype == BISSD_F16) && p.headdim % 8 == 0 && p.dstate % 8 == 0 &&
           p.chunk_size % 8 == 0 && p.headdim <= 256 && p.dstate <= 256;
}
static bool aligned16(const bissd_tensor &t) {
    if (!t.ptr) return true;
    return (reinterpret_cast<uintptr_t>(t.ptr) % 16 == 0) && t.stride_batch % 8 == 0 && t.stride_seq % 8 == 0 &&
           t.stride_head % 8 == 0;
}
static bool all_aligned16(const void *a, const void *b, const void *c) {
    return (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) % 16 == 0;
}
// states_f and states_b: 16-byte pieces, or four elements where the CUDA-core kernels take four at a time
static bool states_aligned(const bissd_problem &p, bool tcp, const void *f, const void *b) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(f) | reinterpret_cast<uintptr_t>(b);
    return at % (tcp || p.x_dtype == BISSD_F32 ? 16 : 8) == 0 || (!tcp && (long long)p.headdim * p.dstate % 4 != 0);
}
static bool force_simt() {
    static const bool v = [] { const char *e = getenv("BISSD_FORCE_SIMT"); return e && e[0] == '1'; }();
    return v;
}

static bool no_ws() {    // BISSD_NO_WS=1: keep the one-tile-per-CTA TMA kernels where a persistent variant exists
    static const bool v = [] { const char *e = getenv("BISSD_NO_WS"); return e && e[0] == '1'; }();
    return v;
}
static bool no_sums() {  // BISSD_NO_SUMS=1: keep the prefix-sweep form of the intra-chunk decay gradient
    static const bool v = [] { const char *e = getenv("BISSD_NO_SUMS"); return e && e[0] == '1'; }();
    return v;
}

static bool no_fused() {  // BISSD_NO_FUSED=1: separate dCB and intra-chunk decay-gradient kernels (for A/B comparisons)
    static const bool v = [] { const char *e = getenv("BISSD_NO_FUSED"); return e && e[0] == '1'; }();
    return v;
}

static bool no_tma() {   // BISSD_NO_TMA=1: keep the thread-staged tcgen05 kernels (for A/B comparisons)
    static const bool v = [] { const char *e = getenv("BISSD_NO_TMA"); return e && e[0] == '1'; }();
    return v;
}

// rank-4 tensor map over a (batch, seq, head, inner) 16-bit tensor; box = [64 inner, 1 head, rows seq, 1 batch]
static bool map_bshd(CUtensorMap *m, int dtype, const void *ptr, long long sb, long long sl, long long sh, int inner,
                     int heads, int seqlen, int batch, unsigned rows) {
    const unsigned long long dims[4] = {(unsigned long long)inner, (unsigned long long)heads, (unsigned long long)seqlen,
                                        (unsigned long long)batch};
    const unsigned long long str[3] = {(unsigned long long)sh * 2, (unsigned long long)sl * 2, (unsigned long long)sb * 2};
    const unsigned box[4] = {64, 1, rows, 1};
    return tc::make_map4(m, dtype, ptr, dims, str, box);
}

// The walk of tc_walk_tma.cuh, where it applies: its tensor maps and whether it is the faster way.
struct Walk {
    bool use = false;
    CUtensorMap mRow, mCol, mSf, mSb;
};
// The walk takes a fixed time per chunk whatever else runs, one CTA an SM; the two kernels it replaces take the time of their
// memory traffic - states in fp32 twice, x or g and their products - and a launch.  So the walk wins unless a long sequence of
// few heads leaves most SMs without one.  Coefficients (us) from 4600 drawn sizes in bf16 and fp16, b 1 - 16, L 200 - 20000, H
// 2 - 64, both headdims, every dstate and chunk, whole passes replayed from a graph with either form: the form taken is more
// than 10 % behind the other at 17 of them forward and 5 in training (22 % at most); by the coefficients of the first walk
// at 242 (43 %) and 141 (38 %).  us a forward call, two kernels and walk: b1 L16747 H24 dstate 64 chunk 128 213, 153; b2 L15326 H16 223,
// 170; and the other way b1 L8192 H8 dstate 128 chunk 256 46, 69, b1 L17397 H2 headdim 128 dstate 256 85, 230.
// A forward pass in two phases (`twice`) would walk twice, where the two kernels repeat the recurrence only: coefficients of its own,
// from 2000 sizes.  More than 10 % behind at 23 of them (22 % at most); with those of one pass at 258, by the first walk's at 147.
static bool walk_pays(const Dims &d, bool twice) {
    struct Cost { double chunk, per128, start, states, rows; };  // a wave's chunk; a chunk's 128 positions; then the two kernels'
    static constexpr Cost cost[2][2] = {{{0.08, 0.41, 1.75, 2.7, 1.75}, {1.0, 0.32, 1.45, 2.7, 1.5}},      // headdim 64, 128
                                        {{0.08, 0.41, 0.15, 1.8, 0.35}, {1.0, 0.32, 0.05, 1.7, 0.7}}};
    const Cost &c = cost[twice][d.P / 64 - 1];
    const double waves = std::ceil(2.0 * d.b * d.H * tc::walk_tiles(d) / sm_count()), rows = 1e-6 * d.b * d.H * d.P;
    return waves * d.nc * (c.chunk + c.per128 * (d.Q / 128)) < c.start + c.states * rows * d.nc * d.N + c.rows * rows * d.L;
}
static bool walk_wanted(const Dims &d, bool twice = false) { return !no_tma() && !no_ws() && tc::walk_ok(d.P, d.N, d.Q) && walk_pays(d, twice); }

// What the sizes alone say of the tensor-core family's kernels, and so which arrays of the workspace a pass does without.
// Operands that no tensor map describes are found out later: such a pass takes other kernels, and needs them all.
static bool ws_wanted(const Dims &d) { return !no_tma() && !no_ws() && tc::scan_ws_ok(d.P, d.N, d.Q); }
static bool fused_wanted(const Dims &d) {                        // tc::intra_dcb_tile, on the bf16 C.B^T tile only
    return ws_wanted(d) && !no_sums() && !no_fused() && tc::scan_tma_ok(d.P, d.N, d.Q) && tc::bmm_cb_tma_ok(d.N, d.Q) && tc::intra_tile_ok(d.P, d.Q);
}
static bool last_wanted(const Dims &d) {                         // dbc_accum_grp finishes dB and dC
    return fused_wanted(d) && head_parts(d) == 1 && tc::bmm_bwd_tma_ok(d.N, d.Q) && tc::dbc_grp_ok(d.P, d.N, d.Q);
}
static FwdWs least_fwd(const Dims &d) { return fwd_layout(d, FwdNeed{!walk_wanted(d), !ws_wanted(d), ws_wanted(d)}); }
static BwdWs least_bwd(const Dims &d) { return bwd_layout(d, true, BwdNeed{!walk_wanted(d), !last_wanted(d), !fused_wanted(d)}); }

static Walk plan_walk(const Dims &d, bool wanted, int dtype, const bissd_tensor &row, const View &col, const float *dt_out,
                      const float *cs_f, const float *cs_b, const void *states_f, const void *states_b) {
    Walk w;
    if (!wanted || !all_aligned16(dt_out, cs_f, cs_b)) return w;
    const unsigned rows = tc::walk_rows(d.P / 64);
    const unsigned long long srows = (unsigned long long)d.b * d.nc * d.H * d.P;
    w.use = map_bshd(&w.mRow, dtype, row.ptr, row.stride_batch, row.stride_seq, row.stride_head, d.N, d.G, d.L, d.b, rows) &&
            map_bshd(&w.mCol, dtype, col.ptr, col.sb, col.sl, col.sh, d.P, d.H, d.L, d.b, rows) &&
            tc::make_map2(&w.mSf, dtype, states_f, d.N, srows, 64, d.P) && tc::make_map2(&w.mSb, dtype, states_b, d.N, srows, 64, d.P);
    return w;
}
template <class T, int MODE>
static int launch_walk(const Dims &d, const Walk &w, const tc::WalkArgs &args, int *status, cudaStream_t s) {
    auto launch = [&](auto kernel) -> int {
        const size_t smem = tc::walk_smem(d.P, MODE);
        const int threads = tc::walk_threads(d.P / 64, MODE, d.N == 64);
        BISSD_ALLOW(kernel, smem);
        BISSD_LAUNCH(MODE ? "tc_dstate_walk" : "tc_state_walk", launch_pdl(kernel, dim3(2 * d.b * d.H * tc::walk_tiles(d)), threads, smem, s,
            d, w.mRow, w.mCol, w.mSf, w.mSb, args, status));
        return BISSD_OK;
    };
    if (d.N == 64) return d.P == 64 ? launch(tc::state_walk<T, MODE, 1, true>) : launch(tc::state_walk<T, MODE, 2, true>);
    return d.P == 64 ? launch(tc::state_walk<T, MODE, 1, false>) : launch(tc::state_walk<T, MODE, 2, false>);
}

template <class T>
static int forward_impl(const bissd_fwd_args &a, const Dims &d, char *ws, size_t ws_bytes, cudaStream_t s) {
    const bool lean = ws_bytes < fwd_layout(d).total;            // no room for what least_fwd leaves out
    const FwdWs w = lean ? least_fwd(d) : fwd_layout(d);
    int *status = reinterpret_cast<int *>(ws);
    float *loc = reinterpret_cast<float *>(ws + w.loc);
    float *CB = reinterpret_cast<float *>(ws + w.cb);
    const View x = view_of(a.x), Bm = view_of(a.B), Cm = view_of(a.C), z = view_of(a.z);
    const int bch = d.b * d.nc * d.H;
    const int ntP = tc::round_up(d.P, 16), ntQ = tc::round_up(d.Q, 16);
    // A FINISH phase with entering states walks again, from the inputs: the decision is the same in both phases.  With the least
    // scratch, which has no room for local states, LOCAL is all that is wanted.
    const bool walks = walk_wanted(d, !lean && a.phases != BISSD_PHASE_ALL);
    const Walk walk = plan_walk(d, walks, a.p.x_dtype, a.B, x, a.dt_out, a.cs_f, a.cs_b, a.states_f, a.states_b);
    if (lean && walks && !walk.use) return BISSD_ERR_WORKSPACE;
    const tc::CumsumFwd cs{a.dt.ptr, a.p.dt_dtype, a.dt.stride_batch, a.dt.stride_seq, a.dt.stride_head, a.A, a.dt_bias, a.dt_out, a.cs_f, a.cs_b,
                           all_aligned16(a.dt_out, a.cs_f, a.cs_b)};
    // C.B^T by TMA: a bf16 copy for the persistent scan, fp32 for the others; in one launch with the cumulative sums where
    // all blocks are resident at once (b1 L384 H8: 20.5 us a forward call with two launches and a memset for the status word)
    const bool ws_path = ws_wanted(d);
    __nv_bfloat16 *CB16 = reinterpret_cast<__nv_bfloat16 *>(ws + w.cb16);
    CUtensorMap mCc, mBc, mCBo;
    const bool cb_tma = !no_tma() && tc::bmm_cb_tma_ok(d.N, d.Q) && make_cb_maps(a, d, &mCc, &mBc) && (!ws_path || make_tile_map(d, CB16, &mCBo));
    if (!ws_path) mCBo = mCc;                                    // not used
    const size_t cb_smem = tc::bmm_cb_tma_smem(d.N, false, !ws_path);
    const tc::CbArgs cb_args{ws_path, 0, nullptr, ws_path ? nullptr : CB, nullptr};
    const long long first_blocks = (long long)d.b * d.nc * d.G * (d.Q / 128) * (d.Q / 128) + tc::cumsum_blocks(d);
    const bool cb_with_cumsum = cb_tma && (a.phases & BISSD_PHASE_LOCAL) && (a.phases & BISSD_PHASE_FINISH) &&
                                first_blocks <= (long long)sm_count() * std::min<size_t>(4, 227 * 1024 / (cb_smem + 2048));
    if (a.phases & BISSD_PHASE_LOCAL) {
        if (cb_with_cumsum) {
            auto launch = [&](auto kernel) -> int {
                const int tiles = d.b * d.nc * d.G * (d.Q / 128) * (d.Q / 128);
                BISSD_ALLOW(kernel, cb_smem);
                BISSD_LAUNCH("cumsum_cb", launch_pdl(kernel, tiles + tc::cumsum_blocks(d), tc::kThreads, cb_smem, s, d, mCc, mBc, mCBo, cb_args, cs, tiles, status));
                return BISSD_OK;
            };
            const int rc = ws_path ? (d.Q == 128 ? launch(tc::cumsum_cb<T, false, 1>) : launch(tc::cumsum_cb<T, false, 2>))
                                   : (d.Q == 128 ? launch(tc::cumsum_cb<T, true, 1>) : launch(tc::cumsum_cb<T, true, 2>));
            if (rc != BISSD_OK) return rc;
        } else {
            BISSD_LAUNCH("cumsum_fwd", launch_pdl(d.Q <= 128 ? tc::cumsum_fwd<1> : tc::cumsum_fwd<2>, tc::cumsum_blocks(d), 32 * tc::kCumsumWarps, 0, s, d, cs, status));
        }
        if (!walk.use) {
            const size_t smem = tc::smem_bytes(ntP, 2 * d.Q);
            bool st_done = false;
            if (!no_tma() && (tc::state_tma_ok(d.P, d.N, d.Q) || (!no_ws() && tc::state_grp_ok(d.P, d.N, d.Q, d.R)))) {
                CUtensorMap mRow, mCol;
                if (map_bshd(&mRow, a.p.x_dtype, a.B.ptr, a.B.stride_batch, a.B.stride_seq, a.B.stride_head, d.N, d.G, d.L, d.b, d.Q) &&
                    map_bshd(&mCol, a.p.x_dtype, a.x.ptr, a.x.stride_batch, a.x.stride_seq, a.x.stride_head, d.P, d.H, d.L, d.b, d.Q)) {
                    if (!no_ws() && tc::state_grp_ok(d.P, d.N, d.Q, d.R)) {
                        const size_t smem_g = tc::state_grp_smem(d.Q);
                        const int ks = tc::state_grp_ksplit(d.b * d.nc * d.G * ceil_div(d.N, 128), d.R, sm_count());
                        BISSD_ALLOW((tc::state_gemm_grp<T, 0>), smem_g);
                        BISSD_LAUNCH("tc_chunk_state_grp", launch_pdl(tc::state_gemm_grp<T, 0>, dim3(d.b * d.nc * d.G * ks, ceil_div(d.N, 128)), tc::kStateGrpThreads, smem_g, s, 
                            d, mRow, mCol, ks, a.dt_out, a.cs_f, a.cs_b, loc, status));
                    } else {
                        const size_t smem_t = tc::state_tma_smem(d.P, d.Q);
                        BISSD_ALLOW((tc::state_gemm_tma<T, 0>), smem_t);
                        BISSD_LAUNCH("tc_chunk_state_tma", tc::state_gemm_tma<T, 0><<<dim3(bch, 2, ceil_div(d.N, 128)), tc::kThreads, smem_t, s>>>(
                            d, mRow, mCol, a.dt_out, a.cs_f, a.cs_b, loc, status));
                    }
                    st_done = true;
                }
            }
            if (st_done) {
            } else if (ntP <= 64) {
                BISSD_ALLOW((tc::state_gemm<T, 0, 2>), smem);
                BISSD_LAUNCH("tc_chunk_state", tc::state_gemm<T, 0, 2><<<dim3(bch, ceil_div(2 * d.N, tc::kTileM)), tc::kThreads, smem, s>>>(
                    d, Bm, x, z, a.dt_out, a.cs_f, a.cs_b, loc, status));
            } else {
                BISSD_ALLOW((tc::state_gemm<T, 0, 8>), smem);
                BISSD_LAUNCH("tc_chunk_state", tc::state_gemm<T, 0, 8><<<dim3(bch, ceil_div(2 * d.N, tc::kTileM)), tc::kThreads, smem, s>>>(
                    d, Bm, x, z, a.dt_out, a.cs_f, a.cs_b, loc, status));
            }
        }
    }
    // the recurrence runs in both phases: from zero (or init_*) in LOCAL, again with init_* in FINISH
    const bool need_pass = (a.phases & BISSD_PHASE_LOCAL) || (a.init_f || a.init_b);
    if (!need_pass) {
    } else if (walk.use) {
        const tc::WalkArgs wa{a.dt_out, a.cs_f, a.cs_b, a.init_f, a.init_b, a.final_f, a.final_b, a.states_f, a.states_b, nullptr, 0};
        const int rc = launch_walk<T, 0>(d, walk, wa, status, s);
        if (rc != BISSD_OK) return rc;
    } else {
        BISSD_LAUNCH("state_passing_fwd", launch_pdl(pass_ahead(d) ? simt::state_passing_fwd4<T, 8> : simt::state_passing_fwd4<T, 1>, pass_grid(d), pass_threads(d), 0, s,
            d, loc, a.cs_f, a.cs_b, a.init_f, a.init_b, a.states_f, a.states_b, a.final_f, a.final_b));
    }
    if (a.phases & BISSD_PHASE_FINISH) {
        {
            const size_t smem_cb = tc::smem_bytes(ntQ, 0), smem_sc = tc::smem_bytes(ntP, 3 * d.Q);
            BISSD_ALLOW(tc::bmm_cb<T>, smem_cb);
            if (cb_with_cumsum) {
            } else if (cb_tma) {
                auto launch = [&](auto kernel) -> int {
                    BISSD_ALLOW(kernel, cb_smem);
                    BISSD_LAUNCH("tc_bmm_cb_tma", launch_pdl(kernel, dim3(d.b * d.nc * d.G, d.Q / 128, d.Q / 128), tc::kThreads, cb_smem, s,
                        d, mCc, mBc, mCBo, mCBo, cb_args, status));
                    return BISSD_OK;
                };
                const int rc = ws_path ? launch(tc::bmm_cb_tma<T, false>) : launch(tc::bmm_cb_tma<T, true>);
                if (rc != BISSD_OK) return rc;
            } else
            BISSD_LAUNCH("tc_bmm_cb", tc::bmm_cb<T><<<dim3(d.b * d.nc * d.G, ceil_div(d.Q, tc::kTileM)), tc::kThreads, smem_cb, s>>>(
                d, Cm, Bm, ws_path ? nullptr : CB, nullptr, ws_path ? CB16 : nullptr, nullptr, nullptr, status));
            bool tma_done = false;
            if (ws_path) {
                CUtensorMap mC, mCB, mSf, mSb, mX, mR;
                const unsigned long long dC[4] = {(unsigned long long)d.N, (unsigned long long)d.G, (unsigned long long)d.L, (unsigned long long)d.b};
                const unsigned long long sC[3] = {(unsigned long long)a.C.stride_head * 2, (unsigned long long)a.C.stride_seq * 2, (unsigned long long)a.C.stride_batch * 2};
                const unsigned bC[4] = {64, 1, 128, 1};
                const unsigned long long rows = (unsigned long long)d.b * d.nc * d.H * d.P;
                bool maps = tc::make_map4(&mC, a.p.x_dtype, a.C.ptr, dC, sC, bC) &&
                            map_bshd(&mX, a.p.x_dtype, a.x.ptr, a.x.stride_batch, a.x.stride_seq, a.x.stride_head, d.P, d.H, d.L, d.b, 64) &&
                            tc::make_map2(&mCB, BISSD_BF16, CB16, d.Q, (unsigned long long)d.b * d.nc * d.G * d.Q, 64, 128) &&
                            tc::make_map2(&mSf, a.p.x_dtype, a.states_f, d.N, rows, 64, d.P) &&
                            tc::make_map2(&mSb, a.p.x_dtype, a.states_b, d.N, rows, 64, d.P);
                // the epilogue's z rows by TMA (a [128 rows x 64] tile per step); without z the map is not used
                const bool z_rows = maps && d.has_z &&
                                    map_bshd(&mR, a.p.x_dtype, a.z.ptr, a.z.stride_batch, a.z.stride_seq, a.z.stride_head, d.P, d.H, d.L, d.b, 128);
                if (maps && !z_rows) mR = mX;
                if (maps) {
                    const size_t smem_t = tc::scan_ws_smem(d.P, d.N, d.Q);
                    const int tiles = bch * (d.Q / tc::kTileM);
                    const int grid = std::min(sm_count(), tiles);
                    auto wide = [](const bissd_tensor &t) {   // 32-byte accesses allowed on every row piece
                        return t.ptr && reinterpret_cast<uintptr_t>(t.ptr) % 32 == 0 && t.stride_batch % 16 == 0 &&
                               t.stride_seq % 16 == 0 && t.stride_head % 16 == 0;
                    };
                    const int wide_z = d.has_z && wide(a.z);
                    const int wide_o = wide(a.out) && (!d.has_z || wide(a.out_x));
                    tc::WsArgs wa{};
                    wa.x = x; wa.z = z; wa.D = a.D; wa.dt_out = a.dt_out; wa.cs_f = a.cs_f; wa.cs_b = a.cs_b;
                    wa.out = mview_of(a.out); wa.out_x = mview_of(a.out_x);
                    wa.wide_z = wide_z; wa.wide_o = wide_o;
                    wa.rows_by_tma = z_rows ? 1 : 0;
#define BISSD_SCAN_WS(NSL, NS)                                                                                          \
do {                                                                                                                \
    BISSD_ALLOW((tc::ws_kernel<T, NSL, NS, 0>), smem_t);                                                            \
    BISSD_LAUNCH("tc_chunk_scan_ws", launch_pdl(tc::ws_kernel<T, NSL, NS, 0>, grid, tc::kWsThreads, smem_t, s,              \
        d, mC, mCB, mSf, mSb, mX, mR, wa, status));                                                                 \
} while (0)
                    if (d.N == 128 && d.Q == 256) BISSD_SCAN_WS(2, 4);
                    else if (d.N == 64 && d.Q == 256) BISSD_SCAN_WS(1, 4);
                    else if (d.N == 128 && d.Q == 128) BISSD_SCAN_WS(2, 2);
                    else BISSD_SCAN_WS(1, 2);
#undef BISSD_SCAN_WS
                    tma_done = true;
                } else {                                     // maps refused: produce the fp32 tile after all
                    if (lean) return BISSD_ERR_WORKSPACE;
                    BISSD_LAUNCH("tc_bmm_cb", tc::bmm_cb<T><<<dim3(d.b * d.nc * d.G, ceil_div(d.Q, tc::kTileM)), tc::kThreads, smem_cb, s>>>(
                        d, Cm, Bm, CB, nullptr, nullptr, nullptr, nullptr, status));
                }
            }
            if (!tma_done && !no_tma() && tc::scan_tma_ok(d.P, d.N, d.Q)) {
                CUtensorMap mC, mSf, mSb, mX;
                const unsigned long long dC[4] = {(unsigned long long)d.N, (unsigned long long)d.G, (unsigned long long)d.L, (unsigned long long)d.b};
                const unsigned long long sC[3] = {(unsigned long long)a.C.stride_head * 2, (unsigned long long)a.C.stride_seq * 2, (unsigned long long)a.C.stride_batch * 2};
                const unsigned bC[4] = {64, 1, 128, 1};
                const unsigned long long dX[4] = {(unsigned long long)d.P, (unsigned long long)d.H, (unsigned long long)d.L, (unsigned long long)d.b};
                const unsigned long long sX[3] = {(unsigned long long)a.x.stride_head * 2, (unsigned long long)a.x.stride_seq * 2, (unsigned long long)a.x.stride_batch * 2};
                const unsigned bX[4] = {64, 1, 64, 1};
                const unsigned long long rows = (unsigned long long)d.b * d.nc * d.H * d.P;
                if (tc::make_map4(&mC, a.p.x_dtype, a.C.ptr, dC, sC, bC) && tc::make_map4(&mX, a.p.x_dtype, a.x.ptr, dX, sX, bX) &&
                    tc::make_map2(&mSf, a.p.x_dtype, a.states_f, d.N, rows, 64, d.P) &&
                    tc::make_map2(&mSb, a.p.x_dtype, a.states_b, d.N, rows, 64, d.P)) {
                    const size_t smem_t = tc::scan_tma_smem(d.P, d.Q);
                    BISSD_ALLOW(tc::chunk_scan_tma<T>, smem_t);
                    BISSD_LAUNCH("tc_chunk_scan_tma", launch_pdl(tc::chunk_scan_tma<T>, dim3(bch, d.Q / tc::kTileM), tc::kThreads, smem_t, s,
                        d, mC, mSf, mSb, mX, x, z, a.D, a.dt_out, a.cs_f, a.cs_b, CB, mview_of(a.out), mview_of(a.out_x), status));
                    tma_done = true;
                }
            }
            if (tma_done) {
            } else if (ntP <= 64) {
                BISSD_ALLOW((tc::chunk_scan<T, 2>), smem_sc);
                BISSD_LAUNCH("tc_chunk_scan", tc::chunk_scan<T, 2><<<dim3(bch, ceil_div(d.Q, tc::kTileM)), tc::kThreads, smem_sc, s>>>(
                    d, x, Cm, z, a.D, a.dt_out, a.cs_f, a.cs_b, CB, a.states_f, a.states_b, mview_of(a.out), mview_of(a.out_x), status));
            } else {
                BISSD_ALLOW((tc::chunk_scan<T, 8>), smem_sc);
                BISSD_LAUNCH("tc_chunk_scan", tc::chunk_scan<T, 8><<<dim3(bch, ceil_div(d.Q, tc::kTileM)), tc::kThreads, smem_sc, s>>>(
                    d, x, Cm, z, a.D, a.dt_out, a.cs_f, a.cs_b, CB, a.states_f, a.states_b, mview_of(a.out), mview_of(a.out_x), status));
            }
        }
    }
    return BISSD_OK;
}

template <class T>
static int backward_impl(const bissd_bwd_args &a, const GradViews &gr, const Dims &d, char *ws, size_t ws_bytes, cudaStream_t s) {
    const bool lean = ws_bytes < bwd_layout(d, true).total;      // no room for what least_bwd leaves out
    const BwdWs w = lean ? least_bwd(d) : bwd_layout(d, true);
    int *status = reinterpret_cast<int *>(ws);
    auto F = [&](size_t off) { return reinterpret_cast<float *>(ws + off); };
    const View x = view_of(a.x), Bm = view_of(a.B), Cm = view_of(a.C), z = view_of(a.z), dout = view_of(a.dout),
               out_x = view_of(a.out_x);
    const int bch = d.b * d.nc * d.H;
    const int ntP = tc::round_up(d.P, 16), ntQ = tc::round_up(d.Q, 16), ntN = std::min(tc::round_up(d.N, 16), 128);
    const int nlt_tc = ceil_div(d.Q, tc::kTileM);
    // Tensor-core family: the gate is applied once (gate_bwd writes g = dout * silu(z) and dz); every later kernel
    // then sees an ungated problem whose output gradient is g.
    Dims dg = d;
    View gv = dout;
    void *E16 = ws + w.E16;
    if (d.has_z) {
        dg.has_z = 0;
        gv = View{ws + w.g, (long long)d.L * d.H * d.P, (long long)d.H * d.P, (long long)d.P};
    }
    Walk walk;                                                   // whole passes only: a split one keeps its local gradients
    if (a.phases == BISSD_PHASE_ALL) walk = plan_walk(d, walk_wanted(d), a.p.x_dtype, a.C, gv, a.dt_out, a.cs_f, a.cs_b, a.states_f, a.states_b);
    if (lean && walk_wanted(d) && !walk.use) return BISSD_ERR_WORKSPACE;
    if (a.phases & BISSD_PHASE_LOCAL) {
        if (!d.has_z && !walk.use) {                             // else the gate kernel or the walk, whichever is first, clears the status word
            const int rc = note_cuda(cudaMemsetAsync(ws, 0, kWsHeader, s), "cudaMemsetAsync");
            if (rc != BISSD_OK) return rc;
        }
        if (d.has_z) {
            const long long chunks = (long long)d.b * d.L * d.H * (d.P / 8);
            BISSD_LAUNCH("gate_bwd", launch_pdl(tc::gate_bwd<T>, (unsigned)((chunks + 255) / 256), 256, 0, s, 
                d, dout, z, out_x, ws + w.g, a.dz, status));
        }
        if (!walk.use) {
            const size_t smem = tc::smem_bytes(ntP, 2 * d.Q);
            bool st_done = false;
            if (!no_tma() && (tc::state_tma_ok(d.P, d.N, d.Q) || (!no_ws() && tc::state_grp_ok(d.P, d.N, d.Q, d.R)))) {
                CUtensorMap mRow, mCol;
                if (map_bshd(&mRow, a.p.x_dtype, a.C.ptr, a.C.stride_batch, a.C.stride_seq, a.C.stride_head, d.N, d.G, d.L, d.b, d.Q) &&
                    map_bshd(&mCol, a.p.x_dtype, gv.ptr, gv.sb, gv.sl, gv.sh, d.P, d.H, d.L, d.b, d.Q)) {
                    if (!no_ws() && tc::state_grp_ok(d.P, d.N, d.Q, d.R)) {
                        const size_t smem_g = tc::state_grp_smem(d.Q);
                        const int ks = tc::state_grp_ksplit(d.b * d.nc * d.G * ceil_div(d.N, 128), d.R, sm_count());
                        BISSD_ALLOW((tc::state_gemm_grp<T, 1>), smem_g);
                        BISSD_LAUNCH("tc_dstates_grp", launch_pdl(tc::state_gemm_grp<T, 1>, dim3(d.b * d.nc * d.G * ks, ceil_div(d.N, 128)), tc::kStateGrpThreads, smem_g, s, 
                            d, mRow, mCol, ks, a.dt_out, a.cs_f, a.cs_b, F(w.gloc), status));
                    } else {
                        const size_t smem_t = tc::state_tma_smem(d.P, d.Q);
                        BISSD_ALLOW((tc::state_gemm_tma<T, 1>), smem_t);
                        BISSD_LAUNCH("tc_dstates_tma", tc::state_gemm_tma<T, 1><<<dim3(bch, 2, ceil_div(d.N, 128)), tc::kThreads, smem_t, s>>>(
                            d, mRow, mCol, a.dt_out, a.cs_f, a.cs_b, F(w.gloc), status));
                    }
                    st_done = true;
                }
            }
            if (st_done) {
            } else if (ntP <= 64) {
                BISSD_ALLOW((tc::state_gemm<T, 1, 2>), smem);
                BISSD_LAUNCH("tc_dstates", tc::state_gemm<T, 1, 2><<<dim3(bch, ceil_div(2 * d.N, tc::kTileM)), tc::kThreads, smem, s>>>(
                    dg, Cm, gv, z, a.dt_out, a.cs_f, a.cs_b, F(w.gloc), status));
            } else {
                BISSD_ALLOW((tc::state_gemm<T, 1, 8>), smem);
                BISSD_LAUNCH("tc_dstates", tc::state_gemm<T, 1, 8><<<dim3(bch, ceil_div(2 * d.N, tc::kTileM)), tc::kThreads, smem, s>>>(
                    dg, Cm, gv, z, a.dt_out, a.cs_f, a.cs_b, F(w.gloc), status));
            }
        }
    }
    const bool need_pass = (a.phases & BISSD_PHASE_LOCAL) || (a.dfinal_f || a.dfinal_b);
    if (walk.use) {
        const tc::WalkArgs wa{a.dt_out, a.cs_f, a.cs_b, a.dfinal_f, a.dfinal_b, a.dinit_f, a.dinit_b, E16,
                              static_cast<char *>(E16) + (size_t)d.b * d.nc * d.H * d.P * d.N * 2, F(w.dTpart), !d.has_z};
        const int rc = launch_walk<T, 1>(d, walk, wa, status, s);
        if (rc != BISSD_OK) return rc;
    } else if (need_pass) {
        auto launch = [&](auto wn) -> int {
            constexpr int WN = decltype(wn)::value;
            const auto kernel = pass_ahead(d) ? simt::state_passing_bwd4<T, 8, WN> : simt::state_passing_bwd4<T, 1, WN>;
            BISSD_LAUNCH("state_passing_bwd", launch_pdl(kernel, pass_grid(d), pass_threads(d), 0, s,
                d, F(w.gloc), a.states_f, a.states_b, a.cs_f, a.cs_b, a.dfinal_f, a.dfinal_b, nullptr, E16, F(w.dTpart), a.dinit_f, a.dinit_b));
            return BISSD_OK;
        };
        int rc;
        if (!tc::walk_ok(d.P, d.N, d.Q)) rc = launch(std::integral_constant<int, 0>());
        else if (d.N == 64) rc = launch(std::integral_constant<int, 64>());
        else if (d.N == 128) rc = launch(std::integral_constant<int, 128>());
        else rc = launch(std::integral_constant<int, 256>());
        if (rc != BISSD_OK) return rc;
    }
    if (!(a.phases & BISSD_PHASE_FINISH)) return BISSD_OK;
    int nlt = w.nlt, nsplit = 1, part_heads = d.H;
    CUtensorMap mEf, mEb, mSf, mSb, mX128, mG128;                // operands of dbc_accum_grp
    bool dbc_last = false;                                       // it finishes dB and dC after the dCB kernel
    auto launch_dbc = [&](auto kernel, const tc::LastMaps &last, cudaStream_t st) -> int {
        const size_t smem_g = tc::dbc_grp_smem(d.Q, std::min(d.N, 128));
        BISSD_ALLOW(kernel, smem_g);
        BISSD_LAUNCH_ON(st, "tc_dbc_accum_grp", launch_pdl(kernel, dim3(d.b * d.nc * d.G * w.nsplit * w.dbc_ks, 1, 2), tc::kDbcGrpThreads, smem_g, st,
            d, mEf, mEb, mSf, mSb, mX128, mG128, a.dt_out, a.cs_f, a.cs_b, F(w.dB_part), F(w.dC_part), w.dbc_ks, last, status));
        return BISSD_OK;
    };
    bool have_fp32_cb = true;                                    // fp32 CB (and its transpose) are in the workspace
    bool use_u4 = false;                                         // decay gradients arrive as u_f / u_b (tc::intra_sums)
    bool fused_cb = false;                                       // the bf16 C.B^T tile for tc::intra_dcb_tile has been written
    SideStream side(s);                                          // where prev_terms_grp and dbc_accum_grp are launched
    int u4_tiles = 2;                                            // (u_f, u_b) vector pairs per chunk in u4
    int dd_slots = 0;                                            // dD partial rows per (b,c,h) when not nlt
    bool dd_compact = false;                                     // per-head D from the persistent dx kernel: dd_slots scalars, no channel axis
    {
        nlt = nlt_tc;
        nsplit = w.nsplit;
        part_heads = d.G;
        const size_t smem_cb = tc::smem_bytes(ntQ, 0), smem_dx = tc::smem_bytes(ntP, 3 * d.Q), smem_n = tc::smem_bytes(ntN, 0);
        BISSD_ALLOW(tc::bmm_cb<T>, smem_cb);
        const bool ws_path = ws_wanted(d);
        const bool sums_path = !no_tma() && !no_sums() && tc::scan_tma_ok(d.P, d.N, d.Q);
        __nv_bfloat16 *CBt16 = reinterpret_cast<__nv_bfloat16 *>(ws + w.cbt16);
        __nv_bfloat16 *CB16b = reinterpret_cast<__nv_bfloat16 *>(ws + w.cb16);
        CUtensorMap mCc, mBc, mCBo, mCBto;
        if (ws_path && sums_path && tc::bmm_cb_tma_ok(d.N, d.Q) && make_cb_maps(a, d, &mCc, &mBc) && make_tile_map(d, CB16b, &mCBo) &&
            make_tile_map(d, CBt16, &mCBto)) {
            // the fused dCB / decay-gradient kernel reads the bf16 tile by TMA; the separate intra_sums kernel
            // reads the fp32 strips
            fused_cb = fused_wanted(d);
            const size_t smem_ct = tc::bmm_cb_tma_smem(d.N, true);
            BISSD_ALLOW((tc::bmm_cb_tma<T, false>), smem_ct);
            BISSD_LAUNCH("tc_bmm_cb_tma", launch_pdl(tc::bmm_cb_tma<T, false>, dim3(d.b * d.nc * d.G, d.Q / 128, d.Q / 128), tc::kThreads, smem_ct, s,
                d, mCc, mBc, mCBo, mCBto, tc::CbArgs{fused_cb, 1, fused_cb ? nullptr : F(w.cbs), nullptr, nullptr}, status));
        } else if (!ws_path && sums_path && tc::bmm_cb_tma_ok(d.N, d.Q) && make_cb_maps(a, d, &mCc, &mBc)) {
            const size_t smem_ct = tc::bmm_cb_tma_smem(d.N, true, true);
            BISSD_ALLOW((tc::bmm_cb_tma<T, true>), smem_ct);
            BISSD_LAUNCH("tc_bmm_cb_tma", launch_pdl(tc::bmm_cb_tma<T, true>, dim3(d.b * d.nc * d.G, d.Q / 128, d.Q / 128), tc::kThreads, smem_ct, s,
                d, mCc, mBc, mCc, mCc, tc::CbArgs{0, 0, F(w.cbs), F(w.cb), F(w.cbt)}, status));
        } else {
            if (lean && fused_wanted(d)) return BISSD_ERR_WORKSPACE;
            BISSD_LAUNCH("tc_bmm_cb", tc::bmm_cb<T><<<dim3(d.b * d.nc * d.G, nlt_tc), tc::kThreads, smem_cb, s>>>(
                d, Cm, Bm, (sums_path && ws_path) ? nullptr : F(w.cb), ws_path ? nullptr : F(w.cbt), nullptr,
                ws_path ? CBt16 : nullptr, sums_path ? F(w.cbs) : nullptr, status));   // only the copies that will be read
        }
        have_fp32_cb = !ws_path;                             // ws path: only the copies its kernels read were written
        auto ensure_fp32_cb = [&]() -> int {                 // for the kernels that read them, should a planned path fall through
            if (have_fp32_cb) return BISSD_OK;
            if (lean && fused_wanted(d)) return BISSD_ERR_WORKSPACE;
            BISSD_LAUNCH("tc_bmm_cb", tc::bmm_cb<T><<<dim3(d.b * d.nc * d.G, nlt_tc), tc::kThreads, smem_cb, s>>>(
                d, Cm, Bm, F(w.cb), F(w.cbt), nullptr, nullptr, nullptr, status));
            have_fp32_cb = true;
            return BISSD_OK;
        };
        bool dx_done = false;
        if (ws_path) {
            CUtensorMap mB, mCBt, mEf, mEb, mG, mR;
            const unsigned long long dB4[4] = {(unsigned long long)d.N, (unsigned long long)d.G, (unsigned long long)d.L, (unsigned long long)d.b};
            const unsigned long long sB4[3] = {(unsigned long long)a.B.stride_head * 2, (unsigned long long)a.B.stride_seq * 2, (unsigned long long)a.B.stride_batch * 2};
            const unsigned bB4[4] = {64, 1, 128, 1};
            const unsigned long long rows = (unsigned long long)d.b * d.nc * d.H * d.P;
            const char *e16 = static_cast<const char *>(E16);
            const bool maps = tc::make_map4(&mB, a.p.x_dtype, a.B.ptr, dB4, sB4, bB4) &&
                              map_bshd(&mG, a.p.x_dtype, gv.ptr, gv.sb, gv.sl, gv.sh, d.P, d.H, d.L, d.b, 64) &&
                              tc::make_map2(&mCBt, BISSD_BF16, CBt16, d.Q, (unsigned long long)d.b * d.nc * d.G * d.Q, 64, 128) &&
                              tc::make_map2(&mEf, a.p.x_dtype, e16, d.N, rows, 64, d.P) &&
                              tc::make_map2(&mEb, a.p.x_dtype, e16 + rows * d.N * 2, d.N, rows, 64, d.P);
            // the epilogue's x rows by TMA (a [128 rows x 64] tile per step)
            const bool x_rows = maps && map_bshd(&mR, a.p.x_dtype, a.x.ptr, a.x.stride_batch, a.x.stride_seq, a.x.stride_head, d.P, d.H, d.L, d.b, 128);
            if (maps && !x_rows) mR = mG;
            if (maps) {
                auto wide = [](const void *ptr, long long sb, long long sl, long long sh) {
                    return ptr && reinterpret_cast<uintptr_t>(ptr) % 32 == 0 && sb % 16 == 0 && sl % 16 == 0 && sh % 16 == 0;
                };
                tc::WsArgs wa{};
                wa.x = x; wa.z = gv; wa.D = a.D; wa.dt_out = a.dt_out; wa.cs_f = a.cs_f; wa.cs_b = a.cs_b;
                wa.out = gr.dx;
                wa.out_x = wa.out;
                wa.ddt_out = F(w.ddt_out); wa.nf = F(w.nf); wa.nb = F(w.nb); wa.dDpart = F(w.dDpart);
                wa.wide_x = wide(x.ptr, x.sb, x.sl, x.sh);
                wa.wide_z = wide(gv.ptr, gv.sb, gv.sl, gv.sh);
                wa.wide_o = wide(gr.dx.ptr, gr.dx.sb, gr.dx.sl, gr.dx.sh);
                wa.rows_by_tma = x_rows ? 1 : 0;
                const size_t smem_t = tc::scan_ws_smem(d.P, d.N, d.Q);
                const int grid = std::min(sm_count(), bch * nlt_tc);
#define BISSD_DX_WS(NSL, NS)                                                                                            \
do {                                                                                                                \
    BISSD_ALLOW((tc::ws_kernel<T, NSL, NS, 1>), smem_t);                                                            \
    BISSD_LAUNCH("tc_dx_ws", launch_pdl(tc::ws_kernel<T, NSL, NS, 1>, grid, tc::kWsThreads, smem_t, s,                      \
        d, mB, mCBt, mEf, mEb, mG, mR, wa, status));                                                                \
} while (0)
                if (d.N == 128 && d.Q == 256) BISSD_DX_WS(2, 4);
                else if (d.N == 64 && d.Q == 256) BISSD_DX_WS(1, 4);
                else if (d.N == 128 && d.Q == 128) BISSD_DX_WS(2, 2);
                else BISSD_DX_WS(1, 2);
#undef BISSD_DX_WS
                dx_done = true;
                if (fused_cb && side_allowed() && side.fork() != cudaSuccess) cudaGetLastError();   // the group-walking kernels branch off here, or stay in line
                dd_slots = nlt_tc * 4;
                if (d.has_D && !d.D_hdim) {
                    dd_slots = nlt_tc * 8;                       // one scalar per epilogue warp and tile
                    dd_compact = true;
                }
            }
        }
        if (!dx_done) {
            const int rc = ensure_fp32_cb();
            if (rc != BISSD_OK) return rc;
        }
        if (!dx_done && !no_tma() && tc::scan_tma_ok(d.P, d.N, d.Q)) {
            CUtensorMap mB, mEf, mEb, mG;
            const unsigned long long dB4[4] = {(unsigned long long)d.N, (unsigned long long)d.G, (unsigned long long)d.L, (unsigned long long)d.b};
            const unsigned long long sB4[3] = {(unsigned long long)a.B.stride_head * 2, (unsigned long long)a.B.stride_seq * 2, (unsigned long long)a.B.stride_batch * 2};
            const unsigned bB4[4] = {64, 1, 128, 1};
            const unsigned long long dG4[4] = {(unsigned long long)d.P, (unsigned long long)d.H, (unsigned long long)d.L, (unsigned long long)d.b};
            const unsigned long long sG4[3] = {(unsigned long long)gv.sh * 2, (unsigned long long)gv.sl * 2, (unsigned long long)gv.sb * 2};
            const unsigned bG4[4] = {64, 1, 64, 1};
            const unsigned long long rows = (unsigned long long)d.b * d.nc * d.H * d.P;
            const char *e16 = static_cast<const char *>(E16);
            if (tc::make_map4(&mB, a.p.x_dtype, a.B.ptr, dB4, sB4, bB4) && tc::make_map4(&mG, a.p.x_dtype, gv.ptr, dG4, sG4, bG4) &&
                tc::make_map2(&mEf, a.p.x_dtype, e16, d.N, rows, 64, d.P) &&
                tc::make_map2(&mEb, a.p.x_dtype, e16 + rows * d.N * 2, d.N, rows, 64, d.P)) {
                const size_t smem_t = tc::dx_tma_smem(d.P, d.Q);
                BISSD_ALLOW(tc::dx_tma<T>, smem_t);
                BISSD_LAUNCH("tc_dx_tma", launch_pdl(tc::dx_tma<T>, dim3(bch, nlt_tc), tc::kThreads, smem_t, s,
                    d, mB, mEf, mEb, mG, x, gv, a.D, a.dt_out, a.cs_f, a.cs_b, F(w.cbt), gr.dx, F(w.ddt_out), F(w.nf), F(w.nb),
                    F(w.dDpart), status));
                dx_done = true;
            }
        }
        if (dx_done) {
        } else if (ntP <= 64) {
            BISSD_ALLOW((tc::dx_kernel<T, 2>), smem_dx);
            BISSD_LAUNCH("tc_dx", tc::dx_kernel<T, 2><<<dim3(bch, nlt_tc), tc::kThreads, smem_dx, s>>>(
                dg, x, Bm, z, gv, out_x, a.D, a.dt_out, a.cs_f, a.cs_b, F(w.cb), E16, gr.dx, a.dz, F(w.ddt_out), F(w.dDpart), status));
        } else {
            BISSD_ALLOW((tc::dx_kernel<T, 8>), smem_dx);
            BISSD_LAUNCH("tc_dx", tc::dx_kernel<T, 8><<<dim3(bch, nlt_tc), tc::kThreads, smem_dx, s>>>(
                dg, x, Bm, z, gv, out_x, a.D, a.dt_out, a.cs_f, a.cs_b, F(w.cb), E16, gr.dx, a.dz, F(w.ddt_out), F(w.dDpart), status));
        }
        bool dbc_done = false;
        if (dx_done) {                                           // the dx kernel has produced nf / nb
            CUtensorMap mC;
            const unsigned long long dC4[4] = {(unsigned long long)d.N, (unsigned long long)d.G, (unsigned long long)d.L, (unsigned long long)d.b};
            const unsigned long long sC4[3] = {(unsigned long long)a.C.stride_head * 2, (unsigned long long)a.C.stride_seq * 2, (unsigned long long)a.C.stride_batch * 2};
            const unsigned bC4[4] = {64, 1, 128, 1};
            const unsigned long long rows = (unsigned long long)d.b * d.nc * d.H * d.P;
            const char *e16 = static_cast<const char *>(E16);
            if (tc::make_map4(&mC, a.p.x_dtype, a.C.ptr, dC4, sC4, bC4) &&
                tc::make_map2(&mEf, a.p.x_dtype, e16, d.N, rows, 64, d.P) &&
                tc::make_map2(&mEb, a.p.x_dtype, e16 + rows * d.N * 2, d.N, rows, 64, d.P) &&
                tc::make_map2(&mSf, a.p.x_dtype, a.states_f, d.N, rows, 64, d.P) &&
                tc::make_map2(&mSb, a.p.x_dtype, a.states_b, d.N, rows, 64, d.P)) {
                const size_t smem_p = tc::prev_tma_smem(d.P), smem_a = tc::dbc_tma_smem(d.P, std::min(d.N, 128));
                if (!map_bshd(&mX128, a.p.x_dtype, a.x.ptr, a.x.stride_batch, a.x.stride_seq, a.x.stride_head, d.P, d.H, d.L, d.b, 128) ||
                    !map_bshd(&mG128, a.p.x_dtype, gv.ptr, gv.sb, gv.sl, gv.sh, d.P, d.H, d.L, d.b, 128))
                    return BISSD_ERR_ALIGN;
                if (!no_ws() && tc::prev_grp_ok(d.P, d.N, d.Q, d.R)) {
                    const size_t smem_g = tc::prev_grp_smem(d.N, d.Q);
                    const int ks = tc::state_grp_ksplit(d.b * d.nc * d.G, d.R, sm_count());
                    BISSD_ALLOW(tc::prev_terms_grp<T>, smem_g);
                    BISSD_LAUNCH_ON(side.stream(), "tc_prev_terms_grp", launch_pdl(tc::prev_terms_grp<T>, dim3(d.b * d.nc * d.G * ks), tc::kPrevGrpThreads, smem_g, side.stream(),
                        d, mC, mSf, mSb, mG128, ks, a.cs_f, a.cs_b, F(w.pf), F(w.pb), status));
                } else {
                    BISSD_ALLOW(tc::prev_terms_tma<T>, smem_p);
                    BISSD_LAUNCH("tc_prev_terms_tma", launch_pdl(tc::prev_terms_tma<T>, dim3(bch, nlt_tc), tc::kThreads, smem_p, s,
                        d, mC, mSf, mSb, gv, a.cs_f, a.cs_b, F(w.pf), F(w.pb), status));
                }
                BISSD_ALLOW(tc::dbc_accum_tma<T>, smem_a);
                if (!no_ws() && tc::dbc_grp_ok(d.P, d.N, d.Q)) {
                    dbc_last = fused_cb && last_wanted(d);       // launched after the dCB kernel, below
                    if (!dbc_last) {
                        const int rc = launch_dbc(tc::dbc_accum_grp<T, false>, tc::LastMaps{}, side.stream());
                        if (rc != BISSD_OK) return rc;
                        part_heads = d.G * dbc_slots(d, w.dbc_ks);
                    }
                } else
                BISSD_LAUNCH("tc_dbc_accum_tma", launch_pdl(tc::dbc_accum_tma<T>, dim3(d.b * d.nc * d.G * w.nsplit, nlt_tc, 2), tc::kDbcTmaThreads, smem_a, s,
                    d, mEf, mEb, mSf, mSb, mX128, mG128, a.dt_out, a.cs_f, a.cs_b, F(w.dB_part), F(w.dC_part), status));
                dbc_done = true;
                nsplit = 1;                                      // nf/nb/pf/pb now hold complete row sums
            }
        }
        if (lean && last_wanted(d) && !dbc_last) return BISSD_ERR_WORKSPACE;
        if (!dbc_done) {
            BISSD_ALLOW(tc::dbc_states<T>, smem_n);
            BISSD_LAUNCH("tc_dbc_states", tc::dbc_states<T><<<dim3(d.b * d.nc * d.G * w.nsplit, nlt_tc, 2), tc::kThreads, smem_n, s>>>(
                dg, x, Bm, Cm, z, gv, a.dt_out, a.cs_f, a.cs_b, E16, a.states_f, a.states_b, F(w.dB_part), F(w.dC_part),
                F(w.nf), F(w.nb), F(w.pf), F(w.pb), status));
        }
    }
    bool bmm_tma = false;                                        // dCB is then a 16-bit array read by TMA
    CUtensorMap mBb, mCb, mDm, mDk;
    {
        const int ntQ128 = std::min(ntQ, 128);
        const size_t smem_dcb = tc::smem_bytes(ntQ128, 3 * d.Q), smem_in = tc::smem_bytes(ntQ, 4 * d.Q + tc::kTileM * 8);
        bool dcb_done = false;
        bool fused_done = false;
        if (fused_cb) {
            // one kernel for dCB and the intra-chunk decay gradients: a CTA per (batch, chunk, group, row tile)
            CUtensorMap mG, mX128, mCB;
            const unsigned long long dBC4[4] = {(unsigned long long)d.N, (unsigned long long)d.G, (unsigned long long)d.L, (unsigned long long)d.b};
            const unsigned long long sB4[3] = {(unsigned long long)a.B.stride_head * 2, (unsigned long long)a.B.stride_seq * 2, (unsigned long long)a.B.stride_batch * 2};
            const unsigned long long sC4b[3] = {(unsigned long long)a.C.stride_head * 2, (unsigned long long)a.C.stride_seq * 2, (unsigned long long)a.C.stride_batch * 2};
            const unsigned bx4[4] = {64, 1, 128, 1};
            const unsigned long long dcb_rows = (unsigned long long)d.b * d.nc * d.G * d.Q;
            if (map_bshd(&mG, a.p.x_dtype, gv.ptr, gv.sb, gv.sl, gv.sh, d.P, d.H, d.L, d.b, 128) &&
                map_bshd(&mX128, a.p.x_dtype, a.x.ptr, a.x.stride_batch, a.x.stride_seq, a.x.stride_head, d.P, d.H, d.L, d.b, 128) &&
                tc::make_map2(&mCB, BISSD_BF16, ws + w.cb16, d.Q, dcb_rows, 64, 128) &&
                tc::bmm_bwd_tma_ok(d.N, d.Q) &&
                tc::make_map4(&mBb, a.p.x_dtype, a.B.ptr, dBC4, sB4, bx4) && tc::make_map4(&mCb, a.p.x_dtype, a.C.ptr, dBC4, sC4b, bx4) &&
                tc::make_map2(&mDm, a.p.x_dtype, F(w.dCB), d.Q, dcb_rows, 64, d.Q) &&
                tc::make_map2(&mDk, a.p.x_dtype, F(w.dCB), d.Q, dcb_rows, 64, 128)) {
                const size_t smem_f = tc::intra_tile_smem();
                const auto intra = tc::intra_dcb_tile<T>;
                const int ks = head_parts(d);                    // one block of a cluster for each part of the heads
                BISSD_ALLOW(intra, smem_f);
                const int rc_regs = check_registers(intra, tc::kIntraLaunchRegs);
                if (rc_regs != BISSD_OK) return rc_regs;
                BISSD_LAUNCH("tc_intra_dcb_tile", launch_cluster(intra, dim3(d.b * d.nc * d.G * ks, nlt_tc, nlt_tc), tc::kIntraTileThreads, smem_f, s, ks,
                    dg, mG, mX128, mCB, a.dt_out, a.cs_f, a.cs_b, F(w.u4), (long long)d.b * d.H * d.nc * d.Q,
                    static_cast<void *>(F(w.dCB)), ks, status));
                u4_tiles = nlt_tc * nlt_tc;
                fused_done = dcb_done = true;
                bmm_tma = true;
                use_u4 = true;
            } else {
                return BISSD_ERR_ALIGN;                      // the bf16 tile was written for this kernel only
            }
        }
        if (!dcb_done && !no_tma() && tc::scan_tma_ok(d.P, d.N, d.Q)) {
            CUtensorMap mG, mX;
            const unsigned long long dX4[4] = {(unsigned long long)d.P, (unsigned long long)d.H, (unsigned long long)d.L, (unsigned long long)d.b};
            const unsigned long long sX4[3] = {(unsigned long long)a.x.stride_head * 2, (unsigned long long)a.x.stride_seq * 2, (unsigned long long)a.x.stride_batch * 2};
            const unsigned long long sG4[3] = {(unsigned long long)gv.sh * 2, (unsigned long long)gv.sl * 2, (unsigned long long)gv.sb * 2};
            const unsigned bx4[4] = {64, 1, 128, 1};
            if (tc::make_map4(&mX, a.p.x_dtype, a.x.ptr, dX4, sX4, bx4) && tc::make_map4(&mG, a.p.x_dtype, gv.ptr, dX4, sG4, bx4)) {
                // the product with B / C reads dCB by TMA from a 16-bit copy when it can
                const unsigned long long dBC4[4] = {(unsigned long long)d.N, (unsigned long long)d.G, (unsigned long long)d.L, (unsigned long long)d.b};
                const unsigned long long sB4[3] = {(unsigned long long)a.B.stride_head * 2, (unsigned long long)a.B.stride_seq * 2, (unsigned long long)a.B.stride_batch * 2};
                const unsigned long long sC4b[3] = {(unsigned long long)a.C.stride_head * 2, (unsigned long long)a.C.stride_seq * 2, (unsigned long long)a.C.stride_batch * 2};
                const unsigned long long dcb_rows = (unsigned long long)d.b * d.nc * d.G * d.Q;
                bmm_tma = !no_ws() && tc::bmm_bwd_tma_ok(d.N, d.Q) &&
                          tc::make_map4(&mBb, a.p.x_dtype, a.B.ptr, dBC4, sB4, bx4) && tc::make_map4(&mCb, a.p.x_dtype, a.C.ptr, dBC4, sC4b, bx4) &&
                          tc::make_map2(&mDm, a.p.x_dtype, F(w.dCB), d.Q, dcb_rows, 64, d.Q) &&
                          tc::make_map2(&mDk, a.p.x_dtype, F(w.dCB), d.Q, dcb_rows, 64, 128);
                const size_t smem_t = tc::dcb_tma_smem(d.P, d.Q);
                BISSD_ALLOW(tc::dcb_tma<T>, smem_t);
                BISSD_LAUNCH("tc_dcb_tma", launch_pdl(tc::dcb_tma<T>, dim3(d.b * d.nc * d.G, nlt_tc, nlt_tc), tc::kThreads, smem_t, s, 
                    d, mG, mX, a.dt_out, a.cs_f, a.cs_b, bmm_tma ? nullptr : F(w.dCB), bmm_tma ? static_cast<void *>(F(w.dCB)) : nullptr, status));
                dcb_done = true;
            }
        }
        if (!dcb_done) {
            BISSD_ALLOW(tc::dcb_kernel<T>, smem_dcb);
            BISSD_LAUNCH("tc_dcb", tc::dcb_kernel<T><<<dim3(d.b * d.nc * d.G, nlt_tc, nlt_tc), tc::kThreads, smem_dcb, s>>>(
                dg, x, z, gv, a.dt_out, a.cs_f, a.cs_b, F(w.dCB), status));
        }
        bool intra_done = fused_done;
        const bool sums_path = !no_tma() && !no_sums() && tc::scan_tma_ok(d.P, d.N, d.Q);
        if (sums_path && !intra_done) {
            CUtensorMap mG, mX;
            if (map_bshd(&mG, a.p.x_dtype, gv.ptr, gv.sb, gv.sl, gv.sh, d.P, d.H, d.L, d.b, 128) &&
                map_bshd(&mX, a.p.x_dtype, a.x.ptr, a.x.stride_batch, a.x.stride_seq, a.x.stride_head, d.P, d.H, d.L, d.b, d.Q)) {
                const size_t smem_s = tc::intra_sums_smem(d.Q);
                BISSD_ALLOW(tc::intra_sums<T>, smem_s);
                BISSD_LAUNCH("tc_intra_sums", launch_pdl(tc::intra_sums<T>, dim3(bch, nlt_tc), tc::kThreads, smem_s, s, 
                    dg, mG, mX, a.dt_out, a.cs_f, a.cs_b, F(w.cbs), F(w.u4), (long long)d.b * d.H * d.nc * d.Q, status));
                intra_done = true;
                use_u4 = true;
            }
        }
        if (!intra_done && !have_fp32_cb) {                  // the prefix-sweep kernels read the fp32 matrix
            if (lean && fused_wanted(d)) return BISSD_ERR_WORKSPACE;
            const size_t smem_cb = tc::smem_bytes(ntQ, 0);
            BISSD_LAUNCH("tc_bmm_cb", tc::bmm_cb<T><<<dim3(d.b * d.nc * d.G, nlt_tc), tc::kThreads, smem_cb, s>>>(
                d, Cm, Bm, F(w.cb), F(w.cbt), nullptr, nullptr, nullptr, status));
            have_fp32_cb = true;
        }
        if (!intra_done && !no_tma() && tc::scan_tma_ok(d.P, d.N, d.Q)) {
            CUtensorMap mG, mX;
            if (map_bshd(&mG, a.p.x_dtype, gv.ptr, gv.sb, gv.sl, gv.sh, d.P, d.H, d.L, d.b, 128) &&
                map_bshd(&mX, a.p.x_dtype, a.x.ptr, a.x.stride_batch, a.x.stride_seq, a.x.stride_head, d.P, d.H, d.L, d.b, d.Q)) {
                BISSD_ALLOW((tc::intra_decay_grad<T, true>), smem_in);
                BISSD_LAUNCH("tc_intra_decay_grad", tc::intra_decay_grad<T, true><<<dim3(bch, nlt_tc), tc::kThreads, smem_in, s>>>(
                    dg, mG, mX, x, z, gv, a.dt_out, a.cs_f, a.cs_b, F(w.cb), F(w.da_f), F(w.da_b), status));
                intra_done = true;
            }
        }
        if (!intra_done) {
            CUtensorMap none{};
            BISSD_ALLOW((tc::intra_decay_grad<T, false>), smem_in);
            BISSD_LAUNCH("tc_intra_decay_grad", tc::intra_decay_grad<T, false><<<dim3(bch, nlt_tc), tc::kThreads, smem_in, s>>>(
                dg, none, none, x, z, gv, a.dt_out, a.cs_f, a.cs_b, F(w.cb), F(w.da_f), F(w.da_b), status));
        }
    }
    // the side stream's kernels rejoin before their results are read
    const bool beside = side.stream() != s;
    int rcj = note_cuda(side.join(), "join of the second stream");
    if (rcj != BISSD_OK) return rcj;
    if (dbc_last) {
        if (!bmm_tma) return BISSD_ERR_ALIGN;                    // its operands are the ones the dCB kernel's branch has mapped
        if (beside) {
            rcj = note_cuda(side.fork(), "fork of the second stream");
            if (rcj != BISSD_OK) return rcj;
        }
        const int rcl = launch_dbc(tc::dbc_accum_grp<T, true>, tc::LastMaps{mDm, mDk, mBb, mCb, gr.dB, gr.dC}, side.stream());
        if (rcl != BISSD_OK) return rcl;
    } else if (bmm_tma) {
        const size_t smem_b = tc::bmm_bwd_tma_smem(d.Q);
        BISSD_ALLOW(tc::bmm_bwd_tma<T>, smem_b);
        BISSD_LAUNCH("tc_bmm_bwd_tma", launch_pdl(tc::bmm_bwd_tma<T>, dim3(d.b * d.nc * d.G * 2, d.Q / 128, d.N / 64), tc::kThreads, smem_b, s,
            d, mDm, mDk, mBb, mCb, F(w.dB_part), F(w.dC_part), part_heads, gr.dB, gr.dC, status));
    } else {
        const size_t smem_n = tc::smem_bytes(ntN, 0);
        BISSD_ALLOW(tc::bmm_bwd<T>, smem_n);
        BISSD_LAUNCH("tc_bmm_bwd", tc::bmm_bwd<T><<<dim3(d.b * d.nc * d.G * 2, nlt_tc, w.nsplit), tc::kThreads, smem_n, s>>>(
            d, Bm, Cm, F(w.dCB), F(w.dB_part), F(w.dC_part), part_heads, gr.dB, gr.dC, status));
    }
    simt::CumsumBwd cs{};
    cs.dt = a.dt.ptr; cs.dt_dtype = a.p.dt_dtype; cs.dsb = a.dt.stride_batch; cs.dsl = a.dt.stride_seq; cs.dsh = a.dt.stride_head;
    cs.A = a.A; cs.dt_bias = a.dt_bias; cs.dt_out = a.dt_out; cs.ddt_out = F(w.ddt_out);
    cs.nf = F(w.nf); cs.nb = F(w.nb); cs.pf = F(w.pf); cs.pb = F(w.pb);
    if (use_u4) { cs.u4 = F(w.u4); cs.u4_tiles = u4_tiles; }
    else { cs.da_f = F(w.da_f); cs.da_b = F(w.da_b); }
    cs.dTpart = F(w.dTpart); cs.nblk = w.nslots; cs.nsplit = nsplit; cs.ddt = gr.ddt; cs.dApart = F(w.dApart); cs.dbiaspart = F(w.dbiaspart);
    BISSD_LAUNCH("cumsum_bwd", launch_pdl(d.Q <= 128 ? tc::cumsum_bwd<1> : tc::cumsum_bwd<2>, tc::cumsum_blocks(d), 32 * tc::kCumsumWarps, 0, s,
        d, cs, all_aligned16(a.dt_out, a.dt_out, a.dt_out)));
    BISSD_LAUNCH("final_reduce", launch_pdl(simt::final_reduce<1024>, d.H, 1024, 0, s, 
        d, F(w.dApart), F(w.dbiaspart), d.has_D ? F(w.dDpart) : nullptr, dd_slots ? dd_slots : nlt, dd_compact ? 1 : 0, a.dA, d.has_bias ? a.ddt_bias : nullptr,
        d.has_D ? a.dD : nullptr));
    return note_cuda(side.join(), "join of the second stream");
}

}  // namespace bissd

using namespace bissd;

extern "C" {

int bissd_abi_version(void) { return BISSD_ABI_VERSION; }

const char *bissd_strerror(int status) {
    switch (status) {
        case BISSD_OK: return "ok";
        case BISSD_ERR_NULL: return "a required pointer is NULL";
        case BISSD_ERR_SHAPE: return "inconsistent or unsupported sizes (need nheads % ngroups == 0, 32 <= chunk_size <= 256)";
        case BISSD_ERR_DTYPE: return "unsupported dtype";
        case BISSD_ERR_ALIGN: return "pointer or stride not sufficiently aligned";
        case BISSD_ERR_WORKSPACE: return "workspace too small or misaligned";
        case BISSD_ERR_LAUNCH: return "CUDA launch or API call failed";
        case BISSD_ERR_ARCH: return "device is not compute capability 10.x (B200)";
        case BISSD_ERR_PHASE: return "invalid phase mask";
        case BISSD_ERR_TOO_LARGE: return "problem needs more scratch than the fixed array of bissd_forward_static_scratch holds";
        default: return "unknown status";
    }
}

const char *bissd_last_cuda_error(void) { return g_cuda_err; }

int bissd_workspace_bytes(const bissd_problem *p, size_t *fwd_bytes, size_t *bwd_bytes) {
    if (!p) return BISSD_ERR_NULL;
    Dims d;
    int rc = make_dims(*p, &d);
    if (rc != BISSD_OK) return rc;
    if (fwd_bytes) *fwd_bytes = fwd_layout(d).total;
    if (bwd_bytes) *bwd_bytes = bwd_layout(d, !force_simt() && tc_shape_ok(*p)).total;
    return BISSD_OK;
}

int bissd_workspace_bytes_least(const bissd_problem *p, size_t *fwd_bytes, size_t *bwd_bytes) {
    if (!p) return BISSD_ERR_NULL;
    Dims d;
    int rc = make_dims(*p, &d);
    if (rc != BISSD_OK) return rc;
    const bool tcp = !force_simt() && tc_shape_ok(*p);
    if (fwd_bytes) *fwd_bytes = (tcp ? least_fwd(d) : fwd_layout(d)).total;
    if (bwd_bytes) *bwd_bytes = (tcp ? least_bwd(d) : bwd_layout(d, false)).total;
    return BISSD_OK;
}

unsigned long long bissd_launch_count(void) { return g_launches.load(); }

int bissd_trace_enable(int on) {
    std::lock_guard<std::mutex> lk(g_trace_mu);
    for (auto &r : g_trace) {
        cudaEventDestroy(r.e0);
        cudaEventDestroy(r.e1);
    }
    g_trace.clear();
    g_trace_on.store(on ? 1 : 0);
    return BISSD_OK;
}

int bissd_trace_read(char *names, size_t names_cap, float *total_ms, int *launches, int cap, int *count) {
    if (!names || !total_ms || !launches || !count) return BISSD_ERR_NULL;
    std::lock_guard<std::mutex> lk(g_trace_mu);
    std::vector<const char *> keys;
    std::vector<float> ms;
    std::vector<int> cnt;
    for (auto &r : g_trace) {
        if (cudaEventSynchronize(r.e1) != cudaSuccess) return note_cuda(cudaGetLastError(), "trace sync");
        float t = 0.f;
        if (cudaEventElapsedTime(&t, r.e0, r.e1) != cudaSuccess) return note_cuda(cudaGetLastError(), "trace elapsed");
        size_t k = 0;
        for (; k < keys.size(); ++k)
            if (strcmp(keys[k], r.name) == 0) break;
        if (k == keys.size()) { keys.push_back(r.name); ms.push_back(0.f); cnt.push_back(0); }
        ms[k] += t;
        cnt[k] += 1;
    }
    size_t used = 0;
    int n = 0;
    names[0] = 0;
    for (size_t k = 0; k < keys.size() && n < cap; ++k) {
        const size_t len = strlen(keys[k]);
        if (used + len + 2 > names_cap) break;
        memcpy(names + used, keys[k], len);
        used += len;
        names[used++] = ';';
        names[used] = 0;
        total_ms[n] = ms[k];
        launches[n] = cnt[k];
        ++n;
    }
    *count = n;
    return BISSD_OK;
}

int bissd_selftest_gemm(int dtype, int a_mn_major, int b_mn_major, int n, int k, const void *A, const void *B, float *C,
                        int *status_dev, void *stream) {
    if (!A || !B || !C || !status_dev) return BISSD_ERR_NULL;
    if (dtype != BISSD_BF16 && dtype != BISSD_F16) return BISSD_ERR_DTYPE;
    if (n < 16 || n > 256 || (n % 16) || k < 8 || (k % 8)) return BISSD_ERR_SHAPE;
    int rc = check_device();
    if (rc != BISSD_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t smem = 2 * tc::kAStageBytes + 2 * 256 * 128 + 1024;
#define BISSD_SELFTEST(T, AM, BM)                                                                          \
    do {                                                                                                   \
        rc = allow_smem(tc::selftest_gemm<T, AM, BM>, smem);                                               \
        if (rc != BISSD_OK) return rc;                                                                     \
        BISSD_LAUNCH("selftest_gemm", tc::selftest_gemm<T, AM, BM><<<1, tc::kThreads, smem, s>>>(          \
                                          static_cast<const T *>(A), static_cast<const T *>(B), C, n, k, status_dev)); \
    } while (0)
#define BISSD_SELFTEST_T(T)                                        \
    do {                                                           \
        if (a_mn_major && b_mn_major) BISSD_SELFTEST(T, true, true);   \
        else if (a_mn_major) BISSD_SELFTEST(T, true, false);       \
        else if (b_mn_major) BISSD_SELFTEST(T, false, true);       \
        else BISSD_SELFTEST(T, false, false);                      \
    } while (0)
    if (dtype == BISSD_BF16) BISSD_SELFTEST_T(__nv_bfloat16);
    else BISSD_SELFTEST_T(__half);
#undef BISSD_SELFTEST_T
#undef BISSD_SELFTEST
    return BISSD_OK;
}

const char *bissd_kernel_path(const bissd_problem *p) {
    if (!p) return "";
    return (!force_simt() && tc_shape_ok(*p)) ? "tcgen05" : "simt";
}

static int static_scratch_if_known(void **out);

int bissd_read_status(const void *workspace, void *stream, int *status_out) {
    if (!status_out) return BISSD_ERR_NULL;
    if (!workspace) {                                            // the library-owned scratch of the current device
        void *scratch = nullptr;
        int rc = static_scratch_if_known(&scratch);
        if (rc != BISSD_OK) return rc;
        workspace = scratch;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int rc = note_cuda(cudaMemcpyAsync(status_out, workspace, sizeof(int), cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
    if (rc != BISSD_OK) return rc;
    return note_cuda(cudaStreamSynchronize(s), "cudaStreamSynchronize");
}

int bissd_forward(const bissd_fwd_args *a, void *workspace, size_t workspace_bytes, void *stream) {
    if (!a) return BISSD_ERR_NULL;
    Dims d;
    int rc = make_dims(a->p, &d);
    if (rc != BISSD_OK) return rc;
    if (a->phases < 1 || a->phases > BISSD_PHASE_ALL) return BISSD_ERR_PHASE;
    if (!a->x.ptr || !a->B.ptr || !a->C.ptr || !a->dt.ptr || !a->A || !a->dt_out || !a->cs_f || !a->cs_b ||
        !a->states_f || !a->states_b)
        return BISSD_ERR_NULL;
    if ((a->phases & BISSD_PHASE_FINISH) && !a->out.ptr) return BISSD_ERR_NULL;
    if (a->p.has_z && (!a->z.ptr || ((a->phases & BISSD_PHASE_FINISH) && !a->out_x.ptr))) return BISSD_ERR_NULL;
    if (a->p.has_D && !a->D) return BISSD_ERR_NULL;
    if (a->p.has_dt_bias && !a->dt_bias) return BISSD_ERR_NULL;
    const bool tcp = !force_simt() && tc_shape_ok(a->p) && aligned16(a->x) && aligned16(a->B) && aligned16(a->C) &&
                     aligned16(a->z) && aligned16(a->out) && aligned16(a->out_x);
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 255) || workspace_bytes < (tcp ? least_fwd(d) : fwd_layout(d)).total)
        return BISSD_ERR_WORKSPACE;
    if (!states_aligned(a->p, tcp, a->states_f, a->states_b)) return BISSD_ERR_ALIGN;
    rc = check_device();
    if (rc != BISSD_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char *ws = static_cast<char *>(workspace);
    if (!tcp) return simt_forward(*a, d, ws, s);
    return a->p.x_dtype == BISSD_BF16 ? forward_impl<__nv_bfloat16>(*a, d, ws, workspace_bytes, s) : forward_impl<__half>(*a, d, ws, workspace_bytes, s);
}

// ---- forward pass on library-owned scratch -------------------------------------------------------------------
// Some hosts may not allocate device memory when they reach this operator: an inference server that hands each
// plug-in a fixed set of buffers and forbids cudaMalloc after start-up, or code that runs while the allocator is
// locked.  For them the scratch of the forward pass lives in this fixed array, part of the library's device image:
// every GPU context that loads libbissd holds these 16 MiB until the process exits, whether or not it uses them.
constexpr size_t kStaticScratchBytes = BISSD_STATIC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// In host code the name g_static_scratch is only a handle for the symbol, not a device address; the address on
// the current device comes from cudaGetSymbolAddress, asked once per device and remembered.
static std::mutex g_static_mu;
static void *g_static_addr[64] = {};

static int static_scratch_on_current_device(void **out) {
    int dev = -1;
    int rc = note_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc != BISSD_OK) return rc;
    if (dev < 0 || dev >= 64) return BISSD_ERR_LAUNCH;
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static_addr[dev]) {
        void *ptr = nullptr;
        rc = note_cuda(cudaGetSymbolAddress(&ptr, g_static_scratch), "cudaGetSymbolAddress");
        if (rc != BISSD_OK) return rc;
        if (!ptr || (reinterpret_cast<uintptr_t>(ptr) & 255)) return BISSD_ERR_WORKSPACE;
        g_static_addr[dev] = ptr;
    }
    *out = g_static_addr[dev];
    return BISSD_OK;
}

// For bissd_read_status(NULL, ...): the address remembered by an earlier bissd_forward_static_scratch call on this
// device; no symbol lookup here, so a status read never triggers the set-up.
static int static_scratch_if_known(void **out) {
    int dev = -1;
    int rc = note_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc != BISSD_OK) return rc;
    if (dev < 0 || dev >= 64) return BISSD_ERR_LAUNCH;
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static_addr[dev]) return BISSD_ERR_NULL;              // bissd_forward_static_scratch has not run here yet
    *out = g_static_addr[dev];
    return BISSD_OK;
}

int bissd_forward_static_scratch(const bissd_fwd_args *a, void *stream) {
    if (!a) return BISSD_ERR_NULL;
    Dims d;
    int rc = make_dims(a->p, &d);
    if (rc != BISSD_OK) return rc;
    if (a->phases != BISSD_PHASE_ALL) return BISSD_ERR_PHASE;      // a split pass needs scratch the caller keeps
    if (fwd_layout(d).total > kStaticScratchBytes) return BISSD_ERR_TOO_LARGE;
    void *scratch = nullptr;
    rc = static_scratch_on_current_device(&scratch);
    if (rc != BISSD_OK) return rc;
    // The array still holds whatever the previous call left.  Only the status word at its start is read before it is written:
    // the first kernel of the pass clears it.
    return bissd_forward(a, scratch, kStaticScratchBytes, stream);
}

int bissd_chain_boundaries(const float *left, const float *right, const float *log_decay, int64_t rank_stride,
                           int64_t log_decay_rank_stride, int world, int rank, int64_t batch_heads, int32_t state_elems,
                           float *out_left, float *out_right, void *stream) {
    if (!left || !right || !log_decay || !out_left || !out_right) return BISSD_ERR_NULL;
    if (world < 1 || rank < 0 || rank >= world || batch_heads <= 0 || state_elems <= 0) return BISSD_ERR_SHAPE;
    int rc = check_device();
    if (rc != BISSD_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const long long n = (long long)batch_heads * state_elems;
    BISSD_LAUNCH("chain_boundaries", simt::chain_boundaries<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(
        left, right, log_decay, rank_stride, log_decay_rank_stride, world, rank, n, state_elems, out_left, out_right));
    return BISSD_OK;
}

int bissd_backward(const bissd_bwd_args *a, void *workspace, size_t workspace_bytes, void *stream) {
    return bissd_backward_into(a, nullptr, workspace, workspace_bytes, stream);
}

int bissd_backward_into(const bissd_bwd_args *a, const bissd_grad_strides *gs, void *workspace, size_t workspace_bytes,
                        void *stream) {
    if (!a) return BISSD_ERR_NULL;
    Dims d;
    int rc = make_dims(a->p, &d);
    if (rc != BISSD_OK) return rc;
    if (a->phases < 1 || a->phases > BISSD_PHASE_ALL) return BISSD_ERR_PHASE;
    if (!a->x.ptr || !a->B.ptr || !a->C.ptr || !a->dt.ptr || !a->dout.ptr || !a->A || !a->dt_out || !a->cs_f ||
        !a->cs_b || !a->states_f || !a->states_b)
        return BISSD_ERR_NULL;
    if (a->phases & BISSD_PHASE_FINISH) {
        if (!a->dx || !a->dB || !a->dC || !a->ddt || !a->dA) return BISSD_ERR_NULL;
        if (a->p.has_z && (!a->dz || !a->out_x.ptr)) return BISSD_ERR_NULL;
        if (a->p.has_D && !a->dD) return BISSD_ERR_NULL;
        if (a->p.has_dt_bias && !a->ddt_bias) return BISSD_ERR_NULL;
    }
    if (a->p.has_z && (!a->z.ptr || !a->dz || !a->out_x.ptr)) return BISSD_ERR_NULL;   // the gate runs in the LOCAL phase
    if (a->p.has_D && !a->D) return BISSD_ERR_NULL;
    if (a->p.has_dt_bias && !a->dt_bias) return BISSD_ERR_NULL;
    // 16-bit tensors that miss the tensor-core family's alignment rules run on the CUDA-core family, which needs the
    // larger workspace that bissd_workspace_bytes reports for the same sizes with fp32 inputs
    const bool tcp = !force_simt() && tc_shape_ok(a->p) && aligned16(a->x) && aligned16(a->B) && aligned16(a->C) &&
                     aligned16(a->z) && aligned16(a->dout) && aligned16(a->out_x);
    const size_t need = (tcp && a->phases == BISSD_PHASE_ALL ? least_bwd(d) : bwd_layout(d, tcp)).total;   // a split pass keeps its local gradients
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 255) || workspace_bytes < need) return BISSD_ERR_WORKSPACE;
    const long long L = d.L, hp = (long long)d.H * d.P, gn = (long long)d.G * d.N;
    GradViews gr{MutView{a->dx, L * hp, hp, d.P}, MutView{a->dB, L * gn, gn, d.N}, MutView{a->dC, L * gn, gn, d.N},
                 MutView{a->ddt, L * d.H, d.H, 1}};
    if (gs) {
        auto set = [](MutView &v, const int64_t *st) { v.sb = st[0]; v.sl = st[1]; v.sh = st[2]; };
        set(gr.dx, gs->dx); set(gr.dB, gs->dB); set(gr.dC, gs->dC); set(gr.ddt, gs->ddt);
    }
    auto al = [](const MutView &v) { return reinterpret_cast<uintptr_t>(v.ptr) % 16 == 0 && v.sb % 8 == 0 && v.sl % 8 == 0 && v.sh % 8 == 0; };
    if (tcp && !(al(gr.dx) && al(gr.dB) && al(gr.dC) && all_aligned16(a->dz, a->dz, a->dz))) return BISSD_ERR_ALIGN;   // 16-byte stores
    if (!states_aligned(a->p, tcp, a->states_f, a->states_b)) return BISSD_ERR_ALIGN;
    rc = check_device();
    if (rc != BISSD_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char *ws = static_cast<char *>(workspace);
    if (!tcp) return simt_backward(*a, gr, d, ws, s);
    return a->p.x_dtype == BISSD_BF16 ? backward_impl<__nv_bfloat16>(*a, gr, d, ws, workspace_bytes, s) : backward_impl<__half>(*a, gr, d, ws, workspace_bytes, s);
}

}  // extern "C"
