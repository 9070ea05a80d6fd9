// Workspace layouts shared by the launch code of the kernel families.  The first 256 bytes hold the device status word
// (nonzero = a bounded device-side wait ran out); everything after it is scratch.
#pragma once
#include "host.cuh"
#include "simt_tile.cuh"

namespace bissd {

constexpr size_t kWsHeader = 256;
struct FwdWs {
    size_t loc, cb, cb16, total;
};
struct BwdWs {
    size_t cb, cbt, cbt16, cb16, cbs, gloc, E, E16, g, dTpart, ddt_out, nf, nb, pf, pb, da_f, da_b, u4, dB_part, dC_part, dCB, dDpart,
        dApart, dbiaspart, total;
    int nslots, nlt, nsplit, hsplit, dbc_ks;
};

// The recurrence over chunks: four elements of the (headdim, dstate) state per thread where their number allows.
inline bool pass_by4(const Dims &d) { return (d.P * d.N) % 4 == 0; }
inline int pass_threads(const Dims &d) {                         // per block: fewer for small states
    const int want = ceil_div(d.P * d.N, pass_by4(d) ? 4 : 1);
    return std::min(simt::TB, (want + 31) / 32 * 32);
}
inline dim3 pass_grid(const Dims &d) { return dim3(d.b * d.H, ceil_div(d.P * d.N, (pass_by4(d) ? 4 : 1) * pass_threads(d)), 2); }
// Few threads (long sequences of small states) wait for memory: they keep eight chunks' loads in flight.  Many threads are
// bound by HBM, and batched loads only cost them residency (b8 H24 nc8 P64 N128: backward 39 us one by one, 49 - 60
// with 4 - 8 in flight, forward 24.5 and 32).
inline bool pass_ahead(const Dims &d) {
    const dim3 g = pass_grid(d);
    return (long long)g.x * g.y * g.z * pass_threads(d) < 256LL * sm_count();
}
inline int pass_slots(const Dims &d) {                           // partial dT per (direction, batch, head, chunk), the walk's included
    return pass_grid(d).y * (pass_by4(d) ? pass_threads(d) / 32 : 1);
}

// Arrays that only some kernels need.  bissd_workspace_bytes reports room for all of them; a pass whose kernels are known to
// do without also runs in less (bissd_workspace_bytes_least).  They lie at the end: the others are where they are either way.
struct FwdNeed {
    bool loc = true, cb = true, cb16 = true;                     // local states; C.B^T in fp32; rounded to bf16 (TMA-fed scan)
};
inline FwdWs fwd_layout(const Dims &d, FwdNeed need = FwdNeed()) {
    FwdWs w;
    size_t o = kWsHeader;
    auto take = [&](size_t bytes) { size_t at = o; o = align256(o + bytes); return at; };
    const size_t qq = (size_t)d.b * d.nc * d.G * d.Q * d.Q;
    w.cb16 = take(need.cb16 ? qq * 2 : 0);
    w.cb = take(need.cb ? qq * 4 : 0);
    w.loc = take(need.loc ? 2 * (size_t)d.b * d.nc * d.H * d.P * d.N * 4 : 0);
    w.total = o;
    return w;
}

// CUDA-core dCB product: are there blocks enough with one for all heads of a group?  Other blocks of the launch fill the SMs
// beside them, so four for five SMs do (us a pass, two blocks an SM asked for and this: b4 L1000 H8 P32 N32 chunk 128,
// 128 blocks, 167, 160; b2 L4000 H4 P64 N64, 256 blocks, 297, 290; b1 L8000 H8 chunk 64, 125 blocks, 267, 260).
inline bool simt_dcb_fills(const Dims &d, int rows) {
    const int nt = ceil_div(d.Q, simt::TILE);
    return 5LL * rows * d.nc * d.G * nt * nt >= 4LL * sm_count();
}
// Parts the heads of a group are summed in: by one row of the batch, so that a row's results do not depend on how many rows
// there are.  A divisor of the heads; enough for two blocks an SM where a row alone does not fill them.
inline int simt_parts(const Dims &d) {
    if (simt_dcb_fills(d, 1)) return 1;
    const int nt = ceil_div(d.Q, simt::TILE);
    const long long blocks = (long long)d.nc * d.G * nt * nt;
    int parts = 1;
    for (int k = 2; k <= d.R && blocks * parts < 2LL * sm_count(); ++k)
        if (d.R % k == 0) parts = k;
    return parts;
}
// Blocks that share the parts, each with a partial dCB of its own that the last product adds to the others: one a part, or
// one for all of them where the rows fill the SMs.
inline int simt_hsplit(const Dims &d) { return simt_dcb_fills(d, d.b) ? 1 : simt_parts(d); }

// Blocks the heads of a group are dealt to in dbc_accum_grp (one block an SM, about 2 us a head), each writing a partial
// dB / dC that the last product adds up again: more than one only where the blocks leave SMs idle.
inline int dbc_ksplit(const Dims &d) {
    const long long tiles = 2LL * d.b * d.nc * d.G * ceil_div(d.N, 128);
    int best = 1;
    float least = 0.f;
    for (int ks = 1; ks <= head_parts(d); ks *= 2) {
        const long long waves = (tiles * ks + sm_count() - 1) / sm_count();
        const float t = waves * (2.f * ceil_div(d.R, ks) + 5.f) + ks;
        if (ks == 1 || t < least) {
            best = ks;
            least = t;
        }
    }
    return best;
}

// tc: sized for the tensor-core family (16-bit inputs that meet its alignment rules): the passed state gradients are
// kept in the input dtype only, and the "states" parts of dB / dC arrive summed over the heads of a group.  The
// CUDA-core family needs the fp32 copy and one partial per head.
struct BwdNeed {
    bool gloc = true, parts = true, cb32 = true;                 // local state gradients; partial dB / dC; C.B^T in fp32 and its copies
};
inline BwdWs bwd_layout(const Dims &d, bool tc, BwdNeed need = BwdNeed()) {
    BwdWs w;
    size_t o = kWsHeader;
    const size_t st = (size_t)d.b * d.nc * d.H * d.P * d.N;
    const size_t hq = (size_t)d.b * d.H * d.nc * d.Q, qq = (size_t)d.b * d.nc * d.G * d.Q * d.Q;
    w.nslots = pass_slots(d);
    w.nlt = ceil_div(d.Q, simt::TILE);
    w.nsplit = tc ? ceil_div(d.N, 128) : 1;
    w.hsplit = tc ? 1 : simt_hsplit(d);
    w.dbc_ks = tc ? dbc_ksplit(d) : 1;
    const int slots = dbc_slots(d, w.dbc_ks);
    auto take = [&](size_t bytes) { size_t at = o; o = align256(o + bytes); return at; };
    w.E = take(tc ? 0 : 2 * st * 4);                                 // fp32 passed state gradients (CUDA-core family)
    w.E16 = take(tc ? 2 * st * 2 : 0);                               // passed state gradients in the input dtype
    w.g = take(tc ? (size_t)d.b * d.L * d.H * d.P * 2 : 0);          // gated output gradient dout * silu(z)
    w.cbt16 = take(tc ? qq * 2 : 0);                                 // CB transposed, rounded to bf16 (TMA-fed dx)
    w.cb16 = take(tc ? qq * 2 : 0);                                  // CB rounded to bf16 (tc::intra_dcb_tile)
    w.dTpart = take((size_t)2 * d.b * d.H * d.nc * w.nslots * 4);
    w.ddt_out = take(hq * 4);
    w.nf = take(hq * 4 * w.nsplit); w.nb = take(hq * 4 * w.nsplit);
    w.pf = take(hq * 4 * w.nsplit); w.pb = take(hq * 4 * w.nsplit);
    w.da_f = take(tc ? hq * 4 : 0); w.da_b = take(tc ? hq * 4 : 0);
    w.u4 = take((tc ? 8 : 4 * w.nlt) * hq * 4);                      // u_f / u_b per tile (tc::intra_sums: 2 row tiles; tc::intra_dcb_tile: 4; simt: 2 nlt)
    w.dCB = take(qq * 4 * w.hsplit);
    w.dDpart = take((size_t)d.b * d.nc * d.H * std::max(w.nlt, 8) * d.P * 4);   // up to 8 partial rows per (b,c,h)
    w.dApart = take((size_t)d.b * d.nc * d.H * 4);
    w.dbiaspart = take((size_t)d.b * d.nc * d.H * 4);
    w.cb = take(need.cb32 ? qq * 4 : 0);
    w.cbt = take(tc && need.cb32 ? qq * 4 : 0);                      // CB transposed
    w.cbs = take(tc && need.cb32 ? qq * 4 : 0);                      // CB in strips of 16 columns (tc::intra_sums)
    const size_t part = need.parts ? (size_t)d.b * d.nc * d.Q * (tc ? d.G * slots : d.H) * d.N * 4 : 0;
    w.dB_part = take(part);
    w.dC_part = take(part);
    w.gloc = take(need.gloc ? 2 * st * 4 : 0);
    w.total = o;
    return w;
}

inline View view_of(const bissd_tensor &t) { return View{t.ptr, t.stride_batch, t.stride_seq, t.stride_head}; }
inline MutView mview_of(const bissd_tensor &t) { return MutView{t.ptr, t.stride_batch, t.stride_seq, t.stride_head}; }

// Where dx, dB, dC and ddt go (bissd_backward: contiguous, bissd_backward_into: the caller's strides).
struct GradViews {
    MutView dx, dB, dC, ddt;
};

// The CUDA-core family (bissd_simt.cu): fp32 inputs, and 16-bit ones outside the tensor-core family's shapes or alignment.
int simt_forward(const bissd_fwd_args &a, const Dims &d, char *ws, cudaStream_t s);
int simt_backward(const bissd_bwd_args &a, const GradViews &gr, const Dims &d, char *ws, cudaStream_t s);

}  // namespace bissd
