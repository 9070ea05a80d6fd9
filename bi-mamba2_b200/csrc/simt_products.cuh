// General-shape CUDA-core kernels for the products of the bidirectional SSD chunk scan, in three launches forward and five
// backward with the recurrence and the reductions (simt_kernels.cuh) between them.
//
// They accept any headdim / dstate / chunk_size (<= 256) / dtype and ragged sequence tails, and compute all products in
// fp32 - the path for fp32 inputs and for shapes the tcgen05 kernels do not cover.  Products that do not depend on one
// another share a launch, as ranges of its blocks ("roles"): a small problem is a handful of blocks per product, bound by
// the latency of a block and of a launch.
//
//   forward1   chunk_state (with the discretisation and the cumulative sums)  |  bmm_cb
//   forward2   chunk_scan
//   backward1  dstates  |  bmm_cb
//   backward2  dcb_intra  |  dx  |  dbc_states
//   backward3  bmm_bwd  |  cumsum_bwd
//
// Decay factors, masks, gates and the two directions are applied while a panel is put into shared memory; where a product
// runs over both directions its depth is simply [forward | reverse].
// Bound by shared-memory reads and instruction issue, small problems by block and launch latency.  Device time of a
// forward + backward pass, fp32, against one product per launch with 64-wide tiles and 16-deep panels filled element by
// element: b1 L256 H4 P32 N16 Q64 156 -> 48 us (17 -> 8 launches), b2 L8192 H4 G4 P16 N16 Q128 1012 -> 311 us.
#pragma once
#include "simt_kernels.cuh"

namespace bissd {
namespace simt {

struct Panels {                                                  // dynamic shared memory of every kernel here
    float a[TILE * LD];
    float b[TILE * LD];
    float v[5][256];                                             // per-position vectors of the chunk (16-byte aligned)
    float red[8][2][TILE];
};

// Which tensors may be read four elements at a time.
enum { VEC_X = 1, VEC_BC = 2, VEC_Q = 4, VEC_N = 8, VEC_P = 16 };

template <class T> __device__ __forceinline__ const T *row_ptr(const View &t, int b, int l, int h) {
    return static_cast<const T *>(t.ptr) + b * t.sb + l * t.sl + h * t.sh;
}
template <class T> __device__ __forceinline__ T *row_ptr(const MutView &t, int b, int l, int h) {
    return static_cast<T *>(t.ptr) + b * t.sb + l * t.sl + h * t.sh;
}
struct Where {                                                   // one (batch, chunk, head)
    int b, c, h, g, l0, lim;
    long long base;                                              // of its per-position vectors
    __device__ __forceinline__ Where(const Dims &d, int i) {
        h = i % d.H; c = (i / d.H) % d.nc; b = i / (d.H * d.nc); g = h / d.R;
        l0 = c * d.Q; lim = min(d.Q, d.L - l0);
        base = ((long long)(b * d.H + h) * d.nc + c) * d.Q;
    }
};
// Four values of row `fw` (columns 0 ... N - 1) and row `bw` (columns N ... 2N - 1) from column m on.
template <class T> __device__ __forceinline__ float4 load_dirs(const T *fw, const T *bw, int m, int N, bool vec) {
    if (m + 4 <= N) return load4<T>(fw + m, 4, vec);
    if (m >= N) return load4<T>(bw + (m - N), 2 * N - m, vec && (m - N) % 4 == 0);
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = m + i < N ? to_f<T>(fw[m + i]) : (m + i < 2 * N ? to_f<T>(bw[m + i - N]) : 0.f);
    return make_float4(v[0], v[1], v[2], v[3]);
}
// g = d(out)/d(y): dout, or dout * silu(z) when gated; rows of one head.
template <class T>
__device__ __forceinline__ void fetch_gated(Frag &fr, int sh, const Dims &d, const View &dout, const View &z, int b, int l, int h, int p0,
                                            int rows, int cols, bool vec) {
    fetch<T>(fr, sh, row_ptr<T>(dout, b, l, h) + p0, dout.sl, rows, cols, vec);
    if (d.has_z) {
        Frag zf;
        fetch<T>(zf, sh, row_ptr<T>(z, b, l, h) + p0, z.sl, rows, cols, vec);
        pieces(sh, [&](int u, int, int) {
            fr.v[u].x *= zf.v[u].x * sigmoidf_(zf.v[u].x);
            fr.v[u].y *= zf.v[u].y * sigmoidf_(zf.v[u].y);
            fr.v[u].z *= zf.v[u].z * sigmoidf_(zf.v[u].z);
            fr.v[u].w *= zf.v[u].w * sigmoidf_(zf.v[u].w);
        });
    }
}
// The chunk's per-position vectors: cumulative sums, Delta, and the decay inside each quad of positions - to its last
// position (reverse: its first), so that four adjacent weights cost one exponential and four products.
struct Vectors {
    const float *sf, *sb, *sd, *qf, *qb;
};
__device__ __forceinline__ Vectors load_vectors(Panels &sm, const Dims &d, const Where &w, const float *dt_out, const float *cs_f, const float *cs_b) {
    const int l = threadIdx.x;                                   // beyond the chunk: finite values that meet zeros only
    const float f = cs_f[w.base + min(l, d.Q - 1)], r = l < d.Q ? cs_b[w.base + l] : 0.f;
    sm.v[0][l] = f;
    sm.v[1][l] = r;
    sm.v[2][l] = l < d.Q ? dt_out[w.base + l] : 0.f;
    // a quad's ends are in this thread's warp
    const float fe = __shfl_sync(0xffffffffu, f, (l & 31) | 3), re = __shfl_sync(0xffffffffu, r, l & 28);
    sm.v[3][l] = expf(fe - f);
    sm.v[4][l] = expf(re - r);
    __syncthreads();
    return Vectors{sm.v[0], sm.v[1], sm.v[2], sm.v[3], sm.v[4]};
}
// Decay from positions from ... from + 3 (a quad) to position `to` of a chunk, both directions (both on the diagonal).
// All exponents are <= 0.
__device__ __forceinline__ float4 decay4(const Vectors &v, int to, int from) {
    const bool below = from + 3 < to, above = from > to;
    if (below || above) {
        const float e = below ? expf(v.sf[to] - v.sf[from + 3]) : expf(v.sb[to] - v.sb[from]);
        const float4 q = *reinterpret_cast<const float4 *>((below ? v.qf : v.qb) + from);
        return make_float4(e * q.x, e * q.y, e * q.z, e * q.w);
    }
    float w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int s = from + i;
        w[i] = (s <= to ? expf(v.sf[to] - v.sf[s]) : 0.f) + (s >= to ? expf(v.sb[to] - v.sb[s]) : 0.f);
    }
    return make_float4(w[0], w[1], w[2], w[3]);
}

// Local chunk states, or their gradients, for both directions: out[dir][b,c,h,p,n] = sum_l X[l,p] Y[l,n] w_dir[l], as a
// (2N x P) tile so that narrow heads fill the tile's rows.
//   chunk_state: X = x, Y = B, w = Delta e^{T - cs};  also dt_out = clamp(softplus(dt + bias)) and the cumulative sums.
//     Takes over _chunk_cumsum_fwd_kernel and _chunk_state_fwd_kernel (src/ssd/bi/ssd_chunk_state.py:34-91, :187-263).
//   dstates:     X = g, Y = C, w = e^{cs}.
//     Takes over _chunk_scan_bwd_dstates_kernel (src/ssd/bi/ssd_chunk_scan.py:457-522).
struct StateArgs {
    View X, Y, z;
    const void *dt;
    int dt_dtype;
    long long dsb, dsl, dsh;
    const float *A, *dt_bias;
    float *dt_out, *cs_f, *cs_b, *out;
};
template <class T, bool GRAD, int TW>
__device__ __forceinline__ void states_role(Panels &sm, const Dims &d, const StateArgs &a, int vec, int block) {
    const int mt = ceil_div(2 * d.N, TILE), pt = ceil_div(d.P, TW), tile = block % (mt * pt);
    const Where w(d, block / (mt * pt));
    const int m0 = tile % mt * TILE, p0 = tile / mt * TW, l = threadIdx.x;
    float *wf = sm.v[0], *wb = sm.v[1];
    if (GRAD) {
        if (l < d.Q) {
            wf[l] = expf(a.cs_f[w.base + l]);
            wb[l] = expf(a.cs_b[w.base + l]);
        }
    } else {
        float v, f, r;
        chunk_cumsum(d, a.dt, a.dt_dtype, a.dsb, a.dsl, a.dsh, a.A, a.dt_bias, w.b, w.c, w.h, w.lim, reinterpret_cast<float(*)[8]>(sm.red), v, f, r);
        if (l < d.Q && tile == 0) {
            a.dt_out[w.base + l] = v;
            a.cs_f[w.base + l] = f;
            a.cs_b[w.base + l] = r;
        }
        if (l == d.Q - 1) sm.v[3][0] = f;
        if (l == 0) sm.v[3][1] = r;
        __syncthreads();
        if (l < d.Q) {
            wf[l] = expf(sm.v[3][0] - f) * v;
            wb[l] = expf(sm.v[3][1] - r) * v;
        }
    }
    __syncthreads();
    const int shA = shift_for(2 * d.N - m0), shB = shift_for(min(d.P - p0, TW));
    Mul mul;
    mul.zero();
    Frag fa, fb;
    panels(w.lim, [&](int k0) {
        pieces(shA, [&](int u, int r, int c) {
            fa.v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            const int k = k0 + r, m = m0 + c;
            if (k >= w.lim || m >= 2 * d.N) return;
            const T *row = row_ptr<T>(a.Y, w.b, w.l0 + k, w.g);
            const float4 v = load_dirs<T>(row, row, m, d.N, vec & VEC_BC);
            fa.v[u] = make_float4(v.x * (m < d.N ? wf : wb)[k], v.y * (m + 1 < d.N ? wf : wb)[k], v.z * (m + 2 < d.N ? wf : wb)[k],
                                  v.w * (m + 3 < d.N ? wf : wb)[k]);
        });
        if (GRAD) fetch_gated<T>(fb, shB, d, a.X, a.z, w.b, w.l0 + k0, w.h, p0, w.lim - k0, d.P - p0, vec & VEC_X);
        else fetch<T>(fb, shB, row_ptr<T>(a.X, w.b, w.l0 + k0, w.h) + p0, a.X.sl, w.lim - k0, d.P - p0, vec & VEC_X);
    }, [&](int) {
        put_rows(fa, shA, sm.a);
        put_rows(fb, shB, sm.b);
    }, [&](int, int depth) { compute_tn<TW>(mul, sm.a, sm.b, depth); });
    const Acc<TW> acc = finish<TW>(mul, sm.a);
    const long long per_dir = (long long)d.b * d.nc * d.H * d.P * d.N;
    float *out = a.out + ((long long)(w.b * d.nc + w.c) * d.H + w.h) * d.P * d.N;
#pragma unroll
    for (int i = 0; i < Acc<TW>::RI; ++i) {
        const int m = m0 + Acc<TW>::row0() + i;
        if (m >= 2 * d.N) continue;
        float *to = out + (m < d.N ? m : per_dir + m - d.N);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int p = p0 + Acc<TW>::col0() + j;
            if (p < d.P) to[(long long)p * d.N] = acc.v[i][j];
        }
    }
}

// CB[b,c,g,l,s] = sum_n C[l,n] B[s,n].  Takes over _bmm_chunk_fwd_kernel (src/ssd/bi/ssd_bmm.py:34-91).
template <class T> __device__ __forceinline__ void cb_role(Panels &sm, const Dims &d, const View &Cm, const View &Bm, float *CB, int vec, int block) {
    const int nt = ceil_div(d.Q, TILE), tile = block % (nt * nt), bcg = block / (nt * nt);
    const int g = bcg % d.G, c = (bcg / d.G) % d.nc, b = bcg / (d.G * d.nc), lim = min(d.Q, d.L - c * d.Q);
    const int l0 = tile / nt * TILE, s0 = tile % nt * TILE, sh = shift_for(min(d.N, TILE));
    Mul mul;
    mul.zero();
    Frag fa, fb;
    panels<false>(d.N, [&](int k0) {
        fetch<T>(fa, sh, row_ptr<T>(Cm, b, c * d.Q + l0, g) + k0, Cm.sl, lim - l0, d.N - k0, vec & VEC_BC);
        fetch<T>(fb, sh, row_ptr<T>(Bm, b, c * d.Q + s0, g) + k0, Bm.sl, lim - s0, d.N - k0, vec & VEC_BC);
    }, [&](int) {
        put_rows(fa, sh, sm.a);
        put_transposed(fb, sh, sm.b);
    }, [&](int, int depth) { compute_nn<64, true>(mul, sm.a, sm.b, depth); });
    const Acc<64> acc = finish<64>(mul, sm.a);
    const int s = s0 + Acc<64>::col0();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int l = l0 + Acc<64>::row0() + i;
        if (l < d.Q)
            store4<float>(CB + ((long long)bcg * d.Q + l) * d.Q + s, d.Q - s, vec & VEC_Q,
                          make_float4(acc.v[i][0], acc.v[i][1], acc.v[i][2], acc.v[i][3]));
    }
}

// Output: y[l,p] = e^{cs_f[l]} C[l].S_f[p] + e^{cs_b[l]} C[l].S_b[p] + sum_s M[l,s] x[s,p] + D x[l,p],
// M[l,s] = CB[l,s] Delta[s] ([s<=l] e^{cs_f[l]-cs_f[s]} + [s>=l] e^{cs_b[l]-cs_b[s]}); out = y silu(z).
// Takes over _chunk_scan_fwd_kernel (src/ssd/bi/ssd_chunk_scan.py:42-189).
// grid (b nc H ceil(Q / 64) ceil(P / TW))
struct ScanArgs {
    View x, Cm, z;
    const float *D, *dt_out, *cs_f, *cs_b, *CB;
    const void *states_f, *states_b;
    MutView out, out_x;
};
template <class T, int TW> __global__ void __launch_bounds__(TB, TW == 64 ? 2 : 3) chunk_scan(Dims d, ScanArgs a, int vec) {
    extern __shared__ char smem[];
    Panels &sm = *reinterpret_cast<Panels *>(smem);
    pdl_begin();
    const int lt = ceil_div(d.Q, TILE), pt = ceil_div(d.P, TW), tile = blockIdx.x % (lt * pt), N = d.N;
    const Where w(d, blockIdx.x / (lt * pt));
    const int l0 = tile % lt * TILE, p0 = tile / lt * TW;
    if (l0 >= w.lim) return;
    const Vectors v = load_vectors(sm, d, w, a.dt_out, a.cs_f, a.cs_b);
    const float *sf = v.sf, *sb = v.sb, *sd = v.sd;
    const float *cb = a.CB + (((long long)w.b * d.nc + w.c) * d.G + w.g) * d.Q * d.Q;
    const long long st = (((long long)w.b * d.nc + w.c) * d.H + w.h) * d.P * N;
    const T *Sf = static_cast<const T *>(a.states_f) + st, *Sb = static_cast<const T *>(a.states_b) + st;
    Mul mul;
    mul.zero();
    Frag fa, fb;
    const int rows = w.lim - l0, shN = shift_for(2 * N);
    panels<false>(2 * N, [&](int k0) {
        pieces(shN, [&](int u, int r, int c) {
            const int k = k0 + c;
            fa.v[u] = fb.v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k >= 2 * N) return;
            if (r < rows) {
                const T *row = row_ptr<T>(a.Cm, w.b, w.l0 + l0 + r, w.g);
                const float4 v = load_dirs<T>(row, row, k, N, vec & VEC_BC);
                const float ef = k < N ? expf(sf[l0 + r]) : 0.f, eb = k + 3 >= N ? expf(sb[l0 + r]) : 0.f;
                fa.v[u] = make_float4(v.x * (k < N ? ef : eb), v.y * (k + 1 < N ? ef : eb), v.z * (k + 2 < N ? ef : eb), v.w * (k + 3 < N ? ef : eb));
            }
            if (r < TW && p0 + r < d.P)
                fb.v[u] = load_dirs<T>(Sf + (long long)(p0 + r) * N, Sb + (long long)(p0 + r) * N, k, N, vec & VEC_N);
        });
    }, [&](int) {
        put_rows(fa, shN, sm.a);
        put_transposed(fb, shN, sm.b);
    }, [&](int, int depth) { compute_nn<TW, true>(mul, sm.a, sm.b, depth); });
    const int shQ = shift_for(w.lim), shP = shift_for(min(d.P - p0, TW));
    panels(w.lim, [&](int k0) {
        fetch<float>(fa, shQ, cb + (long long)l0 * d.Q + k0, d.Q, rows, w.lim - k0, vec & VEC_Q);
        fetch<T>(fb, shP, row_ptr<T>(a.x, w.b, w.l0 + k0, w.h) + p0, a.x.sl, w.lim - k0, d.P - p0, vec & VEC_X);
    }, [&](int k0) {
        pieces(shQ, [&](int u, int r, int c) {
            if (r >= rows || k0 + c >= w.lim) return;            // zeros already
            const float4 e = decay4(v, l0 + r, k0 + c), t = *reinterpret_cast<const float4 *>(sd + k0 + c);
            fa.v[u] = make_float4(fa.v[u].x * (e.x * t.x), fa.v[u].y * (e.y * t.y), fa.v[u].z * (e.z * t.z), fa.v[u].w * (e.w * t.w));
        });
        put_rows(fa, shQ, sm.a);
        put_rows(fb, shP, sm.b);
    }, [&](int, int depth) { compute_nn<TW, false>(mul, sm.a, sm.b, depth); });
    const Acc<TW> acc = finish<TW>(mul, sm.a);
    const int p = p0 + Acc<TW>::col0(), n = d.P - p;
    if (n <= 0) return;
#pragma unroll
    for (int i = 0; i < Acc<TW>::RI; ++i) {
        const int l = l0 + Acc<TW>::row0() + i;
        if (l >= w.lim) continue;
        float y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = acc.v[i][j];
        if (d.has_D) {
            const float4 xv = load4<T>(row_ptr<T>(a.x, w.b, w.l0 + l, w.h) + p, n, vec & VEC_X);
            const float xs[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] += (d.D_hdim ? (j < n ? a.D[w.h * d.P + p + j] : 0.f) : a.D[w.h]) * xs[j];
        }
        if (d.has_z) {
            store4<T>(row_ptr<T>(a.out_x, w.b, w.l0 + l, w.h) + p, n, vec & VEC_X, make_float4(y[0], y[1], y[2], y[3]));
            const float4 zv = load4<T>(row_ptr<T>(a.z, w.b, w.l0 + l, w.h) + p, n, vec & VEC_X);
            const float zs[4] = {zv.x, zv.y, zv.z, zv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] *= zs[j] * sigmoidf_(zs[j]);
        }
        store4<T>(row_ptr<T>(a.out, w.b, w.l0 + l, w.h) + p, n, vec & VEC_X, make_float4(y[0], y[1], y[2], y[3]));
    }
}

// =========================================================================================================
// Backward
// =========================================================================================================
struct BwdArgs {
    View x, Bm, Cm, z, dout, out_x;
    const float *D, *dt_out, *cs_f, *cs_b, *CB, *E;
    const void *states_f, *states_b;
    MutView dx, dB, dC;
    void *dz;
    float *ddt_out, *dDpart, *dB_part, *dC_part, *nf, *nb, *pf, *pb, *dCB, *u;
    int hsplit, parts;                                           // blocks the heads of a group are dealt to in dcb_role, parts they are summed in
};

// dx, ddt_out, dz and per-block dD partials.
//   acc[l,p] = sum_n B[l,n] (E_f[p,n] e^{T-cs_f[l]} + E_b[p,n] e^{T-cs_b[l]})
//            + sum_s CB[s,l] ([s>=l] e^{cs_f[s]-cs_f[l]} + [s<=l] e^{cs_b[s]-cs_b[l]}) g[s,p]
//   dx = acc Delta[l] + D g;  ddt_out[l] = sum_p acc x[l,p];  dD[p] += sum_l g x
// Takes over _chunk_scan_chunk_state_bwd_dx_kernel (src/ssd/bi/ssd_combined.py:59-232) and, for dz,
// _chunk_scan_bwd_dz_kernel (src/ssd/bi/ssd_chunk_scan.py:357-440).  Blocks: b nc H ceil(Q / 64).
template <class T, int TW> __device__ __forceinline__ void dx_role(Panels &sm, const Dims &d, const BwdArgs &a, int vec, int block) {
    const int lt = ceil_div(d.Q, TILE), N = d.N, l0 = block % lt * TILE;
    const Where w(d, block / lt);
    const Vectors v = load_vectors(sm, d, w, a.dt_out, a.cs_f, a.cs_b);
    const float *sf = v.sf, *sb = v.sb, *sd = v.sd;
    const float Tf = sf[d.Q - 1], Tb = sb[0];
    const float *cb = a.CB + (((long long)w.b * d.nc + w.c) * d.G + w.g) * d.Q * d.Q;
    const long long st = (((long long)w.b * d.nc + w.c) * d.H + w.h) * d.P * N;
    const float *Ef = a.E + st, *Eb = Ef + (long long)d.b * d.nc * d.H * d.P * N;
    const int rows = w.lim - l0, shN = shift_for(2 * N), shL = shift_for(rows);
    float rowsum[Acc<TW>::RI];
#pragma unroll
    for (int i = 0; i < Acc<TW>::RI; ++i) rowsum[i] = 0.f;
    for (int p0 = 0; p0 < d.P; p0 += TW) {
        Mul mul;
        mul.zero();
        Frag fa, fb;
        panels<false>(2 * N, [&](int k0) {
            pieces(shN, [&](int u, int r, int c) {
                const int k = k0 + c;
                fa.v[u] = fb.v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k >= 2 * N) return;
                if (r < rows) {
                    const T *row = row_ptr<T>(a.Bm, w.b, w.l0 + l0 + r, w.g);
                    const float4 v = load_dirs<T>(row, row, k, N, vec & VEC_BC);
                    const float ef = k < N ? expf(Tf - sf[l0 + r]) : 0.f, eb = k + 3 >= N ? expf(Tb - sb[l0 + r]) : 0.f;
                    fa.v[u] = make_float4(v.x * (k < N ? ef : eb), v.y * (k + 1 < N ? ef : eb), v.z * (k + 2 < N ? ef : eb), v.w * (k + 3 < N ? ef : eb));
                }
                if (r < TW && p0 + r < d.P)
                    fb.v[u] = load_dirs<float>(Ef + (long long)(p0 + r) * N, Eb + (long long)(p0 + r) * N, k, N, vec & VEC_N);
            });
        }, [&](int) {
            put_rows(fa, shN, sm.a);
            put_transposed(fb, shN, sm.b);
        }, [&](int, int depth) { compute_nn<TW, true>(mul, sm.a, sm.b, depth); });
        const int shP = shift_for(min(d.P - p0, TW));
        panels(w.lim, [&](int k0) {
            fetch<float>(fa, shL, cb + (long long)k0 * d.Q + l0, d.Q, w.lim - k0, rows, vec & VEC_Q);
            fetch_gated<T>(fb, shP, d, a.dout, a.z, w.b, w.l0 + k0, w.h, p0, w.lim - k0, d.P - p0, vec & VEC_X);
        }, [&](int k0) {
            pieces(shL, [&](int u, int r, int c) {
                if (k0 + r >= w.lim || c >= rows) return;        // zeros already
                const float4 e = decay4(v, k0 + r, l0 + c);
                fa.v[u] = make_float4(fa.v[u].x * e.x, fa.v[u].y * e.y, fa.v[u].z * e.z, fa.v[u].w * e.w);
            });
            put_rows(fa, shL, sm.a);
            put_rows(fb, shP, sm.b);
        }, [&](int, int depth) { compute_tn<TW>(mul, sm.a, sm.b, depth); });
        const Acc<TW> acc = finish<TW>(mul, sm.a);
        const int p = p0 + Acc<TW>::col0(), n = d.P - p;
        float colsum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < Acc<TW>::RI; ++i) {
            const int l = l0 + Acc<TW>::row0() + i;
            if (l >= w.lim || n <= 0) continue;
            const float4 xq = load4<T>(row_ptr<T>(a.x, w.b, w.l0 + l, w.h) + p, n, vec & VEC_X);
            const float4 gq = load4<T>(row_ptr<T>(a.dout, w.b, w.l0 + l, w.h) + p, n, vec & VEC_X);
            const float xs[4] = {xq.x, xq.y, xq.z, xq.w};
            float gs[4] = {gq.x, gq.y, gq.z, gq.w}, o[4];
            if (d.has_z) {
                const float4 zq = load4<T>(row_ptr<T>(a.z, w.b, w.l0 + l, w.h) + p, n, vec & VEC_X);
                const float4 yq = load4<T>(row_ptr<T>(a.out_x, w.b, w.l0 + l, w.h) + p, n, vec & VEC_X);
                const float zs[4] = {zq.x, zq.y, zq.z, zq.w}, ys[4] = {yq.x, yq.y, yq.z, yq.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float sg = sigmoidf_(zs[j]);
                    o[j] = gs[j] * ys[j] * sg * (1.f + zs[j] * (1.f - sg));
                    gs[j] *= zs[j] * sg;
                }
                store4<T>(static_cast<T *>(a.dz) + (((long long)w.b * d.L + w.l0 + l) * d.H + w.h) * d.P + p, n, vec & VEC_P,
                          make_float4(o[0], o[1], o[2], o[3]));
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[j] = acc.v[i][j] * sd[l];
                if (d.has_D) o[j] += (d.D_hdim ? (j < n ? a.D[w.h * d.P + p + j] : 0.f) : a.D[w.h]) * gs[j];
                rowsum[i] += acc.v[i][j] * xs[j];
                colsum[j] += gs[j] * xs[j];
            }
            store4<T>(row_ptr<T>(a.dx, w.b, w.l0 + l, w.h) + p, n, vec & VEC_X, make_float4(o[0], o[1], o[2], o[3]));
        }
        if (d.has_D) {                                           // over the tile's rows: lanes with the same columns, then warps
            const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int o = 16; o >= Acc<TW>::NTX; o >>= 1) colsum[j] += __shfl_xor_sync(0xffffffffu, colsum[j], o);
                if (lane < Acc<TW>::NTX) sm.red[warp][0][lane * 4 + j] = colsum[j];
            }
            __syncthreads();
            if (threadIdx.x < TW && p0 + threadIdx.x < d.P) {
                float s = 0.f;
                for (int r = 0; r < 8; ++r) s += sm.red[r][0][threadIdx.x];
                a.dDpart[((((long long)w.b * d.nc + w.c) * d.H + w.h) * lt + block % lt) * d.P + p0 + threadIdx.x] = s;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < Acc<TW>::RI; ++i) {
        const float r = row_sum<TW>(rowsum[i]);
        const int l = l0 + Acc<TW>::row0() + i;
        if (Acc<TW>::col0() == 0 && l < d.Q) a.ddt_out[w.base + l] = r;
    }
}

// Per-head "states" parts of dB / dC and the decay-gradient terms that come with them (which: 0 = dB, 1 = dC).
//   dB: part[l,n] = Delta[l] sum_p x[l,p] (E_f[p,n] e^{T-cs_f[l]} + E_b[p,n] e^{T-cs_b[l]});
//       nf[l] = sum_n (forward part) B[l,n], nb[l] likewise              ("next" terms)
//   dC: part[l,n] = sum_p g[l,p] (S_f[p,n] e^{cs_f[l]} + S_b[p,n] e^{cs_b[l]});
//       pf[l] = sum_n (forward part) C[l,n], pb[l] likewise              ("prev" terms)
// Takes over _chunk_state_bwd_db_kernel (src/ssd/bi/ssd_chunk_state.py:379-495) and _chunk_scan_bwd_dc_kernel
// (src/ssd/bi/ssd_chunk_scan.py:538-636); the sum over the heads of a group happens in bmm_bwd below.
// part layout: [b, nc*Q, H, N] fp32.  Blocks: b nc H ceil(Q / 64) 2.
template <class T, class S, int TW>
__device__ __forceinline__ void dbc_half(Panels &sm, const Dims &d, const BwdArgs &a, int vec, const Where &w, int l0, bool which, const S *Sf,
                                         const S *Sb) {
    const float *sf = sm.v[0], *sb = sm.v[1], *sd = sm.v[2];
    const float Tf = sf[d.Q - 1], Tb = sb[0];
    const int N = d.N, rows = w.lim - l0, shP = shift_for(d.P);
    constexpr int RI = Acc<TW>::RI;
    float rs[2][RI];
#pragma unroll
    for (int i = 0; i < RI; ++i) rs[0][i] = rs[1][i] = 0.f;
    const View &other = which ? a.Cm : a.Bm;
    for (int n0 = 0; n0 < N; n0 += TW) {
        Acc<TW> acc[2];
        const int shN = shift_for(min(N - n0, TW));
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
            Mul mul;
            mul.zero();
            const S *from = (dir ? Sb : Sf) + n0;
            Frag fa, fb;
            panels<false>(d.P, [&](int k0) {
                if (which) fetch_gated<T>(fa, shP, d, a.dout, a.z, w.b, w.l0 + l0, w.h, k0, rows, d.P - k0, vec & VEC_X);
                else fetch<T>(fa, shP, row_ptr<T>(a.x, w.b, w.l0 + l0, w.h) + k0, a.x.sl, rows, d.P - k0, vec & VEC_X);
                fetch<S>(fb, shN, from + (long long)k0 * N, N, d.P - k0, N - n0, vec & VEC_N);
            }, [&](int) {
                put_rows(fa, shP, sm.a);
                put_rows(fb, shN, sm.b);
            }, [&](int, int depth) { compute_nn<TW, false>(mul, sm.a, sm.b, depth); });
            acc[dir] = finish<TW>(mul, sm.a);
        }
        const int nn = n0 + Acc<TW>::col0();
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const int l = l0 + Acc<TW>::row0() + i;
            if (l >= w.lim || nn >= N) continue;
            const float scf = which ? expf(sf[l]) : sd[l] * expf(Tf - sf[l]);
            const float scb = which ? expf(sb[l]) : sd[l] * expf(Tb - sb[l]);
            const float4 oq = load4<T>(row_ptr<T>(other, w.b, w.l0 + l, w.g) + nn, N - nn, vec & VEC_BC);
            const float o[4] = {oq.x, oq.y, oq.z, oq.w};
            float t[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float vf = acc[0].v[i][j] * scf, vb = acc[1].v[i][j] * scb;
                rs[0][i] += vf * o[j];
                rs[1][i] += vb * o[j];
                t[j] = vf + vb;
            }
            float *part = which ? a.dC_part : a.dB_part;
            store4<float>(part + (((long long)w.b * d.nc * d.Q + w.l0 + l) * d.H + w.h) * N + nn, N - nn, vec & VEC_N, make_float4(t[0], t[1], t[2], t[3]));
        }
    }
    float *of = which ? a.pf : a.nf, *ob = which ? a.pb : a.nb;
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        const float rf = row_sum<TW>(rs[0][i]), rb = row_sum<TW>(rs[1][i]);
        const int l = l0 + Acc<TW>::row0() + i;
        if (Acc<TW>::col0() == 0 && l < d.Q) {
            of[w.base + l] = rf;
            ob[w.base + l] = rb;
        }
    }
}
template <class T, int TW> __device__ __forceinline__ void dbc_role(Panels &sm, const Dims &d, const BwdArgs &a, int vec, int block) {
    const int lt = ceil_div(d.Q, TILE), which = block & 1, i = block >> 1;
    const Where w(d, i / lt);
    load_vectors(sm, d, w, a.dt_out, a.cs_f, a.cs_b);
    const long long st = (((long long)w.b * d.nc + w.c) * d.H + w.h) * d.P * d.N;
    if (which) dbc_half<T, T, TW>(sm, d, a, vec, w, i % lt * TILE, true, static_cast<const T *>(a.states_f) + st, static_cast<const T *>(a.states_b) + st);
    else dbc_half<T, float, TW>(sm, d, a, vec, w, i % lt * TILE, false, a.E + st, a.E + (long long)d.b * d.nc * d.H * d.P * d.N + st);
}

// dCB and the intra-chunk decay gradients from one g.x^T product per head and 64 x 64 tile:
//   G2[l,s] = g[l].x[s];   dCB[b,c,g,l,s] = sum_{h in g} G2 Delta_h[s] ([s<=l] e^{cs_f[l]-cs_f[s]} + [s>=l] e^{cs_b[l]-cs_b[s]})
//   W_f[l,s] = G2 CB Delta[s] e^{cs_f[l]-cs_f[s]} (s<l),  W_b likewise (s>l);   the decay gradients
//   da_f[j] = sum_{l>=j} sum_{s<j} W_f[l,s],  da_b[j] = sum_{l<=j} sum_{s>j} W_b[l,s]  are exclusive prefix / suffix sums of
//   u = (column sums - row sums) of W, which cumsum_bwd takes: u[t] for t < ceil(Q/64) holds the column sums over row
//   tile t, the rest minus the row sums over column tile t - ceil(Q/64), forward and reverse in turn.
// Takes over _chunk_scan_bwd_dcb_kernel (src/ssd/bi/ssd_chunk_scan.py:776-859) and the "stable" decay kernels
// (:1361-1446, :1078-1157).  dCB: [b,c,g][hsplit][Q][Q], summed by bmm_bwd; a block with several
// parts adds them up in the same order.  Blocks: b nc G hsplit ceil(Q/64)^2.
template <class T> __device__ __forceinline__ void dcb_role(Panels &sm, const Dims &d, const BwdArgs &a, int vec, int block) {
    const int nt = ceil_div(d.Q, TILE), tile = block % (nt * nt), part = block / (nt * nt) % a.hsplit, bcg = block / (nt * nt) / a.hsplit;
    const int g = bcg % d.G, c = (bcg / d.G) % d.nc, b = bcg / (d.G * d.nc), lim = min(d.Q, d.L - c * d.Q);
    const int lt = tile / nt, st = tile % nt, l0 = lt * TILE, s0 = st * TILE, heads = d.R / a.hsplit, shP = shift_for(d.P);
    const int per = d.R / a.parts;                               // heads a part
    const int lr = l0 + Acc<64>::row0(), sc = s0 + Acc<64>::col0(), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long stride = (long long)d.b * d.H * d.nc * d.Q;
    float tot[4][4], before[4][4];                               // the part's sums, and those of the block's parts before it
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) tot[i][j] = before[i][j] = 0.f;
    for (int r = 0; r < heads; ++r) {
        if (r > 0 && r % per == 0)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    before[i][j] += tot[i][j];
                    tot[i][j] = 0.f;
                }
        Where w(d, (b * d.nc + c) * d.H + g * d.R + part * heads + r);
        __syncthreads();                                         // the vectors' and sums' last readers are done
        const Vectors vec4 = load_vectors(sm, d, w, a.dt_out, a.cs_f, a.cs_b);
        const float *sf = vec4.sf, *sb = vec4.sb, *sd = vec4.sd;
        Mul mul;
        mul.zero();
        Frag fa, fb;
        panels<false>(d.P, [&](int k0) {
            fetch_gated<T>(fa, shP, d, a.dout, a.z, b, w.l0 + l0, w.h, k0, lim - l0, d.P - k0, vec & VEC_X);
            fetch<T>(fb, shP, row_ptr<T>(a.x, b, w.l0 + s0, w.h) + k0, a.x.sl, lim - s0, d.P - k0, vec & VEC_X);
        }, [&](int) {
            put_rows(fa, shP, sm.a);
            put_transposed(fb, shP, sm.b);
        }, [&](int, int depth) { compute_nn<64, true>(mul, sm.a, sm.b, depth); });
        const Acc<64> acc = finish<64>(mul, sm.a);
        float rowf[4], rowb[4], colf[4], colb[4], et[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            rowf[j] = rowb[j] = colf[j] = colb[j] = 0.f;
            et[j] = sc + j < lim ? sd[sc + j] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int l = lr + i;
            if (l >= lim) continue;
            const float4 cq = load4<float>(a.CB + ((long long)bcg * d.Q + l) * d.Q + sc, d.Q - sc, vec & VEC_Q);
            const float cbv[4] = {cq.x, cq.y, cq.z, cq.w};
            if (sc + 3 < l || sc > l) {                          // the four columns lie on one side of the diagonal
                const float4 e = decay4(vec4, l, sc);
                const float es[4] = {e.x, e.y, e.z, e.w};
                float row = 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float v = acc.v[i][j] * (et[j] * es[j]), u = v * cbv[j];
                    tot[i][j] += v;
                    row += u;
                    if (sc > l) colb[j] += u;
                    else colf[j] += u;
                }
                if (sc > l) rowb[i] += row;
                else rowf[i] += row;
                continue;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int s = sc + j;
                const float t = acc.v[i][j] * et[j];
                if (s <= l) {
                    const float v = t * expf(sf[l] - sf[s]);
                    tot[i][j] += v;
                    if (s < l) {
                        rowf[i] += v * cbv[j];
                        colf[j] += v * cbv[j];
                    }
                }
                if (s >= l) {
                    const float v = t * expf(sb[l] - sb[s]);
                    tot[i][j] += v;
                    if (s > l) {
                        rowb[i] += v * cbv[j];
                        colb[j] += v * cbv[j];
                    }
                }
            }
        }
        float *ur = a.u + 2 * (nt + st) * stride + w.base, *uc = a.u + 2 * lt * stride + w.base;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float f = row_sum<64>(rowf[i]), q = row_sum<64>(rowb[i]);
            if (Acc<64>::col0() == 0 && lr + i < d.Q) {
                ur[lr + i] = -f;
                ur[stride + lr + i] = -q;
            }
            colf[i] += __shfl_xor_sync(0xffffffffu, colf[i], 16);
            colb[i] += __shfl_xor_sync(0xffffffffu, colb[i], 16);
            if (lane < 16) {
                sm.red[warp][0][lane * 4 + i] = colf[i];
                sm.red[warp][1][lane * 4 + i] = colb[i];
            }
        }
        __syncthreads();
        if (threadIdx.x < 2 * TILE) {
            const int dir = threadIdx.x / TILE, s = threadIdx.x % TILE;
            float v = 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) v += sm.red[k][dir][s];
            if (s0 + s < d.Q) uc[dir * stride + s0 + s] = v;
        }
    }
    float *out = a.dCB + ((long long)bcg * a.hsplit + part) * d.Q * d.Q;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (lr + i < d.Q)
            store4<float>(out + (long long)(lr + i) * d.Q + sc, d.Q - sc, vec & VEC_Q,
                          make_float4(before[i][0] + tot[i][0], before[i][1] + tot[i][1], before[i][2] + tot[i][2], before[i][3] + tot[i][3]));
}

// dB[s,n] = sum_l dCB[l,s] C[l,n] + sum_{h in g} dB_part[s,h,n];  dC[l,n] = sum_s dCB[l,s] B[s,n] + sum_h dC_part.
// Takes over the two _bmm_chunk_bwd_kernel calls (src/ssd/bi/ssd_bmm.py:108-160; ssd_combined.py:441-442).
// Blocks: b nc G 2 ceil(Q/64) ceil(N/TW).
template <class T, int TW> __device__ __forceinline__ void bmm_bwd_role(Panels &sm, const Dims &d, const BwdArgs &a, int vec, int block) {
    const int nt = ceil_div(d.Q, TILE), ntn = ceil_div(d.N, TW), which = block & 1, i0 = block >> 1;
    const int r0 = i0 % nt * TILE, n0 = i0 / nt % ntn * TW, bcg = i0 / (nt * ntn);
    const int g = bcg % d.G, c = (bcg / d.G) % d.nc, b = bcg / (d.G * d.nc), lim = min(d.Q, d.L - c * d.Q), l00 = c * d.Q;
    const float *dcb = a.dCB + (long long)bcg * a.hsplit * d.Q * d.Q;
    const View &Y = which ? a.Bm : a.Cm;
    const int shR = shift_for(which ? lim : lim - r0), shN = shift_for(min(d.N - n0, TW));
    Mul mul;
    mul.zero();
    Frag fa, fb;
    panels(lim, [&](int k0) {                                    // dC: rows r0 of dCB, depth along them; dB: the other way
        const int fr = which ? r0 : k0, fc = which ? k0 : r0;
        fetch<float>(fa, shR, dcb + (long long)fr * d.Q + fc, d.Q, lim - fr, lim - fc, vec & VEC_Q);
        for (int k = 1; k < a.hsplit; ++k) {
            Frag f2;
            fetch<float>(f2, shR, dcb + ((long long)k * d.Q + fr) * d.Q + fc, d.Q, lim - fr, lim - fc, vec & VEC_Q);
            pieces(shR, [&](int u, int, int) {
                fa.v[u].x += f2.v[u].x; fa.v[u].y += f2.v[u].y; fa.v[u].z += f2.v[u].z; fa.v[u].w += f2.v[u].w;
            });
        }
        fetch<T>(fb, shN, row_ptr<T>(Y, b, l00 + k0, g) + n0, Y.sl, lim - k0, d.N - n0, vec & VEC_BC);
    }, [&](int) {
        put_rows(fa, shR, sm.a);
        put_rows(fb, shN, sm.b);
    }, [&](int, int depth) {
        if (which) compute_nn<TW, false>(mul, sm.a, sm.b, depth);
        else compute_tn<TW>(mul, sm.a, sm.b, depth);
    });
    const Acc<TW> acc = finish<TW>(mul, sm.a);
    const float *part = which ? a.dC_part : a.dB_part;
    const MutView &out = which ? a.dC : a.dB;
    const int nn = n0 + Acc<TW>::col0();
    if (nn >= d.N) return;
#pragma unroll
    for (int i = 0; i < Acc<TW>::RI; ++i) {
        const int l = r0 + Acc<TW>::row0() + i;
        if (l >= lim) continue;
        float4 v = make_float4(acc.v[i][0], acc.v[i][1], acc.v[i][2], acc.v[i][3]);
        const float *pp = part + (((long long)b * d.nc * d.Q + l00 + l) * d.H + g * d.R) * d.N + nn;
        for (int r = 0; r < d.R; ++r) {
            const float4 t = load4<float>(pp + (long long)r * d.N, d.N - nn, vec & VEC_N);
            v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
        }
        store4<T>(row_ptr<T>(out, b, l00 + l, g) + nn, d.N - nn, vec & VEC_BC, v);
    }
}

// ---- the launches ---------------------------------------------------------------------------------------------------
// Blocks of the first role come first; `first` and `second` are the roles' block counts.  The first kernel of a pass
// clears the workspace header (the status word, which these kernels never raise).
template <class T, bool GRAD, int TW>
__global__ void __launch_bounds__(TB, 3) states_and_cb(Dims d, StateArgs a, View Cm, View Bm, float *CB, int vec, int first, int *header) {
    extern __shared__ char smem[];
    Panels &sm = *reinterpret_cast<Panels *>(smem);
    pdl_begin();
    if (header && blockIdx.x == 0 && threadIdx.x < 64) header[threadIdx.x] = 0;
    if ((int)blockIdx.x < first) states_role<T, GRAD, TW>(sm, d, a, vec, blockIdx.x);
    else cb_role<T>(sm, d, Cm, Bm, CB, vec, blockIdx.x - first);
}
template <class T, int TWP, int TWN> __global__ void __launch_bounds__(TB, 2) backward2(Dims d, BwdArgs a, int vec, int first, int second) {
    extern __shared__ char smem[];
    Panels &sm = *reinterpret_cast<Panels *>(smem);
    pdl_begin();
    const int block = blockIdx.x;
    if (block < first) dcb_role<T>(sm, d, a, vec, block);
    else if (block < first + second) dx_role<T, TWP>(sm, d, a, vec, block - first);
    else dbc_role<T, TWN>(sm, d, a, vec, block - first - second);
}
template <class T, int TWN> __global__ void __launch_bounds__(TB, TWN == 64 ? 2 : 3) backward3(Dims d, BwdArgs a, CumsumBwd cs, int vec, int first) {
    extern __shared__ char smem[];
    Panels &sm = *reinterpret_cast<Panels *>(smem);
    pdl_begin();
    if ((int)blockIdx.x < first) bmm_bwd_role<T, TWN>(sm, d, a, vec, blockIdx.x);
    else cumsum_bwd_role(d, cs, blockIdx.x - first, reinterpret_cast<float(*)[8]>(sm.a), reinterpret_cast<float(*)[8]>(sm.b));
}

}  // namespace simt
}  // namespace bissd
