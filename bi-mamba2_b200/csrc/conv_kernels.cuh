// Depthwise, non-causal ("same" padding) conv1d over the sequence followed by SiLU, channels-last, forward and
// backward - the front end of BiMamba2 (src/ssd/modules.py:164-167: conv1d on the transposed tensor, transposed
// back, then the activation).  Working channels-last on (batch, seqlen, channels) removes both transposes and hands
// x / B / C to the scan as strided views of one contiguous tensor, which its TMA maps read in place.
//
//   pre[b,l,c] = bias[c] + sum_k w[c,k] x[b, l + k - K/2, c]      (zero outside 0 <= l < L),   out = silu(pre)
//   dpre = dout silu'(pre);  dx[b,l,c] = sum_k w[c,k] dpre[b, l - k + K/2, c];
//   dw[c,k] = sum_{b,l} dpre[b,l,c] x[b, l + k - K/2, c];  dbias[c] = sum_{b,l} dpre[b,l,c]
//
// A thread owns NP pairs of adjacent channels and walks a run of rows, six rows a round, the next round's loads in flight
// meanwhile, the K - 1 rows it shares with the next round kept in registers (two rounds unrolled, so that for K = 7 they
// never move); multiply-adds are fp32x2 over the pair.
// The backward is one pass: pre is recomputed, dpre stays in registers (fp32) and feeds dx and the weight gradients in
// the same round, so x and dout are read once and dx written once; a run recomputes the K - 1 rows of dpre it needs from
// its neighbours.  Bound by instruction issue (about 75 per pair and row, 16 warps an SM).
// Measured at 16 x 4096 rows of 2176 channels, bf16, K = 7: forward 223 -> 120 us (4.8 TB/s; a pair more per thread or four
// rows a round are slower), backward 632 -> 256 us (three passes over memory before: dpre, dw, dx).
// Weight and bias gradients: registers over the run, one partial row per (batch, run) in the workspace - slot-major, so
// that a warp stores whole lines - summed in a fixed order by conv_bwd_reduce; no float atomics.
// Width K = 1, 3, 5, 7.
#pragma once
#include "vec.cuh"

namespace bissd {
namespace conv {

using namespace vec;

constexpr int kThreads = 128;
constexpr int kStep = 6;                         // rows per round: for K = 7 a round's new rows are the next one's old ones
constexpr int kFwdPairs = 2, kBwdPairs = 1;      // channel pairs per thread

struct ConvDims {
    int batch, seqlen, channels;
    int run, runs;                               // rows per thread, runs per sequence
    long long xsb, xsl;                          // x and dx: batch and row strides in elements; channel stride 1
    long long osb, osl;                          // out and dout
    int has_bias;
};

// Warps, not blocks, are dealt over (channels of a lane's NP pairs, run, batch): channel counts that are no multiple of a
// block's waste lanes of one warp only.
__host__ __device__ inline int warps_across(int channels, int np) { return (channels + 64 * np - 1) / (64 * np); }
template <int NP> __device__ __forceinline__ bool place(const ConvDims &d, int &c0, int &run, int &b) {
    const int across = warps_across(d.channels, NP), i = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5), r = i / across;
    c0 = ((i - r * across) * 32 + (threadIdx.x & 31)) * 2 * NP;
    b = r / d.runs;
    run = r - b * d.runs;
    return c0 < d.channels && b < d.batch;
}
template <class W, int K, int NP> __device__ __forceinline__ void load_weights(const void *weight, int c0, f2 (&w)[NP][K]) {
#pragma unroll
    for (int i = 0; i < NP; ++i)
#pragma unroll
        for (int k = 0; k < K; ++k)
            w[i][k] = pack(ld<W>(weight, (long long)(c0 + 2 * i) * K + k), ld<W>(weight, (long long)(c0 + 2 * i + 1) * K + k));
}

// The NR rows l, l + 1, ... at p (row stride in elements), zero outside 0 <= l < seqlen.
template <class T, int NP, int NR> __device__ __forceinline__ void fetch(Row<T, NP> (&r)[NR], const T *p, long long stride, int l, int seqlen) {
    if (l >= 0 && l + NR <= seqlen) {                            // nearly always; the same for the whole warp
#pragma unroll
        for (int u = 0; u < NR; ++u) r[u] = load_row<T, NP>(p + u * stride);
    } else {
#pragma unroll
        for (int u = 0; u < NR; ++u) r[u] = (l + u >= 0 && l + u < seqlen) ? load_row<T, NP>(p + u * stride) : zero_row<T, NP>();
    }
}

template <class T, class W, int K>
__global__ void __launch_bounds__(kThreads, 4) dwconv_silu_fwd(ConvDims d, const void *x, const void *weight, const void *bias, void *out) {
    constexpr int NP = kFwdPairs, PAD = K / 2, S = kStep;
    pdl_begin();
    int c0, b, run;
    if (!place<NP>(d, c0, run, b)) return;
    const int l0 = run * d.run, l1 = min(d.seqlen, l0 + d.run);
    f2 w[NP][K], bv[NP];
    load_weights<W, K, NP>(weight, c0, w);
#pragma unroll
    for (int i = 0; i < NP; ++i) bv[i] = d.has_bias ? load_pair<W>(bias, c0 + 2 * i) : pack(0.f, 0.f);
    const T *xp = static_cast<const T *>(x) + b * d.xsb + (long long)(l0 + PAD) * d.xsl + c0;
    T *op = static_cast<T *>(out) + b * d.osb + (long long)l0 * d.osl + c0;
    f2 xs[NP][K - 1 + S];                                        // rows lb - PAD ... lb + PAD + S - 1
#pragma unroll
    for (int o = 0; o < K - 1; ++o) {
        const int l = l0 - PAD + o;
        const Row<T, NP> r = (l >= 0 && l < d.seqlen) ? load_row<T, NP>(xp + (o - 2 * PAD) * d.xsl) : zero_row<T, NP>();
#pragma unroll
        for (int i = 0; i < NP; ++i) xs[i][o] = widen<T>(r.v[i]);
    }
    Row<T, NP> xn[S];
    fetch<T, NP, S>(xn, xp, d.xsl, l0 + PAD, d.seqlen);
#pragma unroll 2
    for (int lb = l0; lb < l1; lb += S) {
#pragma unroll
        for (int u = 0; u < S; ++u)
#pragma unroll
            for (int i = 0; i < NP; ++i) xs[i][K - 1 + u] = widen<T>(xn[u].v[i]);
        xp += S * d.xsl;
        if (lb + S < l1) fetch<T, NP, S>(xn, xp, d.xsl, lb + S + PAD, d.seqlen);
#pragma unroll
        for (int u = 0; u < S; ++u) {
            Row<T, NP> o;
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                f2 acc = bv[i];
#pragma unroll
                for (int k = 0; k < K; ++k) acc = fma2(w[i][k], xs[i][u + k], acc);
                o.v[i] = narrow<T>(mul2(acc, sigmoid2(acc)));
            }
            if (lb + u < l1) store_row<T, NP>(op, o);
            op += d.osl;
        }
#pragma unroll
        for (int i = 0; i < NP; ++i)
#pragma unroll
            for (int o = 0; o < K - 1; ++o) xs[i][o] = xs[i][o + S];
    }
}

// part: [batch * runs][K + 1][channels] fp32, slot K holding the bias gradient.
template <class T, class W, int K>
__global__ void __launch_bounds__(kThreads, 4) dwconv_silu_bwd(ConvDims d, const void *x, const void *weight, const void *bias,
                                                            const void *dout, void *dx, float *part) {
    constexpr int PAD = K / 2, S = kStep;
    pdl_begin();
    int c0, b, run;
    if (!place<kBwdPairs>(d, c0, run, b)) return;
    const int l0 = run * d.run, l1 = min(d.seqlen, l0 + d.run);
    f2 w[1][K], dw[K], db = pack(0.f, 0.f);
    load_weights<W, K, 1>(weight, c0, w);
#pragma unroll
    for (int k = 0; k < K; ++k) dw[k] = pack(0.f, 0.f);
    const f2 bv = d.has_bias ? load_pair<W>(bias, c0) : pack(0.f, 0.f);
    // A round makes dpre for rows m ... m + S - 1 (from x rows m - PAD ...) and dx for the rows PAD behind; the rows
    // of dpre outside the run count for dx only.  The first round is at l0 - PAD.
    f2 xs[K - 1 + S], gs[K - 1 + S];                             // x rows m - PAD + j;  dpre rows m - (K - 1) + j
    const T *xp = static_cast<const T *>(x) + b * d.xsb + (long long)l0 * d.xsl + c0;             // row m + PAD
    const T *gp = static_cast<const T *>(dout) + b * d.osb + (long long)(l0 - PAD) * d.osl + c0;  // row m
    T *op = static_cast<T *>(dx) + b * d.xsb + (long long)(l0 - 2 * PAD) * d.xsl + c0;            // row m - PAD
#pragma unroll
    for (int o = 0; o < K - 1; ++o) {
        xs[o] = l0 - 2 * PAD + o >= 0 ? widen<T>(load_row<T, 1>(xp + (o - 2 * PAD) * d.xsl).v[0]) : pack(0.f, 0.f);
        gs[o] = pack(0.f, 0.f);
    }
    Row<T, 1> xn[S], gn[S];
    fetch<T, 1, S>(xn, xp, d.xsl, l0, d.seqlen);
    fetch<T, 1, S>(gn, gp, d.osl, l0 - PAD, d.seqlen);
#pragma unroll 2
    for (int m = l0 - PAD; m < l1 + PAD; m += S) {
        f2 gv[S];
#pragma unroll
        for (int u = 0; u < S; ++u) {
            xs[K - 1 + u] = widen<T>(xn[u].v[0]);
            gv[u] = widen<T>(gn[u].v[0]);
        }
        xp += S * d.xsl;
        gp += S * d.osl;
        if (m + S < l1 + PAD) {                                  // the next round's rows, on their way during this one
            fetch<T, 1, S>(xn, xp, d.xsl, m + S + PAD, d.seqlen);
            fetch<T, 1, S>(gn, gp, d.osl, m + S, d.seqlen);
        }
        const bool inner = m >= l0 && m + S <= l1;               // all of the round's dpre rows belong to the run
#pragma unroll
        for (int u = 0; u < S; ++u) {
            f2 acc = bv;
#pragma unroll
            for (int k = 0; k < K; ++k) acc = fma2(w[0][k], xs[u + k], acc);
            const f2 g = mul2(gv[u], silu_slope2(acc, sigmoid2(acc)));
            gs[K - 1 + u] = g;                                   // zero outside the sequence: dout is
            const f2 own = inner || (m + u >= l0 && m + u < l1) ? g : pack(0.f, 0.f);
            db = add2(db, own);
#pragma unroll
            for (int k = 0; k < K; ++k) dw[k] = fma2(own, xs[u + k], dw[k]);
            f2 o = pack(0.f, 0.f);                               // row m + u - PAD: dpre rows m + u - (K - 1) ... m + u
#pragma unroll
            for (int k = 0; k < K; ++k) o = fma2(w[0][K - 1 - k], gs[u + k], o);
            if (m + u - PAD >= l0 && m + u - PAD < l1) {
                Row<T, 1> r;
                r.v[0] = narrow<T>(o);
                store_row<T, 1>(op, r);
            }
            op += d.xsl;
        }
#pragma unroll
        for (int o = 0; o < K - 1; ++o) {
            xs[o] = xs[o + S];
            gs[o] = gs[o + S];
        }
    }
    float *to = part + (long long)(b * d.runs + run) * (K + 1) * d.channels + c0;
#pragma unroll
    for (int k = 0; k <= K; ++k) {
        float p, q;
        unpack(k < K ? dw[k < K ? k : 0] : db, p, q);
        *reinterpret_cast<float2 *>(to + (long long)k * d.channels) = make_float2(p, q);
    }
}

// dweight[c][k] and dbias[c] = sums of the partial rows.  grid ceil((width + 1) channels / 32).
template <class W>
__global__ void __launch_bounds__(256) conv_bwd_reduce(const float *part, int nparts, int channels, int width, void *dweight,
                                                       void *dbias) {
    pdl_begin();
    column_sums(part, nparts, (width + 1) * channels, [=](int i, float v) {
        const int k = i / channels, c = i % channels;
        if (k < width) st<W>(dweight, (long long)c * width + k, v);
        else if (dbias) st<W>(dbias, c, v);
    });
}

}  // namespace conv
}  // namespace bissd
