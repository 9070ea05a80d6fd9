// Discretisation + both cumulative sums of the tensor-core family, and their backward (formulas at simt::chunk_cumsum and
// simt::cumsum_bwd_role).  Four warps share one (batch, chunk, head), a lane has E consecutive positions: every operand is
// requested at once in wide pieces, the scans are register sums, five shuffles and one barrier.  The block's two heads are
// neighbours, whose dt and ddt values share 32-byte sectors.  Device time by the profiler, us, forward and backward: b16
// L4096 H32 16.5 + 44; b2 L8192 H32 6.5 + 15.2; b8 L2048 H24 5.5 + 12.5 (event brackets around each launch add 3 - 5).  With a
// block of one position a thread: 23 + 88, 7 + 24, 6 + 18 by CUDA events; a warp per chunk 15 + 60 and 5.5 + 16
// for the first and the last.
#pragma once
#include "simt_kernels.cuh"

namespace bissd {
namespace tc {

constexpr int kCumsumWarps = 8, kCumsumShare = 4;              // per block, per chunk
inline int cumsum_blocks(const Dims &d) { return d.b * d.nc * ceil_div(d.H, kCumsumWarps / kCumsumShare); }

template <int E> __device__ __forceinline__ void load_e(const float *p, bool wide, float (&v)[E]) {
    if (E == 2 && wide) {
        const float2 t = *reinterpret_cast<const float2 *>(p);
        v[0] = t.x; v[E - 1] = t.y;
    } else {
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = p[j];
    }
}
template <int E> __device__ __forceinline__ void store_e(float *p, bool wide, const float (&v)[E]) {
    if (E == 2 && wide) *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[E - 1]);
    else
#pragma unroll
        for (int j = 0; j < E; ++j) p[j] = v[j];
}
// dt and ddt, strided and of a type known at run time only: the choice of type stands outside the loop, so that the E loads
// are in flight together (decided element by element, each waited for the one before).  Zero beyond n.
template <int E, class S> __device__ __forceinline__ void load_strided(const void *p, long long at, long long step, int n, float (&v)[E]) {
    const S *q = static_cast<const S *>(p) + at;
    S raw[E];
#pragma unroll
    for (int j = 0; j < E; ++j) raw[j] = j < n ? q[j * step] : from_f<S>(0.f);
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = to_f<S>(raw[j]);
}
template <int E> __device__ __forceinline__ void load_strided(const void *p, int dtype, long long at, long long step, int n, float (&v)[E]) {
    if (dtype == BISSD_F32) load_strided<E, float>(p, at, step, n, v);
    else if (dtype == BISSD_BF16) load_strided<E, __nv_bfloat16>(p, at, step, n, v);
    else load_strided<E, __half>(p, at, step, n, v);
}
template <int E, class S> __device__ __forceinline__ void store_strided(void *p, long long at, long long step, int n, const float (&v)[E]) {
#pragma unroll
    for (int j = 0; j < E; ++j)
        if (j < n) static_cast<S *>(p)[at + j * step] = from_f<S>(v[j]);
}
template <int E> __device__ __forceinline__ void store_strided(void *p, int dtype, long long at, long long step, int n, const float (&v)[E]) {
    if (dtype == BISSD_F32) store_strided<E, float>(p, at, step, n, v);
    else if (dtype == BISSD_BF16) store_strided<E, __nv_bfloat16>(p, at, step, n, v);
    else store_strided<E, __half>(p, at, step, n, v);
}
// v <- inclusive sums over the warp's positions, ascending or descending
template <int E> __device__ __forceinline__ void scan_up(float (&v)[E], int lane) {
#pragma unroll
    for (int j = 1; j < E; ++j) v[j] += v[j - 1];
    float t = v[E - 1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float n = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += n;
    }
    const float before = __shfl_up_sync(0xffffffffu, t, 1);
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] += lane > 0 ? before : 0.f;
}
template <int E> __device__ __forceinline__ void scan_down(float (&v)[E], int lane) {
#pragma unroll
    for (int j = E - 2; j >= 0; --j) v[j] += v[j + 1];
    float t = v[0];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float n = __shfl_down_sync(0xffffffffu, t, o);
        if (lane + o < 32) t += n;
    }
    const float after = __shfl_down_sync(0xffffffffu, t, 1);
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] += lane < 31 ? after : 0.f;
}

// Add the totals of the warps before (ascending scans) or after (descending ones); K scans at once, the first UP
// of them ascending.  last / first positions hold a warp's totals.  One barrier; every warp of the block takes part.
template <int E, int K, int UP> __device__ __forceinline__ void across_warps(float (*const (&v)[K])[E], int lane) {
    constexpr int W = kCumsumShare;
    __shared__ float tot[K][kCumsumWarps];
    const int warp = threadIdx.x >> 5, part = warp % W, first = warp - part;
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (lane == (k < UP ? 31 : 0)) tot[k][warp] = (*v[k])[k < UP ? E - 1 : 0];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        float s = 0.f;
        for (int w = 0; w < W; ++w) s += (k < UP ? w < part : w > part) ? tot[k][first + w] : 0.f;
#pragma unroll
        for (int j = 0; j < E; ++j) (*v[k])[j] += s;
    }
}

// The forward sums as a role of a launch (block of cumsum_blocks).  E = 1 for chunks up to 128, else 2; chunk_size a multiple
// of E.  wide: dt_out, cs_f and cs_b are 16-byte aligned
struct CumsumFwd {
    const void *dt;
    int dt_dtype;
    long long dsb, dsl, dsh;
    const float *A, *dt_bias;
    float *dt_out, *cs_f, *cs_b;
    int wide;
};
template <int E> __device__ __forceinline__ void cumsum_fwd_role(const Dims &d, const CumsumFwd &a, int block) {
    constexpr int W = kCumsumShare, kHeads = kCumsumWarps / W;                    // per block
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l0 = (warp % W * 32 + lane) * E, nhb = (d.H + kHeads - 1) / kHeads;
    const int hw = block % nhb * kHeads + warp / W, c = block / nhb % d.nc, b = block / nhb / d.nc;
    const bool on = l0 < d.Q && hw < d.H;                       // warps beyond the heads redo the last one and store nothing
    const int h = min(hw, d.H - 1);
    const long long base = ((long long)(b * d.H + h) * d.nc + c) * d.Q + l0;
    const int lim = min(d.Q, d.L - c * d.Q);
    const float Ah = a.A[h], bias = d.has_bias ? a.dt_bias[h] : 0.f;
    float v[E], f[E], r[E];
    load_strided(a.dt, a.dt_dtype, b * a.dsb + (long long)(c * d.Q + l0) * a.dsl + h * a.dsh, a.dsl, lim - l0, v);
#pragma unroll
    for (int j = 0; j < E; ++j) {
        float t = v[j] + bias;
        if (d.softplus) t = softplus_ref(t);
        v[j] = l0 + j < lim ? fminf(fmaxf(t, d.dt_min), d.dt_max) : 0.f;
        f[j] = r[j] = v[j] * Ah;
    }
    scan_up(f, lane);
    scan_down(r, lane);
    across_warps<E, 2, 1>({&f, &r}, lane);
    if (on) {
        store_e(a.dt_out + base, a.wide, v);
        store_e(a.cs_f + base, a.wide, f);
        store_e(a.cs_b + base, a.wide, r);
    }
}
// grid cumsum_blocks; the first kernel of a pass: it also clears the status word
template <int E>
__global__ void __launch_bounds__(32 * kCumsumWarps) cumsum_fwd(Dims d, CumsumFwd a, int *status) {
    pdl_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
    cumsum_fwd_role<E>(d, a, blockIdx.x);
}

// a.u4 (with a.u4_tiles) or a.da_f / a.da_b as in simt::cumsum_bwd_role.  wide: dt_out is 16-byte aligned
template <int E>
__global__ void __launch_bounds__(32 * kCumsumWarps)
cumsum_bwd(Dims d, simt::CumsumBwd a, int wide) {
    pdl_begin();
    constexpr int W = kCumsumShare, kHeads = kCumsumWarps / W;                    // per block
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l0 = (warp % W * 32 + lane) * E, nhb = (d.H + kHeads - 1) / kHeads;
    const int hw = blockIdx.x % nhb * kHeads + warp / W, c = blockIdx.x / nhb % d.nc, b = blockIdx.x / nhb / d.nc;
    const bool on = l0 < d.Q && hw < d.H;                       // warps beyond the heads redo the last one and store nothing
    const int h = min(hw, d.H - 1);
    const int lim = min(d.Q, d.L - c * d.Q);
    const long long tix = (long long)(b * d.H + h) * d.nc + c, base = tix * d.Q + l0;
    const long long copies = (long long)d.b * d.H * d.nc * d.Q;        // nf / nb / pf / pb hold nsplit partial copies, u4 its tiles
    const float Ah = a.A[h], bias = d.has_bias ? a.dt_bias[h] : 0.f;
    float v1[E], v2[E], w1[E], w2[E], ex[E], dto[E], dlo[E], pre[E], t[E], u[E];
#pragma unroll
    for (int j = 0; j < E; ++j) v1[j] = v2[j] = w1[j] = w2[j] = ex[j] = dto[j] = dlo[j] = pre[j] = 0.f;
    float ts = 0.f, te = 0.f;                                          // dT_b, dT_f
    for (int k0 = lane; k0 < a.nblk; k0 += 256) {                      // 16 loads in flight: dstate 256 of headdim 128 brings 256 partial values
        float pe[8], ps[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = k0 + 32 * j;
            pe[j] = k < a.nblk ? a.dTpart[tix * a.nblk + k] : 0.f;
            ps[j] = k < a.nblk ? a.dTpart[((long long)d.b * d.H * d.nc + tix) * a.nblk + k] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            te += pe[j];
            ts += ps[j];
        }
    }
    if (l0 < d.Q) {
        load_strided(a.dt, a.dt_dtype, b * a.dsb + (long long)(c * d.Q + l0) * a.dsl + h * a.dsh, a.dsl, lim - l0, pre);
        load_e(a.nf + base, true, v1);
        load_e(a.pb + base, true, v2);
        load_e(a.nb + base, true, w1);
        load_e(a.pf + base, true, w2);
        load_e(a.ddt_out + base, true, dto);
        load_e(a.dt_out + base, wide, dlo);
        if (a.u4) {                                                    // (u_f, u_b) pairs, one per tile of the chunk: at most four
            float uf[4][E], ub[4][E];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < a.u4_tiles) {
                    load_e(a.u4 + (2 * k) * copies + base, true, uf[k]);
                    load_e(a.u4 + (2 * k + 1) * copies + base, true, ub[k]);
                }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < a.u4_tiles)
#pragma unroll
                    for (int j = 0; j < E; ++j) {
                        v1[j] += uf[k][j];
                        w1[j] += ub[k][j];
                    }
        } else {
            load_e(a.da_f + base, true, t);
            load_e(a.da_b + base, true, u);
#pragma unroll
            for (int j = 0; j < E; ++j) ex[j] = t[j] + u[j];
        }
        for (int k = 1; k < a.nsplit; ++k) {
            load_e(a.nf + k * copies + base, true, t);
            load_e(a.nb + k * copies + base, true, u);
#pragma unroll
            for (int j = 0; j < E; ++j) {
                v1[j] += t[j];
                w1[j] += u[j];
            }
            load_e(a.pb + k * copies + base, true, t);
            load_e(a.pf + k * copies + base, true, u);
#pragma unroll
            for (int j = 0; j < E; ++j) {
                v2[j] += t[j];
                w2[j] += u[j];
            }
        }
    }
    ts = simt::warp_sum(ts);
    te = simt::warp_sum(te);
    if (l0 == 0) v2[0] += ts;                                          // dT_b enters at index 0, dT_f at index Q - 1
    if (l0 + E == d.Q) w2[E - 1] += te;
    // ddA = exclusive sums of v1 (ascending) and w1 (descending), inclusive ones of v2 and w2
#pragma unroll
    for (int j = 0; j < E; ++j) ex[j] -= v1[j] + w1[j];
    scan_up(v1, lane);
    scan_up(v2, lane);
    scan_down(w1, lane);
    scan_down(w2, lane);
    across_warps<E, 4, 2>({&v1, &v2, &w1, &w2}, lane);
    float sumA = 0.f, sumB = 0.f, g[E];
#pragma unroll
    for (int j = 0; j < E; ++j) {
        const float ddA = ex[j] + v1[j] + v2[j] + w1[j] + w2[j], at = pre[j] + bias;
        g[j] = ddA * Ah + dto[j];
        const float val = d.softplus ? softplus_ref(at) : at;
        if (val < d.dt_min || val > d.dt_max) g[j] = 0.f;
        if (d.softplus && at <= 20.f) g[j] *= sigmoidf_(at);
        sumA += l0 + j < lim ? ddA * dlo[j] : 0.f;
        sumB += l0 + j < lim ? g[j] : 0.f;
    }
    store_strided(a.ddt.ptr, a.dt_dtype, b * a.ddt.sb + (long long)(c * d.Q + l0) * a.ddt.sl + h * a.ddt.sh, a.ddt.sl, on ? lim - l0 : 0, g);
    sumA = simt::warp_sum(sumA);
    sumB = simt::warp_sum(sumB);
    __shared__ float red[2][kCumsumWarps];
    if (lane == 0) {
        red[0][warp] = sumA;
        red[1][warp] = sumB;
    }
    __syncthreads();
    sumA = sumB = 0.f;
    for (int w = 0; w < W; ++w) {
        sumA += red[0][warp - warp % W + w];
        sumB += red[1][warp - warp % W + w];
    }
    if (lane == 0 && warp % W == 0 && hw < d.H) {
        a.dApart[(long long)(b * d.nc + c) * d.H + h] = sumA;
        a.dbiaspart[(long long)(b * d.nc + c) * d.H + h] = sumB;
    }
}

}  // namespace tc
}  // namespace bissd
