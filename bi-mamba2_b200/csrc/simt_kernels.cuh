// The phases of the scan that every kernel family shares: discretisation and cumulative sums, the recurrence over chunks,
// the last reductions of the parameter gradients, boundary chaining.  The CUDA-core products are in simt_products.cuh.
//
// Notation: Delta = dt_out, a = Delta*A, cs_f[l] = sum_{j<=l} a_j, cs_b[l] = sum_{j>=l} a_j within a chunk,
// T = cs_f[Q-1] = cs_b[0].
#pragma once
#include "common.cuh"
#include "simt_tile.cuh"

namespace bissd {
namespace simt {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_incl_scan(float v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        float t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

__device__ __forceinline__ float warp_incl_scan_rev(float v, int lane) {   // v[lane] + v[lane+1] + ... + v[31]
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        float t = __shfl_down_sync(0xffffffffu, v, o);
        if (lane + o < 32) v += t;
    }
    return v;
}
// Inclusive scans over the 256 threads of a CTA (thread t = position t), ascending for a and b, descending for c and
// e, all four at once: warp scans, the eight warp totals through shared memory (tot[4][8]), fixed order of additions.
__device__ __forceinline__ void block_scan4(float &a, float &b, float &c, float &e, float (*tot)[8]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    a = warp_incl_scan(a, lane);
    b = warp_incl_scan(b, lane);
    c = warp_incl_scan_rev(c, lane);
    e = warp_incl_scan_rev(e, lane);
    if (lane == 31) {
        tot[0][warp] = a;
        tot[1][warp] = b;
    }
    if (lane == 0) {
        tot[2][warp] = c;
        tot[3][warp] = e;
    }
    __syncthreads();
    float pa = 0.f, pb = 0.f, pc = 0.f, pe = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        pa += (w < warp) ? tot[0][w] : 0.f;
        pb += (w < warp) ? tot[1][w] : 0.f;
        pc += (w > warp) ? tot[2][w] : 0.f;
        pe += (w > warp) ? tot[3][w] : 0.f;
    }
    a += pa;
    b += pb;
    c += pc;
    e += pe;
}

// ---------------------------------------------------------------------------------------------------------
// Inter-chunk recurrence, both directions in one launch (blockIdx.z = direction).
// Forward: S_0 = init_f; S_{c+1} = e^{T_c} S_c + loc_f[c]; states_f[c] = S_c; final_f = S_nc.
// Reverse: R_{nc-1} = init_b; R_{c-1} = e^{T_c} R_c + loc_b[c]; states_b[c] = R_c; final_b = R_{-1}.
// Takes over _state_passing_fwd_kernel (src/ssd/bi/ssd_state_passing.py:27-92), called twice by the reference.
// grid (b*H, ceil(P*N/256), 2)
template <class T>
__global__ void __launch_bounds__(TB) state_passing_fwd(Dims d, const float *loc, const float *cs_f, const float *cs_b,
                                                        const float *init_f, const float *init_b, void *states_f,
                                                        void *states_b, float *final_f, float *final_b) {
    const int h = blockIdx.x % d.H, b = blockIdx.x / d.H;
    const int dir = blockIdx.z;
    const int PN = d.P * d.N;
    const int e = blockIdx.y * TB + threadIdx.x;
    if (e >= PN) return;
    const long long per_dir = (long long)d.b * d.nc * d.H * PN;
    const float *lp = loc + dir * per_dir;
    const float *init = dir ? init_b : init_f;
    void *states = dir ? states_b : states_f;
    float *fin = dir ? final_b : final_f;
    float run = init ? init[(long long)(b * d.H + h) * PN + e] : 0.f;
    for (int i = 0; i < d.nc; ++i) {
        const int c = dir ? d.nc - 1 - i : i;
        const long long off = ((long long)(b * d.nc + c) * d.H + h) * PN + e;
        st<T>(states, off, run);
        const long long cb = ((long long)(b * d.H + h) * d.nc + c) * d.Q;
        const float dec = expf(dir ? cs_b[cb] : cs_f[cb + d.Q - 1]);
        run = dec * run + lp[off];
    }
    if (fin) fin[(long long)(b * d.H + h) * PN + e] = run;
}

// ---------------------------------------------------------------------------------------------------------
// State-passing backward, both directions (blockIdx.z).  Per element of the (P,N) state:
//   forward dir: run = dfinal_f; for c = nc-1..0: E_f[c] = run; dT_f[c] += e^{T_c} S_f[c] run; run = e^{T_c} run + gloc_f[c]
//   reverse dir: run = dfinal_b; for c = 0..nc-1: E_b[c] = run; dT_b[c] += e^{T_c} S_b[c] run; run = e^{T_c} run + gloc_b[c]
// and dinit = run at the end.  E[c] is the gradient w.r.t. the local state of chunk c.
// Takes over _state_passing_bwd_kernel (src/ssd/bi/ssd_state_passing.py:106-187); the per-block partial sums
// of dT go to dTpart[dir][b,h,c][blk] and are added in a fixed order later (no atomics).
// grid (b*H, nblk = ceil(P*N/256), 2)
template <class T>
__global__ void __launch_bounds__(TB) state_passing_bwd(Dims d, const float *gloc, const void *states_f,
                                                        const void *states_b, const float *cs_f, const float *cs_b,
                                                        const float *dfinal_f, const float *dfinal_b, float *E,
                                                        void *E16, float *dTpart, float *dinit_f, float *dinit_b) {
    __shared__ float red[TB / 32];
    const int h = blockIdx.x % d.H, b = blockIdx.x / d.H;
    const int dir = blockIdx.z;
    const int PN = d.P * d.N;
    const int nblk = gridDim.y;
    const int e = blockIdx.y * TB + threadIdx.x;
    const bool on = e < PN;
    const long long per_dir = (long long)d.b * d.nc * d.H * PN;
    const float *gp = gloc + dir * per_dir;
    float *Ep = E + dir * per_dir;
    const void *states = dir ? states_b : states_f;
    const float *dfin = dir ? dfinal_b : dfinal_f;
    float *dinit = dir ? dinit_b : dinit_f;
    float run = (on && dfin) ? dfin[(long long)(b * d.H + h) * PN + e] : 0.f;
    for (int i = 0; i < d.nc; ++i) {
        const int c = dir ? i : d.nc - 1 - i;
        const long long off = ((long long)(b * d.nc + c) * d.H + h) * PN + e;
        const long long cb = ((long long)(b * d.H + h) * d.nc + c) * d.Q;
        const float dec = expf(dir ? cs_b[cb] : cs_f[cb + d.Q - 1]);
        float part = 0.f;
        if (on) {
            if (E) Ep[off] = run;                                    // fp32 copy for the CUDA-core kernels
            if (E16) st<T>(E16, dir * per_dir + off, run);           // input-dtype copy for the tensor-core kernels
            part = dec * ld<T>(states, off) * run;
            run = dec * run + gp[off];
        }
        part = warp_sum(part);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
        __syncthreads();
        if (threadIdx.x == 0) {
            float s = 0.f;
            for (int w = 0; w < TB / 32; ++w) s += red[w];
            dTpart[((long long)dir * d.b * d.H * d.nc + (long long)(b * d.H + h) * d.nc + c) * nblk + blockIdx.y] = s;
        }
        __syncthreads();
    }
    if (on && dinit) dinit[(long long)(b * d.H + h) * PN + e] = run;
}

// ---------------------------------------------------------------------------------------------------------
// Discretisation + both cumulative sums, and their backward.  One CTA of 256 threads per (batch, chunk, head), thread
// l holding position l of the chunk (chunk <= 256): every global operand is requested at once and each scan is one
// warp scan plus a combine over the eight warp totals (a warp walking the chunk in eight steps was latency-bound).
// grid (b * nc * H), head fastest.
//
// cumsum_fwd takes over _chunk_cumsum_fwd_kernel (src/ssd/bi/ssd_chunk_state.py:34-91):
//   dt_out = clamp(softplus(dt + bias)), a = dt_out A, cs_f[l] = sum_{j<=l} a_j, cs_b[l] = sum_{j>=l} a_j; zero tail.
// One chunk: v = Delta, f and r the two cumulative sums of Delta A at this thread's position (0 beyond the chunk).
__device__ __forceinline__ void chunk_cumsum(const Dims &d, const void *dt, int dt_dtype, long long dsb, long long dsl, long long dsh,
                                             const float *A, const float *dt_bias, int b, int c, int h, int lim, float (*tot)[8],
                                             float &v, float &f, float &r) {
    const int l = threadIdx.x;
    v = 0.f;
    if (l < lim) {
        v = ld_any(dt, dt_dtype, b * dsb + (long long)(c * d.Q + l) * dsl + h * dsh) + (d.has_bias ? dt_bias[h] : 0.f);
        if (d.softplus) v = softplus_ref(v);
        v = fminf(fmaxf(v, d.dt_min), d.dt_max);
    }
    f = r = (l < d.Q) ? v * A[h] : 0.f;
    float dummy1 = 0.f, dummy2 = 0.f;
    block_scan4(f, dummy1, r, dummy2, tot);
}

// ---------------------------------------------------------------------------------------------------------
// Assemble d(a) from its six terms, go back through the discretisation.  One CTA per (batch, chunk, head), see above.
//   ddA = da_f + da_b + exclcumsum(nf) + exclrevcumsum(nb) + revcumsum(pf, +dT_f at Q-1) + cumsum(pb, +dT_b at 0)
//   ddt = (ddA A + ddt_out), zero where the clamp is active, times sigmoid(pre) when softplus (pre <= 20)
// Takes over the host glue at src/ssd/bi/ssd_combined.py:456-466 and _chunk_cumsum_bwd_kernel
// (src/ssd/bi/ssd_chunk_state.py:106-170).  dA / ddt_bias partials per (b,c,h) are reduced by final_reduce.
// The intra-chunk decay gradients come either as da_f / da_b (already dominance sums) or, when u4 is given, as the
// per-index differences u_f / u_b = column sums - row sums (u4_tiles pairs of arrays: tile 0 f, b, tile 1 f, b, ...), which are
// added to the terms that are prefix-summed (u_f) and suffix-summed (u_b) exclusively; da_f / da_b are then null.
struct CumsumBwd {
    const void *dt;
    int dt_dtype;
    long long dsb, dsl, dsh;
    const float *A, *dt_bias, *dt_out, *ddt_out, *nf, *nb, *pf, *pb, *da_f, *da_b, *u4;
    int u4_tiles;                                                // 0 without u4
    const float *dTpart;
    int nblk, nsplit;
    MutView ddt;
    float *dApart, *dbiaspart;
};
// tot[4][8], red[2][8]: shared memory
__device__ __forceinline__ void cumsum_bwd_role(const Dims &d, const CumsumBwd &a, int block, float (*tot)[8], float (*red)[8]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = block % d.H, c = (block / d.H) % d.nc, b = block / (d.H * d.nc);
    const int l = threadIdx.x;
    const int lim = min(d.Q, d.L - c * d.Q);
    const long long base = ((long long)(b * d.H + h) * d.nc + c) * d.Q;
    const long long tix = (long long)(b * d.H + h) * d.nc + c;
    const long long split_stride = (long long)d.b * d.H * d.nc * d.Q;   // a.nf/a.nb/a.pf/a.pb hold a.nsplit partial copies
    // the four scanned sequences: a.nf (+u_f) and a.pb ascending, a.nb (+u_b) and a.pf descending
    float v1 = 0.f, v2 = 0.f, w1 = 0.f, w2 = 0.f, ex = 0.f, dto = 0.f, dlo = 0.f, pre = 0.f;
    // Every load is requested before the first is used: with the sums next to their loads this kernel was one memory
    // latency per term.
    float ts[4] = {0.f, 0.f, 0.f, 0.f}, te[4] = {0.f, 0.f, 0.f, 0.f};
    const float *slots_b = a.dTpart + ((long long)d.b * d.H * d.nc + tix) * a.nblk, *slots_f = a.dTpart + tix * a.nblk;
    const bool last = warp == (d.Q - 1) >> 5;                    // the warp of position Q - 1
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (warp == 0 && lane + 32 * i < a.nblk) ts[i] = slots_b[lane + 32 * i];
        if (last && lane + 32 * i < a.nblk) te[i] = slots_f[lane + 32 * i];
    }
    if (l < d.Q) {
        const float n0 = a.nf[base + l], p0 = a.pb[base + l], q0 = a.nb[base + l], r0 = a.pf[base + l];
        float uf[4] = {0.f, 0.f, 0.f, 0.f}, ub[4] = {0.f, 0.f, 0.f, 0.f};
        if (a.u4) {                                              // (u_f, u_b) pairs, one per tile of the chunk
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (t < a.u4_tiles) {
                    uf[t] = a.u4[(2 * t) * split_stride + base + l];
                    ub[t] = a.u4[(2 * t + 1) * split_stride + base + l];
                }
        } else {
            ex = a.da_f[base + l] + a.da_b[base + l];
        }
        if (l < lim) {
            dto = a.ddt_out[base + l];
            dlo = a.dt_out[base + l];
            pre = ld_any(a.dt, a.dt_dtype, b * a.dsb + (long long)(c * d.Q + l) * a.dsl + h * a.dsh) + (d.has_bias ? a.dt_bias[h] : 0.f);
        }
        v1 = n0; v2 = p0; w1 = q0; w2 = r0;
        for (int k = 1; k < a.nsplit; ++k) {
            v1 += a.nf[k * split_stride + base + l];
            v2 += a.pb[k * split_stride + base + l];
            w1 += a.nb[k * split_stride + base + l];
            w2 += a.pf[k * split_stride + base + l];
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            v1 += uf[t];
            w1 += ub[t];
        }
        for (int t = 4; t < a.u4_tiles; ++t) {
            v1 += a.u4[(2 * t) * split_stride + base + l];
            w1 += a.u4[(2 * t + 1) * split_stride + base + l];
        }
    }
    // dT_b enters at index 0, dT_f at index Q-1; the warp of that position adds up the slots
    if (warp == 0) {
        float t = (ts[0] + ts[1]) + (ts[2] + ts[3]);
        for (int k = lane + 128; k < a.nblk; k += 32) t += slots_b[k];
        t = warp_sum(t);
        if (lane == 0) v2 += t;
    }
    if (last) {
        float t = (te[0] + te[1]) + (te[2] + te[3]);
        for (int k = lane + 128; k < a.nblk; k += 32) t += slots_f[k];
        t = warp_sum(t);
        if (l == d.Q - 1) w2 += t;
    }
    float s1 = v1, s2 = v2, r1 = w1, r2 = w2;
    block_scan4(s1, s2, r1, r2, tot);
    float sumA = 0.f, sumB = 0.f;
    if (l < lim) {
        const float ddA = (s1 - v1) + s2 + ex + (r1 - w1) + r2;
        float g = ddA * a.A[h] + dto;
        const float val = d.softplus ? softplus_ref(pre) : pre;
        if (val < d.dt_min || val > d.dt_max) g = 0.f;
        if (d.softplus && pre <= 20.f) g *= sigmoidf_(pre);
        st_any(a.ddt.ptr, a.dt_dtype, b * a.ddt.sb + (long long)(c * d.Q + l) * a.ddt.sl + h * a.ddt.sh, g);
        sumA = ddA * dlo;
        sumB = g;
    }
    sumA = warp_sum(sumA);
    sumB = warp_sum(sumB);
    if (lane == 0) {
        red[0][warp] = sumA;
        red[1][warp] = sumB;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float ta = 0.f, tb = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            ta += red[0][w];
            tb += red[1][w];
        }
        a.dApart[(long long)(b * d.nc + c) * d.H + h] = ta;
        a.dbiaspart[(long long)(b * d.nc + c) * d.H + h] = tb;
    }
}

// ---------------------------------------------------------------------------------------------------------
// Sum of v over the block in a fixed order (lanes by butterfly, then the warps' totals by the first warp's butterfly),
// returned to every thread of warp 0; `red` needs NT / 32 entries beyond any the caller still reads.  Two barriers.
template <int NT>
__device__ __forceinline__ float block_sum(float v, float *red) {
    v = warp_sum(v);
    __syncthreads();                                             // earlier readers of red are done
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = 0.f;
    if (threadIdx.x < 32) {
        t = (threadIdx.x < NT / 32) ? red[threadIdx.x] : 0.f;
        t = warp_sum(t);
    }
    return t;
}

// Fixed-order reduction of the per-block partials into dA (H), ddt_bias (H) and dD (H or H*P).  grid (H), NT threads.
// `compact` (per-head D only): dDpart holds nlt scalars per (batch, chunk, head) instead of nlt rows of P channel sums.
template <int NT>
__global__ void __launch_bounds__(NT) final_reduce(Dims d, const float *dApart, const float *dbiaspart,
                                                   const float *dDpart, int nlt, int compact, float *dA, float *ddt_bias,
                                                   float *dD) {
    pdl_begin();
    __shared__ float red[NT];
    const int h = blockIdx.x;
    const int nbc = d.b * d.nc;
    float sa = 0.f, sbias = 0.f;
    for (int i = threadIdx.x; i < nbc; i += NT) {
        sa += dApart[(long long)i * d.H + h];
        sbias += dbiaspart[(long long)i * d.H + h];
    }
    sa = block_sum<NT>(sa, red);
    if (threadIdx.x == 0) dA[h] = sa;
    sbias = block_sum<NT>(sbias, red);
    if (threadIdx.x == 0 && ddt_bias) ddt_bias[h] = sbias;
    if (dD && dDpart && compact) {
        float sd = 0.f;                                          // fixed order: strided per thread, then block_sum
        const int n = nbc * nlt;
        for (int i = threadIdx.x; i < n; i += NT) {
            const int bc = i / nlt, t = i - bc * nlt;
            sd += dDpart[((long long)bc * d.H + h) * nlt + t];
        }
        sd = block_sum<NT>(sd, red);
        if (threadIdx.x == 0) dD[h] = sd;
    } else if (dD && dDpart) {
        // rows of the partial buffer are split over NT / P thread groups, then the groups are added in a fixed order
        const int rows = nbc * nlt;
        const int ngrp = d.P <= NT ? NT / d.P : 1;
        float tot = 0.f;
        for (int p0 = 0; p0 < d.P; p0 += NT) {
            const int p = p0 + (threadIdx.x % (d.P <= NT ? d.P : NT)), grp = d.P <= NT ? threadIdx.x / d.P : 0;
            float s = 0.f;
            if (p < d.P && grp < ngrp) {
                // four independent partial sums keep several loads in flight; they are combined in a fixed order
                float s4[4] = {0.f, 0.f, 0.f, 0.f};
                int r = grp;
                for (; r + 3 * ngrp < rows; r += 4 * ngrp) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int rr = r + u * ngrp, i = rr / nlt, t = rr - i * nlt;
                        s4[u] += dDpart[(((long long)i * d.H + h) * nlt + t) * d.P + p];
                    }
                }
                for (; r < rows; r += ngrp) {
                    const int i = r / nlt, t = r - i * nlt;
                    s4[0] += dDpart[(((long long)i * d.H + h) * nlt + t) * d.P + p];
                }
                s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
            }
            __syncthreads();
            red[threadIdx.x] = s;
            __syncthreads();
            if (grp == 0 && p < d.P) {
                float v = 0.f;
                for (int q = 0; q < ngrp; ++q) v += red[q * d.P + (p - p0)];
                if (d.D_hdim) dD[h * d.P + p] = v;
                tot += v;
            }
        }
        if (!d.D_hdim) {
            __syncthreads();
            tot = block_sum<NT>(tot, red);
            if (threadIdx.x == 0) dD[h] = tot;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------
// Four-elements-per-thread versions of the two state-passing kernels (need headdim*dstate % 4 == 0): 128-bit loads of
// the fp32 chunk quantities, one packed store of the passed values, and the chunk loop unrolled so that several
// chunks' loads are in flight.  Same arithmetic, same order, as state_passing_fwd / state_passing_bwd.
template <class T> __device__ __forceinline__ void st4(void *p, long long i, float a, float b, float c, float e) {
    T v[4] = {from_f<T>(a), from_f<T>(b), from_f<T>(c), from_f<T>(e)};
    if (sizeof(T) == 4) *reinterpret_cast<float4 *>(static_cast<T *>(p) + i) = *reinterpret_cast<float4 *>(v);
    else *reinterpret_cast<uint2 *>(static_cast<T *>(p) + i) = *reinterpret_cast<uint2 *>(v);
}
template <class T> __device__ __forceinline__ float4 ld4(const void *p, long long i) {
    if (sizeof(T) == 4) return *reinterpret_cast<const float4 *>(static_cast<const T *>(p) + i);
    const uint2 u = *reinterpret_cast<const uint2 *>(static_cast<const T *>(p) + i);
    const T *v = reinterpret_cast<const T *>(&u);
    return make_float4(to_f<T>(v[0]), to_f<T>(v[1]), to_f<T>(v[2]), to_f<T>(v[3]));
}

template <class T> __device__ __forceinline__ void st2(void *p, long long i, float a, float b) {   // 16-bit T
    T v[2] = {from_f<T>(a), from_f<T>(b)};
    *reinterpret_cast<uint32_t *>(static_cast<T *>(p) + i) = *reinterpret_cast<uint32_t *>(v);
}
template <class T> __device__ __forceinline__ float2 ld2(const void *p, long long i) {
    const uint32_t u = *reinterpret_cast<const uint32_t *>(static_cast<const T *>(p) + i);
    const T *v = reinterpret_cast<const T *>(&u);
    return make_float2(to_f<T>(v[0]), to_f<T>(v[1]));
}
// The states a pass starts from and ends in are the caller's fp32 arrays, of any alignment; once per thread.
__device__ __forceinline__ float4 load_state4(const float *p) {
    return reinterpret_cast<uintptr_t>(p) % 16 == 0 ? *reinterpret_cast<const float4 *>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __forceinline__ void store_state4(float *p, float4 v) {
    if (reinterpret_cast<uintptr_t>(p) % 16 == 0) {
        *reinterpret_cast<float4 *>(p) = v;
    } else {
        p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w;
    }
}

// grid (b*H, ceil(P*N/4/blockDim), 2)
template <class T, int U>
__global__ void __launch_bounds__(TB) state_passing_fwd4(Dims d, const float *loc, const float *cs_f, const float *cs_b,
                                                         const float *init_f, const float *init_b, void *states_f,
                                                         void *states_b, float *final_f, float *final_b) {
    pdl_begin();
    const int h = blockIdx.x % d.H, b = blockIdx.x / d.H;
    const int dir = blockIdx.z;
    const int PN = d.P * d.N;
    const int e = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
    if (e >= PN) return;
    const long long per_dir = (long long)d.b * d.nc * d.H * PN;
    const float *lp = loc + dir * per_dir;
    const float *init = dir ? init_b : init_f;
    void *states = dir ? states_b : states_f;
    float *fin = dir ? final_b : final_f;
    float4 run = init ? load_state4(init + (long long)(b * d.H + h) * PN + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    const long long cstride = (long long)d.H * PN;
    const long long off0 = ((long long)b * d.nc * d.H + h) * PN + e;
    const long long cb0 = (long long)(b * d.H + h) * d.nc * d.Q;
    for (int i0 = 0; i0 < d.nc; i0 += U) {
        float4 v[U];
        float dec[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = dir ? d.nc - 1 - i0 - u : i0 + u;
            const bool have = i0 + u < d.nc;
            v[u] = have ? __ldg(reinterpret_cast<const float4 *>(lp + off0 + c * cstride)) : make_float4(0.f, 0.f, 0.f, 0.f);
            dec[u] = have ? (dir ? cs_b[cb0 + (long long)c * d.Q] : cs_f[cb0 + (long long)c * d.Q + d.Q - 1]) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (i0 + u >= d.nc) break;
            const int c = dir ? d.nc - 1 - i0 - u : i0 + u;
            const float ed = expf(dec[u]);
            st4<T>(states, off0 + c * cstride, run.x, run.y, run.z, run.w);
            run.x = fmaf(ed, run.x, v[u].x);
            run.y = fmaf(ed, run.y, v[u].y);
            run.z = fmaf(ed, run.z, v[u].z);
            run.w = fmaf(ed, run.w, v[u].w);
        }
    }
    if (fin) store_state4(fin + (long long)(b * d.H + h) * PN + e, run);
}

// grid (b*H, ceil(P*N/4/blockDim), 2), blockDim a multiple of 32; dTpart has one slot per warp of a (dir, b, h): gridDim.y *
// blockDim / 32 - one per warp instead of one per block keeps barriers out of the loop (b8 H24 nc8 P64 N128 bf16: 43 -> 39
// us).  U: chunks whose loads are in flight together, see pass_ahead(); with few threads the instructions of a group of
// chunks are most of the time, so its U sums share their shuffles (b1 L8192 H8 P64 N128 chunk 256: 16.7 -> 14 us).
// WN (dstate, at the sizes of tc::state_walk, 16-bit states; else 0): a thread has the elements, and a slot the sum, that tc::state_walk gives a
// lane and a slot - four columns of 32 n, a lane two adjacent n of two columns - and everything is added up in its order.
// Which of the two runs depends on the batch; dT, and through it ddt and dA, does not.  (dstate is a constant so that the
// distance to a thread's second column is part of the instructions.)
template <class T, int U, int WN>
__global__ void __launch_bounds__(TB) state_passing_bwd4(Dims d, const float *gloc, const void *states_f,
                                                         const void *states_b, const float *cs_f, const float *cs_b,
                                                         const float *dfinal_f, const float *dfinal_b, float *E,
                                                         void *E16, float *dTpart, float *dinit_f, float *dinit_b) {
    pdl_begin();
    const int h = blockIdx.x % d.H, b = blockIdx.x / d.H;
    const int dir = blockIdx.z, lane = threadIdx.x & 31;
    const int PN = d.P * d.N;
    const int nslots = gridDim.y * (blockDim.x >> 5), slot = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int e = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
    constexpr int gap = WN ? 2 * WN : 2;                         // from the first two elements to the others
    if (WN) {
        constexpr bool half = WN == 64;                          // both halves of the 128-row tile are the same 64 n
        const int cols = half ? d.P / 4 : d.P / 2, V = cols / 4, ew = slot / V % 8, quad = ew & 3;
        const int col = (half ? (quad >> 1) * 2 + (ew >> 2) : ew >> 2) * cols + slot % V * 4 + (lane & 1);
        e = col * WN + slot / (8 * V) * 128 + (half ? quad & 1 : quad) * 32 + (lane & ~1);
    }
    const bool on = WN || e < PN;
    const long long per_dir = (long long)d.b * d.nc * d.H * PN;
    const float *gp = gloc + dir * per_dir;
    const void *states = dir ? states_b : states_f;
    const float *dfin = dir ? dfinal_b : dfinal_f;
    float *dinit = dir ? dinit_b : dinit_f;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const long long bh0 = (long long)(b * d.H + h) * PN + e;
    float4 run = zero;
    if (on && dfin) run = WN ? make_float4(dfin[bh0], dfin[bh0 + 1], dfin[bh0 + gap], dfin[bh0 + gap + 1]) : load_state4(dfin + bh0);
    const long long cstride = (long long)d.H * PN;
    const long long off0 = ((long long)b * d.nc * d.H + h) * PN + e;
    const float *total = (dir ? cs_b : cs_f + d.Q - 1) + (long long)(b * d.H + h) * d.nc * d.Q;      // T of chunk 0
    float *slots = dTpart + ((long long)dir * d.b * d.H * d.nc + (long long)(b * d.H + h) * d.nc) * nslots + slot;
    for (int i0 = 0; i0 < d.nc; i0 += U) {
        float4 gv[U], sv[U];
        float dec[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (WN) {                                            // past the last chunk: its values again, not used
                const int k = min(i0 + u, d.nc - 1), c = dir ? k : d.nc - 1 - k;
                const long long off = off0 + c * cstride;
                const float2 lo = __ldg(reinterpret_cast<const float2 *>(gp + off)), hi = __ldg(reinterpret_cast<const float2 *>(gp + off + gap));
                const float2 s0 = ld2<T>(states, off), s1 = ld2<T>(states, off + gap);
                gv[u] = make_float4(lo.x, lo.y, hi.x, hi.y);
                sv[u] = make_float4(s0.x, s0.y, s1.x, s1.y);
                dec[u] = total[(long long)c * d.Q];
                continue;
            }
            const int c = dir ? i0 + u : d.nc - 1 - i0 - u;
            const bool have = on && i0 + u < d.nc;
            gv[u] = have ? __ldg(reinterpret_cast<const float4 *>(gp + off0 + c * cstride)) : zero;
            sv[u] = have ? ld4<T>(states, off0 + c * cstride) : zero;
            dec[u] = i0 + u < d.nc ? total[(long long)c * d.Q] : 0.f;
        }
        float part[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = dir ? i0 + u : d.nc - 1 - i0 - u;
            const long long off = off0 + c * cstride;
            dec[u] = expf(dec[u]);
            // the order is written out: the same whatever U
            if (WN) part[u] = fmaf(sv[u].z, run.z, fmaf(sv[u].w, run.w, fmaf(sv[u].x, run.x, fmaf(sv[u].y, run.y, 0.f))));
            else part[u] = fmaf(sv[u].x, run.x, fmaf(sv[u].y, run.y, fmaf(sv[u].z, run.z, sv[u].w * run.w)));
            if (i0 + u < d.nc) {
                if (on) {
                    if (WN) {
                        st2<T>(E16, dir * per_dir + off, run.x, run.y);
                        st2<T>(E16, dir * per_dir + off + gap, run.z, run.w);
                    } else {
                        if (E) *reinterpret_cast<float4 *>(E + dir * per_dir + off) = run;
                        if (E16) st4<T>(E16, dir * per_dir + off, run.x, run.y, run.z, run.w);
                    }
                }
                run.x = fmaf(dec[u], run.x, gv[u].x);
                run.y = fmaf(dec[u], run.y, gv[u].y);
                run.z = fmaf(dec[u], run.z, gv[u].z);
                run.w = fmaf(dec[u], run.w, gv[u].w);
            }
        }
        // lane 32 u / U writes chunk u's sum, times its decay
        auto value = [&](auto k) -> float { return part[decltype(k)::value]; };
        const float sum = warp_sums<U>(value, lane);
        float ed = dec[0];
#pragma unroll
        for (int u = 1; u < U; ++u) ed = lane == 32 / U * u ? dec[u] : ed;
        const int i = i0 + lane * U / 32;
        if (lane % (32 / U) == 0 && i < d.nc) slots[(long long)(dir ? i : d.nc - 1 - i) * nslots] = ed * sum;
    }
    if (on && dinit) {
        if (WN) {
            dinit[bh0] = run.x; dinit[bh0 + 1] = run.y; dinit[bh0 + gap] = run.z; dinit[bh0 + gap + 1] = run.w;
        } else {
            store_state4(dinit + bh0, run);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------
// Boundary chaining for a sequence sharded over `world` ranks (the single-GPU chunk recurrence of
// src/ssd/bi/ssd_state_passing.py:60,81 continued across ranks, unrolled into weighted sums):
//     out_left[e]  = sum_{r' < rank} exp(sum_{r' < r'' < rank} ld[r''][bh]) left[r'][e]
//     out_right[e] = sum_{r' > rank} exp(sum_{rank < r'' < r'} ld[r''][bh]) right[r'][e]
// with e over (batch*heads) x (headdim*dstate), bh = e / pn, ld[r][bh] = rank r's total log decay (<= 0).  The
// exponent is accumulated rank by rank (no differences of prefix sums), so fp32 is enough: where it is large its
// exponential is zero anyway.  Forward pass: left = F_f -> init_f, right = F_b -> init_b; backward pass:
// left = dinit_b -> dfinal_b, right = dinit_f -> dfinal_f.  All inputs were gathered into local memory beforehand.
static __global__ void __launch_bounds__(256) chain_boundaries(const float *left, const float *right, const float *ld,
                                                        long long rank_stride, long long ld_rank_stride, int world, int rank,
                                                        long long n, int pn, float *out_left, float *out_right) {
    const long long e = (long long)blockIdx.x * 256 + threadIdx.x;
    if (e >= n) return;
    const long long bh = e / pn;
    float a = 0.f, cum = 0.f;
    for (int r = rank - 1; r >= 0; --r) {
        a = fmaf(__expf(cum), left[r * rank_stride + e], a);
        cum += ld[r * ld_rank_stride + bh];
    }
    out_left[e] = a;
    a = 0.f;
    cum = 0.f;
    for (int r = rank + 1; r < world; ++r) {
        a = fmaf(__expf(cum), right[r * rank_stride + e], a);
        cum += ld[r * ld_rank_stride + bh];
    }
    out_right[e] = a;
}

}  // namespace simt
}  // namespace bissd
