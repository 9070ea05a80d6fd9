// Gated RMSNorm, forward and backward, for the layer that follows the scan in BiMamba2
// (takes over _layer_norm_fwd_1pass_kernel / _layer_norm_bwd_kernel of src/ssd/bi/layernorm_gated.py:45-105, :155-268
// in their RMS form; the arithmetic follows rms_norm_ref, :18-41):
//   norm_before_gate:  y = x rstd w;  out = y silu(z)
//   otherwise:         u = x silu(z);  out = u rstd w
// (no bias: the reference's RMSNorm registers none, src/ssd/bi/layernorm_gated.py:424)
//   rstd = rsqrt(mean over the group of (x or u)^2 + eps), one value per (row, group).
//
// Bound by HBM: every tensor is read or written once.  A thread owns 8 adjacent channels (one 16-byte piece of a 16-bit
// row) for all its rows, so the weight and the weight gradient stay in its registers; hidden / 8 threads make a row, a
// block holds Y such rows side by side and takes R rows per thread and step, the next step's loads in flight meanwhile.  Row
// statistics: warp shuffles, one shared-memory exchange and one barrier a step (two exchange buffers).  Groups are whole
// multiples of 256 channels, so the 256 channels of a warp belong to one group.
// 65536 rows of 2048 in bf16 with z: forward 229 -> 173 us (4.7 TB/s), backward 475 -> 235 us (5.7 TB/s); before, a warp
// made a row, the backward read it twice and kept its weight gradient in shared memory.
// Weight gradient: one partial row per block in the workspace, summed by norm_bwd_reduce - no float atomics.
#pragma once
#include "vec.cuh"

namespace bissd {
namespace norm {

using namespace vec;

constexpr int kCh = 8, kPairs = kCh / 2;         // channels per thread
constexpr int kMaxThreads = 512;                 // hidden <= 4096
constexpr int kFwdRows = 2, kBwdRows = 2;        // rows per thread and step

struct NormDims {
    long long rows;
    int hidden, group, ngroups;                  // group = channels per statistics group
    long long sx, sz, so;                        // row strides (elements) of x (and dx), z (and dz), out (and dout)
    float eps;
};

// GATE: 0 none, 1 after the norm, 2 before it
template <class T> __device__ __forceinline__ Row<T, kPairs> row_of(const void *p, long long off, bool on) {
    return on ? load_row<T, kPairs>(static_cast<const T *>(p) + off) : zero_row<T, kPairs>();
}
template <class T> __device__ __forceinline__ void put_row(void *p, long long off, const Row<T, kPairs> &r) {
    store_row<T, kPairs>(static_cast<T *>(p) + off, r);
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ f2 silu2(f2 z) { return mul2(z, sigmoid2(z)); }
// silu and its derivative
__device__ __forceinline__ void silu_grad2(f2 z, f2 &sl, f2 &dsl) {
    const f2 s = sigmoid2(z);
    sl = mul2(z, s);
    dsl = silu_slope2(z, s);
}
__device__ __forceinline__ float hsum(f2 v) {
    float a, b;
    unpack(v, a, b);
    return a + b;
}
// Sum of v[r] over the threads of this thread's statistics group, for each of its R rows.  buf: R x 16 floats a row set.
template <int R> __device__ __forceinline__ void group_sums(float (&v)[R], float *buf, int group) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wpg = group >> 8, first = warp / wpg * wpg;
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = warp_sum(v[r]);
    if (lane < R) {
        float mine = v[0];
#pragma unroll
        for (int r = 1; r < R; ++r) mine = lane == r ? v[r] : mine;
        buf[lane * 16 + warp] = mine;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        float s = 0.f;
        for (int w = first; w < first + wpg; ++w) s += buf[r * 16 + w];
        v[r] = s;
    }
}

// block (hidden / 8, Y); dynamic shared memory 2 * Y * R * 16 floats.  Any grid.
template <class T, class W, int GATE>
__global__ void __launch_bounds__(kMaxThreads) rmsnorm_gated_fwd(NormDims d, const void *x, const void *z, const void *weight,
                                                                 void *out, float *rstd) {
    extern __shared__ float sm[];
    constexpr int R = kFwdRows;
    pdl_begin();
    const int c0 = threadIdx.x * kCh;
    f2 w[kPairs];
#pragma unroll
    for (int i = 0; i < kPairs; ++i) w[i] = load_pair<W>(weight, c0 + 2 * i);
    const long long step = (long long)gridDim.x * blockDim.y * R, first = (long long)blockIdx.x * blockDim.y * R;
    Row<T, kPairs> xr[R], zr[R];
    auto fetch = [&](long long row0) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const bool on = row0 + r < d.rows;
            xr[r] = row_of<T>(x, (row0 + r) * d.sx + c0, on);
            if (GATE) zr[r] = row_of<T>(z, (row0 + r) * d.sz + c0, on);
        }
    };
    fetch(first + threadIdx.y * R);
    int turn = 0;
    for (long long base = first; base < d.rows; base += step, turn ^= 1) {
        const long long row0 = base + threadIdx.y * R;
        float ss[R];
        f2 v[R][kPairs];                                         // the result but for rstd
#pragma unroll
        for (int r = 0; r < R; ++r) {
            f2 s = pack(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < kPairs; ++i) {
                f2 u = widen<T>(xr[r].v[i]), gate;
                if (GATE) gate = silu2(widen<T>(zr[r].v[i]));
                if (GATE == 2) u = mul2(u, gate);
                s = fma2(u, u, s);
                v[r][i] = mul2(u, w[i]);
                if (GATE == 1) v[r][i] = mul2(v[r][i], gate);
            }
            ss[r] = hsum(s);
        }
        if (base + step < d.rows) fetch(row0 + step);
        group_sums<R>(ss, sm + (turn * blockDim.y + threadIdx.y) * R * 16, d.group);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (row0 + r >= d.rows) continue;
            const float rs = rsqrtf(ss[r] / (float)d.group + d.eps);
            if (c0 % d.group == 0) rstd[(row0 + r) * d.ngroups + c0 / d.group] = rs;
            Row<T, kPairs> o;
#pragma unroll
            for (int i = 0; i < kPairs; ++i) o.v[i] = narrow<T>(mul2(v[r][i], pack(rs, rs)));
            put_row<T>(out, (row0 + r) * d.so + c0, o);
        }
    }
}

// Backward.  dw_part: [gridDim.x][hidden] fp32.  Same block; dynamic shared memory as the forward's, or Y * hidden floats
// (the rows of a block's weight gradients) where that is more.
//   xhat = u rstd,  dy = dout (silu(z) if the gate follows the norm),  du = rstd (dy w - xhat mean_group(dy w xhat))
//   gate after the norm:  dx = du,  dz = dout (xhat w) silu'(z);   gate before:  dx = du silu(z),  dz = du x silu'(z)
//   dw = sum over rows of dy xhat
// Only dx (and dz with the gate before) waits for the row's mean.
template <class T, class W, int GATE>
__global__ void __launch_bounds__(kMaxThreads) rmsnorm_gated_bwd(NormDims d, const void *x, const void *z, const void *weight,
                                                                 const void *dout, const float *rstd, void *dx, void *dz,
                                                                 float *dw_part) {
    extern __shared__ float sm[];
    constexpr int R = kBwdRows;
    pdl_begin();
    const int c0 = threadIdx.x * kCh, g = c0 / d.group;
    f2 w[kPairs], dw[kPairs];
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        w[i] = load_pair<W>(weight, c0 + 2 * i);
        dw[i] = pack(0.f, 0.f);
    }
    const long long step = (long long)gridDim.x * blockDim.y * R;
    Row<T, kPairs> xr[R], gr[R], zr[R];
    float rs[R];
    auto fetch = [&](long long row0) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const bool on = row0 + r < d.rows;
            xr[r] = row_of<T>(x, (row0 + r) * d.sx + c0, on);
            gr[r] = row_of<T>(dout, (row0 + r) * d.so + c0, on);
            if (GATE) zr[r] = row_of<T>(z, (row0 + r) * d.sz + c0, on);
            rs[r] = on ? rstd[(row0 + r) * d.ngroups + g] : 0.f;
        }
    };
    const long long first = (long long)blockIdx.x * blockDim.y * R;
    fetch(first + threadIdx.y * R);
    int turn = 0;
    for (long long base = first; base < d.rows; base += step, turn ^= 1) {
        const long long row0 = base + threadIdx.y * R;
        f2 A[R][kPairs], X[R][kPairs], S[R][kPairs], Z[R][kPairs];   // dx = A - X mean (times S), dz = the same times Z
        float dot[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const f2 r2 = pack(rs[r], rs[r]);
            f2 acc = pack(0.f, 0.f);
            Row<T, kPairs> o;
#pragma unroll
            for (int i = 0; i < kPairs; ++i) {
                const f2 xv = widen<T>(xr[r].v[i]), gv = widen<T>(gr[r].v[i]);
                f2 sl, dsl, u = xv, dy = gv;
                if (GATE) silu_grad2(widen<T>(zr[r].v[i]), sl, dsl);
                if (GATE == 1) dy = mul2(gv, sl);
                if (GATE == 2) u = mul2(xv, sl);
                const f2 xhat = mul2(u, r2), dyw = mul2(dy, w[i]);
                acc = fma2(dyw, xhat, acc);
                dw[i] = fma2(dy, xhat, dw[i]);
                A[r][i] = mul2(dyw, r2);
                X[r][i] = mul2(xhat, r2);
                if (GATE == 1) o.v[i] = narrow<T>(mul2(mul2(mul2(gv, xhat), w[i]), dsl));
                if (GATE == 2) {
                    S[r][i] = sl;
                    Z[r][i] = mul2(xv, dsl);
                }
            }
            if (GATE == 1 && row0 + r < d.rows) put_row<T>(dz, (row0 + r) * d.sz + c0, o);
            dot[r] = hsum(acc);
        }
        if (base + step < d.rows) fetch(row0 + step);
        group_sums<R>(dot, sm + (turn * blockDim.y + threadIdx.y) * R * 16, d.group);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (row0 + r >= d.rows) continue;
            const float m = -dot[r] / (float)d.group;
            const f2 m2 = pack(m, m);
            Row<T, kPairs> o, oz;
#pragma unroll
            for (int i = 0; i < kPairs; ++i) {
                const f2 du = fma2(X[r][i], m2, A[r][i]);
                o.v[i] = narrow<T>(GATE == 2 ? mul2(du, S[r][i]) : du);
                if (GATE == 2) oz.v[i] = narrow<T>(mul2(du, Z[r][i]));
            }
            put_row<T>(dx, (row0 + r) * d.sx + c0, o);
            if (GATE == 2) put_row<T>(dz, (row0 + r) * d.sz + c0, oz);
        }
    }
    float v[kCh];
#pragma unroll
    for (int i = 0; i < kPairs; ++i) unpack(dw[i], v[2 * i], v[2 * i + 1]);
    if (blockDim.y > 1) {                                        // the block's rows of gradients are added in order
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kCh; ++i) sm[threadIdx.y * d.hidden + c0 + i] = v[i];
        __syncthreads();
        if (threadIdx.y == 0)
#pragma unroll
            for (int i = 0; i < kCh; ++i)
                for (int y = 1; y < (int)blockDim.y; ++y) v[i] += sm[y * d.hidden + c0 + i];
    }
    if (threadIdx.y == 0) {
        float4 *to = reinterpret_cast<float4 *>(dw_part + (long long)blockIdx.x * d.hidden + c0);
        to[0] = make_float4(v[0], v[1], v[2], v[3]);
        to[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
}

// dw[c] = sum over the partial rows.  grid ceil(hidden / 32).
template <class W> __global__ void __launch_bounds__(256) norm_bwd_reduce(const float *dw_part, int nparts, int hidden, void *dw) {
    pdl_begin();
    column_sums(dw_part, nparts, hidden, [=](int c, float v) { st<W>(dw, c, v); });
}

}  // namespace norm
}  // namespace bissd
