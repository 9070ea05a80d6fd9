// Tile machinery of the CUDA-core kernels (simt_kernels.cuh): 64 x TW output tiles, fp32 multiply-adds, operand panels of
// 64 x 64 in shared memory filled from global memory four elements at a time.
//
// A block has 256 threads.  TW (16, 32 or 64) is the width of what the tile's columns run over - headdim, dstate or
// chunk positions - so that narrow heads do not pay for 64 columns: thread (ty, tx) holds TW / 16 adjacent rows and four
// adjacent columns.  Panels are at most 64 deep; the next panel's global loads are in flight while one is multiplied.
#pragma once
#include "common.cuh"

namespace bissd {
namespace simt {

constexpr int TB = 256;      // threads per block in every kernel of this family
constexpr int TILE = 64;     // rows of a tile, depth of a panel
constexpr int LD = TILE + 4; // floats per panel row: 16-byte rows, and the four-row reads of compute_nn hit distinct banks

__host__ __device__ inline int width_for(int n) { return n <= 16 ? 16 : (n <= 32 ? 32 : 64); }

template <int TW> struct Acc {
    static constexpr int RI = TW / 16, NTX = TW / 4;
    float v[RI][4];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) v[i][j] = 0.f;
    }
    static __device__ __forceinline__ int row0() { return threadIdx.x / NTX * RI; }
    static __device__ __forceinline__ int col0() { return threadIdx.x % NTX * 4; }
};

// acc += A B over kb panel steps.  A row-major: As[m][k];  B: Bs[k][n].
template <int TW> __device__ __forceinline__ void compute_nn(Acc<TW> &acc, const float *As, const float *Bs, int kb) {
    constexpr int RI = Acc<TW>::RI;
    const float *a0 = As + Acc<TW>::row0() * LD, *b0 = Bs + Acc<TW>::col0();
#pragma unroll 2
    for (int k = 0; k < kb; k += 4) {
        float4 a[RI];
#pragma unroll
        for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const float4 *>(a0 + i * LD + k);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 b = *reinterpret_cast<const float4 *>(b0 + (k + q) * LD);
#pragma unroll
            for (int i = 0; i < RI; ++i) {
                const float s = q == 0 ? a[i].x : (q == 1 ? a[i].y : (q == 2 ? a[i].z : a[i].w));
                acc.v[i][0] = fmaf(s, b.x, acc.v[i][0]);
                acc.v[i][1] = fmaf(s, b.y, acc.v[i][1]);
                acc.v[i][2] = fmaf(s, b.z, acc.v[i][2]);
                acc.v[i][3] = fmaf(s, b.w, acc.v[i][3]);
            }
        }
    }
}
// The same with A stored step-major: As[k][m].
template <int TW> __device__ __forceinline__ void compute_tn(Acc<TW> &acc, const float *As, const float *Bs, int kb) {
    constexpr int RI = Acc<TW>::RI;
    const float *a0 = As + Acc<TW>::row0(), *b0 = Bs + Acc<TW>::col0();
#pragma unroll 4
    for (int k = 0; k < kb; ++k) {
        float a[RI];
        if constexpr (RI == 4) {
            const float4 t = *reinterpret_cast<const float4 *>(a0 + k * LD);
            a[0] = t.x; a[1] = t.y; a[2] = t.z; a[3] = t.w;
        } else if constexpr (RI == 2) {
            const float2 t = *reinterpret_cast<const float2 *>(a0 + k * LD);
            a[0] = t.x; a[1] = t.y;
        } else {
            a[0] = a0[k * LD];
        }
        const float4 b = *reinterpret_cast<const float4 *>(b0 + k * LD);
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            acc.v[i][0] = fmaf(a[i], b.x, acc.v[i][0]);
            acc.v[i][1] = fmaf(a[i], b.y, acc.v[i][1]);
            acc.v[i][2] = fmaf(a[i], b.z, acc.v[i][2]);
            acc.v[i][3] = fmaf(a[i], b.w, acc.v[i][3]);
        }
    }
}

// Four adjacent elements as fp32; `n` of them exist (n >= 4: all).  vec: the address is aligned to the four.
template <class T> __device__ __forceinline__ float4 load4(const T *p, int n, bool vec) {
    if (vec && n >= 4) {
        if constexpr (sizeof(T) == 4) {
            return __ldg(reinterpret_cast<const float4 *>(p));
        } else {
            const uint2 u = __ldg(reinterpret_cast<const uint2 *>(p));
            const T *v = reinterpret_cast<const T *>(&u);
            return make_float4(to_f<T>(v[0]), to_f<T>(v[1]), to_f<T>(v[2]), to_f<T>(v[3]));
        }
    }
    return make_float4(n > 0 ? to_f<T>(p[0]) : 0.f, n > 1 ? to_f<T>(p[1]) : 0.f, n > 2 ? to_f<T>(p[2]) : 0.f, n > 3 ? to_f<T>(p[3]) : 0.f);
}
template <class T> __device__ __forceinline__ void store4(T *p, int n, bool vec, float4 v) {
    if (vec && n >= 4) {
        if constexpr (sizeof(T) == 4) {
            *reinterpret_cast<float4 *>(p) = v;
        } else {
            T t[4] = {from_f<T>(v.x), from_f<T>(v.y), from_f<T>(v.z), from_f<T>(v.w)};
            *reinterpret_cast<uint2 *>(p) = *reinterpret_cast<const uint2 *>(t);
        }
        return;
    }
    if (n > 0) p[0] = from_f<T>(v.x);
    if (n > 1) p[1] = from_f<T>(v.y);
    if (n > 2) p[2] = from_f<T>(v.z);
    if (n > 3) p[3] = from_f<T>(v.w);
}

// A panel on its way from global to shared memory: up to four four-element pieces per thread.  Columns are spread over
// 1 << SH pieces a row (SH = 2, 3, 4: up to 16, 32, 64 columns), so narrow panels take one or two pieces per thread.
struct Frag {
    float4 v[4];
};
__device__ __forceinline__ int shift_for(int cols) { return cols <= 16 ? 2 : (cols <= 32 ? 3 : 4); }
// Runs f(piece, row, first column) over this thread's pieces of a 64-row panel.
template <class F> __device__ __forceinline__ void pieces(int sh, F f) {
    const int nu = 1 << (sh - 2), mask = (1 << sh) - 1;
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (u < nu) {
            const int i = threadIdx.x + u * TB;
            f(u, i >> sh, (i & mask) * 4);
        }
}
// rows x cols of a matrix with unit inner stride; zero beyond.
template <class T> __device__ __forceinline__ void fetch(Frag &fr, int sh, const T *p, long long stride, int rows, int cols, bool vec) {
    pieces(sh, [&](int u, int r, int c) {
        fr.v[u] = (r < rows && c < cols) ? load4<T>(p + r * stride + c, cols - c, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
    });
}
__device__ __forceinline__ void put_rows(const Frag &fr, int sh, float *dst) {
    pieces(sh, [&](int u, int r, int c) { *reinterpret_cast<float4 *>(dst + r * LD + c) = fr.v[u]; });
}
__device__ __forceinline__ void put_transposed(const Frag &fr, int sh, float *dst) {
    pieces(sh, [&](int u, int r, int c) {
        dst[c * LD + r] = fr.v[u].x;
        dst[(c + 1) * LD + r] = fr.v[u].y;
        dst[(c + 2) * LD + r] = fr.v[u].z;
        dst[(c + 3) * LD + r] = fr.v[u].w;
    });
}
template <class F> __device__ __forceinline__ void scale(Frag &fr, int sh, F f) {   // f(row, column) multiplies
    pieces(sh, [&](int u, int r, int c) {
        fr.v[u].x *= f(r, c);
        fr.v[u].y *= f(r, c + 1);
        fr.v[u].z *= f(r, c + 2);
        fr.v[u].w *= f(r, c + 3);
    });
}

// The panel loop: load(k0) fetches this thread's pieces of the panels at k0, put(k0) stores them to As / Bs,
// mul(k0, depth) multiplies.
template <class L, class P, class M> __device__ __forceinline__ void panels(int K, L load, P put, M mul) {
    load(0);
    for (int k0 = 0; k0 < K; k0 += TILE) {
        __syncthreads();                                         // the panels' last readers are done
        put(k0);
        __syncthreads();
        if (k0 + TILE < K) load(k0 + TILE);
        mul(k0, min(TILE, K - k0));
    }
}

// sums over the threads that share a row (TW / 4 adjacent lanes)
template <int TW> __device__ __forceinline__ float row_sum(float v) {
#pragma unroll
    for (int o = TW / 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace simt
}  // namespace bissd
