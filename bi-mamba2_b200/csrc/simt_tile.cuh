// Tile machinery of the CUDA-core kernels (simt_kernels.cuh): 64 x TW output tiles, fp32 multiply-adds, operand panels of
// 64 x 64 in shared memory filled from global memory four elements at a time.
//
// A block has 256 threads.  TW (16, 32 or 64) is the width of what the tile's columns run over - headdim, dstate or
// chunk positions - so that narrow heads do not pay for 64 columns.  Panels are at most 64 deep; where several follow one
// another the next one's global loads are in flight while one is multiplied.
#pragma once
#include "common.cuh"

namespace bissd {
namespace simt {

constexpr int TB = 256;      // threads per block in every kernel of this family
constexpr int TILE = 64;     // rows of a tile, depth of a panel
constexpr int LD = TILE + 4; // floats per panel row: 16-byte rows, and the four-row reads of compute_nn hit distinct banks

__host__ __device__ inline int width_for(int n) { return n <= 16 ? 16 : (n <= 32 ? 32 : 64); }

// A finished tile: thread (ty, tx) holds TW / 16 adjacent rows and four adjacent columns.
template <int TW> struct Acc {
    static constexpr int RI = TW / 16, NTX = TW / 4;
    float v[RI][4];
    static __device__ __forceinline__ int row0() { return threadIdx.x / NTX * RI; }
    static __device__ __forceinline__ int col0() { return threadIdx.x % NTX * 4; }
};

// A tile being multiplied: 4 x 4 values per thread whatever TW, so that a shared-memory read feeds four rows or columns
// (a 16-byte read costs a warp four cycles of the shared-memory pipe even where lanes read the same bytes; with TW / 16
// rows per thread that pipe was the limit).  The 64 / TW thread groups this leaves take every (64 / TW)-th step of the
// depth; finish() adds them up.
struct Mul {
    float v[4][4];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) v[i][j] = 0.f;
    }
    __device__ __forceinline__ void step(const float (&a)[4], float4 b) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i][0] = fmaf(a[i], b.x, v[i][0]);
            v[i][1] = fmaf(a[i], b.y, v[i][1]);
            v[i][2] = fmaf(a[i], b.z, v[i][2]);
            v[i][3] = fmaf(a[i], b.w, v[i][3]);
        }
    }
};
template <int TW> struct MulAt {
    static constexpr int NG = 64 / TW, NT = TB / NG, NTX = TW / 4;
    int grp, row, col;
    __device__ __forceinline__ MulAt() {
        const int t = threadIdx.x % NT;
        grp = threadIdx.x / NT; row = t / NTX * 4; col = t % NTX * 4;
    }
};

// m += A B over kb panel steps.  A row-major: As[m][k];  B: Bs[k][n], its columns swizzled by put_transposed where SWZ.
template <int TW, bool SWZ> __device__ __forceinline__ void compute_nn(Mul &m, const float *As, const float *Bs, int kb) {
    const MulAt<TW> at;
    const float *a0 = As + at.row * LD;
#pragma unroll 2
    for (int k = at.grp * 4; k < kb; k += 4 * MulAt<TW>::NG) {
        float4 a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4 *>(a0 + i * LD + k);
        const float *b0 = Bs + k * LD + (SWZ ? at.col ^ (k & 28) : at.col);
        const float ax[4] = {a[0].x, a[1].x, a[2].x, a[3].x}, ay[4] = {a[0].y, a[1].y, a[2].y, a[3].y};
        const float az[4] = {a[0].z, a[1].z, a[2].z, a[3].z}, aw[4] = {a[0].w, a[1].w, a[2].w, a[3].w};
        m.step(ax, *reinterpret_cast<const float4 *>(b0));
        m.step(ay, *reinterpret_cast<const float4 *>(b0 + LD));
        m.step(az, *reinterpret_cast<const float4 *>(b0 + 2 * LD));
        m.step(aw, *reinterpret_cast<const float4 *>(b0 + 3 * LD));
    }
}
// The same with A stored step-major: As[k][m].
template <int TW> __device__ __forceinline__ void compute_tn(Mul &m, const float *As, const float *Bs, int kb) {
    const MulAt<TW> at;
#pragma unroll 4
    for (int k = at.grp; k < kb; k += MulAt<TW>::NG) {
        const float4 a = *reinterpret_cast<const float4 *>(As + k * LD + at.row);
        const float av[4] = {a.x, a.y, a.z, a.w};
        m.step(av, *reinterpret_cast<const float4 *>(Bs + k * LD + at.col));
    }
}
// The groups' partial tiles added in order; buf: 4096 floats that no one reads any more after the barrier.
template <int TW> __device__ __forceinline__ Acc<TW> finish(const Mul &m, float *buf) {
    Acc<TW> acc;
    if constexpr (TW == 64) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc.v[i][j] = m.v[i][j];
    } else {
        const MulAt<TW> at;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i)
            *reinterpret_cast<float4 *>(buf + (at.grp * TILE + at.row + i) * TW + at.col) = make_float4(m.v[i][0], m.v[i][1], m.v[i][2], m.v[i][3]);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < Acc<TW>::RI; ++i) {
            float4 t = *reinterpret_cast<const float4 *>(buf + (Acc<TW>::row0() + i) * TW + Acc<TW>::col0());
#pragma unroll
            for (int g = 1; g < MulAt<TW>::NG; ++g) {
                const float4 o = *reinterpret_cast<const float4 *>(buf + (g * TILE + Acc<TW>::row0() + i) * TW + Acc<TW>::col0());
                t.x += o.x; t.y += o.y; t.z += o.z; t.w += o.w;
            }
            acc.v[i][0] = t.x; acc.v[i][1] = t.y; acc.v[i][2] = t.z; acc.v[i][3] = t.w;
        }
    }
    return acc;
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
// Transposed: source row r becomes column r ^ (step & 28) of the steps c ... c + 3 - without the exclusive or the lanes of a
// warp, four steps apart, would meet in two banks.
__device__ __forceinline__ void put_transposed(const Frag &fr, int sh, float *dst) {
    pieces(sh, [&](int u, int r, int c) {
        float *to = dst + c * LD + (r ^ (c & 28));
        to[0] = fr.v[u].x;
        to[LD] = fr.v[u].y;
        to[2 * LD] = fr.v[u].z;
        to[3 * LD] = fr.v[u].w;
    });
}

// The panel loop: load(k0) fetches this thread's pieces of the panels at k0, put(k0) stores them to As / Bs,
// mul(k0, depth) multiplies.  PREFETCH: the next panel is fetched during the multiplication - for depths that usually take
// several panels; where one is the rule, the registers are better spent otherwise.
template <bool PREFETCH = true, class L, class P, class M> __device__ __forceinline__ void panels(int K, L load, P put, M mul) {
    if (PREFETCH) load(0);
    for (int k0 = 0; k0 < K; k0 += TILE) {
        if (!PREFETCH) load(k0);
        __syncthreads();                                         // the panels' last readers are done
        put(k0);
        __syncthreads();
        if (PREFETCH && k0 + TILE < K) load(k0 + TILE);
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
