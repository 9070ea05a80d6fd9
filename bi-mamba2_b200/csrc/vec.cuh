// Packed access and arithmetic for the element-wise kernels: pairs of channels as fp32x2 (Blackwell's fma.rn.f32x2 does
// two fp32 multiply-adds in one issue slot), and 16-byte row pieces kept as loaded until they are used.
#pragma once
#include <type_traits>

#include "common.cuh"

namespace bissd {
namespace vec {

typedef unsigned long long f2;                                   // two fp32 values, low half first

__device__ __forceinline__ f2 pack(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack(f2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// 1 / (1 + e^-v) from the hardware's 2^x and reciprocal approximations (each within 2 ulp); 0 and 1 at the ends.
__device__ __forceinline__ f2 sigmoid2(f2 v) {
    float a, b;
    unpack(mul2(v, pack(-1.44269504f, -1.44269504f)), a, b);
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(a));
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(b));
    unpack(add2(pack(a, b), pack(1.f, 1.f)), a, b);
    asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(a));
    asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(b));
    return pack(a, b);
}
// silu'(v) from s = sigmoid(v):  s (1 + v (1 - s))
__device__ __forceinline__ f2 silu_slope2(f2 v, f2 s) {
    const f2 one = pack(1.f, 1.f);
    return mul2(s, fma2(v, fma2(s, pack(-1.f, -1.f), one), one));
}

// Two adjacent elements of dtype T as they lie in memory.
template <class T> struct Pair;
template <> struct Pair<float> { using raw = float2; };
template <> struct Pair<__nv_bfloat16> { using raw = uint32_t; };
template <> struct Pair<__half> { using raw = uint32_t; };

__device__ __forceinline__ f2 widen(float2 v, float) { return pack(v.x, v.y); }
__device__ __forceinline__ f2 widen(uint32_t v, __nv_bfloat16) { return pack(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u)); }
__device__ __forceinline__ f2 widen(uint32_t v, __half) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&v));
    return pack(f.x, f.y);
}
template <class T> __device__ __forceinline__ f2 widen(typename Pair<T>::raw v) { return widen(v, T()); }

template <class T> __device__ __forceinline__ typename Pair<T>::raw narrow(f2 v) {
    float a, b;
    unpack(v, a, b);
    if constexpr (sizeof(T) == 4) {
        return make_float2(a, b);
    } else if constexpr (std::is_same<T, __half>::value) {
        const __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<const uint32_t *>(&h);
    } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t *>(&h);
    }
}

// NP adjacent pairs (NP * 2 elements), moved in the widest pieces the size allows (16 bytes at most).
template <class T, int NP> struct Row {
    typename Pair<T>::raw v[NP];
};
template <class T, int NP> __device__ __forceinline__ Row<T, NP> load_row(const T *p) {
    Row<T, NP> r;
    if constexpr (sizeof(T) == 4) {
        static_assert(NP == 1 || NP % 2 == 0, "");
        if constexpr (NP == 1) r.v[0] = __ldg(reinterpret_cast<const float2 *>(p));
#pragma unroll
        for (int i = 0; i + 1 < NP; i += 2) {
            const float4 q = __ldg(reinterpret_cast<const float4 *>(p) + i / 2);
            r.v[i] = make_float2(q.x, q.y);
            r.v[i + 1] = make_float2(q.z, q.w);
        }
    } else {
        static_assert(NP <= 2 || NP % 4 == 0, "");
        if constexpr (NP == 1) r.v[0] = __ldg(reinterpret_cast<const uint32_t *>(p));
        if constexpr (NP == 2) {
            const uint2 q = __ldg(reinterpret_cast<const uint2 *>(p));
            r.v[0] = q.x;
            r.v[1] = q.y;
        }
#pragma unroll
        for (int i = 0; i + 3 < NP; i += 4) {
            const uint4 q = __ldg(reinterpret_cast<const uint4 *>(p) + i / 4);
            r.v[i] = q.x; r.v[i + 1] = q.y; r.v[i + 2] = q.z; r.v[i + 3] = q.w;
        }
    }
    return r;
}
template <class T, int NP> __device__ __forceinline__ Row<T, NP> zero_row() {
    Row<T, NP> r;
#pragma unroll
    for (int i = 0; i < NP; ++i) r.v[i] = typename Pair<T>::raw{};
    return r;
}
template <class T, int NP> __device__ __forceinline__ void store_row(T *p, const Row<T, NP> &r) {
    if constexpr (sizeof(T) == 4) {
        if constexpr (NP == 1) *reinterpret_cast<float2 *>(p) = r.v[0];
#pragma unroll
        for (int i = 0; i + 1 < NP; i += 2)
            reinterpret_cast<float4 *>(p)[i / 2] = make_float4(r.v[i].x, r.v[i].y, r.v[i + 1].x, r.v[i + 1].y);
    } else {
        if constexpr (NP == 1) *reinterpret_cast<uint32_t *>(p) = r.v[0];
        if constexpr (NP == 2) *reinterpret_cast<uint2 *>(p) = make_uint2(r.v[0], r.v[1]);
#pragma unroll
        for (int i = 0; i + 3 < NP; i += 4) reinterpret_cast<uint4 *>(p)[i / 4] = make_uint4(r.v[i], r.v[i + 1], r.v[i + 2], r.v[i + 3]);
    }
}
template <class W> __device__ __forceinline__ f2 load_pair(const void *p, long long i) {   // two weights, any W
    return pack(ld<W>(p, i), ld<W>(p, i + 1));
}

// Sums of the columns of part[rows][cols] (fp32), a fixed order of additions whatever the number of rows: a block takes 32
// columns, its 8 warps every eighth row (the loads of four rows in flight), the eight partial sums are added in warp
// order.  One thread per column walking all rows took 12 us for 296 rows (a chain of loads); this takes 3.
// `put(column, sum)` stores.  grid ceil(cols / 32), 256 threads.
template <class F> __device__ __forceinline__ void column_sums(const float *part, int rows, int cols, F put) {
    __shared__ float red[8][33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, col = blockIdx.x * 32 + lane;
    float s4[4] = {0.f, 0.f, 0.f, 0.f};
    if (col < cols) {
        int p = warp;
        for (; p + 24 < rows; p += 32) {
#pragma unroll
            for (int u = 0; u < 4; ++u) s4[u] += part[(long long)(p + 8 * u) * cols + col];
        }
        for (; p < rows; p += 8) s4[0] += part[(long long)p * cols + col];
    }
    red[warp][lane] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
    __syncthreads();
    if (warp == 0 && col < cols) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[w][lane];
        put(col, v);
    }
}

}  // namespace vec
}  // namespace bissd
