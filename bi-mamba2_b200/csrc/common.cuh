// Shared device/host helpers for libbissd: element types, tensor views, problem dimensions.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "../../include/bissd.h"

namespace bissd {

// Derived sizes of one call, passed by value to every kernel.
struct Dims {
    int b, L, H, P, G, N, Q, nc, R;   // R = heads per group, nc = ceil(L / Q)
    int has_D, D_hdim, has_z, has_bias, softplus;
    float dt_min, dt_max;
};

// (batch, seq, head, inner) view with contiguous inner dimension; strides in elements.
struct View {
    const void *ptr;
    long long sb, sl, sh;
};
struct MutView {
    void *ptr;
    long long sb, sl, sh;
};

__host__ __device__ inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Parts the heads of a group are summed in by the kernels that walk them (dCB, dB, dC): heads R i / S ... R (i + 1) / S of part
// i, the parts' sums then added in a fixed order.  dB and dC: blocks may share the parts or one block take them all.  dCB: a
// block of a cluster for each.  The numbers are the same, and the rule looks at one row of the batch only, so a row's results do
// not depend on how many rows there are.  One part where a row alone brings 32 tiles (b >= 5 such rows fill the chip; summing
// in parts costs one block 5 %) or the heads are few.  dCB with many rows, us: the kernel before, where one block then took all
// parts, and this one in clusters: b8 L1792 H24 143, 99; b16 L1792 276, 177; b64 L256 H24 145, 109; b16 L1500 H16 chunk 128 103, 70.
__host__ __device__ inline int head_parts(const Dims &d) {
    const int nt = ceil_div(d.Q, 128);
    return d.nc * d.G * nt * nt >= 32 ? 1 : (d.R >= 16 ? 4 : (d.R >= 8 ? 2 : 1));
}
// Partial dB / dC of a group that dbc_accum_grp writes when ks blocks share its parts: one per pair of parts, or per part.
__host__ __device__ inline int dbc_slots(const Dims &d, int ks) { const int S = head_parts(d); return ks == S ? S : S / 2; }

template <class T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }

template <class T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }

template <class T> __device__ __forceinline__ float ld(const void *p, long long i) {
    return to_f<T>(static_cast<const T *>(p)[i]);
}
template <class T> __device__ __forceinline__ void st(void *p, long long i, float v) {
    static_cast<T *>(p)[i] = from_f<T>(v);
}

// Load / store with a run-time dtype (used only for dt / ddt, which are tiny).
__device__ __forceinline__ float ld_any(const void *p, int dtype, long long i) {
    if (dtype == BISSD_F32) return static_cast<const float *>(p)[i];
    if (dtype == BISSD_BF16) return __bfloat162float(static_cast<const __nv_bfloat16 *>(p)[i]);
    return __half2float(static_cast<const __half *>(p)[i]);
}
__device__ __forceinline__ void st_any(void *p, int dtype, long long i, float v) {
    if (dtype == BISSD_F32) static_cast<float *>(p)[i] = v;
    else if (dtype == BISSD_BF16) static_cast<__nv_bfloat16 *>(p)[i] = __float2bfloat16_rn(v);
    else static_cast<__half *>(p)[i] = __float2half_rn(v);
}

// softplus with the reference's cut-over: identity above 20 (src/ssd/bi/softplus.py:8-11).
__device__ __forceinline__ float softplus_ref(float v) { return v <= 20.f ? log1pf(expf(v)) : v; }
__device__ __forceinline__ float sigmoidf_(float v) { return 1.f / (1.f + expf(-v)); }

// Sums over the warp of V values a lane, value(integral_constant<G>) the lane's G-th: lane l gets that of value l V / 32.  Each is
// added up in the order of one shuffle per distance 16, 8 ... 1, but the values are dealt to the lanes on the way: V + 4 -
// log2 V shuffles instead of 5 V, and no more than log2 V + 1 values held.
template <int V, int S, int G, class F> __device__ __forceinline__ float dealt_sums(F &value, int lane) {
    if constexpr (S == V) {
        return value(std::integral_constant<int, G>());
    } else {
        const float a = dealt_sums<V, 2 * S, G>(value, lane), b = dealt_sums<V, 2 * S, G + S>(value, lane);
        constexpr int o = 32 * S / V;
        return ((lane & o) ? b : a) + __shfl_xor_sync(0xffffffffu, (lane & o) ? a : b, o);
    }
}
template <int V, class F> __device__ __forceinline__ float warp_sums(F &value, int lane) {
    float v = dealt_sums<V, 1, 0>(value, lane);
#pragma unroll
    for (int o = 16 / V; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Programmatic dependent launch: a kernel launched with the stream-serialisation attribute may be scheduled while
// the kernel before it in the stream is still draining.  Every such kernel opens with pdl_begin(): it lets its own
// successor be scheduled early, then waits until the predecessor grid has completed and its writes are visible -
// before that point the kernel touches nothing but its parameters.  Without the attribute both are no-ops.
__device__ __forceinline__ void pdl_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace bissd
