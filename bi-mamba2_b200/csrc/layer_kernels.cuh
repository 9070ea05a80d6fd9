// The per-head parameters of a BiMamba2 layer on their way into the scan and of their gradients on the way out: one
// launch each instead of an elementwise launch per parameter and conversion (cast, exp, negate; multiply, casts), which
// on a short sequence cost as much as the scan's own small kernels.
#pragma once
#include "common.cuh"

namespace bissd {
namespace layer {

// A32 = A, or -exp(A) where the layer stores log(-A);  D32 = D;  bias32 = dt_bias.  grid ceil(max(H, nD) / 256).
__global__ void __launch_bounds__(256) params_in(int H, int nD, const void *A, int a_dtype, int a_log, const void *D, int d_dtype,
                                                 const void *bias, int b_dtype, float *A32, float *D32, float *bias32) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < H) {
        const float a = ld_any(A, a_dtype, i);
        A32[i] = a_log ? -expf(a) : a;
        if (bias) bias32[i] = ld_any(bias, b_dtype, i);
    }
    if (D && i < nD) D32[i] = ld_any(D, d_dtype, i);
}

// The gradients, in the parameters' dtypes; d(-exp(a)) / da is A itself.
__global__ void __launch_bounds__(256) params_out(int H, int nD, const float *A32, const float *dA32, const float *dD32,
                                                  const float *dbias32, int a_log, void *dA, int a_dtype, void *dD, int d_dtype,
                                                  void *dbias, int b_dtype) {
    pdl_begin();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < H) {
        st_any(dA, a_dtype, i, a_log ? dA32[i] * A32[i] : dA32[i]);
        if (dbias) st_any(dbias, b_dtype, i, dbias32[i]);
    }
    if (dD && i < nD) st_any(dD, d_dtype, i, dD32[i]);
}

}  // namespace layer
}  // namespace bissd
