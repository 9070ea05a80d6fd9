// C ABI of the layer around the scan: gated RMSNorm, depthwise conv1d + SiLU, per-head parameters.
#include <algorithm>

#include "common.cuh"
#include "host.cuh"
#include "conv_kernels.cuh"
#include "layer_kernels.cuh"
#include "norm_kernels.cuh"

using namespace bissd;

// ---- gated RMSNorm ---------------------------------------------------------------------------------------------
static int norm_check(const bissd_norm_args *a, norm::NormDims *d, bool backward) {
    if (!a || !a->x || !a->weight || !a->rstd) return BISSD_ERR_NULL;
    if (!backward && !a->out) return BISSD_ERR_NULL;
    if (backward && (!a->dout || !a->dx || !a->dweight || (a->z && !a->dz))) return BISSD_ERR_NULL;
    if (a->rows <= 0 || a->hidden <= 0 || a->hidden % 256 != 0 || a->hidden > 4096) return BISSD_ERR_SHAPE;
    const int group = a->group_size > 0 ? a->group_size : a->hidden;
    if (group % 256 != 0 || a->hidden % group != 0) return BISSD_ERR_SHAPE;
    if (a->x_dtype < BISSD_F32 || a->x_dtype > BISSD_F16) return BISSD_ERR_DTYPE;
    if (a->w_dtype != BISSD_F32 && a->w_dtype != a->x_dtype) return BISSD_ERR_DTYPE;
    auto al = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    if (!al(a->x) || !al(a->z) || !al(a->weight) || !al(a->out) || !al(a->dout) || !al(a->dx) || !al(a->dz))
        return BISSD_ERR_ALIGN;
    if (a->stride_x % 8 || a->stride_z % 8 || a->stride_out % 8) return BISSD_ERR_ALIGN;
    d->rows = a->rows; d->hidden = a->hidden; d->group = group; d->ngroups = a->hidden / group;
    d->sx = a->stride_x; d->sz = a->stride_z; d->so = a->stride_out;
    d->eps = a->eps;
    return BISSD_OK;
}
// hidden / 8 threads a row, rows side by side up to about 256 threads
static dim3 norm_block(int hidden) { return dim3(hidden / norm::kCh, std::max(1, 256 * norm::kCh / hidden)); }
// Persistent blocks, fewer when the rows run out first; the backward's count is also its number of partial weight-gradient rows.
static int norm_blocks(long long rows, int hidden, int rows_per_thread, int blocks_per_sm) {
    const long long step = (long long)norm_block(hidden).y * rows_per_thread;
    return (int)std::min<long long>((rows + step - 1) / step, (long long)sm_count() * std::max(1, blocks_per_sm));
}
static int norm_bwd_blocks(long long rows, int hidden) {         // 512 threads an SM: what its registers allow
    const dim3 b = norm_block(hidden);
    return norm_blocks(rows, hidden, norm::kBwdRows, 512 / (b.x * b.y));
}

template <class T, class W>
static int norm_forward_impl(const bissd_norm_args *a, const norm::NormDims &d, cudaStream_t s) {
    const dim3 block = norm_block(d.hidden);
    const size_t smem = 2 * block.y * norm::kFwdRows * 16 * sizeof(float);
    const auto kernel = !a->z ? norm::rmsnorm_gated_fwd<T, W, 0>
                              : (a->norm_before_gate ? norm::rmsnorm_gated_fwd<T, W, 1> : norm::rmsnorm_gated_fwd<T, W, 2>);
    // As many blocks as are resident, up to 1024 threads an SM: one block more than fit walks its rows when the others are done.
    // us, 768 threads an SM whatever fits, 1024 whatever fits, this: 16384 rows fp32 without z hidden 1536 34.2, 47.4, 34.0, 2048
    // 44.4, 57.8, 44.6; fp32 with z 1536 53.4, 61.5, 52.8, 2048 76.3, 62.1, 62.2; 65536 rows bf16 with z 2048 174.8, 166.6, 166.7, 4096
    // 424, 345, 345.  (Up to 1536 threads: as 1024.)
    const int threads = block.x * block.y;
    const int grid = norm_blocks(d.rows, d.hidden, norm::kFwdRows, std::min(resident_blocks(kernel, threads, smem), 1024 / threads));
    BISSD_LAUNCH("rmsnorm_gated_fwd", launch_pdl(kernel, grid, block, smem, s, d, a->x, a->z, a->weight, a->out, a->rstd));
    return BISSD_OK;
}
template <class T, class W>
static int norm_backward_impl(const bissd_norm_args *a, const norm::NormDims &d, float *part, cudaStream_t s) {
    const dim3 block = norm_block(d.hidden);
    const int grid = norm_bwd_blocks(d.rows, d.hidden);
    const size_t smem = std::max(2 * block.y * norm::kBwdRows * 16, block.y > 1 ? block.y * d.hidden : 0) * sizeof(float);
    const auto kernel = !a->z ? norm::rmsnorm_gated_bwd<T, W, 0>
                              : (a->norm_before_gate ? norm::rmsnorm_gated_bwd<T, W, 1> : norm::rmsnorm_gated_bwd<T, W, 2>);
    BISSD_LAUNCH("rmsnorm_gated_bwd", launch_pdl(kernel, grid, block, smem, s, d, a->x, a->z, a->weight, a->dout, a->rstd, a->dx,
                                                 a->dz, part));
    BISSD_LAUNCH("norm_bwd_reduce", launch_pdl(norm::norm_bwd_reduce<W>, (d.hidden + 31) / 32, 256, 0, s, part, grid, d.hidden, a->dweight));
    return BISSD_OK;
}
#define BISSD_NORM_DISPATCH(fn, ...)                                                                \
    do {                                                                                            \
        const bool wf = a->w_dtype == BISSD_F32;                                                    \
        switch (a->x_dtype) {                                                                       \
            case BISSD_F32: return fn<float, float>(__VA_ARGS__);                                   \
            case BISSD_BF16: return wf ? fn<__nv_bfloat16, float>(__VA_ARGS__) : fn<__nv_bfloat16, __nv_bfloat16>(__VA_ARGS__); \
            default: return wf ? fn<__half, float>(__VA_ARGS__) : fn<__half, __half>(__VA_ARGS__); \
        }                                                                                           \
    } while (0)


// ---- depthwise conv1d + SiLU -----------------------------------------------------------------------------------
static int conv_check(const bissd_conv_args *a, conv::ConvDims *d, bool backward) {
    if (!a || !a->x || !a->weight) return BISSD_ERR_NULL;
    if (!backward && !a->out) return BISSD_ERR_NULL;
    if (backward && (!a->dout || !a->dx || !a->dweight || (a->bias && !a->dbias))) return BISSD_ERR_NULL;
    if (a->batch <= 0 || a->seqlen <= 0 || a->channels <= 0 || a->channels % 8 != 0) return BISSD_ERR_SHAPE;
    if (a->width <= 0 || a->width > 7 || a->width % 2 == 0) return BISSD_ERR_SHAPE;
    if (a->x_dtype < BISSD_F32 || a->x_dtype > BISSD_F16) return BISSD_ERR_DTYPE;
    if (a->w_dtype != BISSD_F32 && a->w_dtype != a->x_dtype) return BISSD_ERR_DTYPE;
    auto al = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    if (!al(a->x) || !al(a->out) || !al(a->dout) || !al(a->dx) || !al(a->bias)) return BISSD_ERR_ALIGN;
    if (a->x_stride_batch % 8 || a->x_stride_row % 8 || a->out_stride_batch % 8 || a->out_stride_row % 8) return BISSD_ERR_ALIGN;
    d->batch = a->batch; d->seqlen = a->seqlen; d->channels = a->channels; d->run = d->runs = 0;
    d->xsb = a->x_stride_batch; d->xsl = a->x_stride_row; d->osb = a->out_stride_batch; d->osl = a->out_stride_row;
    d->has_bias = a->bias != nullptr;
    return BISSD_OK;
}
// Rows a thread walks: long runs share more (the backward redoes K - 1 rows of dpre per run, and writes a partial row of
// weight gradients), short ones fill the machine; halve from 256 until there are sixteen warps an SM, not below 32.
static int conv_run(int batch, int seqlen, int channels, int pairs) {
    const long long across = conv::warps_across(channels, pairs);
    int run = 256;
    while (run > 32 && across * ((seqlen + run - 1) / run) * batch < 16LL * sm_count()) run /= 2;
    return run;
}
static int conv_blocks(conv::ConvDims &d, int pairs) {
    d.run = conv_run(d.batch, d.seqlen, d.channels, pairs);
    d.runs = (d.seqlen + d.run - 1) / d.run;
    const long long warps = (long long)conv::warps_across(d.channels, pairs) * d.runs * d.batch;
    return (int)((warps + conv::kThreads / 32 - 1) / (conv::kThreads / 32));
}
#define BISSD_BY_WIDTH(width, LAUNCH)          \
    do {                                       \
        switch (width) {                       \
            case 1: LAUNCH(1); break;          \
            case 3: LAUNCH(3); break;          \
            case 5: LAUNCH(5); break;          \
            default: LAUNCH(7); break;         \
        }                                      \
    } while (0)

template <class T, class W>
static int conv_forward_impl(const bissd_conv_args *a, conv::ConvDims d, cudaStream_t s) {
    const int blocks = conv_blocks(d, conv::kFwdPairs);
#define BISSD_CONV_FWD(K)                                                                                                    \
    BISSD_LAUNCH("dwconv_silu_fwd", launch_pdl(conv::dwconv_silu_fwd<T, W, K>, blocks, conv::kThreads, \
                                               0, s, d, a->x, a->weight, a->bias, a->out))
    BISSD_BY_WIDTH(a->width, BISSD_CONV_FWD);
#undef BISSD_CONV_FWD
    return BISSD_OK;
}
template <class T, class W>
static int conv_backward_impl(const bissd_conv_args *a, conv::ConvDims d, char *ws, cudaStream_t s) {
    float *part = reinterpret_cast<float *>(ws);
    const int blocks = conv_blocks(d, conv::kBwdPairs);
#define BISSD_CONV_BWD(K)                                                                                                   \
    BISSD_LAUNCH("dwconv_silu_bwd", launch_pdl(conv::dwconv_silu_bwd<T, W, K>, blocks, conv::kThreads, 0, s, d, a->x,          \
                                               a->weight, a->bias, a->dout, a->dx, part))
    BISSD_BY_WIDTH(a->width, BISSD_CONV_BWD);
#undef BISSD_CONV_BWD
    const int cols = (a->width + 1) * d.channels;
    BISSD_LAUNCH("conv_bwd_reduce", launch_pdl(conv::conv_bwd_reduce<W>, (cols + 31) / 32, 256, 0, s, part, d.runs * d.batch,
                                               d.channels, a->width, a->dweight, a->dbias));
    return BISSD_OK;
}
#undef BISSD_BY_WIDTH

extern "C" {

int bissd_rmsnorm_gated_workspace_bytes(const bissd_norm_args *a, size_t *bwd_bytes) {
    if (!bwd_bytes) return BISSD_ERR_NULL;
    if (!a || a->rows <= 0 || a->hidden <= 0 || a->hidden % 256 != 0) return BISSD_ERR_SHAPE;
    *bwd_bytes = (size_t)norm_bwd_blocks(a->rows, a->hidden) * a->hidden * sizeof(float);
    return BISSD_OK;
}

int bissd_rmsnorm_gated_forward(const bissd_norm_args *a, void *stream) {
    norm::NormDims d;
    int rc = norm_check(a, &d, false);
    if (rc != BISSD_OK) return rc;
    rc = check_device();
    if (rc != BISSD_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    BISSD_NORM_DISPATCH(norm_forward_impl, a, d, s);
}

int bissd_rmsnorm_gated_backward(const bissd_norm_args *a, void *workspace, size_t workspace_bytes, void *stream) {
    norm::NormDims d;
    int rc = norm_check(a, &d, true);
    if (rc != BISSD_OK) return rc;
    if (!workspace) return BISSD_ERR_NULL;
    size_t need = 0;
    bissd_rmsnorm_gated_workspace_bytes(a, &need);
    if (workspace_bytes < need) return BISSD_ERR_WORKSPACE;
    rc = check_device();
    if (rc != BISSD_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float *part = static_cast<float *>(workspace);
    BISSD_NORM_DISPATCH(norm_backward_impl, a, d, part, s);
}

int bissd_dwconv_silu_workspace_bytes(const bissd_conv_args *a, size_t *bwd_bytes) {
    if (!a || !bwd_bytes) return BISSD_ERR_NULL;
    if (a->batch <= 0 || a->seqlen <= 0 || a->channels <= 0 || a->width <= 0) return BISSD_ERR_SHAPE;
    const int run = conv_run(a->batch, a->seqlen, a->channels, conv::kBwdPairs);
    *bwd_bytes = (size_t)a->batch * ((a->seqlen + run - 1) / run) * a->channels * (a->width + 1) * sizeof(float);
    return BISSD_OK;
}

int bissd_dwconv_silu_forward(const bissd_conv_args *a, void *stream) {
    conv::ConvDims d;
    int rc = conv_check(a, &d, false);
    if (rc != BISSD_OK) return rc;
    rc = check_device();
    if (rc != BISSD_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    BISSD_NORM_DISPATCH(conv_forward_impl, a, d, s);
}

int bissd_dwconv_silu_backward(const bissd_conv_args *a, void *workspace, size_t workspace_bytes, void *stream) {
    conv::ConvDims d;
    int rc = conv_check(a, &d, true);
    if (rc != BISSD_OK) return rc;
    if (!workspace) return BISSD_ERR_NULL;
    size_t need = 0;
    bissd_dwconv_silu_workspace_bytes(a, &need);
    if (workspace_bytes < need) return BISSD_ERR_WORKSPACE;
    if (a->out_stride_row != a->channels || a->out_stride_batch != (int64_t)a->seqlen * a->channels)
        return BISSD_ERR_ALIGN;                                  // dout as contiguous rows
    rc = check_device();
    if (rc != BISSD_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    BISSD_NORM_DISPATCH(conv_backward_impl, a, d, static_cast<char *>(workspace), s);
}

static int layer_params_check(const bissd_layer_params *a, bool out) {
    if (!a || !a->A32 || (!out && !a->A) || (out && (!a->dA || !a->dA32))) return BISSD_ERR_NULL;
    if (a->nheads <= 0 || a->d_elems < 0) return BISSD_ERR_SHAPE;
    for (int t : {a->a_dtype, a->d_dtype, a->b_dtype})
        if (t < BISSD_F32 || t > BISSD_F16) return BISSD_ERR_DTYPE;
    if ((a->D && !a->D32) || (a->dt_bias && !a->dt_bias32)) return BISSD_ERR_NULL;
    return check_device();
}

int bissd_layer_params_in(const bissd_layer_params *a, void *stream) {
    const int rc = layer_params_check(a, false);
    if (rc != BISSD_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    BISSD_LAUNCH("layer_params_in", layer::params_in<<<ceil_div(std::max(a->nheads, a->d_elems), 256), 256, 0, s>>>(
        a->nheads, a->d_elems, a->A, a->a_dtype, a->a_log, a->D, a->d_dtype, a->dt_bias, a->b_dtype, a->A32, a->D32, a->dt_bias32));
    return BISSD_OK;
}

int bissd_layer_params_out(const bissd_layer_params *a, void *stream) {
    const int rc = layer_params_check(a, true);
    if (rc != BISSD_OK) return rc;
    if ((a->dD && !a->dD32) || (a->ddt_bias && !a->ddt_bias32)) return BISSD_ERR_NULL;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    BISSD_LAUNCH("layer_params_out", launch_pdl(layer::params_out, ceil_div(std::max(a->nheads, a->d_elems), 256), 256, 0, s,
        a->nheads, a->d_elems, a->A32, a->dA32, a->dD32, a->ddt_bias32, a->a_log, a->dA, a->a_dtype, a->dD, a->d_dtype,
        a->ddt_bias, a->b_dtype));
    return BISSD_OK;
}

}  // extern "C"
