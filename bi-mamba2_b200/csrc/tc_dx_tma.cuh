// Backward, TMA-fed: the gate kernel (g = dout * silu(z), dz) and the fused dx / ddt_out / dD / "next"-term kernel.
//
// dx_tma mirrors chunk_scan_tma: B (as the A operand) and the two passed state gradients E_f / E_b arrive by TMA a dstate slab
// at a time; B.E_f^T and B.E_b^T get their own TMEM accumulators, from which the "next" decay terms nf / nb (dot
// products with the x row) and the sum weighted by e^{T-cs[l]} are taken; the transposed masked-decay product is
// accumulated on top of that sum.  Mt[l,s] = CB[s,l] ([s>l] 2^(f2[s]-f2[l]) + [s<l] 2^(b2[s]-b2[l]) + 2[s=l]) is built by the
// threads, from a transposed copy of CB; the g rows come with it in pieces of 64.  Two CTAs an SM: 113 us at
// headdim 128, dstate 256, b8 L1024 H16 chunk 128 (one: 138).
#pragma once
#include "tc_scan_tma.cuh"

namespace bissd {
namespace tc {

// g = dout * z * sigmoid(z), dz = dout * out_x * sigmoid(z) * (1 + z (1 - sigmoid(z))); 8 elements per thread.
// Takes over _chunk_scan_bwd_dz_kernel (src/ssd/bi/ssd_chunk_scan.py:357-440) except its dD partials.
template <class T>
__global__ void __launch_bounds__(256) gate_bwd(Dims d, View dout, View z, View out_x, void *g_out, void *dz, int *status) {
    pdl_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;        // the first kernel of its pass
    const long long pc = d.P / 8;
    const long long total = (long long)d.b * d.L * d.H * pc;
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    const int p0 = (int)(i % pc) * 8;
    const long long r = i / pc;
    const int h = (int)(r % d.H);
    const long long bl = r / d.H;
    const int l = (int)(bl % d.L), b = (int)(bl / d.L);
    float gv[8], zz[8], ox[8], dzv[8];
    unpack8<T>(ld8v<T>(dout, b, l, h, p0), gv);
    unpack8<T>(ld8v<T>(z, b, l, h, p0), zz);
    unpack8<T>(ld8v<T>(out_x, b, l, h, p0), ox);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float sg = __fdividef(1.f, 1.f + __expf(-zz[j]));
        dzv[j] = gv[j] * ox[j] * sg * (1.f + zz[j] * (1.f - sg));
        gv[j] *= zz[j] * sg;
    }
    const long long o = ((long long)(b * d.L + l) * d.H + h) * d.P + p0;
    *reinterpret_cast<uint4 *>(static_cast<T *>(g_out) + o) = pack8<T>(gv);
    *reinterpret_cast<uint4 *>(static_cast<T *>(dz) + o) = pack8<T>(dzv);
}

inline size_t dx_tma_smem(int P, int Q) { return 1024 + 2 * (size_t)scan_slot_bytes(P) + 2 * (size_t)Q * 4; }

// grid (b*nc*H, Q/128).  g: contiguous (b,L,H,P) gated output gradient (dout itself when there is no z).
template <class T>
__global__ void __launch_bounds__(kThreads, 2)
dx_tma(Dims d, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmEf,
       const __grid_constant__ CUtensorMap tmEb, const __grid_constant__ CUtensorMap tmG, View x, View g, const float *D,
       const float *dt_out, const float *cs_f, const float *cs_b, const float *CBt, MutView dx, float *ddt_out, float *nf,
       float *nb, float *dDpart, int *status) {
    pdl_begin();
    extern __shared__ uint8_t dyn[];
    __shared__ ScanShared sh;
    __shared__ float rowred[3][kTileM];
    __shared__ float colred[4][128];
    const int P = d.P, Q = d.Q;
    uint8_t *base_sm = smem_align1024(dyn);
    float *f2 = reinterpret_cast<float *>(base_sm + 2 * scan_slot_bytes(P)), *b2 = f2 + Q;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.x % d.H, c = (blockIdx.x / d.H) % d.nc, b = blockIdx.x / (d.H * d.nc);
    const int grp = h / d.R;
    const int lim = min(Q, d.L - c * Q);
    const int l0 = blockIdx.y * kTileM;
    const long long base = ((long long)(b * d.H + h) * d.nc + c) * Q;
    const uint32_t ncols = 2 * P;
    ScanFeed feed{sh, d, base_sm, &tmB, &tmEf, &tmEb, &tmG, b, c, h, grp, l0};
    if (warp == 0) tmem_alloc(&sh.tmem_base, ncols);
    if (tid == 32) {                                            // barriers and first loads by the same thread, before the sync
        feed.init_barriers();
        feed.start();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    const float *cbt = CBt + ((long long)(b * d.nc + c) * d.G + grp) * Q * Q;
    // the decay tables are built while the TMA loads are in flight
    for (int i = tid; i < Q; i += kThreads) {
        f2[i] = cs_f[base + i] * 1.4426950408889634f;
        b2[i] = cs_b[base + i] * 1.4426950408889634f;
    }
    __syncthreads();
    uint4 ra[4];
    float4 raw[8];                                              // CB values of the step after next, still in flight
    auto load_raw = [&](int s0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int q = tid + i * kThreads;
            const float *src = cbt + (long long)(l0 + (q >> 3)) * Q + s0 + (q & 7) * 8;
            raw[2 * i] = __ldg(reinterpret_cast<const float4 *>(src));
            raw[2 * i + 1] = __ldg(reinterpret_cast<const float4 *>(src) + 1);
        }
    };
    auto fetch = [&](int s0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int q = tid + i * kThreads;
            const int l = l0 + (q >> 3), sc = s0 + (q & 7) * 8;
            float v[8] = {raw[2 * i].x, raw[2 * i].y, raw[2 * i].z, raw[2 * i].w,
                          raw[2 * i + 1].x, raw[2 * i + 1].y, raw[2 * i + 1].z, raw[2 * i + 1].w};
            const float fl = f2[l], bl = b2[l];
            if (sc > l) {
                const float4 t0 = *reinterpret_cast<const float4 *>(f2 + sc), t1 = *reinterpret_cast<const float4 *>(f2 + sc + 4);
                const float t[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] *= ex2_approx(t[j] - fl);
            } else if (sc + 7 < l) {
                const float4 t0 = *reinterpret_cast<const float4 *>(b2 + sc), t1 = *reinterpret_cast<const float4 *>(b2 + sc + 4);
                const float t[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] *= ex2_approx(t[j] - bl);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int s = sc + j;
                    float w = ex2_approx(s >= l ? f2[s] - fl : b2[s] - bl);
                    if (s == l) w = 2.f;
                    v[j] *= w;
                }
            }
            ra[i] = pack8<T>(v);
        }
    };
    load_raw(0);
    fetch(0);
    if (kStageK < Q) load_raw(kStageK);
    const int quad = warp & 3, half = warp >> 2;
    const int r = quad * 32 + lane, l = l0 + r;                 // this thread's row, in the sums and in the epilogue
    float wf = 0.f, wb = 0.f, dl = 0.f;
    if (l < lim) {
        dl = dt_out[base + l];
        wf = __expf(cs_f[base + Q - 1] - cs_f[base + l]);
        wb = __expf(cs_b[base] - cs_b[base + l]);
    }
    float rs = 0.f, rsf = 0.f, rsb = 0.f;
    const uint32_t tl = tmem_lane_base(tmem);
    // tid 0, not elect_one, which is 1 - 7 % slower at nine shapes (us: b8 L1024 H16 dstate 256 105.5, 112, dstate 64 92.8, 98.8,
    // b4 L2048 H16 dstate 128 chunk 256 112, 119, b2 L8192 H32 dstate 64 310, 328): the kernel is at its 128 registers
    if (tid == 0) feed.products<T>(tmem);
    uint4 xr[4], gr[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) xr[q] = l < lim ? ld8v<T>(x, b, c * Q + l, h, half * 32 + q * 8) : zero8();
    bool ok = mbar_wait(&sh.st_done, 0);
    if (ok) {                                                   // dot products with x; the weighted sum replaces the first product
        tc_fence_after();
        for (int c0 = half * 32; c0 < P; c0 += 64) {
            if (c0 != half * 32) {
#pragma unroll
                for (int q = 0; q < 4; ++q) xr[q] = l < lim ? ld8v<T>(x, b, c * Q + l, h, c0 + q * 8) : zero8();
            }
#pragma unroll
            for (int q = 0; q < 32; q += 8) {
                uint32_t vf[8], vb[8];
                float y[8], xv[8];
                tmem_ld8_nowait(tl + c0 + q, vf);
                tmem_ld8_nowait(tl + P + c0 + q, vb);
                unpack8<T>(xr[q >> 3], xv);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float af = __uint_as_float(vf[j]), ab = __uint_as_float(vb[j]);
                    y[j] = fmaf(wb, ab, wf * af);
                    rsf = fmaf(af, xv[j], rsf);
                    rsb = fmaf(ab, xv[j], rsb);
                }
                tmem_st8(tl + c0 + q, y);
            }
        }
        tmem_st_wait();
        tc_fence_before();
    }
    uint32_t it = 0;
    for (int s0 = 0; s0 < Q; s0 += kStageK, ++it) {
        const int st = it & 1;
        uint8_t *stage = feed.stages() + st * kAStageBytes;
        if (it >= 2) ok = mbar_wait(&sh.free_bar[st], ((it >> 1) - 1) & 1);
        if (ok) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int q = tid + i * kThreads;
                const int rr = q >> 3, cc = q & 7;
                *reinterpret_cast<uint4 *>(stage + rr * 128 + ((cc ^ (rr & 7)) << 4)) = ra[i];
            }
            fence_async_smem();
            if (s0 + kStageK < Q) fetch(s0 + kStageK);
            if (s0 + 2 * kStageK < Q) load_raw(s0 + 2 * kStageK);
        }
        ok = __syncthreads_and(ok) && !sh.fail;
        if (!ok) {
            if (tid == 0) feed.stopped(it);
            break;
        }
        if (tid == 0) {
            tc_fence_after();
            feed.stage_product<T>(tmem, it);
        }
    }
    // epilogue operands of the first strip are requested before waiting for the last MMAs
    const int ec0 = half * 32;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        xr[q] = (ok && l < lim) ? ld8v<T>(x, b, c * Q + l, h, ec0 + q * 8) : zero8();
        gr[q] = (ok && l < lim) ? ld8v<T>(g, b, c * Q + l, h, ec0 + q * 8) : zero8();
    }
    if (ok) {
        if (tid == 0) umma_commit(&sh.done_bar);
        ok = mbar_wait(&sh.done_bar, 0);
        ok = __syncthreads_and(ok) && !sh.fail;
        tc_fence_after();
    }
    if (!ok && tid == 0) atomicExch(status, kErrMmaTimeout);
    if (ok) {
        for (int c0 = half * 32; c0 < P; c0 += 64) {
            if (c0 != ec0) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    xr[q] = (l < lim) ? ld8v<T>(x, b, c * Q + l, h, c0 + q * 8) : zero8();
                    gr[q] = (l < lim) ? ld8v<T>(g, b, c * Q + l, h, c0 + q * 8) : zero8();
                }
            }
#pragma unroll
            for (int hs = 0; hs < 2; ++hs) {                    // two 16-column pieces keep the register footprint down
                const int cc = c0 + hs * 16;
                float av[16];
                tmem_ld16(tl + cc, av);
#pragma unroll
                for (int j = 0; j < 16; j += 8) {
                    const int p0 = cc + j;
                    float xv[8], gv[8], o[8], gx[8];
                    unpack8<T>(xr[hs * 2 + (j >> 3)], xv);
                    unpack8<T>(gr[hs * 2 + (j >> 3)], gv);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float a = av[j + i];
                        o[i] = a * dl;
                        if (d.has_D) o[i] = fmaf(d.D_hdim ? D[h * P + p0 + i] : D[h], gv[i], o[i]);
                        rs = fmaf(a, xv[i], rs);
                        gx[i] = gv[i] * xv[i];
                    }
                    if (l < lim)
                        stg8_once(static_cast<T *>(dx.ptr) + b * dx.sb + (long long)(c * Q + l) * dx.sl + h * dx.sh + p0, pack8<T>(o));
                    if (d.has_D) {                              // column sums of g*x over this warp's 32 rows
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            float sgx = gx[i];
#pragma unroll
                            for (int o2 = 16; o2 > 0; o2 >>= 1) sgx += __shfl_xor_sync(0xffffffffu, sgx, o2);
                            if (lane == 0) colred[quad][p0 + i] = sgx;
                        }
                    }
                }
            }
        }
    }
    if (half == 1) {
        rowred[0][r] = rs;
        rowred[1][r] = rsf;
        rowred[2][r] = rsb;
    }
    tc_fence_before();
    __syncthreads();
    if (ok) {
        if (half == 0 && l < Q) {
            const float hrs = (P > 32) ? rowred[0][r] : 0.f, hf = (P > 32) ? rowred[1][r] : 0.f, hb = (P > 32) ? rowred[2][r] : 0.f;
            ddt_out[base + l] = rs + hrs;
            nf[base + l] = dl * wf * (rsf + hf);
            nb[base + l] = dl * wb * (rsb + hb);
        }
        if (d.has_D && tid < P)
            dDpart[(((long long)(b * d.nc + c) * d.H + h) * gridDim.y + blockIdx.y) * P + tid] =
                colred[0][tid] + colred[1][tid] + colred[2][tid] + colred[3][tid];
    }
    if (warp == 0) {
        if (!ok && tid == 0) feed.leave();
        __syncwarp();
        tmem_dealloc(tmem, ncols);
    }
}

}  // namespace tc
}  // namespace bissd
