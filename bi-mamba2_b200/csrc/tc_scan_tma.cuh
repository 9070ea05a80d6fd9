// Forward chunk scan, TMA-fed variant (see simt::chunk_scan for the formula).
//
// Per CTA: one (batch, chunk, head) and 128 rows l; two CTAs an SM - one tile is a chain of loads, products and sums, and the
// other CTA's work fills the waits (headdim 128, dstate 256, b8 L1024 H16 chunk 128: one CTA an SM, everything resident,
// took 129 us; 111 now).  For that the products C.S_f^T and C.S_b^T take 64 dstate columns at a time: a slot holds a slab of C and
// of both entering states, the next slab lands in the second slot meanwhile.  Both products have a TMEM accumulator; when
// they are complete their sum, weighted by e^{cs_f[l]} and e^{cs_b[l]}, replaces the first of them, and the masked-decay
// product is accumulated on top: 2 P columns of tensor memory instead of 3 P, which would round up to all of it.
// The masked-decay matrix M[l,s] = CB[l,s] Delta[s] (L_f + L_b)[l,s] is built by the threads, 64 columns at a time, in two stage
// buffers in the slot of the last slab; the x rows of the same 64 columns come by TMA into the other slot, two
// pieces in turn.  M is evaluated in the log2 domain with per-column tables tf[s] = cs_f[s] log2e - log2 Delta[s] (tb
// likewise): M = CB * 2^(f2[l] - tf[s]) below the diagonal, CB * 2^(b2[l] - tb[s]) above it, twice that on it.
//
// Shapes: headdim 64 or 128, dstate a multiple of 64 up to 256, chunk 128 or 256.
#pragma once
#include "tc_kernels.cuh"
#include "tc_tma.cuh"

namespace bissd {
namespace tc {

struct ScanShared {
    uint64_t full[2], read[2], x_full[2], st_done, free_bar[2], done_bar;   // full / read: a slot has landed / its MMAs are done
    uint64_t drain_bar;
    uint32_t tmem_base;
    int fail;                                                   // where a wait ran out, as tile_asked reads it
};
__host__ __device__ constexpr int scan_slot_bytes(int P) { return 16384 + 2 * P * 128; }   // [128 x 64] of C, [P x 64] of either state
inline size_t scan_tma_smem(int P, int Q) { return 1024 + 2 * (size_t)scan_slot_bytes(P) + 4 * (size_t)Q * 4; }
inline bool scan_tma_ok(int P, int N, int Q) { return (P == 64 || P == 128) && N % 64 == 0 && N <= 256 && (Q == 128 || Q == 256); }

// The loads and products of one tile, for chunk_scan_tma, dx_tma and prev_terms_tma (which needs no x: mX null); one thread.
struct ScanFeed {
    ScanShared &sh;
    const Dims &d;
    uint8_t *base_sm;
    const CUtensorMap *mA, *mSf, *mSb, *mX;                     // rows (C or B), both states, x or g in boxes of 64 rows
    int b, c, h, grp, l0;
    __device__ __forceinline__ void init_barriers() {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.full[i], 1);
            mbar_init(&sh.read[i], 1);
            mbar_init(&sh.x_full[i], 1);
            mbar_init(&sh.free_bar[i], 1);
        }
        mbar_init(&sh.st_done, 1);
        mbar_init(&sh.done_bar, 1);
        sh.fail = 0;
        fence_mbar_init();
    }
    // Nothing is left in flight by a kernel that gives up: `stopped` notes the stage before which it did, unless a wait of this
    // thread was first, `leave` waits.  Both by the thread that issues the MMAs.  What has been asked for follows from `fail`: kept
    // in shared memory from the first load on, a training pass took 649 us, this way 647 (b8 L1024 H16 P128 N256).
    __device__ __forceinline__ void stopped(int it) {
        if (!sh.fail) sh.fail = kStages + it;
    }
    __device__ __forceinline__ void leave() {
        const Asked asked = tile_asked(sh.fail, d.N / 64, mX ? d.Q / 64 : 0);
        drain_mmas(&sh.drain_bar);
        drain_loads(sh.full, 2, asked.slabs);
        drain_loads(sh.x_full, 2, asked.pieces);
    }
    __device__ __forceinline__ uint8_t *slot(int k) { return base_sm + (k & 1) * scan_slot_bytes(d.P); }
    __device__ __forceinline__ uint8_t *stages() { return slot(d.N / 64 - 1); }   // two M stages, over the last slab
    __device__ __forceinline__ uint8_t *x_piece(int i) { return slot(d.N / 64) + (i & 1) * d.P * 128; }
    __device__ __forceinline__ void load_slab(int k) {
        const int P = d.P, n0 = k * 64, row = ((b * d.nc + c) * d.H + h) * P;
        uint8_t *dst = slot(k);
        mbar_expect_tx(&sh.full[k & 1], (uint32_t)scan_slot_bytes(P));
        tma_load4(dst, mA, n0, grp, c * d.Q + l0, b, &sh.full[k & 1]);
        tma_load2(dst + 16384, mSf, n0, row, &sh.full[k & 1]);
        tma_load2(dst + 16384 + P * 128, mSb, n0, row, &sh.full[k & 1]);
    }
    __device__ __forceinline__ void load_x(int i) {             // rows 64 i ... of the chunk
        if (!mX) return;
        mbar_expect_tx(&sh.x_full[i & 1], (uint32_t)(d.P * 128));
        for (int j = 0; j < d.P / 64; ++j) tma_load4(x_piece(i) + j * 8192, mX, j * 64, h, c * d.Q + i * 64, b, &sh.x_full[i & 1]);
    }
    __device__ __forceinline__ void start() {
        load_slab(0);
        if (d.N > 64) load_slab(1);
        else { load_x(0); load_x(1); }
    }
    template <class T> __device__ __forceinline__ void products(uint32_t tmem) {
        const int P = d.P, ns = d.N / 64;
        const uint32_t idesc = instr_desc(AbFmt<T>::v, false, false, P);
        for (int k = 0; k < ns; ++k) {
            if (!mbar_wait(&sh.full[k & 1], (k >> 1) & 1)) { sh.fail = 1 + k; return; }
            tc_fence_after();
            const uint32_t sa = smem_u32(slot(k));
            for (int dir = 0; dir < 2; ++dir)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    umma(tmem + dir * P, smem_desc(sa + kk * 32, 16, 1024), smem_desc(sa + 16384 + dir * P * 128 + kk * 32, 16, 1024),
                         idesc, (k > 0 || kk > 0) ? 1u : 0u);
            umma_commit(k + 1 < ns ? &sh.read[k & 1] : &sh.st_done);
            if (k >= 1) {                                       // slab k - 1 has been read: its slot takes slab k + 1, or x
                if (!mbar_wait(&sh.read[(k - 1) & 1], ((k - 1) >> 1) & 1)) { sh.fail = 1 + k; return; }
                if (k + 1 < ns) load_slab(k + 1);
                else { load_x(0); load_x(1); }
            }
        }
    }
    // M stage `it` is in place: its product with the x rows of the same columns, on top of the accumulator
    template <class T> __device__ __forceinline__ void stage_product(uint32_t tmem, int it) {
        if (it >= 2) load_x(it);                                // the stage's buffers, x included, were free before it was built
        if (!mbar_wait(&sh.x_full[it & 1], (it >> 1) & 1)) { sh.fail = kStages + it + 1; return; }
        tc_fence_after();
        const uint32_t idesc = instr_desc(AbFmt<T>::v, false, true, d.P);
        const uint32_t sa = smem_u32(stages() + (it & 1) * kAStageBytes), sx = smem_u32(x_piece(it));
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
            umma(tmem, smem_desc(sa + kk * 32, 16, 1024), smem_desc(sx + kk * 16 * 128, 8192, 1024), idesc, 1u);
        umma_commit(&sh.free_bar[it & 1]);
    }
};

template <class T>
__global__ void __launch_bounds__(kThreads, 2)
chunk_scan_tma(Dims d, const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmSf,
               const __grid_constant__ CUtensorMap tmSb, const __grid_constant__ CUtensorMap tmX, View x, View z,
               const float *D, const float *dt_out, const float *cs_f, const float *cs_b, const float *CB, MutView out,
               MutView out_x, int *status) {
    pdl_begin();
    extern __shared__ uint8_t dyn[];
    __shared__ ScanShared sh;
    const int P = d.P, Q = d.Q;
    uint8_t *base_sm = smem_align1024(dyn);
    float *f2 = reinterpret_cast<float *>(base_sm + 2 * scan_slot_bytes(P)), *b2 = f2 + Q, *tf = b2 + Q, *tb = tf + Q;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.x % d.H, c = (blockIdx.x / d.H) % d.nc, b = blockIdx.x / (d.H * d.nc);
    const int g = h / d.R;
    const int lim = min(Q, d.L - c * Q);
    const int l0 = blockIdx.y * kTileM;
    const long long base = ((long long)(b * d.H + h) * d.nc + c) * Q;
    const uint32_t ncols = 2 * P;
    ScanFeed feed{sh, d, base_sm, &tmC, &tmSf, &tmSb, &tmX, b, c, h, g, l0};
    if (warp == 0) tmem_alloc(&sh.tmem_base, ncols);
    if (tid == 32) {                                            // barriers and first loads by the same thread, before the sync
        feed.init_barriers();
        feed.start();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    const float *cbt = CB + ((long long)(b * d.nc + c) * d.G + g) * Q * Q;
    // the decay tables are built while the TMA loads are in flight
    for (int i = tid; i < Q; i += kThreads) {
        const float cf = cs_f[base + i] * 1.4426950408889634f, cb_ = cs_b[base + i] * 1.4426950408889634f;
        const float lg = __log2f(dt_out[base + i]);           // -inf for the zero-padded tail: those columns vanish
        f2[i] = cf;
        b2[i] = cb_;
        tf[i] = cf - lg;
        tb[i] = cb_ - lg;
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
    auto fetch = [&](int s0) {                                  // this thread's four 8-column pieces of M[:, s0:s0+64]
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int q = tid + i * kThreads;
            const int l = l0 + (q >> 3), sc = s0 + (q & 7) * 8;
            float v[8] = {raw[2 * i].x, raw[2 * i].y, raw[2 * i].z, raw[2 * i].w,
                          raw[2 * i + 1].x, raw[2 * i + 1].y, raw[2 * i + 1].z, raw[2 * i + 1].w};
            const float fl = f2[l], bl = b2[l];
            if (sc + 7 < l) {
                const float4 t0 = *reinterpret_cast<const float4 *>(tf + sc), t1 = *reinterpret_cast<const float4 *>(tf + sc + 4);
                const float t[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] *= ex2_approx(fl - t[j]);
            } else if (sc > l) {
                const float4 t0 = *reinterpret_cast<const float4 *>(tb + sc), t1 = *reinterpret_cast<const float4 *>(tb + sc + 4);
                const float t[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] *= ex2_approx(bl - t[j]);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int s = sc + j;
                    float w = ex2_approx(s <= l ? fl - tf[s] : bl - tb[s]);
                    if (s == l) w *= 2.f;
                    v[j] *= w;
                }
            }
            ra[i] = pack8<T>(v);
        }
    };
    load_raw(0);
    fetch(0);
    if (kStageK < Q) load_raw(kStageK);
    const int l = l0 + (warp & 3) * 32 + lane;                  // this thread's row, in the sums and in the epilogue
    const float ef = l < lim ? __expf(cs_f[base + l]) : 0.f, eb = l < lim ? __expf(cs_b[base + l]) : 0.f;
    const uint32_t tl = tmem_lane_base(tmem);
    if (warp == 0 && elect_one()) feed.products<T>(tmem);
    bool ok = mbar_wait(&sh.st_done, 0);
    if (ok) {                                                   // the weighted sum of both products replaces the first
        tc_fence_after();
        for (int c0 = (warp >> 2) * 32; c0 < P; c0 += 64)
#pragma unroll
            for (int q = 0; q < 32; q += 8) {
                uint32_t vf[8], vb[8];
                float y[8];
                tmem_ld8_nowait(tl + c0 + q, vf);
                tmem_ld8_nowait(tl + P + c0 + q, vb);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j) y[j] = fmaf(eb, __uint_as_float(vb[j]), ef * __uint_as_float(vf[j]));
                tmem_st8(tl + c0 + q, y);
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
                const int r = q >> 3, cc = q & 7;
                *reinterpret_cast<uint4 *>(stage + r * 128 + ((cc ^ (r & 7)) << 4)) = ra[i];
            }
            fence_async_smem();
            if (s0 + kStageK < Q) fetch(s0 + kStageK);
            if (s0 + 2 * kStageK < Q) load_raw(s0 + 2 * kStageK);
        }
        ok = __syncthreads_and(ok) && !sh.fail;
        if (!ok) {
            if (warp == 0 && elect_one()) feed.stopped(it);
            break;
        }
        if (warp == 0 && elect_one()) {
            tc_fence_after();
            feed.stage_product<T>(tmem, it);
        }
    }
    // epilogue operands of the first strip are requested before waiting for the last MMAs
    const int ec0 = (warp >> 2) * 32;
    uint4 xr[4], zr[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        xr[q] = (ok && l < lim && d.has_D && ec0 < P) ? ld8v<T>(x, b, c * Q + l, h, ec0 + q * 8) : zero8();
        zr[q] = (ok && l < lim && d.has_z && ec0 < P) ? ld8v<T>(z, b, c * Q + l, h, ec0 + q * 8) : zero8();
    }
    if (ok) {
        if (warp == 0 && elect_one()) umma_commit(&sh.done_bar);
        ok = mbar_wait(&sh.done_bar, 0);
        ok = __syncthreads_and(ok) && !sh.fail;
        tc_fence_after();
    }
    if (!ok && tid == 0) atomicExch(status, kErrMmaTimeout);
    if (ok) {
        for (int c0 = (warp >> 2) * 32; c0 < P; c0 += 64) {
            // all global operands of this strip are requested before anything is consumed: one round trip, not eight
            if (c0 != ec0) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    xr[q] = (l < lim && d.has_D) ? ld8v<T>(x, b, c * Q + l, h, c0 + q * 8) : zero8();
                    zr[q] = (l < lim && d.has_z) ? ld8v<T>(z, b, c * Q + l, h, c0 + q * 8) : zero8();
                }
            }
            float y[32];
            tmem_ld32(tl + c0, y);
            if (l < lim) {
#pragma unroll
                for (int j = 0; j < 32; j += 8) {
                    const int p0 = c0 + j;
                    float o[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) o[i] = y[j + i];
                    if (d.has_D) {
                        float xv[8];
                        unpack8<T>(xr[j >> 3], xv);
#pragma unroll
                        for (int i = 0; i < 8; ++i) o[i] = fmaf(d.D_hdim ? D[h * P + p0 + i] : D[h], xv[i], o[i]);
                    }
                    const long long oo = b * out.sb + (long long)(c * Q + l) * out.sl + h * out.sh + p0;
                    if (d.has_z) {
                        const long long ox = b * out_x.sb + (long long)(c * Q + l) * out_x.sl + h * out_x.sh + p0;
                        stg8_once(static_cast<T *>(out_x.ptr) + ox, pack8<T>(o));
                        float zz[8];
                        unpack8<T>(zr[j >> 3], zz);
#pragma unroll
                        for (int i = 0; i < 8; ++i) o[i] *= __fdividef(zz[i], 1.f + __expf(-zz[i]));
                    }
                    stg8_once(static_cast<T *>(out.ptr) + oo, pack8<T>(o));
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        if (!ok && elect_one()) feed.leave();
        __syncwarp();
        tmem_dealloc(tmem, ncols);
    }
}

}  // namespace tc
}  // namespace bissd
