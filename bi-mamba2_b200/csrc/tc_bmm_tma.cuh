// CB[b,c,g,l,s] = C[l].B[s] with both operands by TMA (see tc::bmm_cb for the thread-staged form and the layouts).
// One shot per CTA: a 128 x 128 tile of (l, s); the C rows and the B rows arrive as K-major tiles of dstate/64 slabs,
// one MMA chain gives the tile, a second one with the operands swapped gives the same tile of the transpose.  Outputs,
// each optional: the bf16 tile (tmO), its transpose (tmOt), CBs (fp32 in strips of 16 columns, [Q/16][Q rows][16]).
// The 16-bit tiles leave by TMA from shared memory, over C and B, which are dead by then: as per-lane row pieces, 32
// different lines per store instruction, they were most of this kernel's time (b2 L8192 G8: 51 us a launch; bound by
// the 67 or 134 MB it writes).  CB and its transpose in fp32, which the headdim 128 kernels read, are likewise turned in shared
// memory into whole rows per warp.  Rows past the end of the sequence read as zeros.
// grid (b*nc*G, Q/128, Q/128).
#pragma once
#include "tc_cumsum.cuh"
#include "tc_scan_tma.cuh"

namespace bissd {
namespace tc {

inline bool bmm_cb_tma_ok(int N, int Q) { return N % 64 == 0 && N <= 256 && (Q == 128 || Q == 256); }
constexpr int kCbRow = 132;                                      // floats a row of the fp32 tile takes in shared memory: no bank conflicts
inline size_t bmm_cb_tma_smem(int N, bool transposed, bool fp32 = false) {   // C and B, then the tile and its transpose, or an fp32 tile
    const size_t in = 2 * (size_t)(N / 64) * 16384, out = fp32 ? 128 * kCbRow * 4 : (transposed ? 65536 : 32768);
    return 1024 + (in > out ? in : out);
}

struct CbArgs {
    int plain, transposed;                                      // which 16-bit tiles
    float *CBs, *CB32, *CBt32;
};
// One tile; bx: (batch, chunk, group), row and column tile.  FP32: CB32 / CBt32 / CBs are written, not the 16-bit tiles
template <class T, bool FP32>
__device__ __forceinline__ void bmm_cb_role(const Dims &d, const CUtensorMap &tmC, const CUtensorMap &tmB, const CUtensorMap &tmO,
                                            const CUtensorMap &tmOt, const CbArgs &a, int bx, int by, int bz, int *status) {
    const bool plain = a.plain, transposed = a.transposed;
    float *CBs = a.CBs, *CB32 = a.CB32, *CBt32 = a.CBt32;
    extern __shared__ uint8_t dyn[];
    __shared__ uint64_t bar_in, bar_done, bar_drain;
    __shared__ uint32_t tmem_slot;
    const int Q = d.Q, nsl = d.N / 64;
    uint8_t *smC = smem_align1024(dyn), *smB = smC + nsl * 16384;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = bx % d.G, c = (bx / d.G) % d.nc, b = bx / (d.G * d.nc);
    const int l0 = by * kTileM, s0 = bz * 128;
    const bool two = FP32 ? CBt32 != nullptr : transposed;                       // the transpose is wanted
    const uint32_t ncols = two ? 256 : 128;
    if (warp == 0) tmem_alloc(&tmem_slot, ncols);
    if (tid == 32) {                                            // barriers and loads by the same thread, before the sync
        mbar_init(&bar_in, 1);
        mbar_init(&bar_done, 1);
        fence_mbar_init();
        mbar_expect_tx(&bar_in, (uint32_t)(2 * nsl * 16384));
        for (int j = 0; j < nsl; ++j) {
            tma_load4(smC + j * 16384, &tmC, j * 64, g, c * Q + l0, b, &bar_in);
            tma_load4(smB + j * 16384, &tmB, j * 64, g, c * Q + s0, b, &bar_in);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    bool ok = true;
    if (warp == 0 && elect_one()) {
        ok = mbar_wait(&bar_in, 0);
        if (ok) {
            tc_fence_after();
            const uint32_t idesc = instr_desc(AbFmt<T>::v, false, false, 128);
            for (int t = 0; t < (two ? 2 : 1); ++t)
                for (int j = 0; j < nsl; ++j)
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        const uint64_t dc = smem_desc(smem_u32(smC + j * 16384) + kk * 32, 16, 1024);
                        const uint64_t db = smem_desc(smem_u32(smB + j * 16384) + kk * 32, 16, 1024);
                        umma(tmem + t * 128, t ? db : dc, t ? dc : db, idesc, (j > 0 || kk > 0) ? 1u : 0u);
                    }
            umma_commit(&bar_done);
        }
    }
    if (ok) ok = mbar_wait(&bar_done, 0);
    ok = __syncthreads_and(ok);
    tc_fence_after();
    if (!ok && tid == 0) atomicExch(status, kErrMmaTimeout);
    if (ok) {
        const int r = (warp & 3) * 32 + lane, half = warp >> 2, c0 = half * 64;   // this thread: row r, columns c0 .. c0 + 63 of either tile
        const long long tile = ((long long)(b * d.nc + c) * d.G + g) * Q * Q;
        const uint32_t tl = tmem_lane_base(tmem) + c0;
        // 32 values of row r as four swizzled 16-byte pieces of slab `half` (rows of 128 bytes)
        auto stage = [&](uint8_t *slab, int hc, const float (&v)[32]) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
                const float o[8] = {v[j], v[j + 1], v[j + 2], v[j + 3], v[j + 4], v[j + 5], v[j + 6], v[j + 7]};
                *reinterpret_cast<uint4 *>(slab + r * 128 + ((((hc + j) >> 3) ^ (r & 7)) << 4)) = pack8<__nv_bfloat16>(o);
            }
        };
        auto rows_out = [&](int t, float *out) {                // accumulator t, to out[rows of Q floats]
            float *buf = reinterpret_cast<float *>(smC);
#pragma unroll
            for (int hc = 0; hc < 64; hc += 32) {
                float v[32];
                tmem_ld32(tl + t * 128 + hc, v);
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    *reinterpret_cast<float4 *>(buf + r * kCbRow + c0 + hc + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            }
            __syncthreads();
            for (int i = warp; i < 128; i += kThreads / 32)
                *reinterpret_cast<float4 *>(out + (long long)i * Q + lane * 4) = *reinterpret_cast<const float4 *>(buf + i * kCbRow + lane * 4);
            __syncthreads();
        };
        if (FP32 && CB32) rows_out(0, CB32 + tile + (long long)l0 * Q + s0);
        if (FP32 && CBt32) rows_out(1, CBt32 + tile + (long long)s0 * Q + l0);
        uint8_t *so = smC, *st = smC + 32768;                   // [2 slabs of 128 x 64]
        if (plain || CBs) {
#pragma unroll
            for (int hc = 0; hc < 64; hc += 32) {
                float v[32];
                tmem_ld32(tl + hc, v);
                const int sc = s0 + c0 + hc;                    // first of these 32 columns
                if (CBs) {
#pragma unroll
                    for (int j = 0; j < 32; j += 4)
                        *reinterpret_cast<float4 *>(CBs + tile + (long long)((sc + j) >> 4) * Q * 16 + (l0 + r) * 16 + ((sc + j) & 15)) =
                            make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                }
                if (plain) stage(so + half * 16384, hc, v);
            }
        }
        if (transposed) {
#pragma unroll
            for (int hc = 0; hc < 64; hc += 32) {
                float v[32];
                tmem_ld32(tl + 128 + hc, v);
                stage(st + half * 16384, hc, v);
            }
        }
        fence_async_smem();
        __syncthreads();
        if (tid == 0 && (plain || transposed)) {
            const int row = ((b * d.nc + c) * d.G + g) * Q;
            for (int k = 0; k < 2; ++k) {
                if (plain) tma_store2(&tmO, so + k * 16384, s0 + k * 64, row + l0);
                if (transposed) tma_store2(&tmOt, st + k * 16384, l0 + k * 64, row + s0);
            }
            tma_store_wait();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        if (!ok && elect_one()) {                               // leave nothing in flight
            drain_mmas(&bar_drain);
            drain_loads(&bar_in, 1, 1);
        }
        __syncwarp();
        tmem_dealloc(tmem, ncols);
    }
}

template <class T, bool FP32>
__global__ void __launch_bounds__(kThreads)
bmm_cb_tma(Dims d, const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmB,
           const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmOt, CbArgs a, int *status) {
    pdl_begin();
    bmm_cb_role<T, FP32>(d, tmC, tmB, tmO, tmOt, a, blockIdx.x, blockIdx.y, blockIdx.z, status);
}

// The cumulative sums and C.B^T of a forward pass in one launch: neither needs the other, and where all blocks are
// resident at once (the caller's rule) the pass is as long as its chain of launches.  The first `tiles` blocks have a C.B^T
// tile each.  The status word is cleared here; a wait that runs out reports long after.
template <class T, bool FP32, int E>
__global__ void __launch_bounds__(kThreads)
cumsum_cb(Dims d, const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmB,
          const __grid_constant__ CUtensorMap tmO, CbArgs a, CumsumFwd cs, int tiles, int *status) {
    pdl_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
    const int nt = d.Q / 128, bcg = tiles / (nt * nt), i = blockIdx.x;
    if (i < tiles) bmm_cb_role<T, FP32>(d, tmC, tmB, tmO, tmO, a, i % bcg, i / bcg % nt, i / bcg / nt, status);
    else cumsum_fwd_role<E>(d, cs, i - tiles);
}

}  // namespace tc
}  // namespace bissd
