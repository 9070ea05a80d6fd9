// dCB and the intra-chunk decay gradients from ONE product per head: a CTA walks the heads of a group.
//
// Both quantities start from G2_h = g_h x_h^T and the same masked decay weights
//     w_h[l,s] = Delta_h[s] ([s<l] e^{cs_f[l]-cs_f[s]} + [s>l] e^{cs_b[l]-cs_b[s]}),   2 Delta_h[l] on the diagonal:
//     dCB[l,s]   = sum_{h in group} G2_h[l,s] w_h[l,s]                       (see simt::dcb_kernel)
//     V_h[l,s]   = G2_h[l,s] w_h[l,s] CB[l,s]  for s != l,  0 on the diagonal
//     u_f[j] = (column sum - row sum) of the part of V_h below the diagonal, u_b[j] the same above it - the
//     differences of the two dominance sums the decay gradient needs (derivation in tc_intra_sums.cuh; cumsum_bwd
//     scans them).
// One CTA per (batch, chunk, group) and 128 x 128 tile of (l, s), two CTAs per SM, the bf16 C.B^T tile resident:
//
//   warps 0-7   weight: a thread owns a row and 64 columns (four strips of 16), reads G2 from tensor memory, adds G2 w to
//               the dCB tile it keeps in registers and writes V as bf16 to shared memory
//   warps 8-11  everything else: the factor tables of the head after next, the read-out of the row and column sums, u_f and
//               u_b; one lane of warp 8 issues the sums' MMAs, one of warp 9 the loads (g and x by TMA) and G2
//
// G2 has two buffers in tensor memory, so the product of head h+1 runs while head h is weighted; V takes the place of the
// g and x it was made from, so that no weighting warp waits for the sums of the head before.  Row and column sums of V
// are products with marks of the positions 16 k ... 16 k + 15 (V as it lies is K-major for the row sums and MN-major for the
// column sums): sums per block of 16, eight of each a lane, sixteen columns over the dead G2 of the same head.  Both are
// sums of the same bf16-rounded values, so that rows and columns telescope exactly.  In a tile on the diagonal the block
// that the diagonal crosses is split by warps 8-11 from V itself.
//
// Weights are row x column factors around a strip's end column; a strip the diagonal crosses pays one ex2 per element.
// There the diagonal counts once in each direction: its weight is doubled once, at the end.  With few tiles a row the heads of
// a group are summed in parts (head_parts), one CTA of a cluster each; they add their dCB tiles through distributed
// shared memory.  (One CTA for all parts, as blocks enough for the chip used to have it, needs the columns of the second G2.)
//
// Bound by instruction issue: about 6900 warp instructions a tile and head, issue slots 54 % busy with two CTAs an SM, and
// by the registers of the weighting warps (64 of 104 hold the tile; at 168 the same code takes 5500 instructions).  us, all
// heads' loads, products, weighting and sums in one chain (256 threads, a triangular ones matrix for the column
// sums) and this form: b8 L2048 H24 136, 84; b2 L8192 H32 G8 194, 142; b16 L4096 H32 dstate 64 732, 441.
// Tried: V in a buffer of its own (106: the weighting warps wait for the sums), the MMAs behind `lane == 0` instead of
// elect_one (1250 cycles for sixteen of them, now 730), strips of 16 columns a load (spills), the next columns of G2 read ahead
// (88: more registers than there are), 96 and 48 registers (91), the warp's number made uniform by a shuffle (90), and, before
// this form, a 128 x Q tile per CTA with sixteen warps (183).
//
// A weight of a strip that the diagonal crosses is one ex2 where that form had a row and a column factor, so that some V round to
// another bf16 value: gradients move by 1e-4 and are no further from fp64 (means over 32 sizes, three seeds each, bf16: dA 2.674e-3,
// 2.671e-3, ddt 2.173e-3 both, dB 2.568e-3 both; fp16: dA 2.288e-3, 2.281e-3, ddt 1.686e-3, dB 3.215e-4 both).
//
// Every blocking point is a bounded mbarrier wait, ids 91-97 in the status word.
//
// Shapes: headdim 64, chunk 128 or 256, 16-bit inputs.
#pragma once
#include "tc_scan_tma.cuh"
#include "vec.cuh"

namespace bissd {
namespace tc {

constexpr int kIntraWorkWarps = 8, kIntraHelpWarps = 4;
constexpr int kIntraTileThreads = 32 * (kIntraWorkWarps + kIntraHelpWarps);
// Registers: 80 a thread at launch (two CTAs of 384 threads), dealt anew as 104 for the weighting warps - 64 of them hold the
// dCB tile - and 32 for the others: 256 * 104 + 128 * 32 = 384 * 80, no more than the CTA was launched with.
constexpr int kIntraWorkRegs = 104, kIntraHelpRegs = 32, kIntraLaunchRegs = 80;
static_assert(32 * (kIntraWorkWarps * kIntraWorkRegs + kIntraHelpWarps * kIntraHelpRegs) <= kIntraTileThreads * kIntraLaunchRegs, "");

// Factors of one head.  Logarithms to base 2.
struct IntraTab {
    float row_f[kTileM], row_b[kTileM];                         // cumulative sums at the tile's rows
    float col_f[kTileM], col_b[kTileM];                         // column factors around the strip's last / first column
    float2 both[kTileM];                                        // cumulative sums less log Delta, forward and reverse
    float ref_f[8], ref_b[8];                                   // cumulative sums at the strips' last / first columns
};
struct IntraGrpShared {
    uint64_t cb_full, v_read, read_done;
    // One per buffer where a role may be a whole head ahead of another that waits: a single barrier could then be two phases on,
    // which a parity wait cannot tell from "not yet".  Two heads ahead nobody gets: G2 of head h + 2 waits for all of head h.
    uint64_t in_full[2], ready[2], v_full[2], sums_full[2], fin_bar[2];   // ready: G2 and the tables
    uint32_t tmem_base;
    int fail;
};

constexpr uint32_t kIntraMarkBytes = 2 * 24 * 128;
inline size_t intra_tile_smem() { return 1024 + 3 * 32768 + kIntraMarkBytes + 2 * sizeof(IntraTab); }
inline bool intra_tile_ok(int P, int Q) { return P == 64 && (Q == 128 || Q == 256); }

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster(uint32_t smem_addr, int rank) {   // 16 bytes at the same address of another block
    uint32_t at;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}

// Shared memory by 32-bit address: registers are short in the weighting warps.
__device__ __forceinline__ uint4 lds16(uint32_t at) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at));
    return v;
}
__device__ __forceinline__ float lds4(uint32_t at) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at));
    return v;
}
__device__ __forceinline__ float lds_bf16(uint32_t at) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(at));
    return __uint_as_float((uint32_t)v << 16);
}
__device__ __forceinline__ void sts4(uint32_t at, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory"); }
__device__ __forceinline__ void sts8(uint32_t at, float a, float b) { asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(at), "f"(a), "f"(b) : "memory"); }
__device__ __forceinline__ void lds_pairs(uint32_t at, vec::f2 &a, vec::f2 &b) { asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(at)); }
__device__ __forceinline__ void sts16(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// The weighting warps (warp = 0..7).  acc: this thread's piece of the dCB tile, the 16 columns of strips chalf, 2 + chalf, 4 + chalf,
// 6 + chalf: dealt alternately, so that in a tile on the diagonal each warp has one of the strips the diagonal crosses.
// cb: shared address of C.B^T, the two buffers of g and x (and V) behind it; g2: this warp's lanes of the G2 buffers.
__device__ __forceinline__ bool intra_weight(IntraGrpShared &sh, uint32_t tabs, uint32_t cb, uint32_t g2,
                                             int nh, int diag, bool below, bool row_on, int warp, int lane, vec::f2 (&acc)[32]) {
    using namespace vec;
    volatile int *fail = &sh.fail;
    const int quad = warp & 3, chalf = warp >> 2, r = quad * 32 + lane;
    const uint32_t own = cb + r * 128 + ((chalf << 5) ^ ((r & 7) << 4));   // the row's first columns of C.B^T
    const int mixed = diag ? quad : -1, edge = diag ? quad : below ? 4 : 0;   // the strip the diagonal crosses; those left of it
    if (!ws_wait_warp(&sh.cb_full, 0, fail, 91)) return false;
    if (diag && chalf == ((r >> 4) & 1))                          // V has no diagonal: the one thread that reads C.B^T[r, r] clears it
        asm volatile("st.shared.u16 [%0], %1;" ::"r"(cb + (r >> 6) * 16384 + r * 128 + ((((r & 63) >> 3) ^ (r & 7)) << 4) + (r & 7) * 2), "h"((short)0) : "memory");
#pragma unroll 1
    for (int h = 0; h < nh; ++h) {
        const uint32_t t = tabs + (h & 1) * (uint32_t)sizeof(IntraTab);
        if (!ws_wait_warp(&sh.ready[h & 1], (h >> 1) & 1, fail, 92)) return false;
        tc_fence_after();
        const float fl = lds4(t + offsetof(IntraTab, row_f) + r * 4), bl = lds4(t + offsetof(IntraTab, row_b) + r * 4);
        const uint32_t g2h = g2 + (h & 1) * 128 + chalf * 16;
        const f2 flbl = pack(fl, bl);
        float rfac = 0.f;
        const uint32_t tc = t + chalf * 64, vo = 32768 + (h & 1) * 32768;
#pragma unroll
        for (int u = 0; u < 8; ++u) {                             // half a strip: 8 columns, the next half on its way
            const int i = u >> 1, p = u & 1;                      // strip 2 i + chalf
            const uint32_t at = (own ^ ((i & 1) * 64 + p * 16)) + (i >> 1) * 16384, ct = (i * 32 + p * 8) * 4;
            const uint4 c4 = lds16(at);
            const uint32_t cw[4] = {c4.x, c4.y, c4.z, c4.w};
            uint32_t v[8], q[4];
            tmem_ld8_nowait(g2h + i * 32 + p * 8, v);
            auto weigh = [&](int j, f2 w) {                       // columns 2 j and 2 j + 1
                const f2 tj = mul2(pack(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), w);
                acc[u * 4 + j] = add2(acc[u * 4 + j], tj);
                q[j] = narrow<__nv_bfloat16>(mul2(tj, widen<__nv_bfloat16>(cw[j])));
            };
            if (i != mixed) {                                    // a strip on one side of the diagonal: row factor x column factor
                const bool fwd = i < edge;
                const uint32_t col = tc + (fwd ? offsetof(IntraTab, col_f) : offsetof(IntraTab, col_b)) + ct;
                if (p == 0) rfac = row_on ? ex2_approx((fwd ? fl : bl) - lds4(t + chalf * 4 + (fwd ? offsetof(IntraTab, ref_f) : offsetof(IntraTab, ref_b)) + i * 8)) : 0.f;
                const f2 rf2 = pack(rfac, rfac);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    f2 ca, cb2;
                    lds_pairs(col + 16 * j, ca, cb2);
                    weigh(2 * j, mul2(ca, rf2));
                    weigh(2 * j + 1, mul2(cb2, rf2));
                }
            } else {                                             // the strip the diagonal crosses: one ex2 per element
                const uint32_t eb = t + offsetof(IntraTab, both) + chalf * 128 + ct * 2;
                const int k = lane - chalf * 16 - p * 8;          // this row's position among the columns
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    f2 ea, ec;
                    lds_pairs(eb + 16 * j, ea, ec);
                    float fa, ba, fc, bc;
                    unpack(fma2(ea, pack(-1.f, -1.f), flbl), fa, ba);
                    unpack(fma2(ec, pack(-1.f, -1.f), flbl), fc, bc);
                    weigh(j, pack(ex2_approx(2 * j <= k ? fa : ba), ex2_approx(2 * j + 1 <= k ? fc : bc)));
                }
            }
            sts16(at + vo, q[0], q[1], q[2], q[3]);
        }
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.v_full[h & 1]);
    }
    return true;
}

// grid (b nc G ks, Q / 128, Q / 128), clusters of ks = head_parts blocks along x.
template <class T>
__global__ void __launch_bounds__(kIntraTileThreads, 2)
intra_dcb_tile(Dims d, const __grid_constant__ CUtensorMap tmG, const __grid_constant__ CUtensorMap tmX,
               const __grid_constant__ CUtensorMap tmCB, const float *dt_out, const float *cs_f, const float *cs_b,
               float *u4, long long hq, void *dCB16, int ks, int *status) {
    pdl_begin();
    extern __shared__ uint8_t dyn[];
    __shared__ IntraGrpShared sh;
    const int Q = d.Q, part = blockIdx.x % ks, bx = blockIdx.x / ks;
    uint8_t *base_sm = smem_align1024(dyn);
    uint8_t *smCB = base_sm;                                      // two slabs [128 x 64] bf16, K-major
    uint8_t *smIn = smCB + 32768;                                 // two buffers: g and x [128 x 64], K-major; then V of that head,
    uint8_t *smT = smIn + 65536;                                  // two slabs [128 rows x 64 columns] bf16; the blocks' marks: two
    IntraTab *tabs = reinterpret_cast<IntraTab *>(smT + kIntraMarkBytes);   // slabs [24 x 64] bf16, K-major; the tables
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = bx % d.G, c = (bx / d.G) % d.nc, b = bx / (d.G * d.nc);
    // Launch order (x, then y, then z) puts the tiles on the diagonal first: they carry the dearer strips, and the
    // second CTA an SM receives is then mostly one off the diagonal.
    const int ty = blockIdx.y ^ blockIdx.z, tz = blockIdx.y;
    const int l0 = ty * kTileM, s0 = tz * kTileM;
    const int h0 = g * d.R + d.R * part / ks, nh = d.R * (part + 1) / ks - d.R * part / ks;
    const int lim = min(Q, d.L - c * Q);
    volatile int *fail = &sh.fail;
    if (warp == 0) tmem_alloc(&sh.tmem_base, 256);
    if (tid == 32) {
        mbar_init(&sh.cb_full, 1);
        mbar_init(&sh.v_read, kIntraHelpWarps);
        mbar_init(&sh.read_done, kIntraHelpWarps);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.v_full[i], kIntraWorkWarps);
            mbar_init(&sh.sums_full[i], 1);
            mbar_init(&sh.in_full[i], 1);
            mbar_init(&sh.fin_bar[i], 1);
            mbar_init(&sh.ready[i], kIntraHelpWarps + 1);
        }
        sh.fail = 0;
        fence_mbar_init();
    }
    for (int i = tid; i < 1536; i += kIntraTileThreads) {         // marks: element (8 + n, k) is one where k / 16 = n, n < 8
        const int slab = i >= 768, n = ((i - slab * 768) >> 5) - 8, k = slab * 64 + (i & 31) * 2;
        *reinterpret_cast<uint32_t *>(smT + slab * 3072 + (n + 8) * 128 + (((((k & 63) >> 3) ^ (n & 7)) << 4) | ((k & 7) * 2))) = (k >> 4) == n ? 0x3F803F80u : 0u;
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    // The two kinds of warps do not meet in common code again: each has its own number of registers.
    if (warp < kIntraWorkWarps) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kIntraWorkRegs));
        const int quad = warp & 3, chalf = warp >> 2, r = quad * 32 + lane;
        vec::f2 acc[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = 0ull;
        const bool ok = intra_weight(sh, smem_u32(tabs), smem_u32(smCB), tmem_lane_base(tmem), nh, ty == tz, ty > tz, l0 + r < lim, warp, lane, acc);
        tc_fence_before();
        __syncthreads();
        if (ty == tz) {                                           // the diagonal counts once per direction in dCB; its weight so far: once
#pragma unroll
            for (int q = 0; q < 32; ++q) {
                const int col = ((q >> 3) * 2 + chalf) * 16 + (q & 7) * 2;
                acc[q] = vec::mul2(acc[q], vec::pack(col == r ? 2.f : 1.f, col + 1 == r ? 2.f : 1.f));
            }
        }
        if (warp == 0) {
            tmem_dealloc(tmem, 256);
            if (sh.fail && lane == 0) atomicExch(status, kErrWsWait + sh.fail);
        }
        if (ks > 1) {
            // The cluster's blocks hold partial sums of the same tile.  Each puts its own into its shared memory in fp32 (over
            // C.B^T, g and x, all dead; 16-byte pieces swizzled by row), then adds up 128 / ks rows over the cluster.
            float4 *mine = reinterpret_cast<float4 *>(base_sm);
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const int col = ((q >> 2) * 2 + chalf) * 16 + (q & 3) * 4;
                float4 v;
                vec::unpack(acc[2 * q], v.x, v.y);
                vec::unpack(acc[2 * q + 1], v.z, v.w);
                mine[r * 32 + ((col >> 2) ^ (r & 31))] = v;
            }
            cluster_sync();
            const int rows = kTileM / ks;
            const uint32_t at = smem_u32(base_sm);
            for (int i = tid; i < rows * 32; i += 32 * kIntraWorkWarps) {
                const int rr = part * rows + (i >> 5), c4 = i & 31;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int k = 0; k < ks; ++k) {
                    const float4 t = ld_cluster(at + (rr * 32 + (c4 ^ (rr & 31))) * 16, k);
                    v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
                }
                const int row = l0 + rr, col = s0 + c4 * 4;
                const bool on = row < lim;                        // zero outside the sequence
                T *out = static_cast<T *>(dCB16) + ((long long)(b * d.nc + c) * d.G + g) * Q * Q + (long long)row * Q + col;
                *reinterpret_cast<uint2 *>(out) = make_uint2(pack2<T>(on && col < lim ? v.x : 0.f, on && col + 1 < lim ? v.y : 0.f),
                                                             pack2<T>(on && col + 2 < lim ? v.z : 0.f, on && col + 3 < lim ? v.w : 0.f));
            }
            cluster_sync();                                       // no block leaves while its tile is being read
        } else if (ok) {                                          // the rounded dCB tile; zero outside the sequence
            const int l = l0 + r;
            T *out = static_cast<T *>(dCB16) + ((long long)(b * d.nc + c) * d.G + g) * Q * Q + (long long)l * Q + s0;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int col = ((q >> 1) * 2 + chalf) * 16 + (q & 1) * 8;
                float o[8];
#pragma unroll
                for (int e = 0; e < 4; ++e) vec::unpack(acc[4 * q + e], o[2 * e], o[2 * e + 1]);
#pragma unroll
                for (int e = 0; e < 8; ++e) o[e] = (l < lim && s0 + col + e < lim) ? o[e] : 0.f;
                *reinterpret_cast<uint4 *>(out + col) = pack8<T>(o);
            }
        }
    } else {
        bool ok = true;
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIntraHelpRegs));
        const int i = tid - 32 * kIntraWorkWarps, kb = i >> 4;    // position in the tile, as a column and as a row
        const bool diag = ty == tz;
        const int role = __shfl_sync(0xffffffffu, warp - kIntraWorkWarps, 0);   // 0: issues the sums' MMAs; 1: loads and G2
        float pcf = 0.f, pcb = 0.f, pdt = 1.f, prf = 0.f, prb = 0.f;
        const int step = d.nc * Q;                                // from a head to the next
        long long base = ((long long)(b * d.H + h0) * d.nc + c) * Q + i;   // of the head whose factors are fetched next
        auto fetch_tab = [&] {
            pcf = cs_f[base + s0];
            pcb = cs_b[base + s0];
            pdt = dt_out[base + s0];
            prf = cs_f[base + l0];
            prb = cs_b[base + l0];
            base += step;
        };
        auto write_tab = [&](int h) {
            const uint32_t t = smem_u32(tabs) + (h & 1) * (uint32_t)sizeof(IntraTab), at = t + i * 4;
            const float cf = pcf * 1.4426950408889634f, cb_ = pcb * 1.4426950408889634f;
            const float lg = __log2f(pdt);                        // -inf on the zero-padded tail: those columns vanish
            const float f1 = __shfl_sync(0xffffffffu, cf, lane | 15), b0 = __shfl_sync(0xffffffffu, cb_, lane & 16);
            sts4(at + offsetof(IntraTab, row_f), prf * 1.4426950408889634f);
            sts4(at + offsetof(IntraTab, row_b), prb * 1.4426950408889634f);
            sts4(at + offsetof(IntraTab, col_f), ex2_approx(f1 - (cf - lg)));
            sts4(at + offsetof(IntraTab, col_b), ex2_approx(b0 - (cb_ - lg)));
            sts8(at + i * 4 + offsetof(IntraTab, both), cf - lg, cb_ - lg);
            if ((i & 15) == 0) {
                const uint32_t k = t + kb * 4;
                sts4(k + offsetof(IntraTab, ref_f), f1);
                sts4(k + offsetof(IntraTab, ref_b), b0);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.ready[h & 1]);
        };
        auto load_head = [&](int h) {                             // g and x of head h
            uint64_t *bar = &sh.in_full[h & 1];
            uint8_t *to = smIn + (h & 1) * 32768;
            mbar_expect_tx(bar, 32768u);
            tma_load4(to, &tmG, 0, h0 + h, c * Q + l0, b, bar);
            tma_load4(to + 16384, &tmX, 0, h0 + h, c * Q + s0, b, bar);
        };
        auto issue_g2 = [&](int h) {                              // G2 of head h, by warp 9
            if (!ws_wait_warp(&sh.in_full[h & 1], (h >> 1) & 1, fail, 93)) return false;
            tc_fence_after();
            if (elect_one()) {
                constexpr uint32_t idesc = instr_desc(AbFmt<T>::v, false, false, 128);
                const uint64_t dG = smem_desc(smem_u32(smIn) + (h & 1) * 32768, 16, 1024);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) umma(tmem + (h & 1) * 128, dG + 2 * kk, dG + 1024 + 2 * kk, idesc, kk > 0 ? 1u : 0u);
                umma_commit(&sh.ready[h & 1]);
            }
            __syncwarp();
            return true;
        };
        int loads = 0;
        if (role == 1) {
            loads = min(nh, 2);
            if (elect_one()) {
                load_head(0);
                mbar_expect_tx(&sh.cb_full, 32768u);
                const int row = ((b * d.nc + c) * d.G + g) * Q + l0;
                for (int k = 0; k < 2; ++k) tma_load2(smCB + k * 16384, &tmCB, s0 + k * 64, row, &sh.cb_full);
                if (nh > 1) load_head(1);
            }
            __syncwarp();
        }
        fetch_tab();
        write_tab(0);
        if (nh > 1) {
            fetch_tab();
            write_tab(1);
        }
        if (role == 1) ok = issue_g2(0) && (nh == 1 || issue_g2(1));
        const uint32_t tl = tmem_lane_base(tmem);
        float *out = u4 + (long long)((ty * (int)gridDim.z + tz) * 2) * hq + ((long long)(b * d.H + h0) * d.nc + c) * Q + s0 + i;
        const int off = (diag ? (s0 ^ kTileM) : l0) - s0;         // the chunk's other half, if there is one
#pragma unroll 1
        for (int h = 0; h < nh && ok; ++h) {
            if (h + 2 < nh) fetch_tab();
            ok = ws_wait_warp(&sh.v_full[h & 1], (h >> 1) & 1, fail, 94);       // V complete, G2 and the tables read
            if (!ok) break;
            if (role == 0) {                                      // columns 0-7: column sums, 8-15: row sums, by block of 16
                tc_fence_after();
                if (elect_one()) {
                    constexpr uint32_t id_r = instr_desc(1, false, false, 16), id_c = instr_desc(1, true, false, 16);
                    const uint32_t v0 = smem_u32(smIn) + (h & 1) * 32768, at = tmem + (h & 1) * 128;
                    const uint64_t dVc = smem_desc(v0, 16384, 1024), dVr = smem_desc(v0, 16, 1024), dT = smem_desc(smem_u32(smT), 16, 1024);
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk) umma(at, dVc + kk * 128, dT + (kk >> 2) * 192 + 64 + (kk & 3) * 2, id_c, kk > 0 ? 1u : 0u);
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk) umma(at, dVr + (kk >> 2) * 1024 + (kk & 3) * 2, dT + (kk >> 2) * 192 + (kk & 3) * 2, id_r, 1u);
                    umma_commit(&sh.sums_full[h & 1]);
                }
                __syncwarp();
            }
            float above = 0.f, left = 0.f;                        // of the block the diagonal crosses: column i above it, row i left of it
            if (diag) {
                const uint32_t slab = smem_u32(smIn) + (h & 1) * 32768 + (i >> 6) * 16384;
                const uint32_t col = slab + kb * 2048 + (i & 7) * 2, ch = (i & 63) >> 3;
#pragma unroll
                for (int j = 0; j < 15; ++j) {                    // rows 16 kb + j of column i
                    const float v = lds_bf16(col + j * 128 + ((ch ^ (j & 7)) << 4));
                    if (j < (i & 15)) above += v;
                }
                const uint32_t row = slab + i * 128 + (((((kb & 3) << 1)) ^ (i & 7)) << 4);
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    float v8[8];
                    unpack8<__nv_bfloat16>(lds16(row ^ (p * 16)), v8);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (p * 8 + j < (i & 15)) left += v8[j];
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.v_read);
            ok = ws_wait_warp(&sh.sums_full[h & 1], (h >> 1) & 1, fail, 95);
            if (!ok) break;
            tc_fence_after();
            if (role == 1 && h + 2 < nh) {                        // V of this head has been read: room for head h + 2
                ok = ws_wait_warp(&sh.v_read, h & 1, fail, 96);
                if (!ok) break;
                if (elect_one()) {
                    fence_async_smem();                           // the warps' reads precede the next TMA write
                    load_head(h + 2);
                }
                __syncwarp();
                ++loads;
            }
            uint32_t sums[16];
            tmem_ld16_nowait(tl + (h & 1) * 128, sums);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.read_done);
            if (h + 2 < nh) write_tab(h);                         // head h + 2 takes the place of head h
            if (diag) {
                float cl = -above, cu = above, rl = left, ru = -left;   // column sums below / above the diagonal, row sums left / right of it
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float cv = __uint_as_float(sums[k]), rv = __uint_as_float(sums[8 + k]);
                    if (k < kb) {
                        cu += cv;
                        rl += rv;
                    } else {
                        cl += cv;
                        ru += rv;
                    }
                }
                out[0] = cl - rl;
                out[hq] = cu - ru;
                if (Q > kTileM) out[off] = out[hq + off] = 0.f;
            } else {                                              // the whole tile lies on one side of the diagonal
                float cv = 0.f, rv = 0.f;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    cv += __uint_as_float(sums[k]);
                    rv += __uint_as_float(sums[8 + k]);
                }
                float *on = out + (ty > tz ? 0 : hq), *no = out + (ty > tz ? hq : 0);
                on[0] = cv;
                on[off] = -rv;
                no[0] = no[off] = 0.f;
            }
            out += step;
            if (role == 1) {                                      // head h + 2's product takes the place of head h's sums
                ok = ws_wait_warp(&sh.read_done, h & 1, fail, 97);
                tc_fence_after();
                if (ok && h + 2 < nh) ok = issue_g2(h + 2);
            }
        }
        if (!ok && role < 2) {                                    // leave no MMA and no load in flight
            if (elect_one()) {
                umma_commit(&sh.fin_bar[role]);
                mbar_wait(&sh.fin_bar[role], 0);
                if (role == 1) {
                    mbar_wait(&sh.cb_full, 0);
                    for (int k = max(0, loads - 2); k < loads; ++k) mbar_wait(&sh.in_full[k & 1], (k >> 1) & 1);
                }
            }
            __syncwarp();
        }
        tc_fence_before();
        __syncthreads();
        if (ks > 1) {                                             // the weighting warps' two meetings over the cluster
            cluster_sync();
            cluster_sync();
        }
    }
}

}  // namespace tc
}  // namespace bissd
