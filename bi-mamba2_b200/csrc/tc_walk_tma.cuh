// Chunk states and the recurrence over chunks in one kernel (and their gradients in the backward pass): a CTA walks the
// chunks of one (batch, head, direction, 128 state columns), the running state in its registers.
//   MODE 0: for every chunk in the direction's order: states[c] = run;  run = e^{T_c} run + sum_l B[l,n] (x[l,p] Delta[l] e^{T_c-cs[l]})
//   MODE 1: in the opposite order: E16[c] = run;  dT_c += e^{T_c} <S_c, run>;  run = e^{T_c} run + sum_l C[l,n] (g[l,p] e^{cs[l]})
// (see simt::chunk_state / simt::dstates and simt::state_passing_fwd / _bwd for the reference line numbers).  As two kernels
// the local states made a round trip through memory in fp32 - 16 bytes for every 4 that are kept - and that was most of the
// two kernels' time.  us, forward + backward, two kernels and walk: b8 L2048 H24 133, 91; b2 L8192 H32 195, 109; b8 L1024 H16
// headdim 128, dstate 256 313, 157 (the last with the 2 - 5 us a launch of event brackets).
//
// Warps 0-3 scale the x / g rows in place; warps 4-11 (4-19) keep the running state (TMEM lane = n, P / 2 or P / 4 columns each)
// and move it from chunk to chunk; one lane of the last warp fills the ring, one of the warp before it issues the MMAs (one
// thread doing both, a stage took 0.75 us whatever was loaded, scaled or multiplied).  Stages are 128 positions (64 at P = 128): [128 x 128 n] of
// B / C and [128 x P] of x / g, both MN-major as they land, with the rows' cumulative sums and Delta beside them (read from
// global memory by the scaling warps, their latency was the length of a stage).  Accumulators and, in MODE 1, the entering
// states that come by TMA are double-buffered.  dstate 64: the second 64 rows of the tile repeat the first, and each half of
// the lanes keeps half of the columns.
// Every blocking point is a bounded mbarrier wait, ids 71-78 in the status word.
#pragma once
#include "tc_state_tma.cuh"

namespace bissd {
namespace tc {

// Threads that keep the running state.  Sixteen warps in the backward walk at headdim 128 with dstate 128 and 256, where eight are
// what it waits for (dot products with the entering states); elsewhere eight are as good or better.  us, eight and sixteen warps,
// backward, headdim 128: dstate 256 b8 L1024 H16 102.9, 85.1, b2 L4096 H24 chunk 256 109, 93.6; dstate 128 b8 L1024 H16 55.8, 45.5,
// b1 L2048 H8 51.6, 38.8; dstate 64 (half the columns a thread) b8 L1024 H16 35.3, 37.4, b2 L8192 H32 101.5, 103.5.  Forward, b8 L1024
// H16 dstate 256: 69.6, 70.9.  Headdim 64, b8 L2048 H24 dstate 128: forward 45.2, 45.5, backward 53.6, 55.4.
constexpr int kWalkScale = 128;
__host__ __device__ constexpr int walk_state_threads(int pb, int mode, bool half) { return pb == 2 && mode == 1 && !half ? 512 : 256; }
__host__ __device__ constexpr int walk_threads(int pb, int mode, bool half) { return kWalkScale + walk_state_threads(pb, mode, half) + 64; }   // 14 or 22 warps
__host__ __device__ constexpr int walk_rows(int pb) { return pb == 1 ? 128 : 64; }   // positions per stage
__host__ __device__ constexpr int walk_ring(int pb, int mode) { return pb == 1 ? (mode ? 3 : 4) : (mode ? 4 : 6); }
__host__ __device__ constexpr int walk_stage_bytes(int pb) { return walk_rows(pb) * (256 + pb * 128) + 2048; }
inline bool walk_ok(int P, int N, int Q) {
    return (P == 64 || P == 128) && (N == 64 || (N % 128 == 0 && N <= 256)) && (Q == 128 || Q == 256);
}
inline size_t walk_smem(int P, int mode) {
    return 1024 + (size_t)walk_ring(P / 64, mode) * walk_stage_bytes(P / 64) + (mode ? 2 * (size_t)P * 256 : 0);
}
inline int walk_tiles(const Dims &d) { return d.N == 64 ? 1 : d.N / 128; }

struct WalkShared {
    uint64_t full[6], scaled[6], empty[6], acc[2], acc_free[2], s_full[2], s_free[2], drain_bar;
    uint32_t tmem_base;
    int fail, loads, s_loads;                                   // stages, and chunks whose entering states, requested
};
struct WalkArgs {
    const float *dt_out, *cs_f, *cs_b;
    const float *start_f, *start_b;                             // init_* or dfinal_*: (b, H, P, N) fp32 or null
    float *end_f, *end_b;                                       // final_* or dinit_*: the same, or null
    void *out_f, *out_b;                                        // states_* or E16 per direction: (b, nc, H, P, N) 16-bit
    float *dTpart;                                              // MODE 1
    int first;                                                  // first kernel of its pass: clears the status word (a wait that runs out reports long after)
};

// grid 2 b H tiles; tmRow: B or C, box [64 n x a stage's positions]; tmCol: x or g, the same; tmS*: states, box [64 n x P
// rows].  PB = P / 64; HALF: dstate 64.  cs_* and dt_out are 16-byte aligned.
template <class T, int MODE, int PB, bool HALF>
__global__ void __launch_bounds__(walk_threads(PB, MODE, HALF), 1)
state_walk(Dims d, const __grid_constant__ CUtensorMap tmRow, const __grid_constant__ CUtensorMap tmCol,
           const __grid_constant__ CUtensorMap tmSf, const __grid_constant__ CUtensorMap tmSb, WalkArgs a, int *status) {
    pdl_begin();
    if (a.first && blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
    extern __shared__ uint8_t dyn[];
    __shared__ WalkShared sh;
    constexpr int P = 64 * PB, SR = walk_rows(PB), NS = walk_ring(PB, MODE);
    constexpr int kA = 2 * SR * 128, kX = PB * SR * 128, kStage = walk_stage_bytes(PB);   // + the rows' cs, Delta and the chunk's T
    constexpr int kState = walk_state_threads(PB, MODE, HALF), CS = kState / 128;   // CS warps share a row quarter's columns
    constexpr int NC = (HALF ? P / 2 : P) / CS;                 // columns a thread keeps
    const int N = d.N, Q = d.Q, nc = d.nc, spc = Q / SR;        // stages per chunk
    uint8_t *base_sm = smem_align1024(dyn), *smS = base_sm + NS * kStage;   // smS: [2 buffers][2][P rows x 128 B]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles = HALF ? 1 : N / 128;
    const int dir = blockIdx.x & 1, tile = (blockIdx.x >> 1) % tiles, bh = (blockIdx.x >> 1) / tiles;
    const int h = bh % d.H, b = bh / d.H, grp = h / d.R, n0 = tile * 128;
    const bool up = MODE == 0 ? dir == 0 : dir == 1;            // chunks ascending
    const float *cs = dir ? a.cs_b : a.cs_f;
    const long long vec0 = ((long long)b * d.H + h) * nc * Q;   // this head's per-position vectors
    auto chunk = [&](int i) { return up ? i : nc - 1 - i; };
    volatile int *fail = &sh.fail;
    const int total = nc * spc;
    // Position in the walk, advanced stage by stage (no divisions in the single-thread loops).
    struct Pos {
        int chunk = 0, part = 0, slot = 0, phase = 0;           // chunk of the walk, stage in it, ring slot, its phase parity
    };
    auto advance = [&](Pos &p) {
        if (++p.part == spc) { p.part = 0; ++p.chunk; }
        if (++p.slot == NS) { p.slot = 0; p.phase ^= 1; }
    };
    auto load_stage = [&](const Pos &p) {
        uint8_t *dst = base_sm + p.slot * kStage;
        uint64_t *bar = &sh.full[p.slot];
        const int c = chunk(p.chunk), row = c * Q + p.part * SR;
        const float *v = cs + vec0 + (long long)c * Q;
        mbar_expect_tx(bar, (uint32_t)(kA + kX + (MODE == 0 ? SR * 8 + 16 : SR * 4)));
        for (int j = 0; j < 2; ++j) tma_load4(dst + j * SR * 128, &tmRow, HALF ? 0 : n0 + j * 64, grp, row, b, bar);
        for (int j = 0; j < PB; ++j) tma_load4(dst + kA + j * SR * 128, &tmCol, j * 64, h, row, b, bar);
        bulk_load(dst + kA + kX, v + p.part * SR, SR * 4, bar);
        if (MODE == 0) {
            bulk_load(dst + kA + kX + SR * 4, a.dt_out + vec0 + (long long)c * Q + p.part * SR, SR * 4, bar);
            bulk_load(dst + kA + kX + SR * 8, v + (dir ? 0 : Q - 4), 16, bar);
        }
    };
    auto load_states = [&](int i) {                             // MODE 1: the states entering chunk i of the walk
        mbar_expect_tx(&sh.s_full[i & 1], (uint32_t)(P * (HALF ? 128 : 256)));
        const int row = ((b * nc + chunk(i)) * d.H + h) * P;
        for (int j = 0; j < (HALF ? 1 : 2); ++j)
            tma_load2(smS + (i & 1) * P * 256 + j * P * 128, dir ? &tmSb : &tmSf, n0 + j * 64, row, &sh.s_full[i & 1]);
    };
    if (warp == 0) tmem_alloc(&sh.tmem_base, 2 * P);
    if (tid == kWalkScale + kState + 32) {
        for (int i = 0; i < NS; ++i) {
            mbar_init(&sh.full[i], 1);
            mbar_init(&sh.scaled[i], kWalkScale / 32);
            mbar_init(&sh.empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.acc[i], 1);
            mbar_init(&sh.acc_free[i], kState / 32);
            mbar_init(&sh.s_full[i], 1);
            mbar_init(&sh.s_free[i], kState / 32);
        }
        sh.fail = 0;
        fence_mbar_init();
        if (MODE == 1)
            for (int i = 0; i < 2 && i < nc; ++i) load_states(i);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    // At headdim 128 the walk is bound elsewhere, and no faster with elect_one but for dstate 64 (us, lane 0 and elect_one, forward:
    // b8 L1024 H16 dstate 256 65.7, 68.0, dstate 128 35.4, 37.2, dstate 64 30.1, 29.2; b2 L8192 H32 dstate 64 88.7, 94.0; backward
    // within 1.5 % but for b1 L2048 H8 38.7, 37.3).  Headdim 64, b8 L2048 H24 dstate 128: 48.7, 45.2.
    auto one_lane = [&] { return PB == 1 ? elect_one() : lane == 0; };
    if (warp == (kWalkScale + kState) / 32) {
        if (one_lane()) {
            const uint32_t idesc = instr_desc(AbFmt<T>::v, true, true, P);
            bool ok = true;
            Pos m;
            int states = min(2, nc);
            for (int s = 0; s < total; ++s, advance(m)) {
                const int i = m.chunk;
                if (m.part == 0 && i >= 2) {                    // the accumulator of chunk i - 2 (and its states) have been used
                    ok = ws_wait(&sh.acc_free[i & 1], ((i >> 1) - 1) & 1, fail, 73);
                    if (MODE == 1 && ok) ok = ws_wait(&sh.s_free[i & 1], ((i >> 1) - 1) & 1, fail, 74);
                    if (MODE == 1 && ok) load_states(states++);
                }
                ok = ok && ws_wait(&sh.scaled[m.slot], m.phase, fail, 72);
                if (!ok) break;
                tc_fence_after();
                const uint32_t sa = smem_u32(base_sm + m.slot * kStage), acc = tmem + (i & 1) * P;
                const uint64_t da = smem_desc(sa, SR * 128, 1024), db = smem_desc(sa + kA, SR * 128, 1024);
                umma(acc, da, db, idesc, m.part > 0 ? 1u : 0u);
#pragma unroll
                for (int kk = 1; kk < SR / 16; ++kk) umma(acc, da + kk * 128, db + kk * 128, idesc, 1u);   // 2048 bytes a step, in 16-byte units
                umma_commit(&sh.empty[m.slot]);
                if (m.part == spc - 1) umma_commit(&sh.acc[i & 1]);
            }
            sh.s_loads = states;
        }
    } else if (warp > (kWalkScale + kState) / 32) {             // the ring's loads
        if (one_lane()) {
            Pos p;
            int s = 0;
            for (; s < total; ++s, advance(p)) {
                if (s >= NS && !ws_wait(&sh.empty[p.slot], p.phase ^ 1, fail, 71)) break;
                load_stage(p);
            }
            sh.loads = s;
        }
    } else if (warp < 4) {
        // this thread scales 16-byte pieces of rows r0 + 16 k of a stage (in each of the PB blocks)
        constexpr int K = SR / 16;
        const int r0 = tid >> 3;
        Pos p;
#pragma unroll 1
        for (int s = 0; s < total; ++s, advance(p)) {
            if (!ws_wait_warp(&sh.full[p.slot], p.phase, fail, 76)) break;
            uint4 *x = reinterpret_cast<uint4 *>(base_sm + p.slot * kStage + kA);
            const float *pc = reinterpret_cast<const float *>(base_sm + p.slot * kStage + kA + kX), *pd = pc + SR;
            const float T_ = MODE == 0 ? pc[2 * SR + (dir ? 0 : 3)] : 0.f;
            float w[K];
            uint4 v[K * PB];
#pragma unroll
            for (int k = 0; k < K * PB; ++k) v[k] = x[tid + k * kWalkScale];
#pragma unroll
            for (int k = 0; k < K; ++k) w[k] = MODE == 0 ? pd[r0 + 16 * k] * __expf(T_ - pc[r0 + 16 * k]) : __expf(pc[r0 + 16 * k]);
#pragma unroll
            for (int k = 0; k < K * PB; ++k) x[tid + k * kWalkScale] = scale8_packed<T>(v[k], w[k % K]);
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.scaled[p.slot]);
        }
    } else {
        const int quad = warp & 3, colq = (warp - 4) >> 2, odd = lane & 1;
        const int n = HALF ? (quad & 1) * 32 + lane : quad * 32 + lane;       // within the 128-column tile
        const int col0 = HALF ? ((quad >> 1) * CS + colq) * NC : colq * NC;
        const long long hp = ((long long)b * d.H + h) * P * N, cstride = (long long)d.H * P * N;
        const long long off0 = (long long)b * nc * cstride + (long long)h * P * N;
        const float *start = dir ? a.start_b : a.start_f;
        float *end = dir ? a.end_b : a.end_f;
        T *out = static_cast<T *>(dir ? a.out_b : a.out_f) + off0 + (long long)(col0 + odd) * N + n0 + (n & ~1);
        float run[NC];
#pragma unroll
        for (int j = 0; j < NC; ++j) run[j] = start ? start[hp + (long long)(col0 + j) * N + n0 + n] : 0.f;
        float T_next = cs[vec0 + (long long)chunk(0) * Q + (dir ? 0 : Q - 1)];
        bool ok = true;
#pragma unroll 1
        for (int i = 0; i < nc; ++i) {                          // chunk i of the walk: what enters it leaves as output, then the update
            const int c = chunk(i);
            const float e = expf(T_next);
            if (i + 1 < nc) T_next = cs[vec0 + (long long)chunk(i + 1) * Q + (dir ? 0 : Q - 1)];
            if (MODE == 1) {
                ok = ws_wait_warp(&sh.s_full[i & 1], (i >> 1) & 1, fail, 77);
                if (!ok) break;
            }
            // Neighbouring lanes swap one of two columns, so that each has two adjacent n of one column: half as many
            // stores (and reads of the entering states), of twice the width.
            T *o = out + c * cstride;
            const uint8_t *sp = smS + (i & 1) * P * 256 + (n >> 6) * P * 128 + (n & 6) * 2;
            auto put = [&](int j, float part) -> float {        // columns j and j + 1; part + their share of <S, run>
                const float got = __shfl_xor_sync(0xffffffffu, odd ? run[j] : run[j + 1], 1);
                const float lo = odd ? got : run[j], hi = odd ? run[j + 1] : got;   // column j + odd, at n & ~1 and n | 1
                *reinterpret_cast<uint32_t *>(o + (long long)j * N) = pack2<T>(lo, hi);
                if (MODE == 0) return 0.f;
                const int p = col0 + j + odd;
                float s0, s1;
                unpack2<T>(*reinterpret_cast<const uint32_t *>(sp + p * 128 + ((((n & 63) >> 3) ^ (p & 7)) << 4)), s0, s1);
                return fmaf(s0, lo, fmaf(s1, hi, part));
            };
            if constexpr (MODE == 0) {
#pragma unroll
                for (int j = 0; j < NC; j += 2) put(j, 0.f);
            } else {
                // A partial dT per four columns and 32 n: a warp's worth of simt::state_passing_bwd4, in its order
                constexpr int V = NC / 4;
                auto four = [&](auto k) -> float { return put(4 * decltype(k)::value + 2, put(4 * decltype(k)::value, 0.f)); };
                const float part = warp_sums<V>(four, lane);
                if (lane == 0) mbar_arrive(&sh.s_free[i & 1]);
                if (lane % (32 / V) == 0) {
                    const long long hc = ((long long)dir * d.b * d.H + (long long)b * d.H + h) * nc + c;
                    a.dTpart[(hc * tiles + tile) * (4 * CS * V) + ((quad + 4 * (colq / (CS / 2))) * (CS / 2) + colq % (CS / 2)) * V + lane * V / 32] = e * part;
                }
            }
            ok = ws_wait_warp(&sh.acc[i & 1], (i >> 1) & 1, fail, 78);
            if (!ok) break;
            tc_fence_after();
            constexpr int LD = CS == 4 ? NC : 16;                // columns read at once: what the registers allow
#pragma unroll
            for (int q = 0; q < NC; q += LD) {
                uint32_t v[LD];
#pragma unroll
                for (int k = 0; k < LD; k += 8) tmem_ld8_nowait(tmem_lane_base(tmem) + (i & 1) * P + col0 + q + k, *reinterpret_cast<uint32_t(*)[8]>(&v[k]));
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < LD; ++j) run[q + j] = fmaf(e, run[q + j], __uint_as_float(v[j]));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.acc_free[i & 1]);
        }
        if (ok && end)
#pragma unroll
            for (int j = 0; j < NC; ++j) end[hp + (long long)(col0 + j) * N + n0 + n] = run[j];
    }
    tc_fence_before();
    __syncthreads();
    if (sh.fail) {                                              // leave nothing in flight
        if (tid == 0) atomicExch(status, kErrWsWait + sh.fail);
        if (warp == (kWalkScale + kState) / 32 && one_lane()) drain_mmas(&sh.drain_bar);
        if (tid == 0) {
            drain_loads(sh.full, NS, sh.loads);
            if (MODE == 1) drain_loads(sh.s_full, 2, sh.s_loads);
        }
        __syncthreads();
    }
    if (warp == 0) {
        __syncwarp();
        tmem_dealloc(tmem, 2 * P);
    }
}

}  // namespace tc
}  // namespace bissd
