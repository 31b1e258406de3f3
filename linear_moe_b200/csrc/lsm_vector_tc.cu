// The kernels of lsm_vector.cu for 128-wide heads and groups of several chunks on the 5th-generation tensor cores: chunks of 64 tokens, tiles by TMA, products as tcgen05.mma
// with accumulators in tensor memory.  The arithmetic is the same, operands rescaled around the middle of a chunk: with chunks of 128 the factors
// e^{+-(b_i - b_m)} would overflow twice as early.  A tile of 64 tokens stands where an instruction wants 128 rows: the lower half of its
// accumulator holds the tile's rows, the upper half products of whatever follows the tile in shared memory, and nobody reads it (an
// instruction with 64 rows takes as long).
//
//   gla_state_tc_kernel   group summaries.
//   gla_sweep_tc_kernel   outputs and dq, chunks in order.
//   gla_dkv_tc_kernel     dk and dv, chunks in reverse order.
//
// Warps: one brings tiles and gates, one issues products, one stores results.  Two sets of four make the rescaled operands of every other chunk: a
// thread owns two channels of the 32 tokens on one side of the chunk's middle and walks away from it, so one running sum is all it needs.  Eight keep
// the chain over the chunks: the state lives in tensor memory, is scaled there row by row and published as a bf16 tile, and the chunk's
// increment accumulates onto it.  (Four of them for the state alone and four for scores and outputs took as long: a row's 128 columns then come
// one half after the other.)
// The summaries' chain is one product a chunk onto the state, which eight warps scale row by row in between.
// Sweeps are bound by the latency of a chunk, 4000 - 5000 cycles of which the tensor cores need 2000 - 3500 (a group has only cpg chunks), summaries
// by memory.  8 x 2048 tokens of 8 heads, against mma.sync: outputs 97 -> 49 us (201 MB, 31 us at the copy rate), dq 102 -> 58, dk and dv
// 141 -> 73, summaries 43 -> 31 and 41 -> 27 (134 MB, 20 us).  With gates in registers and the walks written out: 67, 73 and 82, summaries 41 and 64.
#include <cstddef>
#include "flash_tc_utils.cuh"
#include "lsm_vector.cuh"

namespace lmoe {
namespace lvt {
using namespace lmoe::tc;
using fatc::mbar_wait_suspend;
using fatc::tma_load_4d;
using fatc::tmem_st16;
using fatc::tmem_st_wait;
using fatc::elect_one;
using fatc::umma_ss;
using fatc::umma_ts;

constexpr int D = 128, CT = 64;
constexpr int TILE = CT * D * 2, BLOCK = CT * 128;                       // a tile: two blocks of [64 rows x 64 columns], 128-byte swizzled rows
constexpr int SBLOCK = D * 128, STILE = 2 * SBLOCK;                      // the state's tile: two blocks of [128 rows x 64 columns]
constexpr int EW = 8, CW = 8, E0 = 3, C0 = E0 + EW, THREADS = 32 * (C0 + CW);     // warps 0: TMA, 1: MMA, 2: stores, then operands, then chain
constexpr uint32_t TMEM_COLS = 512;

// The rows of a tile of BL-byte blocks as the K dimension (MN) or as M / N; K-steps of 16.
template <bool MN, int BL>
__device__ __forceinline__ uint32_t tile_lo(const uint8_t* tile) { return ((s32(tile) >> 4) & 0x3FFFu) | ((MN ? (uint32_t)(BL >> 4) : 1u) << 16); }
template <bool MN, int BL>
__device__ __forceinline__ constexpr uint32_t step_lo(int kk) { return MN ? (kk * 2048) >> 4 : ((kk / 4) * BL + (kk % 4) * 32) >> 4; }
template <bool A_MN, bool B_MN, int N>
__host__ __device__ constexpr uint32_t idesc() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((A_MN ? 1u : 0u) << 15) | ((B_MN ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// [128 x N] (+)= A B over 16 STEPS; A a tile of 64 tokens, B one (BB = BLOCK) or the state's (BB = SBLOCK)
template <bool A_MN, bool B_MN, int N, int STEPS, int BB>
__device__ __forceinline__ void product(uint32_t tmem_d, const uint8_t* a, const uint8_t* b, bool add) {
    if (!elect_one()) return;
    const uint32_t al = tile_lo<A_MN, BLOCK>(a), bl = tile_lo<B_MN, BB>(b);
#pragma unroll
    for (int kk = 0; kk < STEPS; ++kk)
        umma_ss(tmem_d, al + step_lo<A_MN, BLOCK>(kk), bl + step_lo<B_MN, BB>(kk), idesc<A_MN, B_MN, N>(), add || kk > 0);
}
// [128 x 128] (+)= P X: P in tensor memory (two tokens per column, 32 tokens from every STRIDE-th column on), X's 64 rows are K
template <int STRIDE>
__device__ __forceinline__ void product_p(uint32_t tmem_d, uint32_t tmem_p, const uint8_t* x, bool add) {
    if (!elect_one()) return;
    const uint32_t bl = tile_lo<true, BLOCK>(x);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) umma_ts(tmem_d, tmem_p + kk / 2 * STRIDE + kk % 2 * 8, bl + step_lo<true, BLOCK>(kk), idesc<false, true, 128>(), add || kk > 0);
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tma_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int h, int t0, int b) {
    tma_load_4d(dst, map, bar, 0, h, t0, b);
    tma_load_4d(dst + BLOCK, map, bar, 64, h, t0, b);
}
__device__ __forceinline__ void tma_store(const CUtensorMap* map, const uint8_t* src, int h, int t0, int b) {       // rows behind T are cut off
    fatc::tma_store_4d(map, src, 0, h, t0, b);
    fatc::tma_store_4d(map, src + BLOCK, 64, h, t0, b);
}
// 16-byte piece i (0 .. 7) of row r of a block
__device__ __forceinline__ uint4* piece(uint8_t* block, int r, int i) { return reinterpret_cast<uint4*>(block + r * 128 + ((i ^ (r & 7)) << 4)); }
// 32 numbers times f as bf16 into row r of a block, from 16-byte piece i0 on
__device__ __forceinline__ void store32(uint8_t* block, int r, int i0, const uint32_t (&v)[32], float f) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = pack_bf16(f * __uint_as_float(v[8 * i + 2 * e]), f * __uint_as_float(v[8 * i + 2 * e + 1]));
        *piece(block, r, i0 + i) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}
// this thread's N scores (row, column: tokens of the chunk) from column c0 on -> P times `scale`, packed over them; LOWER: columns up to the row, else
// from it on
template <bool LOWER, int N>
__device__ __forceinline__ void mask_scores(uint32_t taddr, int row, int c0, float scale) {
#pragma unroll 1
    for (int c = 0; c < N; c += 32) {
        uint32_t x[32], p[16];
        tmem_ld32(taddr + c, x);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const int j = c0 + c + 2 * e;
            p[e] = pack_bf16((LOWER ? j <= row : j >= row) ? scale * __uint_as_float(x[2 * e]) : 0.f,
                             (LOWER ? j + 1 <= row : j + 1 >= row) ? scale * __uint_as_float(x[2 * e + 1]) : 0.f);
        }
        tmem_st16(taddr + c / 2, p);
    }
    tmem_st_wait();
}
// this thread's 64 columns of the state times f, in place, and in bf16 (times `scale` too) to the state's tile; loops over columns stay loops, as in Walk
__device__ __forceinline__ void publish(uint32_t taddr, uint8_t* block, int r, float f, float scale) {
#pragma unroll 1
    for (int c = 0; c < 64; c += 32) {
        uint32_t x[32];
        tmem_ld32(taddr + c, x);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; ++e) x[e] = __float_as_uint(f * __uint_as_float(x[e]));
        tmem_st16(taddr + c, reinterpret_cast<uint32_t(&)[16]>(x[0]));
        tmem_st16(taddr + c + 16, reinterpret_cast<uint32_t(&)[16]>(x[16]));
        store32(block, r, c / 8, x, scale);
    }
    tmem_st_wait();
    fence_async();
}
// rows of the group's entering state, 64 columns, times f into tensor memory
__device__ __forceinline__ void load_state(uint32_t taddr, const float* src, float f) {
#pragma unroll
    for (int c = 0; c < 64; c += 16) {
        uint32_t x[16];
#pragma unroll
        for (int e = 0; e < 16; e += 4) {
            const float4 v = *reinterpret_cast<const float4*>(src + c + e);
            x[e] = __float_as_uint(f * v.x); x[e + 1] = __float_as_uint(f * v.y); x[e + 2] = __float_as_uint(f * v.z); x[e + 3] = __float_as_uint(f * v.w);
        }
        tmem_st16(taddr + c, x);
    }
    tmem_st_wait();
}
__device__ __forceinline__ void arrive(uint64_t* bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
__device__ __forceinline__ void init_tmem(uint32_t* base, int warp, uint32_t cols) {
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(s32(base)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
}
__device__ __forceinline__ void free_tmem(uint32_t base, int warp, uint32_t cols) {
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(base), "r"(cols) : "memory");
    }
}

__device__ __forceinline__ uint32_t lds32(uint32_t p) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ float2 lds64(uint32_t p) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ void sts32(uint32_t p, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" :: "r"(p), "r"(v) : "memory"); }
// two bf16 numbers times fx and fy
__device__ __forceinline__ uint32_t times(uint32_t x, float fx, float fy) { return pack_bf16(__uint_as_float(x << 16) * fx, __uint_as_float(x & 0xffff0000u) * fy); }

// A thread's walk away from the middle of a chunk: channels 2 p and 2 p + 1 of the 32 tokens before (SIDE 0) or behind (SIDE 1) it, eight at a time.  The
// loop stays a loop: with 32 rows written out the warps waited for instructions more than for anything else (7.4 of 17.6 cycles between two
// instructions of a warp), a walk over two tiles taking 6000 cycles.  So the gates cannot stay in registers and come from a tile of their own.
// Sums are kept in units of ln 2, for ex2.
constexpr float LOG2E = 1.4426950408889634f;
template <int SIDE>
struct Walk {
    static constexpr int side = SIDE;
    uint32_t at, gat;              // this thread's bytes of a row of a tile, and of the gates' tile from the first row on
    __device__ __forceinline__ explicit Walk(int p) : at((p >> 5) * BLOCK + ((p & 31) >> 2 << 4) + (p & 3) * 4), gat((SIDE ? 32 : 31) * 512 + p * 8) {}
    // Rows of the tile at `minus` times e^{-(b_t - b_m)} (MINUS), of the one DELTA bytes behind it times e^{b_t - b_m} (PLUS).  Returns e^ the sum of the gates.
    template <bool PLUS, bool MINUS, int DELTA>
    __device__ __forceinline__ float2 go(uint32_t minus, uint32_t gates) const {
        constexpr uint32_t STEP = SIDE ? 1024u : 0u - 1024u;
        uint32_t p[8], gp = gates + gat;
#pragma unroll
        for (int e = 0; e < 8; ++e) p[e] = minus + (at ^ ((SIDE ? e : 7 - e) << 4)) + (SIDE ? 32 + e : 31 - e) * 128;
        float2 s = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
            float2 g[8];
            uint32_t v[8], w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) g[e] = lds64(gp + (SIDE ? (uint32_t)(e * 512) : 0u - (uint32_t)(e * 512)));
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                if (MINUS) v[e] = lds32(p[e]);
                if (PLUS) w[e] = lds32(p[e] + (uint32_t)DELTA);
            }
            // b_t - b_m: behind the middle with the token's own gate, before it without
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float2 before = s;
                s.x = fmaf(g[e].x, LOG2E, s.x); s.y = fmaf(g[e].y, LOG2E, s.y);
                const float2 x = SIDE ? s : make_float2(-before.x, -before.y);
                if (MINUS) sts32(p[e], times(v[e], exp2f(-x.x), exp2f(-x.y)));
                if (PLUS) sts32(p[e] + (uint32_t)DELTA, times(w[e], exp2f(x.x), exp2f(x.y)));
                p[e] += STEP;
            }
            gp += 4 * STEP;
        }
        return make_float2(exp2f(s.x), exp2f(s.y));
    }
};
// A thread's channels, its set of warps and f(its walk, pair, set) (the walk's side is a constant in f)
template <typename F>
__device__ __forceinline__ void operand_warps(int tid, F f) {
    if ((tid >> 6) & 1) f(Walk<1>(tid & 63), tid & 63, tid >> 7);
    else f(Walk<0>(tid & 63), tid & 63, tid >> 7);
}

// ---------------------------------------------------------------------------------------------------------------------
constexpr int SS = 3, GTILE = CT * D * 4;                                // stages of the summaries; bytes of a chunk's gates
constexpr int ST_E0 = 2, ST_C0 = ST_E0 + 8, ST_THREADS = 32 * (ST_C0 + 8);   // warps 0: TMA, 1: MMA, then two sets of operand warps, then the state
struct __align__(1024) SmemState {
    uint8_t x[SS][TILE], y[SS][TILE], gk[SS][GTILE];
    float tab[SS][D];                               // the sum of a chunk's gates
    uint64_t full[SS], empty[SS], e_ready[SS], s_ready, s_done;
    uint32_t tmem_base;
    int abort_flag;
};

// The operand of a summary: 32 rows of a tile times e^ the sum of the gates between them and the chunk's end (REV 0, without their own) or its start (REV 1,
// with their own, times `mul` too), in the order away from there.  FAR: the rows behind the other 32, whose gates are summed first.  Returns the sum.
template <int REV>
__device__ __forceinline__ float2 summary_rows(uint32_t tile, uint32_t gates, int pair, bool far, float mul) {
    constexpr uint32_t STEP = REV ? 1024u : 0u - 1024u;
    const uint32_t at = (pair >> 5) * BLOCK + ((pair & 31) >> 2 << 4) + (pair & 3) * 4, first = (REV ? 0 : 63);
    uint32_t gp = gates + first * 512 + pair * 8;
    float2 z = make_float2(0.f, 0.f);
    auto gate = [&](int e) { return lds64(gp + (REV ? (uint32_t)(e * 512) : 0u - (uint32_t)(e * 512))); };
    if (far) {
#pragma unroll 1
        for (int j = 0; j < 4; ++j, gp += 4 * STEP) {
            float2 g[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) g[e] = gate(e);
#pragma unroll
            for (int e = 0; e < 8; ++e) { z.x += g[e].x; z.y += g[e].y; }
        }
    }
    uint32_t p[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) p[e] = tile + (at ^ ((REV ? e : 7 - e) << 4)) + (REV ? e : 63 - e) * 128 + (far ? 4 * STEP : 0u);
#pragma unroll 1
    for (int j = 0; j < 4; ++j, gp += 4 * STEP) {
        float2 g[8];
        uint32_t v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) g[e] = gate(e);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = lds32(p[e]);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if (REV) { z.x += g[e].x; z.y += g[e].y; }
            sts32(p[e], REV ? times(v[e], __expf(z.x) * mul, __expf(z.y) * mul) : times(v[e], __expf(z.x), __expf(z.y)));
            if (!REV) { z.x += g[e].x; z.y += g[e].y; }
            p[e] += STEP;
        }
    }
    return z;
}

// Group summaries.  REV 0: S <- e^{b_C} S + (e^{b_C - b_j} K)^T V.  REV 1: dS <- e^{b_C} dS + (scale e^{b_i} Q)^T dO, chunks in reverse order.
template <int REV>
__global__ void __launch_bounds__(ST_THREADS, 1)
gla_state_tc_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmGk, GlaArgs a) {
    extern __shared__ uint8_t smem_raw[];
    SmemState& sm = *reinterpret_cast<SmemState*>(smem_raw + ((1024 - (s32(smem_raw) & 1023)) & 1023));
    const int warp = fatc::uniform_warp(), lane = threadIdx.x & 31;
    const int grp = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int chunks = (a.T + CT - 1) / CT, c_lo = grp * a.cpg, n = max(0, min(chunks, c_lo + a.cpg) - c_lo);
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    if (threadIdx.x == 0) {
        for (int s = 0; s < SS; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); mbar_init(&sm.e_ready[s], 4); }
        mbar_init(&sm.s_ready, 8); mbar_init(&sm.s_done, 1);
        sm.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    init_tmem(&sm.tmem_base, warp, 128);
    const uint32_t tmem_base = fatc::uniform(sm.tmem_base);

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < n; ++i) {
                const int s = i % SS, t0 = (REV ? c_lo + n - 1 - i : c_lo + i) * CT;
                if (!mbar_wait_suspend(&sm.empty[s], ((i / SS) & 1) ^ 1, abort_flag, err, 0xa100 | s)) break;
                mbar_expect_tx(&sm.full[s], 2 * TILE + GTILE);
                tma_load_4d(sm.gk[s], &tmGk, &sm.full[s], 0, h, t0, b);
                tma_tile(sm.x[s], &tmX, &sm.full[s], h, t0, b);
                tma_tile(sm.y[s], &tmY, &sm.full[s], h, t0, b);
            }
        }
    } else if (warp == 1) {
        for (int i = 0; i < n; ++i) {
            const int s = i % SS;
            if (!fatc::mbar_wait_warp(&sm.e_ready[s], (i / SS) & 1, abort_flag, err, 0xa200 | s)) break;
            if (!fatc::mbar_wait_warp(&sm.full[s], (i / SS) & 1, abort_flag, err, 0xa210 | s)) break;
            if (!fatc::mbar_wait_warp(&sm.s_ready, i & 1, abort_flag, err, 0xa220)) break;
            tc_fence_after();
            product<true, true, 128, 4, BLOCK>(tmem_base, sm.x[s], sm.y[s], i > 0);
            if (elect_one()) { umma_commit(&sm.empty[s]); umma_commit(&sm.s_done); }
        }
    } else if (warp < ST_C0) {                      // rescaled operands; a set of four warps takes every other chunk
        const int tid = threadIdx.x - ST_E0 * 32, pair = tid & 63, set = tid >> 7;
        const bool far = (tid >> 6) & 1;
        for (int i = set; i < n; i += 2) {
            const int s = i % SS;
            // The other set has this stage's chunk before: until that one's tiles are there, full[s] looks as it will when this one's are.
            if (i >= SS && !mbar_wait_suspend(&sm.e_ready[s], (i / SS - 1) & 1, abort_flag, err, 0xa310 | s)) break;
            if (!mbar_wait_suspend(&sm.full[s], (i / SS) & 1, abort_flag, err, 0xa300 | s)) break;
            const float2 sum = summary_rows<REV>(s32(sm.x[s]), s32(sm.gk[s]), pair, far, a.scale);
            if (far) *reinterpret_cast<float2*>(&sm.tab[s][2 * pair]) = sum;
            fence_async();
            arrive(&sm.e_ready[s]);
        }
    } else {
        const int qd = warp & 3, part = (warp - ST_C0) >> 2, r = qd * 32 + lane;
        const uint32_t st = tmem_base + ((uint32_t)(qd * 32) << 16) + part * 64;
        float decay = 0.f;
        bool ok = true;
        for (int i = 0; ok && i < n; ++i) {
            const int s = i % SS;
            ok = mbar_wait_suspend(&sm.e_ready[s], (i / SS) & 1, abort_flag, err, 0xa400 | s);
            if (!ok) break;
            const float sum = sm.tab[s][r], f = __expf(sum);
            decay += sum;
            if (i > 0) {
                ok = mbar_wait_suspend(&sm.s_done, (i - 1) & 1, abort_flag, err, 0xa410);
                if (!ok) break;
                tc_fence_after();
#pragma unroll 1
                for (int c = 0; c < 64; c += 32) {
                    uint32_t x[32];
                    tmem_ld32(st + c, x);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) x[e] = __float_as_uint(f * __uint_as_float(x[e]));
                    tmem_st16(st + c, reinterpret_cast<uint32_t(&)[16]>(x[0]));
                    tmem_st16(st + c + 16, reinterpret_cast<uint32_t(&)[16]>(x[16]));
                }
                tmem_st_wait();
                tc_fence_before();
            }
            arrive(&sm.s_ready);
        }
        if (ok && n > 0) ok = mbar_wait_suspend(&sm.s_done, (n - 1) & 1, abort_flag, err, 0xa420);
        tc_fence_after();
        float* out = a.states + (((int64_t)bh * a.G + grp) * D + r) * D + part * 64;
#pragma unroll 1
        for (int c = 0; c < 64; c += 32) {
            uint32_t v[32];
            tmem_ld32(st + c, v);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; e += 4)
                *reinterpret_cast<float4*>(out + c + e) = n > 0 ? make_float4(__uint_as_float(v[e]), __uint_as_float(v[e + 1]), __uint_as_float(v[e + 2]), __uint_as_float(v[e + 3]))
                                                                : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (a.gdecay != nullptr && part == 0) a.gdecay[((int64_t)bh * a.G + grp) * D + r] = decay;
    }
    free_tmem(tmem_base, warp, 128);
}

// ---------------------------------------------------------------------------------------------------------------------
constexpr int FS = 2;              // stages, one for each set of operand warps
struct __align__(1024) SmemSweep {
    uint8_t t0[FS][TILE], k[FS][TILE], v[FS][TILE], sb[STILE], gk[FS][GTILE];
    float tab[FS][2][D];                            // e^{b_m}, e^{b_C - b_m}
    uint64_t full[FS], empty[FS], e_ready[FS], o_ready[FS], st_ready[FS], sc_full, p_ready, sb_ready, o_full;
    uint32_t tmem_base;
    int abort_flag;
};

// MODE 0: t0 = Q, scores Q K^T, out = o = scale (P V + q~ (e^{b_m} S)).  MODE 1: t0 = dO, scores dO V^T, out = dq = e^{b_i - b_m} scale (P k~ + dO (e^{b_m} S)^T).
template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
gla_sweep_tc_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                    const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmGk, GlaArgs a) {
    extern __shared__ uint8_t smem_raw[];
    SmemSweep& sm = *reinterpret_cast<SmemSweep*>(smem_raw + ((1024 - (s32(smem_raw) & 1023)) & 1023));
    constexpr uint32_t SC = 0, OUT = 128, ST = 256, OP = 384;                    // scores, then P, of two chunks; X0 times the state; the state; P times X2
    const int warp = fatc::uniform_warp(), lane = threadIdx.x & 31;
    const int grp = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int chunks = (a.T + CT - 1) / CT, c_lo = grp * a.cpg, n = max(0, min(chunks, c_lo + a.cpg) - c_lo);
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    if (threadIdx.x == 0) {
        for (int s = 0; s < FS; ++s) {
            mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); mbar_init(&sm.e_ready[s], EW / 2);
            mbar_init(&sm.o_ready[s], CW / 2); mbar_init(&sm.st_ready[s], EW / 2);
        }
        mbar_init(&sm.sc_full, 1); mbar_init(&sm.p_ready, CW / 2); mbar_init(&sm.sb_ready, CW); mbar_init(&sm.o_full, 1);
        sm.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    init_tmem(&sm.tmem_base, warp, TMEM_COLS);
    const uint32_t tmem_base = fatc::uniform(sm.tmem_base);

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < n; ++i) {
                const int s = i % FS, t0 = (c_lo + i) * CT;
                if (!mbar_wait_suspend(&sm.empty[s], ((i / FS) & 1) ^ 1, abort_flag, err, 0xb100 | s)) break;
                mbar_expect_tx(&sm.full[s], 3 * TILE + GTILE);
                tma_load_4d(sm.gk[s], &tmGk, &sm.full[s], 0, h, t0, b);
                tma_tile(sm.k[s], &tmK, &sm.full[s], h, t0, b);
                tma_tile(sm.t0[s], &tm0, &sm.full[s], h, t0, b);
                tma_tile(sm.v[s], &tmV, &sm.full[s], h, t0, b);
            }
        }
    } else if (warp == 1) {
        auto scores = [&](int i) -> bool {          // into the columns that P of chunk i - 2 had: its product has completed, the state came behind it
            const int s = i % FS;
            if (!fatc::mbar_wait_warp(&sm.full[s], (i / FS) & 1, abort_flag, err, 0xb200 | s) ||
                !fatc::mbar_wait_warp(&sm.e_ready[s], (i / FS) & 1, abort_flag, err, 0xb210 | s)) return false;
            tc_fence_after();
            product<false, false, 64, 8, BLOCK>(tmem_base + SC + (i & 1) * 64, sm.t0[s], MODE == 0 ? sm.k[s] : sm.v[s], false);
            if (elect_one()) umma_commit(&sm.sc_full);
            return true;
        };
        bool ok = n > 0 && scores(0);
        for (int i = 0; ok && i < n; ++i) {
            const int s = i % FS;
            ok = fatc::mbar_wait_warp(&sm.sb_ready, i & 1, abort_flag, err, 0xb220);
            if (!ok) break;
            tc_fence_after();
            product<false, MODE == 0, 128, 8, SBLOCK>(tmem_base + OUT, sm.t0[s], sm.sb, false);
            product<true, true, 128, 4, BLOCK>(tmem_base + ST, sm.k[s], sm.v[s], true);                       // S += k~^T V
            ok = fatc::mbar_wait_warp(&sm.p_ready, i & 1, abort_flag, err, 0xb230);
            if (!ok) break;
            tc_fence_after();
            product_p<32>(tmem_base + OP, tmem_base + SC + (i & 1) * 64, MODE == 0 ? sm.v[s] : sm.k[s], false);
            if (elect_one()) umma_commit(&sm.o_full);
            if (i + 1 < n) ok = scores(i + 1);
        }
    } else if (warp == 2) {
        for (int i = 0; i < n; ++i) {
            const int s = i % FS;
            if (!mbar_wait_suspend(MODE == 0 ? &sm.o_ready[s] : &sm.st_ready[s], (i / FS) & 1, abort_flag, err, 0xb300 | s)) break;
            if (lane == 0) {
                tma_store(&tmO, sm.t0[s], h, (c_lo + i) * CT, b);
                fatc::tma_store_commit();
                fatc::tma_store_wait_read();
                mbar_arrive(&sm.empty[s]);
            }
            __syncwarp();
        }
        if (lane == 0) fatc::tma_store_wait();
    } else if (warp < C0) {                        // rescaled operands; a set of four warps takes every other chunk
        operand_warps(threadIdx.x - E0 * 32, [&](auto walk, int pair, int set) {
            constexpr int K_T0 = -FS * TILE;         // from a stage's K to its first tile
            static_assert(offsetof(SmemSweep, t0) - offsetof(SmemSweep, k) == (size_t)(int64_t)K_T0);
            for (int i = set; i < n; i += 2) {
                const int s = i % FS;
                const uint32_t ph = (i / FS) & 1;
                if (!mbar_wait_suspend(&sm.full[s], ph, abort_flag, err, 0xb400 | s)) break;
                *reinterpret_cast<float2*>(&sm.tab[s][walk.side][2 * pair]) = walk.template go<MODE == 0, true, K_T0>(s32(sm.k[s]), s32(sm.gk[s]));   // k~, q~
                fence_async();
                arrive(&sm.e_ready[s]);
                if (MODE == 1) {                    // dq <- e^{b_i - b_m} dq, by the threads that know the factors
                    if (!mbar_wait_suspend(&sm.o_ready[s], ph, abort_flag, err, 0xb410 | s)) break;
                    walk.template go<true, false, K_T0>(s32(sm.k[s]), s32(sm.gk[s]));
                    fence_async();
                    arrive(&sm.st_ready[s]);
                }
            }
        });
    } else {                                        // the chain
        const int qd = warp & 3, part = (warp - C0) >> 2, r = qd * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16), st = lane_addr + ST + part * 64;
        load_state(st, a.states + (((int64_t)bh * a.G + grp) * D + r) * D + part * 64, 1.f);
        float pend = 1.f;                           // e^{b_C - b_m} of the chunk before, which the state still wants
        for (int i = 0; i < n; ++i) {
            const int s = i % FS;
            if (!mbar_wait_suspend(&sm.e_ready[s], (i / FS) & 1, abort_flag, err, 0xb500 | s)) break;
            // e^{b_m} S; the increment before it and the product that read the tile are done (o_full)
            publish(st, sm.sb + part * SBLOCK, r, pend * sm.tab[s][0][r], 1.f);
            pend = sm.tab[s][1][r];
            tc_fence_before();
            arrive(&sm.sb_ready);
            if (qd < 2) {                           // scores -> P
                if (!mbar_wait_suspend(&sm.sc_full, i & 1, abort_flag, err, 0xb510)) break;
                tc_fence_after();
                mask_scores<true, 32>(lane_addr + SC + (i & 1) * 64 + part * 32, r, part * 32, a.scale);
                tc_fence_before();
                arrive(&sm.p_ready);
            }
            if (!mbar_wait_suspend(&sm.o_full, i & 1, abort_flag, err, 0xb520)) break;
            tc_fence_after();
            if (qd < 2) {
#pragma unroll 1
                for (int c = 0; c < 64; c += 32) {
                    uint32_t x[32], y[32];
                    tmem_ld32(lane_addr + OUT + part * 64 + c, x);
                    tmem_ld32(lane_addr + OP + part * 64 + c, y);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) x[e] = __float_as_uint(fmaf(a.scale, __uint_as_float(x[e]), __uint_as_float(y[e])));
                    store32(sm.t0[s] + part * BLOCK, r, c / 8, x, 1.f);                                   // every product has read X0
                }
                fence_async();
                arrive(&sm.o_ready[s]);
            }
        }
    }
    free_tmem(tmem_base, warp, TMEM_COLS);
}

// ---------------------------------------------------------------------------------------------------------------------
struct __align__(1024) SmemDkv {
    uint8_t q[FS][TILE], g[FS][TILE], k[FS][TILE], v[FS][TILE], sb[STILE], gk[FS][GTILE];
    float tab[2][2][D];                             // e^{b_m}, e^{b_C - b_m}
    uint64_t full[FS], empty[FS], e_ready[FS], o_ready[FS], st_ready[FS], sc_full, p_ready, sb_ready, o_full;
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(SmemDkv) == 227 * 1024, "all that a block can have");

// dv = P1 dO + k~ Db,  dk = e^{b_m - b_j} (P2 q~ + V Db^T),  P1 = (scale k~ q~^T . mask), P2 = (scale V dO^T . mask), Db = e^{b_C - b_m} dS; the state in
// tensor memory is dS / scale.
__global__ void __launch_bounds__(THREADS, 1)
gla_dkv_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                  const __grid_constant__ CUtensorMap tmG, const __grid_constant__ CUtensorMap tmDK, const __grid_constant__ CUtensorMap tmDV,
                  const __grid_constant__ CUtensorMap tmGk, GlaArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_tiles[];
    SmemDkv& sm = *reinterpret_cast<SmemDkv*>(smem_tiles);
    if ((s32(smem_tiles) & 1023) != 0) {              // nothing is left to round it up with
        if (threadIdx.x == 0) atomicExch(a.err, 0xc001);
        return;
    }
    constexpr uint32_t SC = 0, DV = 128, DK = 256, ST = 384;                     // two tiles of scores, then P1 and P2
    const int warp = fatc::uniform_warp(), lane = threadIdx.x & 31;
    const int grp = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int chunks = (a.T + CT - 1) / CT, c_lo = grp * a.cpg, n = max(0, min(chunks, c_lo + a.cpg) - c_lo), c_last = c_lo + n - 1;
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    if (threadIdx.x == 0) {
        for (int s = 0; s < FS; ++s) {
            mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); mbar_init(&sm.e_ready[s], EW / 2);
            mbar_init(&sm.o_ready[s], CW / 2); mbar_init(&sm.st_ready[s], EW / 2);
        }
        mbar_init(&sm.sc_full, 1); mbar_init(&sm.p_ready, CW / 2); mbar_init(&sm.sb_ready, CW); mbar_init(&sm.o_full, 1);
        sm.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    init_tmem(&sm.tmem_base, warp, TMEM_COLS);
    const uint32_t tmem_base = fatc::uniform(sm.tmem_base);

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < n; ++i) {
                const int s = i % FS, t0 = (c_last - i) * CT;
                if (!mbar_wait_suspend(&sm.empty[s], ((i / FS) & 1) ^ 1, abort_flag, err, 0xc100 | s)) break;
                mbar_expect_tx(&sm.full[s], 4 * TILE + GTILE);
                tma_load_4d(sm.gk[s], &tmGk, &sm.full[s], 0, h, t0, b);
                tma_tile(sm.q[s], &tmQ, &sm.full[s], h, t0, b);
                tma_tile(sm.k[s], &tmK, &sm.full[s], h, t0, b);
                tma_tile(sm.v[s], &tmV, &sm.full[s], h, t0, b);
                tma_tile(sm.g[s], &tmG, &sm.full[s], h, t0, b);
            }
        }
    } else if (warp == 1) {
        bool ok = true;
        for (int i = 0; ok && i < n; ++i) {
            const int s = i % FS;
            ok = fatc::mbar_wait_warp(&sm.full[s], (i / FS) & 1, abort_flag, err, 0xc200 | s) &&
                 fatc::mbar_wait_warp(&sm.e_ready[s], (i / FS) & 1, abort_flag, err, 0xc210 | s) &&
                 (i == 0 || fatc::mbar_wait_warp(&sm.o_full, (i - 1) & 1, abort_flag, err, 0xc220));         // P1 and P2 have been read
            if (!ok) break;
            tc_fence_after();
            product<false, false, 64, 8, BLOCK>(tmem_base + SC, sm.k[s], sm.q[s], false);          // k~ q~^T
            product<false, false, 64, 8, BLOCK>(tmem_base + SC + 64, sm.v[s], sm.g[s], false);     // V dO^T
            if (elect_one()) umma_commit(&sm.sc_full);
            ok = fatc::mbar_wait_warp(&sm.sb_ready, i & 1, abort_flag, err, 0xc230);
            if (!ok) break;
            tc_fence_after();
            product<false, true, 128, 8, SBLOCK>(tmem_base + DV, sm.k[s], sm.sb, false);           // k~ Db
            product<false, false, 128, 8, SBLOCK>(tmem_base + DK, sm.v[s], sm.sb, false);          // V Db^T
            product<true, true, 128, 4, BLOCK>(tmem_base + ST, sm.q[s], sm.g[s], true);            // += q~^T dO
            ok = fatc::mbar_wait_warp(&sm.p_ready, i & 1, abort_flag, err, 0xc240);
            if (!ok) break;
            tc_fence_after();
            product_p<16>(tmem_base + DV, tmem_base + SC, sm.g[s], true);
            product_p<16>(tmem_base + DK, tmem_base + SC + 64, sm.q[s], true);
            if (elect_one()) umma_commit(&sm.o_full);
        }
    } else if (warp == 2) {
        for (int i = 0; i < n; ++i) {
            const int s = i % FS, t0 = (c_last - i) * CT;
            if (!mbar_wait_suspend(&sm.st_ready[s], (i / FS) & 1, abort_flag, err, 0xc300 | s)) break;
            if (lane == 0) {
                tma_store(&tmDV, sm.v[s], h, t0, b);
                tma_store(&tmDK, sm.k[s], h, t0, b);
                fatc::tma_store_commit();
                fatc::tma_store_wait_read();
                mbar_arrive(&sm.empty[s]);
            }
            __syncwarp();
        }
        if (lane == 0) fatc::tma_store_wait();
    } else if (warp < C0) {                        // rescaled operands; set 0 takes the even chunks
        operand_warps(threadIdx.x - E0 * 32, [&](auto walk, int pair, int set) {
            constexpr int K_Q = -2 * FS * TILE;      // from a stage's K to its Q
            static_assert(offsetof(SmemDkv, q) - offsetof(SmemDkv, k) == (size_t)(int64_t)K_Q);
            for (int i = set; i < n; i += 2) {
                const int s = i % FS;
                const uint32_t ph = (i / FS) & 1;
                if (!mbar_wait_suspend(&sm.full[s], ph, abort_flag, err, 0xc400 | s)) break;
                *reinterpret_cast<float2*>(&sm.tab[s][walk.side][2 * pair]) = walk.template go<true, true, K_Q>(s32(sm.k[s]), s32(sm.gk[s]));      // k~, q~
                fence_async();
                arrive(&sm.e_ready[s]);
                if (!mbar_wait_suspend(&sm.o_ready[s], ph, abort_flag, err, 0xc410 | s)) break;
                walk.template go<false, true, K_Q>(s32(sm.k[s]), s32(sm.gk[s]));      // dk <- e^{b_m - b_j} dk
                fence_async();
                arrive(&sm.st_ready[s]);
            }
        });
    } else {                                        // the chain
        const int qd = warp & 3, part = (warp - C0) >> 2, r = qd * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16), st = lane_addr + ST + part * 64;
        load_state(st, a.states + (((int64_t)bh * a.G + grp) * D + r) * D + part * 64, 1.f / a.scale);
        float pend = 1.f;                           // e^{b_m} of the chunk behind, which the state still wants
        for (int i = 0; i < n; ++i) {
            const int s = i % FS;
            if (!mbar_wait_suspend(&sm.e_ready[s], (i / FS) & 1, abort_flag, err, 0xc500 | s)) break;
            publish(st, sm.sb + part * SBLOCK, r, pend * sm.tab[s][1][r], a.scale);
            pend = sm.tab[s][0][r];
            tc_fence_before();
            arrive(&sm.sb_ready);
            if (qd < 2) {                           // part 0: P1, part 1: P2
                if (!mbar_wait_suspend(&sm.sc_full, i & 1, abort_flag, err, 0xc510)) break;
                tc_fence_after();
                mask_scores<false, 64>(lane_addr + SC + part * 64, r, 0, a.scale);
                tc_fence_before();
                arrive(&sm.p_ready);
            }
            if (!mbar_wait_suspend(&sm.o_full, i & 1, abort_flag, err, 0xc520)) break;
            tc_fence_after();
            if (qd < 2) {
#pragma unroll 1
                for (int c = 0; c < 64; c += 32) {  // every product has read K and V
                    uint32_t x[32], y[32];
                    tmem_ld32(lane_addr + DV + part * 64 + c, x);
                    tmem_ld32(lane_addr + DK + part * 64 + c, y);
                    tmem_ld_wait();
                    store32(sm.v[s] + part * BLOCK, r, c / 8, x, 1.f);
                    store32(sm.k[s] + part * BLOCK, r, c / 8, y, 1.f);
                }
                fence_async();
                arrive(&sm.o_ready[s]);
            }
        }
    }
    free_tmem(tmem_base, warp, TMEM_COLS);
}

// [B, T, H, D] bf16 with element strides; dimensions of size one take a stride of their own (theirs may be anything)
static int map_of(CUtensorMap* m, const bf16* p, const GlaArgs& a, int64_t sb, int64_t st, int64_t sh) {
    if (a.H == 1) sh = D;
    if (a.T == 1) st = sh * a.H;
    if (a.B == 1) sb = st * a.T;
    return fatc::make_map_4d(m, p, a.B, a.T, a.H, D, sb, st, sh, CT);
}
// the gates: [B, T, H, D] fp32, dense, tokens of a chunk by TMA
static int gates_map(CUtensorMap* m, const GlaArgs& a) {
    auto enc = fatc::get_encode();
    if (enc == nullptr) return -10;
    const cuuint64_t row = (cuuint64_t)D * 4, dims[4] = {D, (cuuint64_t)a.H, (cuuint64_t)a.T, (cuuint64_t)a.B}, strides[3] = {row, row * a.H, row * a.H * a.T};
    const cuuint32_t box[4] = {D, 1, CT, 1}, estr[4] = {1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(a.gk), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -11;
}
template <typename K>
static int set_smem(K kernel, size_t bytes) { return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); }

// which as in lmoe_gla_launch; positive strides
int launch(int which, const GlaArgs& a, Maps& m, cudaStream_t st) {
    if (a.err == nullptr) return -1;
    dim3 grid(a.G, a.B * a.H);
    CUtensorMap o, dk, dv;
    int rc = 0;
    auto want = [&](unsigned bit, auto make) { if (!(m.made & bit)) { rc |= make(); m.made |= bit; } };
    want(1, [&] { return gates_map(&m.gk, a); });
    if (which == 1 || which == 2 || which == 4) want(2, [&] { return map_of(&m.q, a.q, a, a.qs_b, a.qs_t, a.qs_h); });
    if (which != 1) {
        want(4, [&] { return map_of(&m.k, a.k, a, a.ks_b, a.ks_t, a.ks_h); });
        want(8, [&] { return map_of(&m.v, a.v, a, a.vs_b, a.vs_t, a.vs_h); });
    }
    if (which == 1 || which == 3 || which == 4) want(16, [&] { return map_of(&m.g, a.d_o, a, (int64_t)a.T * a.H * D, (int64_t)a.H * D, D); });
    if (which == 2) rc |= map_of(&o, a.o, a, (int64_t)a.T * a.H * D, (int64_t)a.H * D, D);
    if (which == 3) rc |= map_of(&o, a.dq, a, a.dqs_b, a.dqs_t, a.dqs_h);
    if (which == 4) { rc |= map_of(&dk, a.dk, a, a.dks_b, a.dks_t, a.dks_h); rc |= map_of(&dv, a.dv, a, a.dvs_b, a.dvs_t, a.dvs_h); }
    if (rc) return -11;
    if (which == 0 || which == 1) {
        const size_t smem = sizeof(SmemState) + 1024;
        rc = which == 0 ? set_smem(gla_state_tc_kernel<0>, smem) : set_smem(gla_state_tc_kernel<1>, smem);
        if (rc) return rc;
        if (which == 0) gla_state_tc_kernel<0><<<grid, ST_THREADS, smem, st>>>(m.k, m.v, m.gk, a);
        else gla_state_tc_kernel<1><<<grid, ST_THREADS, smem, st>>>(m.q, m.g, m.gk, a);
    } else if (which == 2 || which == 3) {
        const size_t smem = sizeof(SmemSweep) + 1024;
        rc = which == 2 ? set_smem(gla_sweep_tc_kernel<0>, smem) : set_smem(gla_sweep_tc_kernel<1>, smem);
        if (rc) return rc;
        if (which == 2) gla_sweep_tc_kernel<0><<<grid, THREADS, smem, st>>>(m.q, m.k, m.v, o, m.gk, a);
        else gla_sweep_tc_kernel<1><<<grid, THREADS, smem, st>>>(m.g, m.k, m.v, o, m.gk, a);
    } else if (which == 4) {
        const size_t smem = sizeof(SmemDkv);
        rc = set_smem(gla_dkv_tc_kernel, smem);
        if (rc) return rc;
        gla_dkv_tc_kernel<<<grid, THREADS, smem, st>>>(m.q, m.k, m.v, m.g, dk, dv, m.gk, a);
    } else return -1;
    return (int)cudaGetLastError();
}

}  // namespace lvt
}  // namespace lmoe
