// The kernels of lsm_scalar.cu for 128-wide heads on the 5th-generation tensor cores: chunks of 128 tokens, every product a
// tcgen05.mma with its accumulator in tensor memory, tiles staged by TMA (4-D tensor maps over [B, T, H, D], 128-byte swizzle).
//
//   lsm_state_tc_kernel   group summaries.  Rows of X are scaled by the decay to the group's end (its start in the reverse
//                         direction), a running sum of log decays from chunk to chunk, so the sum over the whole group is one accumulation
//                         in tensor memory that nothing rescales.
//   lsm_sweep_tc_kernel   outputs and dq.  Per chunk, with S the state in front of it in fp32 registers and as a bf16 tile:
//                             scores X0 X1^T and X0 S | the threads: P = decayed, masked scores (bf16, over X0's tile), X0 S scaled in tensor
//                             memory, X1's rows by the decay to the chunk's end | state increment X2^T X1 (X1^T X2 for the outputs), + P X2 | S, output
//   lsm_dkv_tc_kernel     dk and dv, chunks in reverse order, with the state's gradient in registers: K Q^T, V dO^T, K dS, V dS^T | the threads:
//                             both decayed score tiles go back into tensor memory in bf16 as A operands, K dS and V dS^T are scaled there,
//                             Q scaled into V's tile | += P1 dO, += P2 Q, increment Q^T dO | dS, dk, dv
//
// 16 warps share a tile: the four with equal (w & 3) own the 32 rows of a tensor-memory lane quarter and split the 128 columns.
// A factor e^{b_i - b_j} of a score is one exponential per element only in the 32 x 32 blocks on the diagonal; in the others it is a row
// factor times a column factor around the block's edge, both at most one.
//
// A chunk brings 96 - 128 KB of tiles and takes away 32 - 64 KB, so memory is the bound that they approach: outputs and dq run at 0.49 of the DRAM
// peak, dk / dv at 0.44, with the tensor pipe active for 0.3 of the cycles; between that and the bound stands a chunk's score products waiting for
// the state of the chunk before.  mma.sync fragments of 16 x 64 tiles read shared memory 2.5 cycles per 2 cycles of tensor pipe with three
// to four barriers per 64 tokens: those kernels were at 18 - 22 % of DRAM.
// 16 heads of 16384 tokens: outputs 125 -> 59 us, dq 125 -> 63, dk / dv 232 -> 98, group summaries 50 -> 32 each.
#include "flash_tc_utils.cuh"
#include "lsm_scalar.cuh"

namespace lmoe {
namespace lst {
using namespace lmoe::tc;
using fatc::mbar_wait_suspend;
using fatc::tmem_st16;
using fatc::tmem_st_wait;
using fatc::tma_load_4d;
using fatc::umma_commit_if;
using fatc::umma_lo;

constexpr int D = 128, CT = 128, PARTS = 4, PW = CT / PARTS;           // PW: columns of a tile per thread
constexpr int TILE = CT * D * 2, BLOCK = CT * 128;                      // a tile: two blocks of [128 rows x 64 columns], 128-byte swizzled rows
constexpr int WARPS = 16, THREADS = 96 + 32 * WARPS;                    // warps 0: TMA, 1: MMA, 2: decay tables, 3..18: the rest
constexpr int SWARPS = 8, STHREADS = 96 + 32 * SWARPS, SSTAGES = 3;
constexpr uint32_t TMEM_COLS = 512;

// A tile's rows as the K dimension (MN-major) or as M / N (K-major); K-steps of 16.
template <bool MN>
__device__ __forceinline__ uint32_t tile_lo(uint32_t saddr) { return ((saddr >> 4) & 0x3FFFu) | ((MN ? (uint32_t)(BLOCK >> 4) : 1u) << 16); }
template <bool MN>
__device__ __forceinline__ constexpr uint32_t step_lo(int kk) { return MN ? (kk * 2048) >> 4 : ((kk / 4) * BLOCK + (kk % 4) * 32) >> 4; }
template <bool A_MN, bool B_MN>
__host__ __device__ constexpr uint32_t idesc() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((A_MN ? 1u : 0u) << 15) | ((B_MN ? 1u : 0u) << 16) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// [128 x 128] (+)= A B over 128
template <bool A_MN, bool B_MN>
__device__ __forceinline__ void product(uint32_t tmem_d, const void* a, const void* b, bool add, uint32_t issue) {
    const uint32_t al = tile_lo<A_MN>(s32(a)), bl = tile_lo<B_MN>(s32(b));
#pragma unroll
    for (int kk = 0; kk < 8; ++kk)
        umma_lo(tmem_d, al + step_lo<A_MN>(kk), bl + step_lo<B_MN>(kk), idesc<A_MN, B_MN>(), (add || kk > 0) ? 1u : 0u, issue);
}
// [128 x 128] += A B over 128 with A in tensor memory as the threads' parts leave it: 16 packed columns at the start of every 32
__device__ __forceinline__ void product_ta(uint32_t tmem_d, uint32_t tmem_a, const void* b, uint32_t issue) {
    const uint32_t bl = tile_lo<true>(s32(b));
#pragma unroll
    for (int kk = 0; kk < 8; ++kk)
        fatc::umma_ta(tmem_d, tmem_a + kk / 2 * 32 + kk % 2 * 8, bl + step_lo<true>(kk), idesc<false, true>(), 1u, issue);
}
__device__ __forceinline__ void load_half(float (&v)[16], uint32_t taddr) {
    uint32_t x[16];
    fatc::tmem_ld16(taddr, x);
    tmem_ld_wait();
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(x[e]);
}
// the thread's 32 columns, in place
__device__ __forceinline__ void scale_part(uint32_t taddr, float f) {
#pragma unroll
    for (int c = 0; c < PW; c += 16) {
        uint32_t x[16];
        fatc::tmem_ld16(taddr + c, x);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = __float_as_uint(f * __uint_as_float(x[e]));
        tmem_st16(taddr + c, x);
    }
}
// S = gamma S + increment
__device__ __forceinline__ void update_state(float (&S)[PW], uint32_t taddr, float gamma) {
#pragma unroll
    for (int c = 0; c < PW; c += 16) {
        uint32_t x[16];
        fatc::tmem_ld16(taddr + c, x);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) S[c + e] = gamma * S[c + e] + __uint_as_float(x[e]);
    }
}
__device__ __forceinline__ uint4 packed8(const uint32_t* v) {
    return make_uint4(pack_bf16(__uint_as_float(v[0]), __uint_as_float(v[1])), pack_bf16(__uint_as_float(v[2]), __uint_as_float(v[3])),
                      pack_bf16(__uint_as_float(v[4]), __uint_as_float(v[5])), pack_bf16(__uint_as_float(v[6]), __uint_as_float(v[7])));
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
// the 64 bytes (four 16-byte chunks) of a tile that belong to row r and column part `part`
__device__ __forceinline__ uint4* chunk(uint8_t* tile, int r, int part, int i) {
    return reinterpret_cast<uint4*>(tile + (part >> 1) * BLOCK + r * 128 + ((((part & 1) * 4 + i) ^ (r & 7)) << 4));
}
__device__ __forceinline__ uint4 scaled(uint4 x, float f) {
    uint32_t* u = reinterpret_cast<uint32_t*>(&x);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[e]));
        u[e] = pack_bf16(v.x * f, v.y * f);
    }
    return x;
}
// numbers as bf16 into the tile, from 16-byte chunk `first` of the part on
template <int N>
__device__ __forceinline__ void store_part(uint8_t* tile, int r, int part, const float (&v)[N], int first = 0) {
#pragma unroll
    for (int i = 0; i < N / 8; ++i)
        *chunk(tile, r, part, first + i) = make_uint4(pack_bf16(v[8 * i], v[8 * i + 1]), pack_bf16(v[8 * i + 2], v[8 * i + 3]),
                                                      pack_bf16(v[8 * i + 4], v[8 * i + 5]), pack_bf16(v[8 * i + 6], v[8 * i + 7]));
}

// Inclusive sums of the log decays of chunk `c`: four tokens per lane, into `b` (tokens 4 l .. 4 l + 3); returns the chunk's total.
__device__ __forceinline__ float chunk_decays(const LsmArgs& a, int bi, int h, int c, float (&b)[4]) {
    const int l = threadIdx.x & 31, t0 = c * CT + 4 * l;
    float g[4] = {0.f, 0.f, 0.f, 0.f};
    if (a.gmode != 0) {
        const float gh = a.gmode == 1 ? a.g[h] : 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (t0 + e < a.T) g[e] = a.gmode == 1 ? gh : a.g[((int64_t)bi * a.T + t0 + e) * a.H + h];
    }
    g[1] += g[0]; g[2] += g[1]; g[3] += g[2];
    float s = g[3];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float x = __shfl_up_sync(0xffffffffu, s, o);
        if (l >= o) s += x;
    }
    const float before = s - g[3];
#pragma unroll
    for (int e = 0; e < 4; ++e) b[e] = before + g[e];
    return __shfl_sync(0xffffffffu, s, 31);
}

// 16 score columns (from column c of its part) of a thread's row, decayed and masked: LOWER (rows are queries): columns up to the row, else
// from it on.  `tab`: the column factors; `row`: this block's row factor; `lb`: the sums, used in the blocks on the diagonal.
template <bool LOWER>
__device__ __forceinline__ void decay_scores(float (&v)[16], uint32_t taddr, int c, int r, int qd, int part, const float* lb, const float* tab, float row, float b_r, float scale) {
    if (LOWER ? part > qd : part < qd) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = 0.f;
        return;
    }
    load_half(v, taddr + c);
    if (part != qd) {
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
            const float4 f = *reinterpret_cast<const float4*>(tab + part * PW + c + j);
            v[j] *= row * f.x; v[j + 1] *= row * f.y; v[j + 2] *= row * f.z; v[j + 3] *= row * f.w;
        }
    } else {
        const int own = r - part * PW - c;
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
            const float4 f = *reinterpret_cast<const float4*>(lb + part * PW + c + j);
            const float* fp = reinterpret_cast<const float*>(&f);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float x = LOWER ? b_r - fp[e] : fp[e] - b_r;
                v[j + e] = (LOWER ? j + e <= own : j + e >= own) ? v[j + e] * (__expf(x) * scale) : 0.f;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------
struct __align__(1024) SmemState {
    uint8_t x[SSTAGES][TILE], y[SSTAGES][TILE];
    float tab[SSTAGES][CT];
    uint64_t full[SSTAGES], empty[SSTAGES], tab_full[SSTAGES], ready[SSTAGES], done;
    uint32_t tmem_base;
    int abort_flag;
};

template <int REV>
__global__ void __launch_bounds__(STHREADS, 1)
lsm_state_tc_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmY, LsmArgs a) {
    extern __shared__ uint8_t smem_raw[];
    SmemState& sm = *reinterpret_cast<SmemState*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = fatc::uniform_warp(), lane = threadIdx.x & 31;
    const int grp = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int nchunks = (a.T + CT - 1) / CT, cpg = a.cpg / 2;                    // cpg counts chunks of 64
    const int c_lo = grp * cpg, n = max(0, min(nchunks, c_lo + cpg) - c_lo);
    // towards the group's end (forward) or start (reverse): the running sum covers the chunks that are done
    auto at = [&](int i) { return REV ? c_lo + i : c_lo + n - 1 - i; };
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    if (threadIdx.x == 0) {
        for (int s = 0; s < SSTAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); mbar_init(&sm.tab_full[s], 1); mbar_init(&sm.ready[s], SWARPS); }
        mbar_init(&sm.done, 1);
        sm.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(s32(&sm.tmem_base)), "r"(128) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = fatc::uniform(sm.tmem_base);

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < n; ++i) {
                const int s = i % SSTAGES;
                if (!mbar_wait_suspend(&sm.empty[s], ((i / SSTAGES) & 1) ^ 1, abort_flag, err, 0x7100 | s)) break;
                mbar_expect_tx(&sm.full[s], 2 * TILE);
                tma_tile(sm.x[s], &tmX, &sm.full[s], h, at(i) * CT, b);
                tma_tile(sm.y[s], &tmY, &sm.full[s], h, at(i) * CT, b);
            }
        }
    } else if (warp == 1) {
        const uint32_t issue = lane == 0 ? 1u : 0u;
        bool ok = true;
        for (int i = 0; ok && i < n; ++i) {
            const int s = i % SSTAGES;
            ok = fatc::mbar_wait_warp(&sm.ready[s], (i / SSTAGES) & 1, abort_flag, err, 0x7200 | s);
            if (!ok) break;
            tc_fence_after();
            product<true, true>(tmem_base, sm.x[s], sm.y[s], i > 0, issue);
            umma_commit_if(&sm.empty[s], issue);
        }
        if (ok) umma_commit_if(&sm.done, issue);
    } else if (warp == 2) {
        float run = 0.f;
        bool ok = true;
        for (int i = 0; ok && i < n; ++i) {
            const int s = i % SSTAGES;
            float bl[4];
            const float tot = chunk_decays(a, b, h, at(i), bl);
            ok = mbar_wait_suspend(&sm.empty[s], ((i / SSTAGES) & 1) ^ 1, abort_flag, err, 0x7300 | s);
            if (!ok) break;
            float4 f;
            f.x = __expf(REV ? run + bl[0] : run + (tot - bl[0])); f.y = __expf(REV ? run + bl[1] : run + (tot - bl[1]));
            f.z = __expf(REV ? run + bl[2] : run + (tot - bl[2])); f.w = __expf(REV ? run + bl[3] : run + (tot - bl[3]));
            *reinterpret_cast<float4*>(&sm.tab[s][4 * lane]) = f;
            run += tot;
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.tab_full[s]);
        }
        if (lane == 0 && a.gdecay != nullptr) a.gdecay[(int64_t)bh * a.G + grp] = run;
    } else if (warp >= 3) {
        const int tid = threadIdx.x - 96;
        bool ok = true;
        for (int i = 0; ok && i < n; ++i) {
            const int s = i % SSTAGES;
            const uint32_t ph = (i / SSTAGES) & 1;
            ok = mbar_wait_suspend(&sm.full[s], ph, abort_flag, err, 0x7400 | s) && mbar_wait_suspend(&sm.tab_full[s], ph, abort_flag, err, 0x7500 | s);
            if (!ok) break;
            if (a.gmode != 0) {                                                  // row factors; a chunk's place inside its row does not matter
#pragma unroll
                for (int x = 0; x < TILE / 16; x += 32 * SWARPS) {
                    uint4* p = reinterpret_cast<uint4*>(sm.x[s]) + x + tid;
                    *p = scaled(*p, sm.tab[s][((x + tid) >> 3) & (CT - 1)]);
                }
                fence_async();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.ready[s]);
        }
        const int r = (warp & 3) * 32 + lane, half = (warp - 3) >> 2;
        float* out = a.states + (((int64_t)bh * a.G + grp) * D + r) * D + half * 64;
        const float mul = REV ? a.scale : 1.f;
        if (ok && n > 0) ok = mbar_wait_suspend(&sm.done, 0, abort_flag, err, 0x7600);
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
            uint32_t v[32];
            tmem_ld32(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + half * 64 + c, v);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; e += 4)
                *reinterpret_cast<float4*>(out + c + e) = n > 0 ? make_float4(mul * __uint_as_float(v[e]), mul * __uint_as_float(v[e + 1]),
                                                                              mul * __uint_as_float(v[e + 2]), mul * __uint_as_float(v[e + 3])) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(128) : "memory");
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Two stages of three tiles and the state fill the 227 KB: the dynamic shared memory starts on a 1024-byte boundary (there is no static one),
// which the kernel checks before anything else.
struct __align__(1024) SmemSweep {
    uint8_t t0[2][TILE], t1[2][TILE], t2[2][TILE], sb[TILE];
    float lb[2][CT], tab[2][CT];                    // sums of the log decays; column factors e^{b of the block's last - b_j}
    uint64_t full[2], empty[2], tab_full[2], tab_empty[2], sb_ready, c1, p_ready, c2, o_full, o_ready[2];
    uint32_t tmem_base;
    int abort_flag;
};

// MODE 0: X0 = Q, X1 = K, X2 = V, out = o.  MODE 1: X0 = dO, X1 = V, X2 = K, out = dq (and the state is read transposed).
template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
lsm_sweep_tc_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1, const __grid_constant__ CUtensorMap tm2,
                    const __grid_constant__ CUtensorMap tmO, LsmArgs a) {
    extern __shared__ uint8_t smem_raw[];
    SmemSweep& sm = *reinterpret_cast<SmemSweep*>(smem_raw);
    if ((s32(smem_raw) & 1023u) != 0) {             // the swizzled tiles need it
        if (threadIdx.x == 0) atomicCAS(a.err, 0, 0x8001);
        return;
    }
    constexpr uint32_t SC = 0, DS = 128, OUT = 256;                              // columns of tensor memory; two outputs take turns
    const int warp = fatc::uniform_warp(), lane = threadIdx.x & 31;
    const int grp = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int nchunks = (a.T + CT - 1) / CT, cpg = a.cpg / 2;
    const int c_lo = grp * cpg, n = max(0, min(nchunks, c_lo + cpg) - c_lo);
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); mbar_init(&sm.tab_full[s], 1); mbar_init(&sm.tab_empty[s], WARPS); mbar_init(&sm.o_ready[s], WARPS); }
        mbar_init(&sm.sb_ready, WARPS); mbar_init(&sm.p_ready, WARPS);
        mbar_init(&sm.c1, 1); mbar_init(&sm.c2, 1); mbar_init(&sm.o_full, 1);
        sm.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(s32(&sm.tmem_base)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = fatc::uniform(sm.tmem_base);

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < n; ++i) {
                const int s = i & 1, t0 = (c_lo + i) * CT;
                if (!mbar_wait_suspend(&sm.empty[s], ((i >> 1) & 1) ^ 1, abort_flag, err, 0x8100 | s)) break;
                mbar_expect_tx(&sm.full[s], 3 * TILE);
                tma_tile(sm.t0[s], &tm0, &sm.full[s], h, t0, b);
                tma_tile(sm.t1[s], &tm1, &sm.full[s], h, t0, b);
                tma_tile(sm.t2[s], &tm2, &sm.full[s], h, t0, b);
            }
        }
    } else if (warp == 1) {
        const uint32_t issue = lane == 0 ? 1u : 0u;
        for (int i = 0; i < n; ++i) {
            const int s = i & 1;
            if (!fatc::mbar_wait_warp(&sm.full[s], (i >> 1) & 1, abort_flag, err, 0x8200 | s)) break;
            if (!fatc::mbar_wait_warp(&sm.sb_ready, i & 1, abort_flag, err, 0x8210)) break;
            tc_fence_after();
            product<false, false>(tmem_base + SC, sm.t0[s], sm.t1[s], false, issue);
            product<false, MODE == 0>(tmem_base + OUT + s * 128, sm.t0[s], sm.sb, false, issue);      // X0 S: rows of S are K; X0 S^T: rows of S are N
            umma_commit_if(&sm.c1, issue);
            if (!fatc::mbar_wait_warp(&sm.p_ready, i & 1, abort_flag, err, 0x8220)) break;
            tc_fence_after();
            if (MODE == 0) product<true, true>(tmem_base + DS, sm.t1[s], sm.t2[s], false, issue);
            else product<true, true>(tmem_base + DS, sm.t2[s], sm.t1[s], false, issue);
            umma_commit_if(&sm.c2, issue);
            product<false, true>(tmem_base + OUT + s * 128, sm.t0[s], sm.t2[s], true, issue);   // + P X2
            umma_commit_if(&sm.o_full, issue);
        }
    } else if (warp == 2) {                         // decay tables, and the outputs' way to memory
        auto tables = [&](int i) -> bool {
            const int s = i & 1;
            float bl[4];
            chunk_decays(a, b, h, c_lo + i, bl);
            if (!mbar_wait_suspend(&sm.tab_empty[s], ((i >> 1) & 1) ^ 1, abort_flag, err, 0x8300 | s)) return false;
            *reinterpret_cast<float4*>(&sm.lb[s][4 * lane]) = make_float4(bl[0], bl[1], bl[2], bl[3]);
            const float ref = __shfl_sync(0xffffffffu, bl[3], lane | 7);                        // last token of the block of 32
            *reinterpret_cast<float4*>(&sm.tab[s][4 * lane]) = make_float4(__expf(ref - bl[0]), __expf(ref - bl[1]), __expf(ref - bl[2]), __expf(ref - bl[3]));
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.tab_full[s]);
            return true;
        };
        bool ok = n < 1 || tables(0);
        if (ok && n > 1) ok = tables(1);
        for (int i = 0; ok && i < n; ++i) {
            const int s = i & 1;
            ok = mbar_wait_suspend(&sm.o_ready[s], (i >> 1) & 1, abort_flag, err, 0x8310 | s);
            if (!ok) break;
            if (lane == 0) {
                tma_store(&tmO, sm.t0[s], h, (c_lo + i) * CT, b);
                fatc::tma_store_commit();
                fatc::tma_store_wait_read();
                mbar_arrive(&sm.empty[s]);
            }
            __syncwarp();
            if (i + 2 < n) ok = tables(i + 2);
        }
        if (lane == 0) fatc::tma_store_wait();
    } else if (warp >= 3) {
        const int qd = warp & 3, part = (warp - 3) >> 2, r = qd * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16) + part * PW;
        float S[PW];                                                                            // row r of the state, the part's columns
        {
            const float* src = a.states + (((int64_t)bh * a.G + grp) * D + r) * D + part * PW;
#pragma unroll
            for (int e = 0; e < PW; e += 4) {
                const float4 x = *reinterpret_cast<const float4*>(src + e);
                S[e] = x.x; S[e + 1] = x.y; S[e + 2] = x.z; S[e + 3] = x.w;
            }
        }
        auto publish_state = [&]() {
            store_part(sm.sb, r, part, S);
            fence_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.sb_ready);
        };
        publish_state();
        for (int i = 0; i < n; ++i) {
            const int s = i & 1;
            if (!mbar_wait_suspend(&sm.tab_full[s], (i >> 1) & 1, abort_flag, err, 0x8400 | s)) break;
            const float* lb = sm.lb[s];
            const float b_r = lb[r], b_c = lb[CT - 1];
            const float row = __expf(b_r - lb[part * PW + PW - 1]) * a.scale;                   // meaningful where the block lies below the row
            const float into = __expf(b_r) * a.scale, gamma = __expf(b_c), rest = __expf(b_c - b_r);
            if (!mbar_wait_suspend(&sm.c1, i & 1, abort_flag, err, 0x8410)) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < PW; c += 16) {
                float o[16];
                decay_scores<true>(o, lane_addr + SC, c, r, qd, part, lb, sm.tab[s], row, b_r, a.scale);
                store_part(sm.t0[s], r, part, o, c / 8);                                        // X0 has been read: P over it
            }
            scale_part(lane_addr + OUT + s * 128, into);                                        // X0 S, row by row
            if (a.gmode != 0) {
#pragma unroll
                for (int e = 0; e < 4; ++e) { uint4* p = chunk(sm.t1[s], r, part, e); *p = scaled(*p, rest); }
            }
            tmem_st_wait();
            fence_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&sm.p_ready); mbar_arrive(&sm.tab_empty[s]); }
            if (!mbar_wait_suspend(&sm.c2, i & 1, abort_flag, err, 0x8420)) break;
            tc_fence_after();
            update_state(S, lane_addr + DS, gamma);
            publish_state();                                                                    // the next chunk's products may start
            if (!mbar_wait_suspend(&sm.o_full, i & 1, abort_flag, err, 0x8430)) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < PW; c += 16) {
                float o[16];
                load_half(o, lane_addr + OUT + s * 128 + c);
                store_part(sm.t0[s], r, part, o, c / 8);                                        // P has been read
            }
            fence_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.o_ready[s]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Q and dO in two stages, K and V in one: V's tile holds scaled Q once V has been read, K's and V's next tiles come in as soon as their
// readers are done.
struct __align__(1024) SmemDkv {
    uint8_t q[2][TILE], g[2][TILE], k[TILE], v[TILE], db[TILE];
    float lb[2][CT], tab[2][CT];                    // sums of the log decays; column factors e^{b_i - b of the block's first}
    uint64_t qg_full[2], qg_empty[2], k_full, k_empty, v_full, v_empty, tab_full[2], tab_empty[2], db_ready, c1, p_ready, p1_done, acc_full, o_ready[2];
    uint32_t tmem_base;
    int abort_flag;
};

__global__ void __launch_bounds__(THREADS, 1)
lsm_dkv_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                  const __grid_constant__ CUtensorMap tmG, const __grid_constant__ CUtensorMap tmDK, const __grid_constant__ CUtensorMap tmDV, LsmArgs a) {
    extern __shared__ uint8_t smem_raw[];
    SmemDkv& sm = *reinterpret_cast<SmemDkv*>(smem_raw);
    if ((s32(smem_raw) & 1023u) != 0) {
        if (threadIdx.x == 0) atomicCAS(a.err, 0, 0x9001);
        return;
    }
    constexpr uint32_t AT = 0, BT = 128, DV = 256, DK = 384;                     // AT: K Q^T, P1, then the state increment
    const int warp = fatc::uniform_warp(), lane = threadIdx.x & 31;
    const int grp = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int nchunks = (a.T + CT - 1) / CT, cpg = a.cpg / 2;
    const int c_lo = grp * cpg, n = max(0, min(nchunks, c_lo + cpg) - c_lo), c_last = c_lo + n - 1;
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) { mbar_init(&sm.qg_full[s], 1); mbar_init(&sm.qg_empty[s], 1); mbar_init(&sm.tab_full[s], 1); mbar_init(&sm.tab_empty[s], WARPS); mbar_init(&sm.o_ready[s], WARPS); }
        mbar_init(&sm.k_full, 1); mbar_init(&sm.k_empty, 1); mbar_init(&sm.v_full, 1); mbar_init(&sm.v_empty, 1);
        mbar_init(&sm.db_ready, WARPS); mbar_init(&sm.p_ready, WARPS);
        mbar_init(&sm.c1, 1); mbar_init(&sm.p1_done, 1); mbar_init(&sm.acc_full, 1);
        sm.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(s32(&sm.tmem_base)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = fatc::uniform(sm.tmem_base);

    if (warp == 0) {
        if (lane == 0) {
            auto load_qg = [&](int i) -> bool {
                const int s = i & 1, t0 = (c_last - i) * CT;
                if (!mbar_wait_suspend(&sm.qg_empty[s], ((i >> 1) & 1) ^ 1, abort_flag, err, 0x9100 | s)) return false;
                mbar_expect_tx(&sm.qg_full[s], 2 * TILE);
                tma_tile(sm.q[s], &tmQ, &sm.qg_full[s], h, t0, b);
                tma_tile(sm.g[s], &tmG, &sm.qg_full[s], h, t0, b);
                return true;
            };
            bool ok = n > 0 && load_qg(0);
            for (int i = 0; ok && i < n; ++i) {
                const int t0 = (c_last - i) * CT;
                ok = mbar_wait_suspend(&sm.k_empty, (i & 1) ^ 1, abort_flag, err, 0x9110);
                if (!ok) break;
                mbar_expect_tx(&sm.k_full, TILE);
                tma_tile(sm.k, &tmK, &sm.k_full, h, t0, b);
                ok = mbar_wait_suspend(&sm.v_empty, (i & 1) ^ 1, abort_flag, err, 0x9120);
                if (!ok) break;
                mbar_expect_tx(&sm.v_full, TILE);
                tma_tile(sm.v, &tmV, &sm.v_full, h, t0, b);
                if (i + 1 < n) ok = load_qg(i + 1);
            }
        }
    } else if (warp == 1) {
        const uint32_t issue = lane == 0 ? 1u : 0u;
        for (int i = 0; i < n; ++i) {
            const int s = i & 1;
            if (!fatc::mbar_wait_warp(&sm.qg_full[s], (i >> 1) & 1, abort_flag, err, 0x9200 | s)) break;
            if (!fatc::mbar_wait_warp(&sm.k_full, i & 1, abort_flag, err, 0x9210)) break;
            if (!fatc::mbar_wait_warp(&sm.v_full, i & 1, abort_flag, err, 0x9220)) break;
            if (!fatc::mbar_wait_warp(&sm.db_ready, i & 1, abort_flag, err, 0x9230)) break;       // also: the accumulators of chunk i - 1 have been read
            tc_fence_after();
            product<false, false>(tmem_base + AT, sm.k, sm.q[s], false, issue);                // K Q^T
            product<false, true>(tmem_base + DV, sm.k, sm.db, false, issue);                   // K dS
            umma_commit_if(&sm.k_empty, issue);
            product<false, false>(tmem_base + BT, sm.v, sm.g[s], false, issue);                // V dO^T
            product<false, false>(tmem_base + DK, sm.v, sm.db, false, issue);                  // V dS^T
            umma_commit_if(&sm.c1, issue);
            if (!fatc::mbar_wait_warp(&sm.p_ready, i & 1, abort_flag, err, 0x9240)) break;
            tc_fence_after();
            product_ta(tmem_base + DV, tmem_base + AT, sm.g[s], issue);                        // += P1 dO
            umma_commit_if(&sm.p1_done, issue);
            product_ta(tmem_base + DK, tmem_base + BT, sm.q[s], issue);                        // += P2 Q
            if (!fatc::mbar_wait_warp(&sm.p1_done, i & 1, abort_flag, err, 0x9250)) break;        // over P1 goes
            product<true, true>(tmem_base + AT, sm.v, sm.g[s], false, issue);                  // (scaled Q)^T dO
            umma_commit_if(&sm.v_empty, issue);
            umma_commit_if(&sm.acc_full, issue);
        }
    } else if (warp == 2) {
        auto tables = [&](int i) -> bool {
            const int s = i & 1;
            float bl[4];
            chunk_decays(a, b, h, c_last - i, bl);
            if (!mbar_wait_suspend(&sm.tab_empty[s], ((i >> 1) & 1) ^ 1, abort_flag, err, 0x9300 | s)) return false;
            *reinterpret_cast<float4*>(&sm.lb[s][4 * lane]) = make_float4(bl[0], bl[1], bl[2], bl[3]);
            const float ref = __shfl_sync(0xffffffffu, bl[0], lane & 24);                       // first token of the block of 32
            *reinterpret_cast<float4*>(&sm.tab[s][4 * lane]) = make_float4(__expf(bl[0] - ref), __expf(bl[1] - ref), __expf(bl[2] - ref), __expf(bl[3] - ref));
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.tab_full[s]);
            return true;
        };
        bool ok = n < 1 || tables(0);
        if (ok && n > 1) ok = tables(1);
        for (int i = 0; ok && i < n; ++i) {
            const int s = i & 1;
            ok = mbar_wait_suspend(&sm.o_ready[s], (i >> 1) & 1, abort_flag, err, 0x9310 | s);
            if (!ok) break;
            if (lane == 0) {
                tma_store(&tmDV, sm.g[s], h, (c_last - i) * CT, b);
                tma_store(&tmDK, sm.q[s], h, (c_last - i) * CT, b);
                fatc::tma_store_commit();
                fatc::tma_store_wait_read();
                mbar_arrive(&sm.qg_empty[s]);
            }
            __syncwarp();
            if (i + 2 < n) ok = tables(i + 2);
        }
        if (lane == 0) fatc::tma_store_wait();
    } else if (warp >= 3) {
        const int qd = warp & 3, part = (warp - 3) >> 2, r = qd * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16) + part * PW;
        float S[PW];                                                                            // row r of dS, the part's columns
        {
            const float* src = a.states + (((int64_t)bh * a.G + grp) * D + r) * D + part * PW;
#pragma unroll
            for (int e = 0; e < PW; e += 4) {
                const float4 x = *reinterpret_cast<const float4*>(src + e);
                S[e] = x.x; S[e + 1] = x.y; S[e + 2] = x.z; S[e + 3] = x.w;
            }
        }
        auto publish_state = [&]() {
            store_part(sm.db, r, part, S);
            fence_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.db_ready);
        };
        publish_state();
        for (int i = 0; i < n; ++i) {
            const int s = i & 1;
            if (!mbar_wait_suspend(&sm.tab_full[s], (i >> 1) & 1, abort_flag, err, 0x9400 | s)) break;
            const float* lb = sm.lb[s];
            const float b_r = lb[r], b_c = lb[CT - 1];
            const float row = __expf(lb[part * PW] - b_r) * a.scale;                            // meaningful where the block lies right of the row
            const float into = __expf(b_r) * a.scale, gamma = __expf(b_c), rest = __expf(b_c - b_r);
            if (!mbar_wait_suspend(&sm.c1, i & 1, abort_flag, err, 0x9410)) break;
            tc_fence_after();
#pragma unroll
            for (int which = 0; which < 2; ++which) {                                           // K Q^T -> P1, V dO^T -> P2
                const uint32_t at = lane_addr + (which == 0 ? AT : BT);
                uint32_t p[16];                                                                 // packed over the first half of the scores
#pragma unroll
                for (int c = 0; c < PW; c += 16) {
                    float o[16];
                    decay_scores<false>(o, at, c, r, qd, part, lb, sm.tab[s], row, b_r, a.scale);
#pragma unroll
                    for (int e = 0; e < 8; ++e) p[c / 2 + e] = pack_bf16(o[2 * e], o[2 * e + 1]);
                }
                tmem_st16(at, p);
            }
            if (a.gmode != 0) {                                                                 // K dS and V dS^T, row by row
                scale_part(lane_addr + DV, rest);
                scale_part(lane_addr + DK, rest);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) *chunk(sm.v, r, part, e) = scaled(*chunk(sm.q[s], r, part, e), into);
            tmem_st_wait();
            fence_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&sm.p_ready); mbar_arrive(&sm.tab_empty[s]); }
            if (!mbar_wait_suspend(&sm.acc_full, i & 1, abort_flag, err, 0x9420)) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < PW; c += 16) {                                                  // every product has read Q and dO: dk and dv over them
                uint32_t x[16], y[16];
                fatc::tmem_ld16(lane_addr + DV + c, x);
                fatc::tmem_ld16(lane_addr + DK + c, y);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    *chunk(sm.g[s], r, part, c / 8 + e) = packed8(x + 8 * e);
                    *chunk(sm.q[s], r, part, c / 8 + e) = packed8(y + 8 * e);
                }
            }
            update_state(S, lane_addr + AT, gamma);
            publish_state();                                                                    // the next chunk's products may start
            fence_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.o_ready[s]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// [B, T, H, D] bf16 with element strides; dimensions of size one take a stride of their own (theirs may be anything)
static int map_of(CUtensorMap* m, const bf16* p, const LsmArgs& a, int64_t sb, int64_t st, int64_t sh) {
    if (a.H == 1) sh = D;
    if (a.T == 1) st = sh * a.H;
    if (a.B == 1) sb = st * a.T;
    return fatc::make_map_4d(m, p, a.B, a.T, a.H, D, sb, st, sh, CT);
}
template <typename K>
static int set_smem(K kernel, size_t bytes) { return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); }

// which as in lmoe_lsm_scalar_launch; 128-wide heads, groups of an even number of 64-token chunks, positive strides
int launch(int which, const LsmArgs& a, cudaStream_t st) {
    if (a.cpg % 2 || a.err == nullptr) return -1;
    dim3 grid(a.G, a.B * a.H);
    CUtensorMap q, k, v, g, o, dk, dv;
    int rc = 0;
    if (which != 0 && which != 3) rc |= map_of(&q, a.q, a, a.qs_b, a.qs_t, a.qs_h);
    if (which != 1) { rc |= map_of(&k, a.k, a, a.ks_b, a.ks_t, a.ks_h); rc |= map_of(&v, a.v, a, a.vs_b, a.vs_t, a.vs_h); }
    if (which == 1 || which == 3 || which == 4) rc |= map_of(&g, a.d_o, a, (int64_t)a.T * a.H * D, (int64_t)a.H * D, D);
    if (which == 2) rc |= map_of(&o, a.o, a, (int64_t)a.T * a.H * D, (int64_t)a.H * D, D);
    if (which == 3) rc |= map_of(&o, a.dq, a, a.dqs_b, a.dqs_t, a.dqs_h);
    if (which == 4) { rc |= map_of(&dk, a.dk, a, a.dks_b, a.dks_t, a.dks_h); rc |= map_of(&dv, a.dv, a, a.dvs_b, a.dvs_t, a.dvs_h); }
    if (rc) return -11;
    if (which == 0 || which == 1) {
        const size_t smem = sizeof(SmemState) + 1024;
        rc = which == 0 ? set_smem(lsm_state_tc_kernel<0>, smem) : set_smem(lsm_state_tc_kernel<1>, smem);
        if (rc) return rc;
        if (which == 0) lsm_state_tc_kernel<0><<<grid, STHREADS, smem, st>>>(k, v, a);
        else lsm_state_tc_kernel<1><<<grid, STHREADS, smem, st>>>(q, g, a);
    } else if (which == 2 || which == 3) {
        const size_t smem = sizeof(SmemSweep);
        rc = which == 2 ? set_smem(lsm_sweep_tc_kernel<0>, smem) : set_smem(lsm_sweep_tc_kernel<1>, smem);
        if (rc) return rc;
        if (which == 2) lsm_sweep_tc_kernel<0><<<grid, THREADS, smem, st>>>(q, k, v, o, a);
        else lsm_sweep_tc_kernel<1><<<grid, THREADS, smem, st>>>(g, v, k, o, a);
    } else if (which == 4) {
        const size_t smem = sizeof(SmemDkv);
        rc = set_smem(lsm_dkv_tc_kernel, smem);
        if (rc) return rc;
        lsm_dkv_tc_kernel<<<grid, THREADS, smem, st>>>(q, k, v, g, dk, dv, a);
    } else return -1;
    return (int)cudaGetLastError();
}

}  // namespace lst
}  // namespace lmoe
