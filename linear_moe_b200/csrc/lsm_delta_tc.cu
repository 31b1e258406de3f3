// The scans of lsm_delta.cu for 128-wide keys on the 5th-generation tensor cores: every product is a tcgen05.mma with its accumulator in tensor memory,
// the state stays there in fp32, tiles come and go by TMA.
//
//   forward, per chunk:  X = W S | Vn = U - X | S = gamma S + Kd^T Vn;  beside the chain O = Qd S + A Vn
//   reverse, per chunk:  X = A^T dO + Kd dS' | dVn = X | dS = gamma dS' + Qd^T dO - W^T dVn
//
// Both are chains over the chunks: a step is two products that wait for one another, with the threads' conversions between them (the state and Vn
// as bf16 tiles), so its latency is all that counts.  With mma.sync a step was 2900 cycles, most of it fragments from shared memory and two
// barriers of eight warps.  Here a product is eight instructions of one thread, a CTA takes 64 value columns instead of 32 (the tiles are read by half as
// many CTAs), and the outputs are made while the next step's first product runs.
// A tile of 64 rows stands where an instruction wants 128: the upper half of its accumulator holds products of what follows the tile in shared
// memory, and nobody reads it.
// 2 x 4096 tokens, 16 heads of 128 (64 CTAs, 64 chunks each): outputs 97 -> 90 us, reverse 95 -> 89, Vn and the states alone 82 -> 82 (with fewer heads, 2 x 64
// chunks, 71 -> 81: such scans stay with lsm_delta.cu); 2700 cycles a chunk, of which the two products of the chain and their latencies are about half.
// 64 heads x 26 chunks (128 CTAs against 256): outputs 82 -> 42, reverse 80 -> 42, Vn and the states 55 -> 37.
#include "flash_tc_utils.cuh"
#include "lsm_delta.cuh"

namespace lmoe {
namespace dr {
namespace tcs {
using namespace lmoe::tc;
using fatc::mbar_wait_suspend;
using fatc::tma_load_4d;
using fatc::tmem_st16;
using fatc::tmem_st_wait;
using fatc::elect_one;
using fatc::umma_ss;

constexpr int DK = 128, VS = 64;                                          // key width, value columns of a CTA
constexpr int BLOCK = C * 128;                                            // [64 rows x 64 columns], 128-byte swizzled rows
constexpr int TK = 2 * BLOCK, SBLOCK = DK * 128;                          // a tile of keys: two blocks; the state's tile: [128 x 64]
constexpr int STAGES = 3, WORKERS = 8, THREADS = 32 * (4 + WORKERS);      // warps 0: loads, 1: products, 2 and 3: stores, then the threads

template <bool MN, int BL>
__device__ __forceinline__ uint32_t tile_lo(const uint8_t* tile) { return ((s32(tile) >> 4) & 0x3FFFu) | ((MN ? (uint32_t)(BL >> 4) : 1u) << 16); }
template <bool MN, int BL>
__device__ __forceinline__ constexpr uint32_t step_lo(int kk) { return MN ? (kk * 2048) >> 4 : ((kk / 4) * BL + (kk % 4) * 32) >> 4; }
// [128 x 64] (+)= A B over 16 STEPS; B's rows are K
template <bool A_MN, int STEPS>
__device__ __forceinline__ void product(uint32_t tmem_d, const uint8_t* a, const uint8_t* b, bool add) {
    if (!elect_one()) return;
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((A_MN ? 1u : 0u) << 15) | (1u << 16) | ((uint32_t)(VS >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    const uint32_t al = tile_lo<A_MN, BLOCK>(a), bl = tile_lo<true, BLOCK>(b);
#pragma unroll
    for (int kk = 0; kk < STEPS; ++kk)
        umma_ss(tmem_d, al + step_lo<A_MN, BLOCK>(kk), bl + step_lo<true, BLOCK>(kk), idesc, add || kk > 0);
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void store_2d(const CUtensorMap* map, const uint8_t* src, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" :: "l"(map), "r"(s32(src)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void key_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int row) {
    tma_load_2d(dst, map, bar, 0, row);
    tma_load_2d(dst + BLOCK, map, bar, 64, row);
}
__device__ __forceinline__ void arrive(uint64_t* bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
// 32 numbers as bf16 into columns 32 part .. of row r of a tile of 64 columns
__device__ __forceinline__ void store32(uint8_t* tile, int r, int part, const float (&v)[32], float f = 1.f) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = pack_bf16(f * v[8 * i + 2 * e], f * v[8 * i + 2 * e + 1]);
        *reinterpret_cast<uint4*>(tile + r * 128 + (((part * 4 + i) ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}
__device__ __forceinline__ void load_tmem(float (&v)[32], uint32_t taddr) {
    uint32_t x[32];
    tmem_ld32(taddr, x);
    tmem_ld_wait();
#pragma unroll
    for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(x[e]);
}
__device__ __forceinline__ void store_tmem(uint32_t taddr, const float (&v)[32], float f) {
#pragma unroll
    for (int c = 0; c < 32; c += 16) {
        uint32_t x[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = __float_as_uint(f * v[c + e]);
        tmem_st16(taddr + c, x);
    }
}
__device__ __forceinline__ void load_row(float (&v)[32], const float* src) {
#pragma unroll
    for (int e = 0; e < 32; e += 4) {
        const float4 x = src == nullptr ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(src + e);
        v[e] = x.x; v[e + 1] = x.y; v[e + 2] = x.z; v[e + 3] = x.w;
    }
}
__device__ __forceinline__ void save_row(float* dst, const float (&v)[32]) {
#pragma unroll
    for (int e = 0; e < 32; e += 4) *reinterpret_cast<float4*>(dst + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
}

template <bool OUT> struct Stage;
template <> struct Stage<true> { uint8_t w[TK], kd[TK], qd[TK], a[BLOCK], x[BLOCK]; };       // x: U (then O), or dO
template <> struct Stage<false> { uint8_t w[TK], kd[TK], x[BLOCK]; };
template <bool OUT>
struct __align__(1024) Smem {
    Stage<OUT> st[STAGES];
    uint8_t sb[SBLOCK], vb[BLOCK], vneg[BLOCK];
    // Every wait goes by the parity of a phase, so a barrier must not be two phases ahead of whoever waits for it.  What keeps it from that, chunk n:
    //   full     its next phase wants empty, which comes behind everybody's use of the stage; empty: behind the one load that waits for it
    //   sb_ready the next is for chunk n + 1 and wants s_full (from the warp that issues products) and, where Sn and Vn are kept, kept (from the one that
    //            stores them); x_full, s_full, kept: the next wants sb_ready n + 1, where all eight warps of threads arrive behind these waits
    //   v_ready  the next wants x_full n + 1, and kept, so both of its waiters; o_full: the next wants v_ready n + 1, behind the outputs of chunk n
    //   o_ready  one per stage: the next of a stage wants full, so empty, so the store of the stage's outputs.  (With one for all of them the threads could get two
    //            chunks ahead of a slow store, which then waited for ever.)
    uint64_t full[STAGES], empty[STAGES], sb_ready, x_full, v_ready, s_full, o_full, o_ready[STAGES], kept;
    uint32_t tmem_base;
    int abort_flag;
};
template <bool OUT>
__device__ __forceinline__ uint32_t setup(Smem<OUT>& sm, int warp) {
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); mbar_init(&sm.o_ready[s], WORKERS / 2); }
        mbar_init(&sm.sb_ready, WORKERS); mbar_init(&sm.x_full, 1); mbar_init(&sm.v_ready, WORKERS / 2); mbar_init(&sm.s_full, 1);
        mbar_init(&sm.o_full, 1); mbar_init(&sm.kept, 1);
        sm.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(s32(&sm.tmem_base)), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    return fatc::uniform(sm.tmem_base);
}
__device__ __forceinline__ void finish(uint32_t base, int warp) {
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(base), "r"(256) : "memory");
    }
}
constexpr uint32_t ST = 0, X = 64, O = 128;                               // columns of tensor memory: state, first product, two outputs

struct Maps { CUtensorMap w, kd, qd, a, x, o, vn, sn; };                  // x: U or dO;  vn, sn: Vn and Sn, or dVn and dSn

// OUT: the outputs O are wanted (the forward pass); without: Vn and the entering states only (what the backward pass rebuilds).
template <bool OUT>
__global__ void __launch_bounds__(THREADS, 1) delta_scan_fwd_tc_kernel(const __grid_constant__ Maps m, Args a) {
    extern __shared__ uint8_t smem_raw[];
    Smem<OUT>& sm = *reinterpret_cast<Smem<OUT>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = fatc::uniform_warp(), lane = threadIdx.x & 31, col0 = blockIdx.x * VS, bh = blockIdx.y, row0 = bh * a.N * C;
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    const uint32_t tmem = setup(sm, warp);
    const bool keep = a.Vn != nullptr;

    if (warp == 0) {
        if (lane == 0) {
            for (int n = 0; n < a.N; ++n) {
                const int s = n % STAGES, row = row0 + n * C;
                if (!mbar_wait_suspend(&sm.empty[s], ((n / STAGES) & 1) ^ 1, abort_flag, err, 0xd100 | s)) break;
                mbar_expect_tx(&sm.full[s], sizeof(Stage<OUT>));
                Stage<OUT>& t = sm.st[s];
                key_tile(t.w, &m.w, &sm.full[s], row);
                tma_load_2d(t.x, &m.x, &sm.full[s], col0, row);
                key_tile(t.kd, &m.kd, &sm.full[s], row);
                if constexpr (OUT) {
                    key_tile(t.qd, &m.qd, &sm.full[s], row);
                    tma_load_2d(t.a, &m.a, &sm.full[s], 0, row);
                }
            }
        }
    } else if (warp == 1) {
        for (int n = 0; n < a.N; ++n) {
            const int s = n % STAGES;
            Stage<OUT>& t = sm.st[s];
            if (!fatc::mbar_wait_warp(&sm.full[s], (n / STAGES) & 1, abort_flag, err, 0xd200 | s)) break;
            if (!fatc::mbar_wait_warp(&sm.sb_ready, n & 1, abort_flag, err, 0xd210)) break;
            tc_fence_after();
            product<false, 8>(tmem + X, t.w, sm.sb, false);
            if (elect_one()) umma_commit(&sm.x_full);
            if constexpr (OUT) product<false, 8>(tmem + O + (n & 1) * VS, t.qd, sm.sb, false);
            if (!fatc::mbar_wait_warp(&sm.v_ready, n & 1, abort_flag, err, 0xd220)) break;
            tc_fence_after();
            product<true, 4>(tmem + ST, t.kd, sm.vb, true);
            if (elect_one()) umma_commit(&sm.s_full);
            if constexpr (OUT) {
                product<false, 4>(tmem + O + (n & 1) * VS, t.a, sm.vb, true);
                if (elect_one()) umma_commit(&sm.o_full);
            } else if (elect_one()) umma_commit(&sm.empty[s]);
        }
    } else if (warp == 2) {                                               // Sn and Vn
        for (int n = 0; keep && n < a.N; ++n) {
            if (!mbar_wait_suspend(&sm.sb_ready, n & 1, abort_flag, err, 0xd300)) break;
            if (lane == 0) { store_2d(&m.sn, sm.sb, col0, (bh * a.N + n) * DK); fatc::tma_store_commit(); }
            __syncwarp();
            if (!mbar_wait_suspend(&sm.v_ready, n & 1, abort_flag, err, 0xd310)) break;
            if (lane == 0) {
                store_2d(&m.vn, sm.vb, col0, row0 + n * C);
                fatc::tma_store_commit();
                fatc::tma_store_wait_read();
                mbar_arrive(&sm.kept);
            }
            __syncwarp();
        }
        if (lane == 0) fatc::tma_store_wait();
    } else if (warp == 3) {                                               // O
        if constexpr (OUT) {
            for (int n = 0; n < a.N; ++n) {
                const int s = n % STAGES;
                if (!mbar_wait_suspend(&sm.o_ready[s], (n / STAGES) & 1, abort_flag, err, 0xd400 | s)) break;
                if (lane == 0) {
                    fatc::tma_store_4d(&m.o, sm.st[s].x, col0, bh % a.H, n * C, bh / a.H);       // rows behind T are cut off
                    fatc::tma_store_commit();
                    fatc::tma_store_wait_read();
                    mbar_arrive(&sm.empty[s]);
                }
                __syncwarp();
            }
            if (lane == 0) fatc::tma_store_wait();
        }
    } else {
        const int qd = warp & 3, part = (warp - 4) >> 2, r = qd * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)(qd * 32) << 16) + part * 32;
        const long long at = ((long long)bh * DK + r) * a.dv + col0 + part * 32;
        // O of chunk n, over its U
        auto output = [&](int n) -> bool {
            if constexpr (OUT) {
                if (qd >= 2) return true;
                if (!mbar_wait_suspend(&sm.o_full, n & 1, abort_flag, err, 0xd500)) return false;
                tc_fence_after();
                float o[32];
                load_tmem(o, lane_addr + O + (n & 1) * VS);
                store32(sm.st[n % STAGES].x, r, part, o);
                fence_async();
                tc_fence_before();
                arrive(&sm.o_ready[n % STAGES]);
            }
            return true;
        };
        float S[32];
        load_row(S, a.S0 == nullptr ? nullptr : a.S0 + at);
        bool ok = true;
        for (int n = 0; ok && n < a.N; ++n) {
            const int s = n % STAGES;
            const float gamma = __ldg(a.gamma + (long long)bh * a.N + n);
            if (n > 0) {
                ok = mbar_wait_suspend(&sm.s_full, (n - 1) & 1, abort_flag, err, 0xd510) &&
                     (!keep || mbar_wait_suspend(&sm.kept, (n - 1) & 1, abort_flag, err, 0xd520));
                if (!ok) break;
                tc_fence_after();
                load_tmem(S, lane_addr + ST);
            }
            store32(sm.sb, r, part, S);                                   // the state in front of the chunk; its last readers are done
            store_tmem(lane_addr + ST, S, gamma);
            tmem_st_wait();
            fence_async();
            tc_fence_before();
            arrive(&sm.sb_ready);
            if (n > 0) ok = output(n - 1);
            if (ok && qd < 2) {                                           // Vn = U - W S
                ok = mbar_wait_suspend(&sm.full[s], (n / STAGES) & 1, abort_flag, err, 0xd530 | s) && mbar_wait_suspend(&sm.x_full, n & 1, abort_flag, err, 0xd540);
                if (!ok) break;
                tc_fence_after();
                float x[32];
                load_tmem(x, lane_addr + X);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 u = *reinterpret_cast<const uint4*>(sm.st[s].x + r * 128 + (((part * 4 + i) ^ (r & 7)) << 4));
                    const __nv_bfloat162* up = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = __bfloat1622float2(up[e]);
                        x[8 * i + 2 * e] = f.x - x[8 * i + 2 * e];
                        x[8 * i + 2 * e + 1] = f.y - x[8 * i + 2 * e + 1];
                    }
                }
                store32(sm.vb, r, part, x);
                fence_async();
                tc_fence_before();
                arrive(&sm.v_ready);
            }
        }
        if (ok && a.N > 0) {
            ok = mbar_wait_suspend(&sm.s_full, (a.N - 1) & 1, abort_flag, err, 0xd550);
            tc_fence_after();
            load_tmem(S, lane_addr + ST);
            if (ok) output(a.N - 1);
        }
        if (ok) save_row(a.Sfinal + at, S);
    }
    finish(tmem, warp);
}

// Reverse walk: dS' enters from the right (gradient of the state leaving the chunk).
__global__ void __launch_bounds__(THREADS, 1) delta_scan_bwd_tc_kernel(const __grid_constant__ Maps m, Args a) {
    extern __shared__ uint8_t smem_raw[];
    Smem<true>& sm = *reinterpret_cast<Smem<true>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = fatc::uniform_warp(), lane = threadIdx.x & 31, col0 = blockIdx.x * VS, bh = blockIdx.y, row0 = bh * a.N * C;
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    const uint32_t tmem = setup(sm, warp);

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < a.N; ++i) {
                const int n = a.N - 1 - i, s = i % STAGES, row = row0 + n * C;
                if (!mbar_wait_suspend(&sm.empty[s], ((i / STAGES) & 1) ^ 1, abort_flag, err, 0xe100 | s)) break;
                mbar_expect_tx(&sm.full[s], sizeof(Stage<true>));
                Stage<true>& t = sm.st[s];
                tma_load_2d(t.a, &m.a, &sm.full[s], 0, row);
                tma_load_4d(t.x, &m.x, &sm.full[s], col0, bh % a.H, n * C, bh / a.H);            // rows behind T are zeros
                key_tile(t.kd, &m.kd, &sm.full[s], row);
                key_tile(t.qd, &m.qd, &sm.full[s], row);
                key_tile(t.w, &m.w, &sm.full[s], row);
            }
        }
    } else if (warp == 1) {
        for (int i = 0; i < a.N; ++i) {
            const int s = i % STAGES;
            Stage<true>& t = sm.st[s];
            if (!fatc::mbar_wait_warp(&sm.full[s], (i / STAGES) & 1, abort_flag, err, 0xe200 | s)) break;
            tc_fence_after();
            product<true, 4>(tmem + X, t.a, t.x, false);                                   // A^T dO, ahead of the state (X has been read: v_ready)
            if (!fatc::mbar_wait_warp(&sm.sb_ready, i & 1, abort_flag, err, 0xe210)) break;
            tc_fence_after();
            product<false, 8>(tmem + X, t.kd, sm.sb, true);
            if (elect_one()) umma_commit(&sm.x_full);
            product<true, 4>(tmem + ST, t.qd, t.x, true);
            if (!fatc::mbar_wait_warp(&sm.v_ready, i & 1, abort_flag, err, 0xe220)) break;
            tc_fence_after();
            product<true, 4>(tmem + ST, t.w, sm.vneg, true);
            if (elect_one()) { umma_commit(&sm.s_full); umma_commit(&sm.empty[s]); }
        }
    } else if (warp == 2) {                                               // dSn and dVn
        for (int i = 0; i < a.N; ++i) {
            const int n = a.N - 1 - i;
            if (!mbar_wait_suspend(&sm.sb_ready, i & 1, abort_flag, err, 0xe300)) break;
            if (lane == 0) { store_2d(&m.sn, sm.sb, col0, (bh * a.N + n) * DK); fatc::tma_store_commit(); }
            __syncwarp();
            if (!mbar_wait_suspend(&sm.v_ready, i & 1, abort_flag, err, 0xe310)) break;
            if (lane == 0) {
                store_2d(&m.vn, sm.vb, col0, row0 + n * C);
                fatc::tma_store_commit();
                fatc::tma_store_wait_read();
                mbar_arrive(&sm.kept);
            }
            __syncwarp();
        }
        if (lane == 0) fatc::tma_store_wait();
    } else if (warp >= 4) {
        const int qd = warp & 3, part = (warp - 4) >> 2, r = qd * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)(qd * 32) << 16) + part * 32;
        const long long at = ((long long)bh * DK + r) * a.dv + col0 + part * 32;
        float S[32];
        load_row(S, a.dSfinal == nullptr ? nullptr : a.dSfinal + at);
        bool ok = true;
        for (int i = 0; ok && i < a.N; ++i) {
            const float gamma = __ldg(a.gamma + (long long)bh * a.N + a.N - 1 - i);
            if (i > 0) {
                ok = mbar_wait_suspend(&sm.s_full, (i - 1) & 1, abort_flag, err, 0xe500) && mbar_wait_suspend(&sm.kept, (i - 1) & 1, abort_flag, err, 0xe510);
                if (!ok) break;
                tc_fence_after();
                load_tmem(S, lane_addr + ST);
            }
            store32(sm.sb, r, part, S);
            store_tmem(lane_addr + ST, S, gamma);
            tmem_st_wait();
            fence_async();
            tc_fence_before();
            arrive(&sm.sb_ready);
            if (qd < 2) {
                ok = mbar_wait_suspend(&sm.x_full, i & 1, abort_flag, err, 0xe520);
                if (!ok) break;
                tc_fence_after();
                float x[32];
                load_tmem(x, lane_addr + X);
                store32(sm.vneg, r, part, x, -1.f);
                store32(sm.vb, r, part, x);
                fence_async();
                tc_fence_before();
                arrive(&sm.v_ready);
            }
        }
        if (ok && a.N > 0) {
            ok = mbar_wait_suspend(&sm.s_full, (a.N - 1) & 1, abort_flag, err, 0xe530);
            tc_fence_after();
            load_tmem(S, lane_addr + ST);
        }
        if (ok) save_row(a.dS0 + at, S);
    }
    finish(tmem, warp);
}

// [B, T, H, dv] with element strides; dimensions of size one take a stride of their own (theirs may be anything)
static int rows_map(CUtensorMap* m, const bf16* p, const Args& a, int B, long long sb, long long st, long long sh) {
    if (a.H == 1) sh = a.dv;
    if (a.T == 1) st = sh * a.H;
    if (B == 1) sb = st * a.T;
    return fatc::make_map_4d(m, p, B, a.T, a.H, a.dv, sb, st, sh, C);
}
}  // namespace tcs

int scan_tc(int dir, int BH, const Args& a, cudaStream_t st) {
    using namespace tcs;
    const uint64_t rows = (uint64_t)BH * a.N * C, states = (uint64_t)BH * a.N * DK;
    const bool out = dir != 0 || a.O != nullptr, keep = dir != 0 || a.Vn != nullptr;
    Maps m = {};
    int rc = make_map(&m.w, a.W, rows, DK, a.ldw, C) | make_map(&m.kd, a.Kd, rows, DK, a.ldw, C);
    if (out) rc |= make_map(&m.qd, a.Qd, rows, DK, a.ldw, C) | make_map(&m.a, a.A, rows, C, a.lda, C);
    if (dir != 0) rc |= rows_map(&m.x, a.dO, a, BH / a.H, a.gs_b, a.gs_t, a.gs_h);
    else rc |= make_map(&m.x, a.U, rows, a.dv, a.dv, C);
    if (dir == 0 && out) rc |= rows_map(&m.o, a.O, a, BH / a.H, a.os_b, a.os_t, a.os_h);
    if (keep) rc |= make_map(&m.vn, dir ? a.dVn : a.Vn, rows, a.dv, a.dv, C) | make_map(&m.sn, dir ? a.dSn : a.Sn, states, a.dv, a.dv, DK);
    if (rc) return -11;
    const dim3 grid(a.dv / VS, BH);
#define LMOE_SCAN_TC(KERNEL, FULL)                                                                                       \
    do {                                                                                                                 \
        const size_t smem = sizeof(Smem<FULL>) + 1024;                                                                   \
        rc = (int)cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                  \
        if (rc) return rc;                                                                                               \
        KERNEL<<<grid, THREADS, smem, st>>>(m, a);                                                                       \
    } while (0)
    if (dir != 0) LMOE_SCAN_TC(delta_scan_bwd_tc_kernel, true);
    else if (out) LMOE_SCAN_TC(delta_scan_fwd_tc_kernel<true>, true);
    else LMOE_SCAN_TC(delta_scan_fwd_tc_kernel<false>, false);
#undef LMOE_SCAN_TC
    return (int)cudaGetLastError();
}

}  // namespace dr
}  // namespace lmoe
