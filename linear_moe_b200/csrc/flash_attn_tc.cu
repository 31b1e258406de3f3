// Flash-attention forward on the 5th-generation tensor cores: S = Q K^T and O_j = P_j V_j are tcgen05.mma instructions
// with accumulators in tensor memory, operands staged by TMA (4-D tensor maps over [B, T, H, D], 128-byte swizzle).
//
// One CTA = 128 queries of one head.  640 threads:
//   warp 0      TMA producer: Q once, then K_j / V_j tiles of 128 keys through two 2-stage rings
//   warp 1      MMA issuer:   S_{j+1} = Q K_{j+1}^T is issued before O += P_j V_j
//   warps 4..19 softmax, two groups of eight: group g works on the tiles j = g (mod 2), so that one group's exponentials run while the
//               other one waits for its scores, exchanges maxima or hands over P.  (With all warps on the same tile every stage of
//               it was exposed: 3900 cycles a tile against 1024 of exponentials.)  Inside a group the two warps with equal (w & 3) own the 32 rows
//               of a tensor-memory lane quarter and half of the columns each.
// Each group has its own running maximum, sum and output, which are joined at the end.  Its output accumulates in tensor memory in
// units of a maximum that may lag behind by up to 2^LAG; only when a row runs ahead of that the output is rescaled there.  P_j goes
// back over its scores in bf16 and is read as the A operand from tensor memory.
// Tensor memory: 2 x 128 columns of scores, 2 x D of outputs.
// B=2, T=4096, 16 query and 4 kv heads of 128: 242 -> 190 us; B=1, 1531 queries over 2552 keys, 32 / 8 heads of 64: 86 -> 66 us.
// Masking (causal with a query offset, sliding window, key length) is applied only on tiles that cross a boundary.
// Every mbarrier wait is bounded (clock64 budget); on expiry the error word is set and the CTA drains and frees its
// tensor memory.  Writes O (bf16) and the natural-log row log-sum-exp, which the backward kernels of flash_attn.cu use.
//
// Replaces dot_product_attention.py:139-183 (baddbmm + softmax + bmm) and the flash_attn / TransformerEngine back ends
// of the reference (llama3/transformer_legacy.py:446-505).
#include "flash_tc_utils.cuh"

namespace lmoe {
namespace fatc {

struct Args {
    bf16* out;            // [B, Tq, Hq, D]
    float* lse;           // [B, Hq, Tq]
    int B, Tq, Tk, Hq, Hkv;
    int q_offset, window; // window <= 0: none
    float scale;
    int* err;
};

constexpr float LAG = 8.f;            // how far, as a power of two, a row's weights may run ahead of the maximum they are measured in

template <int D>
struct __align__(1024) Smem {
    uint8_t q[BM * D * 2];
    uint8_t k[2][BN * D * 2];
    uint8_t v[2][BN * D * 2];
    uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_ready[2], pv_done[2];
    float mx[2][2][2][BM];            // [parity of the group's tile][group][half of the columns]
    float ls[2][2][BM], ms[2][BM];    // sums and maxima at the end
    uint32_t tmem_base;
    int abort_flag;
};

template <int D>
__global__ void __launch_bounds__(THREADS, 1)
fa_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, Args a) {
    extern __shared__ uint8_t smem_raw[];
    Smem<D>& sm = *reinterpret_cast<Smem<D>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int DK = D / 64;                              // 64-element blocks along the head dimension
    constexpr uint32_t TMEM_COLS = 512;
    constexpr uint32_t O_COL = 2 * BN;                      // the groups' outputs behind the two score buffers
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int qb = gridDim.x - 1 - blockIdx.x;              // long (late) query tiles first
    const int h = blockIdx.y, b = blockIdx.z;
    const int hk = h / (a.Hq / a.Hkv);
    const int q0 = qb * BM;
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;

    // visible key range of this query tile -> key tiles [nb_lo, nb_hi)
    const int last_q = min(a.Tq, q0 + BM) - 1;
    const int k_hi = min(a.Tk, a.q_offset + last_q + 1);
    const int k_lo = a.window > 0 ? max(0, a.q_offset + q0 - a.window + 1) : 0;
    const int nb_lo = k_lo / BN, nb_hi = (k_hi + BN - 1) / BN;
    const int n_it = max(nb_hi - nb_lo, 0);

    if (threadIdx.x == 0) {
        mbar_init(&sm.q_full, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&sm.k_full[s], 1); mbar_init(&sm.k_empty[s], 1);
            mbar_init(&sm.v_full[s], 1); mbar_init(&sm.v_empty[s], 1);
            mbar_init(&sm.s_full[s], 1); mbar_init(&sm.pv_done[s], 1);
            mbar_init(&sm.p_ready[s], 8);
        }
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
    const uint32_t tmem_base = sm.tmem_base;

    if (warp == 0) {
        if (lane == 0 && n_it > 0) {
            mbar_expect_tx(&sm.q_full, BM * D * 2);
#pragma unroll
            for (int kb = 0; kb < DK; ++kb) tma_load_4d(sm.q + kb * BM * 128, &tmQ, &sm.q_full, kb * 64, h, q0, b);
            for (int j = 0; j < n_it; ++j) {
                const int s = j & 1;
                const uint32_t ph = (j >> 1) & 1;
                const int key0 = (nb_lo + j) * BN;
                if (!mbar_wait_suspend(&sm.k_empty[s], ph ^ 1, abort_flag, err, 0x1100 | s)) break;
                mbar_expect_tx(&sm.k_full[s], BN * D * 2);
#pragma unroll
                for (int kb = 0; kb < DK; ++kb) tma_load_4d(sm.k[s] + kb * BN * 128, &tmK, &sm.k_full[s], kb * 64, hk, key0, b);
                if (!mbar_wait_suspend(&sm.v_empty[s], ph ^ 1, abort_flag, err, 0x1200 | s)) break;
                mbar_expect_tx(&sm.v_full[s], BN * D * 2);
                // MN-major operand: per 64 keys, D/64 boxes of {64 d, 64 keys} (8 KiB each)
#pragma unroll
                for (int kk = 0; kk < BN / 64; ++kk)
#pragma unroll
                    for (int nb = 0; nb < DK; ++nb)
                        tma_load_4d(sm.v[s] + (kk * DK + nb) * 8192, &tmV, &sm.v_full[s], nb * 64, hk, key0 + kk * 64, b);
            }
        }
    } else if (warp == 1) {
        if (n_it > 0) {
            const uint32_t issue = lane == 0 ? 1u : 0u;
            constexpr uint32_t idesc_s = idesc_bf16<false, BN>();
            constexpr uint32_t idesc_o = idesc_bf16<true, D>();
            bool ok = mbar_wait_suspend(&sm.q_full, 0, abort_flag, err, 0x2000);
            auto issue_s = [&](int j) -> bool {
                const int s = j & 1;
                if (!mbar_wait_suspend(&sm.k_full[s], (j >> 1) & 1, abort_flag, err, 0x2100 | s)) return false;
                tc_fence_after();
                const uint32_t ql = desc_lo<false>(s32(sm.q)), kl = desc_lo<false>(s32(sm.k[s]));
#pragma unroll
                for (int kk = 0; kk < D / UMMA_K; ++kk) {
                    const uint32_t off = ((kk / 4) * (BM * 128) + (kk % 4) * 32) >> 4;
                    umma_lo(tmem_base + s * BN, ql + off, kl + off, idesc_s, kk > 0 ? 1u : 0u, issue);
                }
                umma_commit_if(&sm.k_empty[s], issue);
                umma_commit_if(&sm.s_full[s], issue);
                return true;
            };
            if (ok) ok = issue_s(0);
            for (int j = 0; ok && j < n_it; ++j) {
                const int s = j & 1;
                if (j + 1 < n_it) {
                    // the other score buffer holds P_{j-1}: its product has to complete
                    if (j > 0 && !mbar_wait_suspend(&sm.pv_done[s ^ 1], ((j - 1) >> 1) & 1, abort_flag, err, 0x2400)) break;
                    ok = issue_s(j + 1);
                    if (!ok) break;
                }
                if (!mbar_wait_suspend(&sm.v_full[s], (j >> 1) & 1, abort_flag, err, 0x2200 | s)) break;
                if (!mbar_wait_suspend(&sm.p_ready[s], (j >> 1) & 1, abort_flag, err, 0x2300 | s)) break;
                tc_fence_after();
                const uint32_t vl = desc_lo<true>(s32(sm.v[s]));
#pragma unroll
                for (int kk = 0; kk < BN / UMMA_K; ++kk) {
                    // every half of the columns left its 32 columns of P at its beginning
                    const uint32_t boff = ((kk / 4) * (DK * 8192) + (kk % 4) * 2048) >> 4;
                    umma_ta(tmem_base + O_COL + s * D, tmem_base + s * BN + kk / 4 * 64 + kk % 4 * 8, vl + boff, idesc_o, (j > 1 || kk > 0) ? 1u : 0u, issue);
                }
                umma_commit_if(&sm.v_empty[s], issue);
                umma_commit_if(&sm.pv_done[s], issue);
            }
        }
    } else if (warp >= 4) {
        const int qd = warp & 3, quarter = (warp - 4) >> 2, grp = quarter >> 1, part = quarter & 1;
        const int r = qd * 32 + lane;                         // query row inside the tile
        const int qi = a.q_offset + q0 + r;                   // absolute position of this query
        const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16);
        const uint32_t s_addr = lane_addr + grp * BN + part * 64, o_addr = lane_addr + O_COL + grp * D + part * (D / 2);
        const float sc = a.scale * LOG2E, lag = LAG / sc;
        float m = -INFINITY, l = 0.f;
        bool ok = true;                                       // after a wait that ran out only the barriers are kept up with
        for (int j = grp; j < n_it; j += 2) {
            const int k = j >> 1;
            const int tile_key0 = (nb_lo + j) * BN;
            if (ok) ok = mbar_wait_suspend(&sm.s_full[grp], k & 1, abort_flag, err, 0x3100 | grp);
            if (!ok) {
                asm volatile("bar.sync %0, 64;" :: "r"(1 + grp * 4 + qd) : "memory");
                continue;
            }
            tc_fence_after();
            uint32_t v[64];
            tmem_ld64(s_addr, v);
            tmem_ld_wait();
            const bool need_mask = (tile_key0 + BN - 1 > a.q_offset + q0) || (tile_key0 + BN > a.Tk) ||
                                   (a.window > 0 && tile_key0 <= a.q_offset + q0 + BM - 1 - a.window);
            if (need_mask) {
                const int key0 = tile_key0 + part * 64;
                const int hi = min(qi, a.Tk - 1) - key0, lo = a.window > 0 ? qi - a.window - key0 : -1;      // visible: lo < c <= hi
#pragma unroll
                for (int c = 0; c < 64; ++c)
                    if (c > hi || c <= lo) v[c] = 0xff800000u;                                               // -inf
            }
            float mx4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                mx4[e] = fmaxf(__uint_as_float(v[e]), __uint_as_float(v[e + 4]));
#pragma unroll
                for (int c = 8; c < 64; c += 8) mx4[e] = max3(mx4[e], __uint_as_float(v[c + e]), __uint_as_float(v[c + e + 4]));
            }
            float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            sm.mx[k & 1][grp][part][r] = mx;
            asm volatile("bar.sync %0, 64;" :: "r"(1 + grp * 4 + qd) : "memory");
            mx = fmaxf(mx, sm.mx[k & 1][grp][part ^ 1][r]);
            // both halves of a row see the same numbers and decide alike
            const bool grow = mx > m + lag;                   // also the first visible key of the row (m = -inf)
            const bool scaled = grow && m != -INFINITY;
            const float corr = scaled ? exp2f((m - mx) * sc) : 1.f;
            if (grow) m = mx;
            l *= corr;
            if (__any_sync(0xffffffffu, scaled)) {            // k > 0; the scores of tile j were issued behind the last product of this group
                ok = mbar_wait_suspend(&sm.pv_done[grp], (k - 1) & 1, abort_flag, err, 0x3200 | grp);
                if (!ok) continue;
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < D / 2; c += 16) {
                    uint32_t o[16];
                    tmem_ld16(o_addr + c, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                    tmem_st16(o_addr + c, o);
                }
            }
            const float nm = m == -INFINITY ? 0.f : -m * sc;
            const float2 sc2 = make_float2(sc, sc), nm2 = make_float2(nm, nm);
            float2 sum0 = make_float2(0.f, 0.f), sum1 = make_float2(0.f, 0.f);
#pragma unroll
            for (int c = 0; c < 64; c += 32) {
                uint32_t p[16];
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float2 x01 = __ffma2_rn(make_float2(__uint_as_float(v[c + i]), __uint_as_float(v[c + i + 1])), sc2, nm2);
                    const float2 x23 = __ffma2_rn(make_float2(__uint_as_float(v[c + i + 2]), __uint_as_float(v[c + i + 3])), sc2, nm2);
                    const float p0 = exp2f(x01.x), p1 = exp2f(x01.y), p2 = exp2f(x23.x), p3 = exp2f(x23.y);
                    sum0 = __fadd2_rn(sum0, make_float2(p0, p1));
                    sum1 = __fadd2_rn(sum1, make_float2(p2, p3));
                    p[i >> 1] = pack_bf16(p0, p1);
                    p[(i >> 1) + 1] = pack_bf16(p2, p3);
                }
                tmem_st16(s_addr + (c >> 1), p);              // over scores that are in registers
            }
            l += (sum0.x + sum0.y) + (sum1.x + sum1.y);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.p_ready[grp]);
        }
        // join the groups: every warp takes a quarter of the columns of both outputs
        sm.ls[grp][part][r] = l;
        if (part == 0) sm.ms[grp][r] = m;
        asm volatile("bar.sync 9, 512;" ::: "memory");        // behind it at most the last product of each group is outstanding
        float w[2], mm = fmaxf(sm.ms[0][r], sm.ms[1][r]);
        l = 0.f;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const float mg = sm.ms[g][r];
            w[g] = mg == -INFINITY ? 0.f : exp2f((mg - mm) * sc);
            l += w[g] * (sm.ls[g][0][r] + sm.ls[g][1][r]);
        }
        constexpr int OW = D / 4;
        float o[OW];
#pragma unroll
        for (int i = 0; i < OW; ++i) o[i] = 0.f;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            if (g >= n_it) break;
            const int last = n_it - 1 - ((n_it - 1 - g) & 1);                    // the group's last tile
            if (!mbar_wait_suspend(&sm.pv_done[g], (last >> 1) & 1, abort_flag, err, 0x3300 | g)) break;
            tc_fence_after();
            uint32_t x[OW];
            tmem_ld<OW>(lane_addr + O_COL + g * D + quarter * OW, x);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < OW; ++i) o[i] += w[g] * __uint_as_float(x[i]);
        }
        const int row = q0 + r;
        if (row < a.Tq) {
            const float inv = l > 0.f ? 1.f / l : 0.f;
            bf16* og = a.out + (((long long)b * a.Tq + row) * a.Hq + h) * D + quarter * OW;
#pragma unroll
            for (int c = 0; c < OW; c += 8) {
                uint4 y;
                y.x = pack_bf16(o[c] * inv, o[c + 1] * inv);
                y.y = pack_bf16(o[c + 2] * inv, o[c + 3] * inv);
                y.z = pack_bf16(o[c + 4] * inv, o[c + 5] * inv);
                y.w = pack_bf16(o[c + 6] * inv, o[c + 7] * inv);
                *reinterpret_cast<uint4*>(og + c) = y;
            }
            if (quarter == 0) a.lse[((long long)b * a.Hq + h) * a.Tq + row] = l > 0.f ? mm * a.scale + logf(l) : -INFINITY;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}


// =====================================================================================================================
// Backward on tcgen05, two kernels that recompute the scores (7 GEMMs per tile pair instead of 5, no atomics):
//   fa_bwd_dq_tc_kernel    one CTA = 128 queries of one head; loops over tiles of 64 keys:
//                          S = Q K^T and dP = dO V^T into tensor memory -> dS = P (dP - delta) scale (softmax warps,
//                          thread = query row) -> shared memory -> dQ += dS K accumulated in tensor memory.
//   fa_bwd_dkv_tc_kernel   one CTA = 128 keys of one KV head; loops over the query heads of the group and tiles of 64
//                          queries: S^T = K Q^T and dP^T = V dO^T -> P^T, dS^T (thread = key row) -> shared memory ->
//                          dV += P^T dO and dK += dS^T Q accumulated in tensor memory.
// A [64 x D] tile loaded as D/64 boxes of {64 d, 64 rows} serves both as a K-major operand (rows = N) of the score GEMMs
// and as an MN-major operand (rows = K) of the gradient GEMMs.  Same warp roles, barriers and bounded waits as the forward:
// two groups of eight warps take turns with the iterations, each with its own dS (and P^T) tile, so that one group's
// exponentials run while the other's tile is read by the gradient GEMMs.  (All sixteen warps on one iteration and one tile: 4300
// cycles an iteration against 1280 of tensor-core time.)
// B=2, T=4096, 16 query and 4 kv heads of 128: dQ 335 -> 332 us, dK / dV 538 -> 509 us.
// =====================================================================================================================
constexpr int BT = 64;                                       // tile of the looped dimension (keys for dQ, queries for dK/dV)
constexpr int NST = 3;                                       // TMA stages of the looped tiles: a stage is released only after the
                                                             // gradient MMAs of its iteration, so two stages would expose the load latency

struct BwdArgs {
    const float* lse;     // [B, Hq, Tq] natural-log sum-exp from the forward
    const float* delta;   // [B, Hq, Tq] rowsum(dO * O)
    bf16* dq;             // [B, Tq, Hq, D]
    bf16* dk;             // [B, Tk, Hkv, D]
    bf16* dv;             // [B, Tk, Hkv, D]
    int B, Tq, Tk, Hq, Hkv;
    int q_offset, window;
    float scale;
    int* err;
};

template <int D>
struct __align__(1024) SmemBwd {
    uint8_t big0[BM * D * 2];          // dQ kernel: Q tile      | dK/dV kernel: K tile
    uint8_t big1[BM * D * 2];          // dQ kernel: dO tile     | dK/dV kernel: V tile
    uint8_t st0[NST][BT * D * 2];        // dQ kernel: K stages    | dK/dV kernel: Q stages
    uint8_t st1[NST][BT * D * 2];        // dQ kernel: V stages    | dK/dV kernel: dO stages
    uint8_t p[2][BM * BT * 2];         // per group: dS (dQ kernel) | P^T (dK/dV kernel), K-major, 128 rows x 128 bytes
    uint8_t ds[2][BM * BT * 2];        // dS^T (dK/dV kernel)
    float lse2[NST][BT], delta[NST][BT];     // of the looped queries (dK/dV kernel)
    uint64_t big_full, st_full[NST], st_empty[NST], stat_full[NST], s_full[2], p_ready[2], acc_done[2];
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ bool visible(int key, int qi, int Tk, int window) {
    return key <= qi && key < Tk && (window <= 0 || key > qi - window);
}

template <int D>
__global__ void __launch_bounds__(THREADS, 1)
fa_bwd_dq_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmG,
                    const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, BwdArgs a) {
    extern __shared__ uint8_t smem_raw[];
    SmemBwd<D>& sm = *reinterpret_cast<SmemBwd<D>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int DK = D / 64;
    constexpr uint32_t TMEM_COLS = 512, ACC_COL = 256;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int qb = gridDim.x - 1 - blockIdx.x;
    const int h = blockIdx.y, b = blockIdx.z;
    const int hk = h / (a.Hq / a.Hkv);
    const int q0 = qb * BM;
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    const int last_q = min(a.Tq, q0 + BM) - 1;
    const int k_hi = min(a.Tk, a.q_offset + last_q + 1);
    const int k_lo = a.window > 0 ? max(0, a.q_offset + q0 - a.window + 1) : 0;
    const int nb_lo = k_lo / BT, nb_hi = (k_hi + BT - 1) / BT;
    const int n_it = max(nb_hi - nb_lo, 0);

    if (threadIdx.x == 0) {
        mbar_init(&sm.big_full, 1);
        for (int s = 0; s < NST; ++s) { mbar_init(&sm.st_full[s], 1); mbar_init(&sm.st_empty[s], 1); mbar_init(&sm.stat_full[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&sm.s_full[s], 1); mbar_init(&sm.p_ready[s], 8); mbar_init(&sm.acc_done[s], 1); }
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
    const uint32_t tmem_base = sm.tmem_base;

    if (warp == 0) {
        if (lane == 0 && n_it > 0) {
            mbar_expect_tx(&sm.big_full, 2 * BM * D * 2);
#pragma unroll
            for (int kb = 0; kb < DK; ++kb) {
                tma_load_4d(sm.big0 + kb * BM * 128, &tmQ, &sm.big_full, kb * 64, h, q0, b);
                tma_load_4d(sm.big1 + kb * BM * 128, &tmG, &sm.big_full, kb * 64, h, q0, b);
            }
            for (int j = 0; j < n_it; ++j) {
                const int s = j % NST;
                const int key0 = (nb_lo + j) * BT;
                if (!mbar_wait_suspend(&sm.st_empty[s], ((j / NST) & 1) ^ 1, abort_flag, err, 0x4100 | s)) break;
                mbar_expect_tx(&sm.st_full[s], 2 * BT * D * 2);
#pragma unroll
                for (int kb = 0; kb < DK; ++kb) {
                    tma_load_4d(sm.st0[s] + kb * 8192, &tmK, &sm.st_full[s], kb * 64, hk, key0, b);
                    tma_load_4d(sm.st1[s] + kb * 8192, &tmV, &sm.st_full[s], kb * 64, hk, key0, b);
                }
            }
        }
    } else if (warp == 1) {
        if (n_it > 0) {
            const uint32_t issue = lane == 0 ? 1u : 0u;
            constexpr uint32_t idesc_s = idesc_bf16<false, BT>();       // [128 q] x [64 keys], both K-major
            constexpr uint32_t idesc_a = idesc_bf16<true, D>();         // dQ += dS K: B = K tile read MN-major
            bool ok = mbar_wait_suspend(&sm.big_full, 0, abort_flag, err, 0x4200);
            auto issue_sd = [&](int j) -> bool {
                const int s = j & 1, g = j % NST;                    // tensor-memory buffer, shared-memory stage
                if (!mbar_wait_suspend(&sm.st_full[g], (j / NST) & 1, abort_flag, err, 0x4300 | g)) return false;
                tc_fence_after();
                const uint32_t ql = desc_lo<false>(s32(sm.big0)), gl = desc_lo<false>(s32(sm.big1));
                const uint32_t kl = desc_lo<false>(s32(sm.st0[g])), vl = desc_lo<false>(s32(sm.st1[g]));
#pragma unroll
                for (int kk = 0; kk < D / UMMA_K; ++kk) {
                    const uint32_t ao = ((kk / 4) * (BM * 128) + (kk % 4) * 32) >> 4, bo = ((kk / 4) * 8192 + (kk % 4) * 32) >> 4;
                    umma_lo(tmem_base + s * 128, ql + ao, kl + bo, idesc_s, kk > 0 ? 1u : 0u, issue);
                }
#pragma unroll
                for (int kk = 0; kk < D / UMMA_K; ++kk) {
                    const uint32_t ao = ((kk / 4) * (BM * 128) + (kk % 4) * 32) >> 4, bo = ((kk / 4) * 8192 + (kk % 4) * 32) >> 4;
                    umma_lo(tmem_base + s * 128 + 64, gl + ao, vl + bo, idesc_s, kk > 0 ? 1u : 0u, issue);
                }
                umma_commit_if(&sm.s_full[s], issue);
                return true;
            };
            if (ok) ok = issue_sd(0);
            for (int j = 0; ok && j < n_it; ++j) {
                if (j + 1 < n_it) { ok = issue_sd(j + 1); if (!ok) break; }
                const int s = j % NST;
                if (!mbar_wait_suspend(&sm.p_ready[j & 1], (j >> 1) & 1, abort_flag, err, 0x4400)) break;
                tc_fence_after();
                const uint32_t pl = desc_lo<false>(s32(sm.p[j & 1])), kl = desc_lo<true>(s32(sm.st0[s]));
#pragma unroll
                for (int kk = 0; kk < BT / UMMA_K; ++kk)
                    umma_lo(tmem_base + ACC_COL, pl + kk * 2, kl + kk * 128, idesc_a, (j > 0 || kk > 0) ? 1u : 0u, issue);
                umma_commit_if(&sm.st_empty[s], issue);
                umma_commit_if(&sm.acc_done[j & 1], issue);
            }
        }
    } else if (warp >= 4) {
        const int qd = warp & 3, quarter = (warp - 4) >> 2, grp = quarter >> 1, part = quarter & 1;
        const int r = qd * 32 + lane;
        const int row = q0 + r;
        const int qi = a.q_offset + row;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16);
        const float sc = a.scale * LOG2E;
        constexpr int CW = BT / 2;                               // 32 keys per thread
        const long long stat = ((long long)b * a.Hq + h) * a.Tq + row;
        const float lse2 = row < a.Tq ? a.lse[stat] * LOG2E : INFINITY;
        const float dl = row < a.Tq ? a.delta[stat] : 0.f;
        uint8_t* prow = sm.p[grp] + (r >> 3) * 1024 + (r & 7) * 128;
        bool alive = n_it > 0;
        for (int j = grp; alive && j < n_it; j += 2) {
            const int k = j >> 1;
            const int key0 = (nb_lo + j) * BT + part * CW;
            if (!mbar_wait_suspend(&sm.s_full[grp], k & 1, abort_flag, err, 0x4500 | grp)) { alive = false; break; }
            tc_fence_after();
            // masking is needed only on tiles that cross the causal diagonal, the window edge or the key length
            const int tile_key0 = (nb_lo + j) * BT;
            const bool need_mask = (tile_key0 + BT - 1 > a.q_offset + q0) || (tile_key0 + BT > a.Tk) ||
                                   (a.window > 0 && tile_key0 <= a.q_offset + q0 + BM - 1 - a.window);
            uint32_t pk[CW / 2];
#pragma unroll
            for (int c = 0; c < CW; c += 16) {
                uint32_t sv[16], dv[16];
                tmem_ld16(lane_addr + grp * 128 + part * CW + c, sv);
                tmem_ld16(lane_addr + grp * 128 + 64 + part * CW + c, dv);
                tmem_ld_wait();
                if (need_mask) {
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (!visible(key0 + c + i, qi, a.Tk, a.window)) sv[i] = 0xff800000u;      // -inf -> p = 0
                }
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    const float p0 = exp2f(fmaf(__uint_as_float(sv[i]), sc, -lse2)), p1 = exp2f(fmaf(__uint_as_float(sv[i + 1]), sc, -lse2));
                    pk[(c + i) >> 1] = pack_bf16(p0 * (__uint_as_float(dv[i]) - dl), p1 * (__uint_as_float(dv[i + 1]) - dl));   // the softmax scale is applied to dQ at the end
                }
            }
            if (k > 0 && !mbar_wait_suspend(&sm.acc_done[grp], (k - 1) & 1, abort_flag, err, 0x4600 | grp)) { alive = false; break; }
#pragma unroll
            for (int c = 0; c < 4; ++c)
                *reinterpret_cast<uint4*>(prow + (((part * 4 + c) ^ (r & 7)) << 4)) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
            tc_fence_before();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.p_ready[grp]);
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");           // behind it at most the last gradient GEMM of each group is outstanding
        constexpr int OW = D / SPLIT;
        uint32_t acc[OW];
#pragma unroll
        for (int i = 0; i < OW; ++i) acc[i] = 0u;
        if (alive && n_it > 0 && mbar_wait_suspend(&sm.acc_done[(n_it - 1) & 1], ((n_it - 1) >> 1) & 1, abort_flag, err, 0x4700)) {
            tc_fence_after();
            tmem_ld<OW>(lane_addr + ACC_COL + quarter * OW, acc);
            tmem_ld_wait();
        }
        if (row < a.Tq) {
            bf16* og = a.dq + (((long long)b * a.Tq + row) * a.Hq + h) * D + quarter * OW;
#pragma unroll
            for (int c = 0; c < OW; c += 8)
                *reinterpret_cast<uint4*>(og + c) = make_uint4(pack_bf16(a.scale * __uint_as_float(acc[c]), a.scale * __uint_as_float(acc[c + 1])),
                                                               pack_bf16(a.scale * __uint_as_float(acc[c + 2]), a.scale * __uint_as_float(acc[c + 3])),
                                                               pack_bf16(a.scale * __uint_as_float(acc[c + 4]), a.scale * __uint_as_float(acc[c + 5])),
                                                               pack_bf16(a.scale * __uint_as_float(acc[c + 6]), a.scale * __uint_as_float(acc[c + 7])));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}


template <int D>
__global__ void __launch_bounds__(THREADS, 1)
fa_bwd_dkv_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmG,
                     const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, BwdArgs a) {
    extern __shared__ uint8_t smem_raw[];
    SmemBwd<D>& sm = *reinterpret_cast<SmemBwd<D>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int DK = D / 64;
    constexpr uint32_t TMEM_COLS = 512, DV_COL = 256, DK_COL = 256 + D;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kb_tile = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
    const int rep = a.Hq / a.Hkv;
    const int k0 = kb_tile * BM;
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    // query tiles (of 64) that can see a key of this tile: q >= k0 - q_offset, and with a window q < k0 + 127 + window - q_offset
    const int i_lo = max(0, k0 - a.q_offset) / BT;
    int q_end = a.Tq;
    if (a.window > 0) q_end = min(a.Tq, max(0, k0 + BM - 1 + a.window - a.q_offset));
    const int i_hi = (q_end + BT - 1) / BT;
    const int ni = max(i_hi - i_lo, 0);
    const int n_it = ni * rep;

    if (threadIdx.x == 0) {
        mbar_init(&sm.big_full, 1);
        for (int s = 0; s < NST; ++s) { mbar_init(&sm.st_full[s], 1); mbar_init(&sm.st_empty[s], 1); mbar_init(&sm.stat_full[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&sm.s_full[s], 1); mbar_init(&sm.p_ready[s], 8); mbar_init(&sm.acc_done[s], 1); }
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
    const uint32_t tmem_base = sm.tmem_base;

    if (warp == 0) {
        if (lane == 0 && n_it > 0) {
            mbar_expect_tx(&sm.big_full, 2 * BM * D * 2);
#pragma unroll
            for (int kb = 0; kb < DK; ++kb) {
                tma_load_4d(sm.big0 + kb * BM * 128, &tmK, &sm.big_full, kb * 64, hk, k0, b);
                tma_load_4d(sm.big1 + kb * BM * 128, &tmV, &sm.big_full, kb * 64, hk, k0, b);
            }
            for (int it = 0; it < n_it; ++it) {
                const int s = it % NST;
                const int h = hk * rep + it / ni, q0 = (i_lo + it % ni) * BT;
                if (!mbar_wait_suspend(&sm.st_empty[s], ((it / NST) & 1) ^ 1, abort_flag, err, 0x5100 | s)) break;
                mbar_expect_tx(&sm.st_full[s], 2 * BT * D * 2);
#pragma unroll
                for (int kb = 0; kb < DK; ++kb) {
                    tma_load_4d(sm.st0[s] + kb * 8192, &tmQ, &sm.st_full[s], kb * 64, h, q0, b);
                    tma_load_4d(sm.st1[s] + kb * 8192, &tmG, &sm.st_full[s], kb * 64, h, q0, b);
                }
            }
        }
    } else if (warp == 1) {
        if (n_it > 0) {
            const uint32_t issue = lane == 0 ? 1u : 0u;
            constexpr uint32_t idesc_s = idesc_bf16<false, BT>();       // [128 keys] x [64 queries], both K-major
            constexpr uint32_t idesc_a = idesc_bf16<true, D>();         // B = dO / Q tile read MN-major
            bool ok = mbar_wait_suspend(&sm.big_full, 0, abort_flag, err, 0x5200);
            auto issue_sd = [&](int it) -> bool {
                const int s = it & 1, g = it % NST;                  // tensor-memory buffer, shared-memory stage
                if (!mbar_wait_suspend(&sm.st_full[g], (it / NST) & 1, abort_flag, err, 0x5300 | g)) return false;
                tc_fence_after();
                const uint32_t kl = desc_lo<false>(s32(sm.big0)), vl = desc_lo<false>(s32(sm.big1));
                const uint32_t ql = desc_lo<false>(s32(sm.st0[g])), gl = desc_lo<false>(s32(sm.st1[g]));
#pragma unroll
                for (int kk = 0; kk < D / UMMA_K; ++kk) {
                    const uint32_t ao = ((kk / 4) * (BM * 128) + (kk % 4) * 32) >> 4, bo = ((kk / 4) * 8192 + (kk % 4) * 32) >> 4;
                    umma_lo(tmem_base + s * 128, kl + ao, ql + bo, idesc_s, kk > 0 ? 1u : 0u, issue);
                }
#pragma unroll
                for (int kk = 0; kk < D / UMMA_K; ++kk) {
                    const uint32_t ao = ((kk / 4) * (BM * 128) + (kk % 4) * 32) >> 4, bo = ((kk / 4) * 8192 + (kk % 4) * 32) >> 4;
                    umma_lo(tmem_base + s * 128 + 64, vl + ao, gl + bo, idesc_s, kk > 0 ? 1u : 0u, issue);
                }
                umma_commit_if(&sm.s_full[s], issue);
                return true;
            };
            if (ok) ok = issue_sd(0);
            for (int it = 0; ok && it < n_it; ++it) {
                if (it + 1 < n_it) { ok = issue_sd(it + 1); if (!ok) break; }
                const int s = it % NST;
                if (!mbar_wait_suspend(&sm.p_ready[it & 1], (it >> 1) & 1, abort_flag, err, 0x5400)) break;
                tc_fence_after();
                const uint32_t pl = desc_lo<false>(s32(sm.p[it & 1])), dl_ = desc_lo<false>(s32(sm.ds[it & 1]));
                const uint32_t ql = desc_lo<true>(s32(sm.st0[s])), gl = desc_lo<true>(s32(sm.st1[s]));
#pragma unroll
                for (int kk = 0; kk < BT / UMMA_K; ++kk)        // dV += P^T dO
                    umma_lo(tmem_base + DV_COL, pl + kk * 2, gl + kk * 128, idesc_a, (it > 0 || kk > 0) ? 1u : 0u, issue);
#pragma unroll
                for (int kk = 0; kk < BT / UMMA_K; ++kk)        // dK += dS^T Q
                    umma_lo(tmem_base + DK_COL, dl_ + kk * 2, ql + kk * 128, idesc_a, (it > 0 || kk > 0) ? 1u : 0u, issue);
                umma_commit_if(&sm.st_empty[s], issue);
                umma_commit_if(&sm.acc_done[it & 1], issue);
            }
        }
    } else if (warp == 2) {                                      // log-sum-exp and delta of the looped queries
        for (int it = 0; it < n_it; ++it) {
            const int s = it % NST;
            const int h = hk * rep + it / ni, q0 = (i_lo + it % ni) * BT;
            const long long row = ((long long)b * a.Hq + h) * a.Tq;
            float x[2], y[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int q = q0 + lane + 32 * e;
                x[e] = q < a.Tq ? __ldg(a.lse + row + q) * LOG2E : INFINITY;
                y[e] = q < a.Tq ? __ldg(a.delta + row + q) : 0.f;
            }
            if (!mbar_wait_suspend(&sm.st_empty[s], ((it / NST) & 1) ^ 1, abort_flag, err, 0x5110 | s)) break;
#pragma unroll
            for (int e = 0; e < 2; ++e) { sm.lse2[s][lane + 32 * e] = x[e]; sm.delta[s][lane + 32 * e] = y[e]; }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.stat_full[s]);
        }
    } else if (warp >= 4) {
        const int qd = warp & 3, quarter = (warp - 4) >> 2, grp = quarter >> 1, part = quarter & 1;
        const int r = qd * 32 + lane;                            // key row inside the tile
        const int key = k0 + r;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16);
        const float sc = a.scale * LOG2E;
        uint8_t* prow = sm.p[grp] + (r >> 3) * 1024 + (r & 7) * 128;
        uint8_t* drow = sm.ds[grp] + (r >> 3) * 1024 + (r & 7) * 128;
        bool alive = n_it > 0;
        for (int it = grp; alive && it < n_it; it += 2) {
            const int k = it >> 1, g = it % NST;
            const int tile_q0 = (i_lo + it % ni) * BT;
            if (!mbar_wait_suspend(&sm.stat_full[g], (it / NST) & 1, abort_flag, err, 0x5510 | g)) { alive = false; break; }
            if (!mbar_wait_suspend(&sm.s_full[grp], k & 1, abort_flag, err, 0x5500 | grp)) { alive = false; break; }
            tc_fence_after();
            const bool need_mask = (k0 + BM - 1 > a.q_offset + tile_q0) || (k0 + BM > a.Tk) ||
                                   (a.window > 0 && k0 <= a.q_offset + tile_q0 + BT - 1 - a.window);
            uint32_t pk[16], dk2[16];
#pragma unroll
            for (int c = 0; c < 32; c += 16) {                   // 32 queries per thread, 16 at a time
                uint32_t sv[16], dv[16];
                tmem_ld16(lane_addr + grp * 128 + part * 32 + c, sv);
                tmem_ld16(lane_addr + grp * 128 + 64 + part * 32 + c, dv);
                tmem_ld_wait();
                if (need_mask) {
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (!visible(key, a.q_offset + tile_q0 + part * 32 + c + i, a.Tk, a.window)) sv[i] = 0xff800000u;
                }
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 l2 = *reinterpret_cast<const float4*>(&sm.lse2[g][part * 32 + c + i]), dl = *reinterpret_cast<const float4*>(&sm.delta[g][part * 32 + c + i]);
                    const float p0 = exp2f(fmaf(__uint_as_float(sv[i]), sc, -l2.x)), p1 = exp2f(fmaf(__uint_as_float(sv[i + 1]), sc, -l2.y));
                    const float p2 = exp2f(fmaf(__uint_as_float(sv[i + 2]), sc, -l2.z)), p3 = exp2f(fmaf(__uint_as_float(sv[i + 3]), sc, -l2.w));
                    const int o = (c + i) >> 1;
                    pk[o] = pack_bf16(p0, p1);
                    pk[o + 1] = pack_bf16(p2, p3);
                    dk2[o] = pack_bf16(p0 * (__uint_as_float(dv[i]) - dl.x), p1 * (__uint_as_float(dv[i + 1]) - dl.y));          // scale applied to dK at the end
                    dk2[o + 1] = pack_bf16(p2 * (__uint_as_float(dv[i + 2]) - dl.z), p3 * (__uint_as_float(dv[i + 3]) - dl.w));
                }
            }
            if (k > 0 && !mbar_wait_suspend(&sm.acc_done[grp], (k - 1) & 1, abort_flag, err, 0x5600 | grp)) { alive = false; break; }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int at = ((part * 4 + c) ^ (r & 7)) << 4;
                *reinterpret_cast<uint4*>(prow + at) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
                *reinterpret_cast<uint4*>(drow + at) = make_uint4(dk2[4 * c], dk2[4 * c + 1], dk2[4 * c + 2], dk2[4 * c + 3]);
            }
            tc_fence_before();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.p_ready[grp]);
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");           // behind it at most the last gradient GEMMs of each group are outstanding
        constexpr int OW = D / SPLIT;
        uint32_t av[OW], ak[OW];
#pragma unroll
        for (int i = 0; i < OW; ++i) { av[i] = 0u; ak[i] = 0u; }
        if (alive && n_it > 0 && mbar_wait_suspend(&sm.acc_done[(n_it - 1) & 1], ((n_it - 1) >> 1) & 1, abort_flag, err, 0x5700)) {
            tc_fence_after();
            tmem_ld<OW>(lane_addr + DV_COL + quarter * OW, av);
            tmem_ld<OW>(lane_addr + DK_COL + quarter * OW, ak);
            tmem_ld_wait();
        }
        if (key < a.Tk) {
            const long long off = (((long long)b * a.Tk + key) * a.Hkv + hk) * D + quarter * OW;
#pragma unroll
            for (int c = 0; c < OW; c += 8) {
                *reinterpret_cast<uint4*>(a.dv + off + c) = make_uint4(pack_bf16(__uint_as_float(av[c]), __uint_as_float(av[c + 1])),
                                                                       pack_bf16(__uint_as_float(av[c + 2]), __uint_as_float(av[c + 3])),
                                                                       pack_bf16(__uint_as_float(av[c + 4]), __uint_as_float(av[c + 5])),
                                                                       pack_bf16(__uint_as_float(av[c + 6]), __uint_as_float(av[c + 7])));
                *reinterpret_cast<uint4*>(a.dk + off + c) = make_uint4(pack_bf16(a.scale * __uint_as_float(ak[c]), a.scale * __uint_as_float(ak[c + 1])),
                                                                       pack_bf16(a.scale * __uint_as_float(ak[c + 2]), a.scale * __uint_as_float(ak[c + 3])),
                                                                       pack_bf16(a.scale * __uint_as_float(ak[c + 4]), a.scale * __uint_as_float(ak[c + 5])),
                                                                       pack_bf16(a.scale * __uint_as_float(ak[c + 6]), a.scale * __uint_as_float(ak[c + 7])));
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// delta[b,h,t] = sum_d dO[b,t,h,d] * O[b,t,h,d]; one warp per (b,t,h)
template <int D>
__global__ void fa_delta_tc_kernel(const bf16* __restrict__ o, const bf16* __restrict__ d_o, float* __restrict__ delta, int B, int Tq, int Hq) {
    const int l = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= (long long)B * Tq * Hq) return;
    const int h = row % Hq;
    const long long bt = row / Hq;
    const int t = bt % Tq, b = bt / Tq;
    float s = 0.f;
    for (int c = l * 2; c < D; c += 64) {
        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(o + row * D + c));
        const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(d_o + row * D + c));
        s += x.x * y.x + x.y * y.y;
    }
    s = warp_sum(s);
    if (l == 0) delta[((long long)b * Hq + h) * Tq + t] = s;
}

}  // namespace fatc
}  // namespace lmoe

using namespace lmoe;
using namespace lmoe::fatc;

// q [B,Tq,Hq,D], k/v [B,Tk,Hkv,D] bf16 with element strides (batch, token, head); 16-byte aligned bases, strides % 8 == 0.
LMOE_API int lmoe_flash_attn_fwd_tc(const void* q, const long long* qs, const void* k, const long long* ks, const void* v,
                                    const long long* vs, const Args* ap, int D, cudaStream_t st) {
    const Args a = *ap;
    CUtensorMap mq, mk, mv;
    int rc = make_map_4d(&mq, q, a.B, a.Tq, a.Hq, D, qs[0], qs[1], qs[2], BM);
    if (rc) return rc;
    rc = make_map_4d(&mk, k, a.B, a.Tk, a.Hkv, D, ks[0], ks[1], ks[2], BN);
    if (rc) return rc;
    rc = make_map_4d(&mv, v, a.B, a.Tk, a.Hkv, D, vs[0], vs[1], vs[2], 64);
    if (rc) return rc;
    dim3 grid((a.Tq + BM - 1) / BM, a.Hq, a.B);
    if (D == 128) {
        const size_t smem = sizeof(Smem<128>) + 1024;
        cudaFuncSetAttribute(fa_fwd_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        fa_fwd_tc_kernel<128><<<grid, THREADS, smem, st>>>(mq, mk, mv, a);
    } else if (D == 64) {
        const size_t smem = sizeof(Smem<64>) + 1024;
        cudaFuncSetAttribute(fa_fwd_tc_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        fa_fwd_tc_kernel<64><<<grid, THREADS, smem, st>>>(mq, mk, mv, a);
    } else return -1;
    return (int)cudaGetLastError();
}

template <int D>
static int launch_bwd_tc(const CUtensorMap& q128, const CUtensorMap& g128, const CUtensorMap& k64, const CUtensorMap& v64,
                         const CUtensorMap& q64, const CUtensorMap& g64, const CUtensorMap& k128, const CUtensorMap& v128,
                         const BwdArgs& a, const bf16* o, const bf16* d_o, float* delta, cudaStream_t st) {
    const long long rows = (long long)a.B * a.Tq * a.Hq;
    fa_delta_tc_kernel<D><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(o, d_o, delta, a.B, a.Tq, a.Hq);
    const size_t smem = sizeof(SmemBwd<D>) + 1024;
    cudaFuncSetAttribute(fa_bwd_dq_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaFuncSetAttribute(fa_bwd_dkv_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    fa_bwd_dq_tc_kernel<D><<<dim3((a.Tq + BM - 1) / BM, a.Hq, a.B), THREADS, smem, st>>>(q128, g128, k64, v64, a);
    fa_bwd_dkv_tc_kernel<D><<<dim3((a.Tk + BM - 1) / BM, a.Hkv, a.B), THREADS, smem, st>>>(q64, g64, k128, v128, a);
    return (int)cudaGetLastError();
}

// Backward of lmoe_flash_attn_fwd_tc.  o, d_o: contiguous [B,Tq,Hq,D]; ap->delta is scratch [B,Hq,Tq]; writes dq, dk, dv.
LMOE_API int lmoe_flash_attn_bwd_tc(const void* q, const long long* qs, const void* k, const long long* ks, const void* v,
                                    const long long* vs, const void* o, const void* d_o, float* delta, const BwdArgs* ap, int D,
                                    cudaStream_t st) {
    BwdArgs a = *ap;
    a.delta = delta;
    const long long gs[3] = {(long long)a.Tq * a.Hq * D, (long long)a.Hq * D, (long long)D};
    CUtensorMap q128, g128, k64, v64, q64, g64, k128, v128;
    int rc = 0;
    rc |= make_map_4d(&q128, q, a.B, a.Tq, a.Hq, D, qs[0], qs[1], qs[2], BM);
    rc |= make_map_4d(&g128, d_o, a.B, a.Tq, a.Hq, D, gs[0], gs[1], gs[2], BM);
    rc |= make_map_4d(&k64, k, a.B, a.Tk, a.Hkv, D, ks[0], ks[1], ks[2], BT);
    rc |= make_map_4d(&v64, v, a.B, a.Tk, a.Hkv, D, vs[0], vs[1], vs[2], BT);
    rc |= make_map_4d(&q64, q, a.B, a.Tq, a.Hq, D, qs[0], qs[1], qs[2], BT);
    rc |= make_map_4d(&g64, d_o, a.B, a.Tq, a.Hq, D, gs[0], gs[1], gs[2], BT);
    rc |= make_map_4d(&k128, k, a.B, a.Tk, a.Hkv, D, ks[0], ks[1], ks[2], BM);
    rc |= make_map_4d(&v128, v, a.B, a.Tk, a.Hkv, D, vs[0], vs[1], vs[2], BM);
    if (rc) return -11;
    if (D == 128) return launch_bwd_tc<128>(q128, g128, k64, v64, q64, g64, k128, v128, a, (const bf16*)o, (const bf16*)d_o, delta, st);
    if (D == 64) return launch_bwd_tc<64>(q128, g128, k64, v64, q64, g64, k128, v128, a, (const bf16*)o, (const bf16*)d_o, delta, st);
    return -1;
}
