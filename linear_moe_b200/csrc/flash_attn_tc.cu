// Flash-attention forward on the 5th-generation tensor cores: S = Q K^T and O_j = P_j V_j are tcgen05.mma instructions
// with accumulators in tensor memory, operands staged by TMA (4-D tensor maps over [B, T, H, D], 128-byte swizzle).
//
// One CTA = 128 queries of one head.  640 threads:
//   warp 0      TMA producer: Q once, then K_j / V_j tiles of 128 keys through rings of four (D 128: two) and two stages
//   warps 1, 2  MMA issuers, one per softmax group: S_j = Q K_j^T, then O += P_j V_j.  (One warp for both spent 1.3 of 2.4 thousand cycles a tile waiting
//               for one group's product to complete before it could issue the other group's next one.)
//   warps 4..19 softmax, two groups of eight: group g works on the tiles j = g (mod 2), so that one group's exponentials run while the
//               other one waits for its scores, exchanges maxima or hands over P.  (With all warps on the same tile every stage of
//               it was exposed: 3900 cycles a tile against 1024 of exponentials.)  Inside a group the two warps with equal (w & 3) own the 32 rows
//               of a tensor-memory lane quarter and half of the columns each.
// Each group has its own running maximum, sum and output, which are joined at the end.  Its output accumulates in tensor memory in
// units of a maximum that may lag behind by up to 2^LAG; only when a row runs ahead of that the output is rescaled there.  P_j goes
// back over its scores in bf16 and is read as the A operand from tensor memory.
// Tensor memory: 2 x 128 columns of scores, 2 x D of outputs.
// B=2, T=4096, 16 query and 4 kv heads of 128: 242 -> 180 us; B=1, 1531 queries over 2552 keys, 32 / 8 heads of 64: 86 -> 60 us (with one issuing warp and two stages of K 63).
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
    // The scores of a tile wait for its K at once, its V only behind the exponentials.  An even number of stages: a stage's tiles are all of one group, whose
    // warp has waited for the one before (else a wait by parity could take the tile before for this one).
    static constexpr int KS = D == 64 ? 4 : 2;
    uint8_t k[KS][BN * D * 2];
    uint8_t v[2][BN * D * 2];
    uint64_t q_full, k_full[KS], k_empty[KS], v_full[2], v_empty[2], s_full[2], p_ready[2], pv_done[2];
    float mx[2][2][2][BM];            // [parity of the group's tile][group][half of the columns]
    float ls[2][2][BM], ms[2][BM];    // sums and maxima at the end
    uint32_t tmem_base;
    int abort_flag;
};

// Which tile a CTA takes.  CTAs start in the order of their index, so the longest tiles of all (batch, head) pairs come first and the short ones
// fill the end: with the tile as the fastest dimension inside a head, the last heads' longest tiles started when the others were done
// (SM busy for 0.61 of the dk / dv launch, 0.85 of the others).  Only `group` pairs are mixed at a time: their streamed rows share the L2.
// B=2, T=4096, 16 / 4 heads of 128, forward and backward: 901 -> 752 us; 1531 queries over 2552 keys, 32 / 8 heads of 64: 67 -> 61.
struct TileOf { int rank, pair; };
__device__ __forceinline__ TileOf longest_first(int idx, int tiles, int pairs, int group) {
    const int sec = idx / (tiles * group), rem = idx - sec * tiles * group;
    const int n = min(group, pairs - sec * group);
    return {rem / n, sec * group + rem % n};
}
// Pairs whose streamed tensors (two of `rows` x D bf16 per `share` pairs) stay within half of the L2 together.
static int pairs_in_l2(int pairs, long long rows, int D, int share) {
    const long long n = (64LL << 20) / max(rows * D * 4, 1LL);
    return (int)min((long long)pairs, max(n, 1LL) * share);
}

template <int D>
__global__ void __launch_bounds__(THREADS, 1)
fa_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, Args a, int group) {
    extern __shared__ uint8_t smem_raw[];
    Smem<D>& sm = *reinterpret_cast<Smem<D>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int KS = Smem<D>::KS;
    constexpr int DK = D / 64;                              // 64-element blocks along the head dimension
    constexpr uint32_t TMEM_COLS = 512;
    constexpr uint32_t O_COL = 2 * BN;                      // the groups' outputs behind the two score buffers
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int n_qb = (a.Tq + BM - 1) / BM;
    const TileOf t = longest_first(blockIdx.x, n_qb, a.B * a.Hq, group);
    const int qb = n_qb - 1 - t.rank;                       // late query tiles see the most keys
    const int h = t.pair % a.Hq, b = t.pair / a.Hq;
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
        for (int s = 0; s < KS; ++s) { mbar_init(&sm.k_full[s], 1); mbar_init(&sm.k_empty[s], 1); }
        for (int s = 0; s < 2; ++s) {
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
    const uint32_t tmem_base = uniform(sm.tmem_base);

    if (warp == 0) {
        if (lane == 0 && n_it > 0) {
            mbar_expect_tx(&sm.q_full, BM * D * 2);
#pragma unroll
            for (int kb = 0; kb < DK; ++kb) tma_load_4d(sm.q + kb * BM * 128, &tmQ, &sm.q_full, kb * 64, h, q0, b);
            for (int j = 0; j < n_it; ++j) {
                const int s = j & 1, sk = j % KS;
                const uint32_t ph = (j >> 1) & 1;
                const int key0 = (nb_lo + j) * BN;
                if (!mbar_wait_suspend(&sm.k_empty[sk], ((j / KS) & 1) ^ 1, abort_flag, err, 0x1100 | sk)) break;
                mbar_expect_tx(&sm.k_full[sk], BN * D * 2);
#pragma unroll
                for (int kb = 0; kb < DK; ++kb) tma_load_4d(sm.k[sk] + kb * BN * 128, &tmK, &sm.k_full[sk], kb * 64, hk, key0, b);
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
    } else if (warp == 1 || warp == 2) {                       // a group's products, each group's in a warp of its own
        const int g = warp - 1;
        if (g < n_it) {
            constexpr uint32_t idesc_s = idesc_bf16<false, BN>();
            constexpr uint32_t idesc_o = idesc_bf16<true, D>();
            bool ok = mbar_wait_warp(&sm.q_full, 0, abort_flag, err, 0x2000);
            for (int j = g; ok && j < n_it; j += 2) {
                const int sk = j % KS;
                const uint32_t ph = (j >> 1) & 1;
                // the scores go over the group's last P: its product has to complete
                ok = mbar_wait_warp(&sm.k_full[sk], (j / KS) & 1, abort_flag, err, 0x2100 | sk) &&
                     (j < 2 || mbar_wait_warp(&sm.pv_done[g], ph ^ 1, abort_flag, err, 0x2400));
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t ql = desc_lo<false>(s32(sm.q)), kl = desc_lo<false>(s32(sm.k[sk]));
#pragma unroll
                    for (int kk = 0; kk < D / UMMA_K; ++kk) {
                        const uint32_t off = ((kk / 4) * (BM * 128) + (kk % 4) * 32) >> 4;
                        umma_ss(tmem_base + g * BN, ql + off, kl + off, idesc_s, kk > 0);
                    }
                    umma_commit(&sm.k_empty[sk]);
                    umma_commit(&sm.s_full[g]);
                }
                ok = mbar_wait_warp(&sm.v_full[g], ph, abort_flag, err, 0x2200 | g) && mbar_wait_warp(&sm.p_ready[g], ph, abort_flag, err, 0x2300 | g);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t vl = desc_lo<true>(s32(sm.v[g]));
#pragma unroll
                    for (int kk = 0; kk < BN / UMMA_K; ++kk) {
                        // every half of the columns left its 32 columns of P at its beginning
                        const uint32_t boff = ((kk / 4) * (DK * 8192) + (kk % 4) * 2048) >> 4;
                        umma_ts(tmem_base + O_COL + g * D, tmem_base + g * BN + kk / 4 * 64 + kk % 4 * 8, vl + boff, idesc_o, j > 1 || kk > 0);
                    }
                    umma_commit(&sm.v_empty[g]);
                    umma_commit(&sm.pv_done[g]);
                }
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
// Backward on tcgen05, two kernels that recompute the scores (7 GEMMs per tile pair instead of 5, no atomics), on tiles of
// 128 queries x 128 keys:
//   fa_bwd_dq_tc_kernel    one CTA = 128 queries of one head, looping over the key tiles:
//                          S = Q K^T and dP = dO V^T into tensor memory -> dS = P (dP - delta) (softmax warps, thread = query row), in bf16
//                          over S -> dQ += dS K accumulated in tensor memory.
//   fa_bwd_dkv_tc_kernel   one CTA = 128 keys of one KV head, looping over the query heads of the group and their query
//                          tiles: S^T = K Q^T and dP^T = V dO^T -> P^T, dS^T (thread = key row), in bf16 over the two ->
//                          dV += P^T dO and dK += dS^T Q accumulated in tensor memory.
// A tile of 128 rows loaded as D/64 boxes of {64 d, 128 rows} serves both as a K-major operand (rows = N) of the score GEMMs
// and as an MN-major operand (rows = K) of the gradient GEMMs.  Same warp roles and bounded waits as the forward; all sixteen softmax
// warps share a tile, four per 32 rows with 32 columns each.  The order of the products keeps the tensor core busy while
// the warps work: a score GEMM is issued as soon as its scores have been read, ahead of the gradient GEMM of the tile before.
// The 64-wide tiles that stood here first issued 24 instructions per 128 x 64 scores, these 32 per 128 x 128.  B=2, T=4096, 16 query and 4 kv heads of
// 128 (16896 pairs of 128 x 128): dk / dv 514 -> 396 us, dq 335 -> 288 (at the measured 1654 TFLOP/s: 166 and 125), with the tensor pipe active for
// 0.53 and 0.39 of the cycles of a busy SM; the order of the tiles then took another 120 us off the two.
// P^T and dS as operands in tensor memory (a trip through shared memory before, with a fence and an eighth of the traffic of its products) leave room for
// dO in two stages: forward and backward 752 -> 738 us, dk / dv 277, dq 247.  A third stage of K in the dq kernel (a tile's K is read by its first and its
// last product, and the next scores waited for a load that could start only then), its exponentials ahead of the wait for dP instead of
// behind it, where the compiler had moved them, and MMA operands that look uniform: 738 -> 695, dk / dv 257, dq 208.
// =====================================================================================================================
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

constexpr int BLK = BM * 128;                                // one 64-column block of a 128-row tile

__device__ __forceinline__ bool visible(int key, int qi, int Tk, int window) {
    return key <= qi && key < Tk && (window <= 0 || key > qi - window);
}
template <int D>
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int h, int row, int b) {
#pragma unroll
    for (int kb = 0; kb < D / 64; ++kb) tma_load_4d(dst + kb * BLK, map, bar, kb * 64, h, row, b);
}
// [128 x 128] = A B^T over D, both tiles K-major
template <int D>
__device__ __forceinline__ void score_product(uint32_t tmem_d, const uint8_t* A, const uint8_t* B) {
    if (!elect_one()) return;
    const uint32_t al = desc_lo<false>(s32(A)), bl = desc_lo<false>(s32(B));
#pragma unroll
    for (int kk = 0; kk < D / UMMA_K; ++kk) {
        const uint32_t off = ((kk / 4) * BLK + (kk % 4) * 32) >> 4;
        umma_ss(tmem_d, al + off, bl + off, idesc_bf16<false, 128>(), kk > 0);
    }
}
// [128 x D] (+)= A B over 128: A in tensor memory as the warps left it (16 packed columns at the beginning of every part's 32), B's rows are K
template <int D>
__device__ __forceinline__ void grad_product(uint32_t tmem_d, uint32_t tmem_a, const uint8_t* B, bool add) {
    if (!elect_one()) return;
    const uint32_t bl = ((s32(B) >> 4) & 0x3FFFu) | ((uint32_t)(BLK >> 4) << 16);
#pragma unroll
    for (int kk = 0; kk < 128 / UMMA_K; ++kk)
        umma_ts(tmem_d, tmem_a + kk / 2 * 32 + kk % 2 * 8, bl + ((kk * 2048) >> 4), idesc_bf16<true, D>(), add || kk > 0);
}
// this thread's 32 columns of an operand, over scores that it has read
__device__ __forceinline__ void hand_over(uint32_t taddr, const uint32_t (&v)[16], uint64_t* bar) {
    tmem_st16(taddr, v);
    tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
// a thread's part of an accumulator row, times `scale`, to memory
template <int OW>
__device__ __forceinline__ void write_row(bf16* out, uint32_t taddr, float scale, bool valid, bool empty) {
    uint32_t v[OW];
    tmem_ld<OW>(taddr, v);
    tmem_ld_wait();
    if (!valid) return;
#pragma unroll
    for (int c = 0; c < OW; c += 8) {
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = empty ? 0.f : scale * __uint_as_float(v[c + e]);
        *reinterpret_cast<uint4*>(out + c) = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
    }
}

// With 128-wide heads the tiles fill the shared memory: it has to start on a 1024-byte boundary (there is no static one), which the
// kernels check before anything else.
template <int D>
struct __align__(1024) SmemDq {
    uint8_t q[BM * D * 2], g[BM * D * 2], k[3][BM * D * 2], v[2][BM * D * 2];      // K: read by a tile's first and last product
    uint64_t qg_full, k_full[3], k_empty[3], v_full[2], v_empty[2], s_full[2], dp_full, ds_ready, dq_done, all_done;
    uint32_t tmem_base;
    int abort_flag;
};

template <int D>
__global__ void __launch_bounds__(THREADS, 1)
fa_bwd_dq_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmG,
                    const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, BwdArgs a, int group) {
    extern __shared__ uint8_t smem_raw[];
    SmemDq<D>& sm = *reinterpret_cast<SmemDq<D>*>(smem_raw);
    if ((s32(smem_raw) & 1023u) != 0) {
        if (threadIdx.x == 0) atomicCAS(a.err, 0, 0x4001);
        return;
    }
    constexpr uint32_t TMEM_COLS = 512, DP = 256, DQ = 384;                  // two buffers of scores in front
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int n_qb = (a.Tq + BM - 1) / BM;
    const TileOf t = longest_first(blockIdx.x, n_qb, a.B * a.Hq, group);
    const int qb = n_qb - 1 - t.rank;
    const int h = t.pair % a.Hq, b = t.pair / a.Hq;
    const int hk = h / (a.Hq / a.Hkv);
    const int q0 = qb * BM;
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    const int last_q = min(a.Tq, q0 + BM) - 1;
    const int k_hi = min(a.Tk, a.q_offset + last_q + 1);
    const int k_lo = a.window > 0 ? max(0, a.q_offset + q0 - a.window + 1) : 0;
    const int nb_lo = k_lo / BN, nb_hi = (k_hi + BN - 1) / BN;
    const int n_it = max(nb_hi - nb_lo, 0);

    if (threadIdx.x == 0) {
        mbar_init(&sm.qg_full, 1);
        for (int s = 0; s < 3; ++s) { mbar_init(&sm.k_full[s], 1); mbar_init(&sm.k_empty[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&sm.v_full[s], 1); mbar_init(&sm.v_empty[s], 1); mbar_init(&sm.s_full[s], 1); }
        mbar_init(&sm.dp_full, 1); mbar_init(&sm.ds_ready, 4 * SPLIT); mbar_init(&sm.dq_done, 1); mbar_init(&sm.all_done, 1);
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
    const uint32_t tmem_base = uniform(sm.tmem_base);

    if (warp == 0) {
        if (lane == 0 && n_it > 0) {
            mbar_expect_tx(&sm.qg_full, 2 * BM * D * 2);
            load_tile<D>(sm.q, &tmQ, &sm.qg_full, h, q0, b);
            load_tile<D>(sm.g, &tmG, &sm.qg_full, h, q0, b);
            for (int j = 0; j < n_it; ++j) {
                const int s = j & 1, s3 = j % 3, key0 = (nb_lo + j) * BN;
                if (!mbar_wait_suspend(&sm.k_empty[s3], ((j / 3) & 1) ^ 1, abort_flag, err, 0x4100 | s3)) break;
                mbar_expect_tx(&sm.k_full[s3], BM * D * 2);
                load_tile<D>(sm.k[s3], &tmK, &sm.k_full[s3], hk, key0, b);
                if (!mbar_wait_suspend(&sm.v_empty[s], ((j >> 1) & 1) ^ 1, abort_flag, err, 0x4110 | s)) break;
                mbar_expect_tx(&sm.v_full[s], BM * D * 2);
                load_tile<D>(sm.v[s], &tmV, &sm.v_full[s], hk, key0, b);
            }
        }
    } else if (warp == 1) {
        if (n_it > 0) {
            bool ok = mbar_wait_warp(&sm.qg_full, 0, abort_flag, err, 0x4200);
            auto scores = [&](int j) -> bool {
                const int s = j & 1, s3 = j % 3;
                if (!mbar_wait_warp(&sm.k_full[s3], (j / 3) & 1, abort_flag, err, 0x4300 | s3)) return false;
                tc_fence_after();
                score_product<D>(tmem_base + s * 128, sm.q, sm.k[s3]);
                if (elect_one()) umma_commit(&sm.s_full[s]);
                return true;
            };
            auto dprobs = [&](int j) -> bool {
                const int s = j & 1;
                if (!mbar_wait_warp(&sm.v_full[s], (j >> 1) & 1, abort_flag, err, 0x4310 | s)) return false;
                tc_fence_after();
                score_product<D>(tmem_base + DP, sm.g, sm.v[s]);
                if (elect_one()) { umma_commit(&sm.v_empty[s]); umma_commit(&sm.dp_full); }
                return true;
            };
            if (ok) ok = scores(0) && dprobs(0);
            if (ok && n_it > 1) ok = scores(1);
            for (int j = 0; ok && j < n_it; ++j) {
                const int s = j & 1;
                if (!mbar_wait_warp(&sm.ds_ready, j & 1, abort_flag, err, 0x4400)) break;
                if (j + 1 < n_it && !dprobs(j + 1)) break;
                tc_fence_after();
                grad_product<D>(tmem_base + DQ, tmem_base + s * 128, sm.k[j % 3], j > 0);
                if (elect_one()) { umma_commit(&sm.k_empty[j % 3]); umma_commit(j + 1 < n_it ? &sm.dq_done : &sm.all_done); }
                // the next scores of this buffer go over dS_j: the product that reads it has to complete
                if (j + 2 < n_it) ok = mbar_wait_warp(&sm.dq_done, j & 1, abort_flag, err, 0x4600) && scores(j + 2);
            }
        }
    } else if (warp >= 4) {
        const int qd = warp & 3, part = (warp - 4) >> 2;
        const int r = qd * 32 + lane;
        const int row = q0 + r;
        const int qi = a.q_offset + row;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16);
        const float sc = a.scale * LOG2E;
        const long long stat = ((long long)b * a.Hq + h) * a.Tq + row;
        const float lse2 = row < a.Tq ? a.lse[stat] * LOG2E : INFINITY;
        const float dl = row < a.Tq ? a.delta[stat] : 0.f;
        bool alive = n_it > 0;
        for (int j = 0; alive && j < n_it; ++j) {
            const int s = j & 1;
            const int tile_key0 = (nb_lo + j) * BN, key0 = tile_key0 + part * 32;
            // masking is needed only on tiles that cross the causal diagonal, the window edge or the key length
            const bool need_mask = (tile_key0 + BN - 1 > a.q_offset + q0) || (tile_key0 + BN > a.Tk) ||
                                   (a.window > 0 && tile_key0 <= a.q_offset + q0 + BM - 1 - a.window);
            if (!mbar_wait_suspend(&sm.s_full[s], (j >> 1) & 1, abort_flag, err, 0x4500 | s)) { alive = false; break; }
            tc_fence_after();
            uint32_t v[32];
            tmem_ld32(lane_addr + s * 128 + part * 32, v);
            tmem_ld_wait();
            if (need_mask) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (!visible(key0 + i, qi, a.Tk, a.window)) v[i] = 0xff800000u;              // -inf -> p = 0
            }
            float2 p[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float2 x = __ffma2_rn(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), make_float2(sc, sc), make_float2(-lse2, -lse2));
                p[i] = make_float2(exp2f(x.x), exp2f(x.y));
                asm volatile("" : "+f"(p[i].x), "+f"(p[i].y));                                     // here, not behind the wait
            }
            if (!mbar_wait_suspend(&sm.dp_full, j & 1, abort_flag, err, 0x4510)) { alive = false; break; }
            tc_fence_after();
            tmem_ld32(lane_addr + DP + part * 32, v);
            tmem_ld_wait();
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {                                                       // the softmax scale is applied to dQ at the end
                const float2 d = __fmul2_rn(p[i], __fadd2_rn(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), make_float2(-dl, -dl)));
                pk[i] = pack_bf16(d.x, d.y);
            }
            hand_over(lane_addr + s * 128 + part * 32, pk, &sm.ds_ready);
        }
        if (alive) alive = mbar_wait_suspend(&sm.all_done, 0, abort_flag, err, 0x4700);
        tc_fence_after();
        constexpr int OW = D / SPLIT;
        write_row<OW>(a.dq + (((long long)b * a.Tq + row) * a.Hq + h) * D + part * OW, lane_addr + DQ + part * OW, a.scale, row < a.Tq, !alive);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}


template <int D>
struct __align__(1024) SmemDkv {
    uint8_t k[BM * D * 2], v[BM * D * 2], q[2][BM * D * 2], g[2][BM * D * 2];
    float lse2[2][BM], delta[2][BM];                                         // of the looped queries
    uint64_t kv_full, q_full[2], q_empty[2], stat_full[2], g_full[2], g_empty[2], s_full, dp_full, p_ready, ds_ready, dv_done, dk_done, all_done;
    uint32_t tmem_base;
    int abort_flag;
};

template <int D>
__global__ void __launch_bounds__(THREADS, 1)
fa_bwd_dkv_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmG,
                     const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, BwdArgs a, int group) {
    extern __shared__ uint8_t smem_raw[];
    SmemDkv<D>& sm = *reinterpret_cast<SmemDkv<D>*>(smem_raw);
    if ((s32(smem_raw) & 1023u) != 0) {
        if (threadIdx.x == 0) atomicCAS(a.err, 0, 0x5001);
        return;
    }
    constexpr uint32_t TMEM_COLS = 512, ST = 0, DP = 128, DV = 256, DKC = 384;
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const TileOf t = longest_first(blockIdx.x, (a.Tk + BM - 1) / BM, a.B * a.Hkv, group);
    const int kb_tile = t.rank, hk = t.pair % a.Hkv, b = t.pair / a.Hkv;      // early key tiles are seen by the most queries
    const int rep = a.Hq / a.Hkv;
    const int k0 = kb_tile * BM;
    volatile int* abort_flag = &sm.abort_flag;
    int* err = a.err;
    // query tiles that can see a key of this tile: q >= k0 - q_offset, and with a window q < k0 + 127 + window - q_offset
    const int i_lo = max(0, k0 - a.q_offset) / BM;
    int q_end = a.Tq;
    if (a.window > 0) q_end = min(a.Tq, max(0, k0 + BM - 1 + a.window - a.q_offset));
    const int i_hi = (q_end + BM - 1) / BM;
    const int ni = max(i_hi - i_lo, 0);
    const int n_it = ni * rep;

    if (threadIdx.x == 0) {
        mbar_init(&sm.kv_full, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&sm.q_full[s], 1); mbar_init(&sm.q_empty[s], 1); mbar_init(&sm.stat_full[s], 1);
            mbar_init(&sm.g_full[s], 1); mbar_init(&sm.g_empty[s], 1);
        }
        mbar_init(&sm.s_full, 1); mbar_init(&sm.dp_full, 1);
        mbar_init(&sm.p_ready, 4 * SPLIT); mbar_init(&sm.ds_ready, 4 * SPLIT);
        mbar_init(&sm.dv_done, 1); mbar_init(&sm.dk_done, 1); mbar_init(&sm.all_done, 1);
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
    const uint32_t tmem_base = uniform(sm.tmem_base);

    if (warp == 0) {
        if (lane == 0 && n_it > 0) {
            mbar_expect_tx(&sm.kv_full, 2 * BM * D * 2);
            load_tile<D>(sm.k, &tmK, &sm.kv_full, hk, k0, b);
            load_tile<D>(sm.v, &tmV, &sm.kv_full, hk, k0, b);
            for (int it = 0; it < n_it; ++it) {
                const int s = it & 1;
                const int h = hk * rep + it / ni, q0 = (i_lo + it % ni) * BM;
                if (!mbar_wait_suspend(&sm.q_empty[s], ((it >> 1) & 1) ^ 1, abort_flag, err, 0x5100 | s)) break;
                mbar_expect_tx(&sm.q_full[s], BM * D * 2);
                load_tile<D>(sm.q[s], &tmQ, &sm.q_full[s], h, q0, b);
                if (!mbar_wait_suspend(&sm.g_empty[s], ((it >> 1) & 1) ^ 1, abort_flag, err, 0x5120 | s)) break;
                mbar_expect_tx(&sm.g_full[s], BM * D * 2);
                load_tile<D>(sm.g[s], &tmG, &sm.g_full[s], h, q0, b);
            }
        }
    } else if (warp == 1) {
        if (n_it > 0) {
            bool ok = mbar_wait_warp(&sm.kv_full, 0, abort_flag, err, 0x5200);
            auto scores = [&](int it) -> bool {
                if (!mbar_wait_warp(&sm.q_full[it & 1], (it >> 1) & 1, abort_flag, err, 0x5300 | (it & 1))) return false;
                tc_fence_after();
                score_product<D>(tmem_base + ST, sm.k, sm.q[it & 1]);
                if (elect_one()) umma_commit(&sm.s_full);
                return true;
            };
            auto dprobs = [&](int it) -> bool {
                if (!mbar_wait_warp(&sm.g_full[it & 1], (it >> 1) & 1, abort_flag, err, 0x5310 | (it & 1))) return false;
                tc_fence_after();
                score_product<D>(tmem_base + DP, sm.v, sm.g[it & 1]);
                if (elect_one()) umma_commit(&sm.dp_full);
                return true;
            };
            if (ok) ok = scores(0) && dprobs(0);
            for (int it = 0; ok && it < n_it; ++it) {
                if (!mbar_wait_warp(&sm.p_ready, it & 1, abort_flag, err, 0x5400)) break;
                tc_fence_after();
                const bool more = it + 1 < n_it;
                grad_product<D>(tmem_base + DV, tmem_base + ST, sm.g[it & 1], it > 0);   // dV += P^T dO
                if (elect_one()) umma_commit(&sm.g_empty[it & 1]);
                if (more) {
                    // the next scores go over P^T: the product that reads it has to complete
                    if (elect_one()) umma_commit(&sm.dv_done);
                    if (!mbar_wait_warp(&sm.dv_done, it & 1, abort_flag, err, 0x5600) || !scores(it + 1)) break;
                }
                if (!mbar_wait_warp(&sm.ds_ready, it & 1, abort_flag, err, 0x5410)) break;
                tc_fence_after();
                grad_product<D>(tmem_base + DKC, tmem_base + DP, sm.q[it & 1], it > 0);  // dK += dS^T Q
                if (elect_one()) { umma_commit(&sm.q_empty[it & 1]); umma_commit(more ? &sm.dk_done : &sm.all_done); }
                if (more) ok = mbar_wait_warp(&sm.dk_done, it & 1, abort_flag, err, 0x5610) && dprobs(it + 1);
            }
        }
    } else if (warp == 2) {                                      // log-sum-exp and delta of the looped queries
        for (int it = 0; it < n_it; ++it) {
            const int s = it & 1;
            const int h = hk * rep + it / ni, q0 = (i_lo + it % ni) * BM;
            const long long row = ((long long)b * a.Hq + h) * a.Tq;
            float x[4], y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int q = q0 + lane + 32 * e;
                x[e] = q < a.Tq ? __ldg(a.lse + row + q) * LOG2E : INFINITY;
                y[e] = q < a.Tq ? __ldg(a.delta + row + q) : 0.f;
            }
            if (!mbar_wait_suspend(&sm.q_empty[s], ((it >> 1) & 1) ^ 1, abort_flag, err, 0x5110 | s)) break;
#pragma unroll
            for (int e = 0; e < 4; ++e) { sm.lse2[s][lane + 32 * e] = x[e]; sm.delta[s][lane + 32 * e] = y[e]; }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.stat_full[s]);
        }
    } else if (warp >= 4) {
        const int qd = warp & 3, part = (warp - 4) >> 2;
        const int r = qd * 32 + lane;                            // key row inside the tile
        const int key = k0 + r;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16);
        const float sc = a.scale * LOG2E;
        bool alive = n_it > 0;
        for (int it = 0; alive && it < n_it; ++it) {
            const int s = it & 1;
            const int tile_q0 = (i_lo + it % ni) * BM;
            const bool need_mask = (k0 + BM - 1 > a.q_offset + tile_q0) || (k0 + BM > a.Tk) ||
                                   (a.window > 0 && k0 <= a.q_offset + tile_q0 + BM - 1 - a.window);
            if (!mbar_wait_suspend(&sm.stat_full[s], (it >> 1) & 1, abort_flag, err, 0x5510 | s)) { alive = false; break; }
            if (!mbar_wait_suspend(&sm.s_full, it & 1, abort_flag, err, 0x5500)) { alive = false; break; }
            tc_fence_after();
            uint32_t v[32], pk[16];
            float2 p[16];
            tmem_ld32(lane_addr + ST + part * 32, v);
            tmem_ld_wait();
            if (need_mask) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (!visible(key, a.q_offset + tile_q0 + part * 32 + i, a.Tk, a.window)) v[i] = 0xff800000u;
            }
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const float4 l2 = *reinterpret_cast<const float4*>(&sm.lse2[s][part * 32 + 2 * i]);
                const float2 x = __ffma2_rn(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), make_float2(sc, sc), make_float2(-l2.x, -l2.y));
                const float2 y = __ffma2_rn(make_float2(__uint_as_float(v[2 * i + 2]), __uint_as_float(v[2 * i + 3])), make_float2(sc, sc), make_float2(-l2.z, -l2.w));
                p[i] = make_float2(exp2f(x.x), exp2f(x.y));
                p[i + 1] = make_float2(exp2f(y.x), exp2f(y.y));
                pk[i] = pack_bf16(p[i].x, p[i].y);
                pk[i + 1] = pack_bf16(p[i + 1].x, p[i + 1].y);
            }
            hand_over(lane_addr + ST + part * 32, pk, &sm.p_ready);
            if (!mbar_wait_suspend(&sm.dp_full, it & 1, abort_flag, err, 0x5520)) { alive = false; break; }
            tc_fence_after();
            tmem_ld32(lane_addr + DP + part * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; i += 2) {                                                   // scale applied to dK at the end
                const float4 dl = *reinterpret_cast<const float4*>(&sm.delta[s][part * 32 + 2 * i]);
                const float2 x = __fmul2_rn(p[i], __fadd2_rn(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), make_float2(-dl.x, -dl.y)));
                const float2 y = __fmul2_rn(p[i + 1], __fadd2_rn(make_float2(__uint_as_float(v[2 * i + 2]), __uint_as_float(v[2 * i + 3])), make_float2(-dl.z, -dl.w)));
                pk[i] = pack_bf16(x.x, x.y);
                pk[i + 1] = pack_bf16(y.x, y.y);
            }
            hand_over(lane_addr + DP + part * 32, pk, &sm.ds_ready);
        }
        if (alive) alive = mbar_wait_suspend(&sm.all_done, 0, abort_flag, err, 0x5700);        // covers dV, which was issued before dK
        tc_fence_after();
        constexpr int OW = D / SPLIT;
        const long long off = (((long long)b * a.Tk + key) * a.Hkv + hk) * D + part * OW;
        write_row<OW>(a.dv + off, lane_addr + DV + part * OW, 1.f, key < a.Tk, !alive);
        write_row<OW>(a.dk + off, lane_addr + DKC + part * OW, a.scale, key < a.Tk, !alive);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// delta[b,h,t] = sum_d dO[b,t,h,d] * O[b,t,h,d].  Bound by reading both tensors once: D / 8 lanes take a row 16 bytes at a time, and a thread asks
// for its pieces of four rows before it uses the first (a warp per row with 4-byte loads had too little in flight).
template <int D>
__global__ void __launch_bounds__(256) fa_delta_tc_kernel(const bf16* __restrict__ o, const bf16* __restrict__ d_o, float* __restrict__ delta, int B, int Tq, int Hq) {
    constexpr int LANES = D / 8, PER = 256 / LANES, U = 4;       // lanes of a row, rows of a block at a time
    const int l = threadIdx.x % LANES;
    const long long rows = (long long)B * Tq * Hq, row0 = (long long)blockIdx.x * (PER * U) + threadIdx.x / LANES;
    Vec<bf16> x[U], y[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long at = min(row0 + u * PER, rows - 1) * D + l * 8;
        x[u].load(o + at);
        y[u].load(d_o + at);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long row = row0 + u * PER;
        float s = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) s += x[u].get(e) * y[u].get(e);
#pragma unroll
        for (int w = LANES / 2; w > 0; w >>= 1) s += __shfl_xor_sync(0xffffffffu, s, w);
        if (l == 0 && row < rows) {
            const long long bt = row / Hq;
            delta[((bt / Tq) * Hq + row % Hq) * Tq + bt % Tq] = s;
        }
    }
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
    const unsigned grid = (unsigned)((a.Tq + BM - 1) / BM) * a.Hq * a.B;
    const int group = pairs_in_l2(a.B * a.Hq, a.Tk, D, a.Hq / a.Hkv);
    if (D == 128) {
        const size_t smem = sizeof(Smem<128>) + 1024;
        cudaFuncSetAttribute(fa_fwd_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        fa_fwd_tc_kernel<128><<<grid, THREADS, smem, st>>>(mq, mk, mv, a, group);
    } else if (D == 64) {
        const size_t smem = sizeof(Smem<64>) + 1024;
        cudaFuncSetAttribute(fa_fwd_tc_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        fa_fwd_tc_kernel<64><<<grid, THREADS, smem, st>>>(mq, mk, mv, a, group);
    } else return -1;
    return (int)cudaGetLastError();
}

template <int D>
static int launch_bwd_tc(const CUtensorMap& q, const CUtensorMap& g, const CUtensorMap& k, const CUtensorMap& v, const BwdArgs& a, const bf16* o,
                         const bf16* d_o, float* delta, cudaStream_t st) {
    const long long rows = (long long)a.B * a.Tq * a.Hq;
    constexpr int per_block = 4 * 256 / (D / 8);
    fa_delta_tc_kernel<D><<<(unsigned)((rows + per_block - 1) / per_block), 256, 0, st>>>(o, d_o, delta, a.B, a.Tq, a.Hq);
    int rc = (int)cudaFuncSetAttribute(fa_bwd_dq_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemDq<D>));
    if (rc) return rc;
    rc = (int)cudaFuncSetAttribute(fa_bwd_dkv_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemDkv<D>));
    if (rc) return rc;
    fa_bwd_dq_tc_kernel<D><<<(unsigned)((a.Tq + BM - 1) / BM) * a.Hq * a.B, THREADS, sizeof(SmemDq<D>), st>>>(
        q, g, k, v, a, pairs_in_l2(a.B * a.Hq, a.Tk, D, a.Hq / a.Hkv));
    // a CTA goes through its query heads one after the other, so one of them counts
    fa_bwd_dkv_tc_kernel<D><<<(unsigned)((a.Tk + BM - 1) / BM) * a.Hkv * a.B, THREADS, sizeof(SmemDkv<D>), st>>>(
        q, g, k, v, a, pairs_in_l2(a.B * a.Hkv, a.Tq, D, 1));
    return (int)cudaGetLastError();
}

// Backward of lmoe_flash_attn_fwd_tc.  o, d_o: contiguous [B,Tq,Hq,D]; ap->delta is scratch [B,Hq,Tq]; writes dq, dk, dv.
LMOE_API int lmoe_flash_attn_bwd_tc(const void* q, const long long* qs, const void* k, const long long* ks, const void* v,
                                    const long long* vs, const void* o, const void* d_o, float* delta, const BwdArgs* ap, int D,
                                    cudaStream_t st) {
    BwdArgs a = *ap;
    a.delta = delta;
    const long long gs[3] = {(long long)a.Tq * a.Hq * D, (long long)a.Hq * D, (long long)D};
    CUtensorMap mq, mg, mk, mv;
    int rc = 0;
    rc |= make_map_4d(&mq, q, a.B, a.Tq, a.Hq, D, qs[0], qs[1], qs[2], BM);
    rc |= make_map_4d(&mg, d_o, a.B, a.Tq, a.Hq, D, gs[0], gs[1], gs[2], BM);
    rc |= make_map_4d(&mk, k, a.B, a.Tk, a.Hkv, D, ks[0], ks[1], ks[2], BM);
    rc |= make_map_4d(&mv, v, a.B, a.Tk, a.Hkv, D, vs[0], vs[1], vs[2], BM);
    if (rc) return -11;
    if (D == 128) return launch_bwd_tc<128>(mq, mg, mk, mv, a, (const bf16*)o, (const bf16*)d_o, delta, st);
    if (D == 64) return launch_bwd_tc<64>(mq, mg, mk, mv, a, (const bf16*)o, (const bf16*)d_o, delta, st);
    return -1;
}
