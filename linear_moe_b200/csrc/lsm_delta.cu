// (Gated) delta rule: the recurrence over chunks, forward and backward, as hand-written kernels.
//
//   S_t = e^{g_t} S_{t-1} + beta_t k_t^T (v_t - k_t e^{g_t} S_{t-1}),      o_t = scale * q_t S_t
//
// In the chunked (WY / UT-transform) form every chunk of C = 64 tokens is described by tiles that do not depend on
// the state (computed chunk-parallel before this kernel):
//   W  [C,dk]  pseudo keys      T (beta e^{b} K),        T = (I + tril(diag(beta) (K K^T . Gamma), -1))^{-1}
//   U  [C,dv]  pseudo values    T (beta V)
//   Qd [C,dk]  scale * e^{b_i} q_i           Kd [C,dk]  e^{b_C - b_j} k_j
//   A  [C,C]   scale * tril((Q K^T) . Gamma)  (diagonal included),   Gamma_ij = e^{b_i - b_j},   gamma = e^{b_C}
// and the state-dependent part is, per chunk with entering state S,
//   Vn = U - W S,        O = Qd S + A Vn,        S' = gamma S + Kd^T Vn.
// The columns of S are independent, so a (batch, head) sequence is split over dv / 32 CTAs (value slices) to fill the
// machine; a CTA walks the chunks in order with its [dk x 32] state slice in fp32 registers and a bf16 copy in shared
// memory as the B operand.  The forward kernel also writes Vn and the entering state of every chunk (bf16): with them
// the gradients of W, U, Qd, Kd, A and gamma are chunk-parallel products; only the state gradient
//   dVn = A^T dO + Kd dS',      dS = gamma dS' + Qd^T dO - W^T dVn
// is a recurrence, walked in reverse by the backward kernel, which writes dVn and the dS' of every chunk.
//
// Reference counterpart: fla.ops.gated_delta_rule / delta_rule chunk kernels called by
// sequence_modeling/gated_deltanet/gated_deltanet.py:99-116 and deltanet/deltanet.py:127-130.
#include <algorithm>
#include "lsm_delta.cuh"
#include "mma_utils.cuh"
#include "tcgen05_utils.cuh"

namespace lmoe {
namespace dr {

constexpr int DVS = 32;          // value columns per CTA
constexpr int NT = 256;          // threads

// Both walks are chains over the chunks, bound by the latency of a step: two products with a barrier behind each.  Eight warps share the
// products and a ninth brings the tiles, up to two chunks ahead.  The tile kernel writes them with the padded rows they have in shared memory, so
// that a tile is one bulk copy; dense tiles (built with torch ops) and U or dO come 16 bytes at a time.  (As 16-byte copies of all threads the issue alone took 2000
// of a step's 4100 cycles, and 400 as bulk copies of one of the working threads; with the outputs in four warps of their own the others
// waited 600 cycles for the longest of them.)
// 2 x 4096 tokens, 16 heads of 128 (64 chunks, 128 CTAs): forward 98 us, without outputs 83, reverse 96
// (with four warps and everything on the chain: 169, 169 and 150).
template <int DK> struct Cfg {
    static constexpr int LDK = DK + 8;
    static constexpr int LDC = C + 8;
    static constexpr int LDV = DVS + 8;
    static constexpr int SN = DK == 128 ? 4 : 2;    // the state's n-tiles per warp: 16 rows x 32 columns (dk = 128) or x 16 (dk = 64)
    // a stage (bf16 elements): W, Kd: C x LDK; X (U or dO): C x LDV; Qd: C x LDK; A: C x LDC (the last two not where no output is wanted)
    static constexpr int QD = 2 * C * LDK + C * LDV, AQ = QD + C * LDK;
    static constexpr int FULL = AQ + C * LDC;
    // Stages: three where one CTA fills an SM's shared memory anyway, else two, and a second CTA fits.
    static __host__ __device__ constexpr int stages(bool out) { return DK == 128 && out ? 3 : 2; }
    static __host__ __device__ constexpr size_t smem(bool out) {                          // + two states, Vn, O
        return (size_t)(stages(out) * (out ? FULL : QD) + 2 * DK * LDV + (out ? 2 : 1) * C * LDV) * 2;
    }
};

__device__ __forceinline__ void bulk_copy(bf16* dst, const bf16* src, int elements, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(smem_u32(dst)), "l"(src), "r"(elements * 2), "r"(smem_u32(bar)) : "memory");
}
// a tile of C rows in shared memory (row stride LD) by one warp: one bulk copy by lane `which` if memory has the same rows, else 16 bytes per
// copy; rows from `rows` on become zeros
template <int COLS, int LD>
__device__ __forceinline__ void warp_tile(bf16* dst, const bf16* src, long long ld_src, int rows, int lane) {
#pragma unroll 8
    for (int i = lane; i < C * (COLS / 8); i += 32) {
        const int r = i / (COLS / 8), c = (i % (COLS / 8)) * 8;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                     :: "r"(smem_u32(dst + r * LD + c)), "l"(src + (r < rows ? r : 0) * ld_src + c), "r"(r < rows ? 16 : 0) : "memory");
    }
}
template <int COLS, int LD>
__device__ __forceinline__ void produce_tile(bf16* dst, const bf16* src, int ld_src, int lane, int which, uint64_t* bar) {
    if (ld_src != LD) warp_tile<COLS, LD>(dst, src, ld_src, C, lane);
    else if (lane == which) bulk_copy(dst, src, C * LD, bar);
}

struct Pipe {
    uint64_t full[3], empty[3];
    int aborted;
};
template <int STAGES>
__device__ __forceinline__ void init_pipe(Pipe& p) {
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { tc::mbar_init(&p.full[s], 33); tc::mbar_init(&p.empty[s], NT / 32); }
        p.aborted = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}
// The producer warp: the tiles of the steps in order, each as soon as its stage is free.  x: U or dO; rows past x_rows are zeros.
template <int DK, bool FULL, int STAGES, bool REV>
__device__ __forceinline__ void produce(bf16* stage, const Args& a, Pipe& p, const bf16* x, long long xs_t, int x_rows, long long bh) {
    using F = Cfg<DK>;
    constexpr int STAGE = FULL ? F::FULL : F::QD;
    const int lane = threadIdx.x & 31;
    for (int i = 0; i < a.N; ++i) {
        const int n = REV ? a.N - 1 - i : i, s = i % STAGES;
        if (!tc::mbar_wait(&p.empty[s], ((i / STAGES) & 1) ^ 1, &p.aborted, a.err, 0x6c00 | s)) break;
        const long long cn = bh * a.N + n;
        bf16* st = stage + s * STAGE;
        bf16* xt = st + 2 * C * F::LDK;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // what was written and read here comes before the copies
        if (lane == 0) {
            constexpr int TILE = C * F::LDK, TA = C * F::LDC;
            tc::mbar_expect_tx(&p.full[s], ((a.ldw == F::LDK ? (FULL ? 3 : 2) * TILE : 0) + (FULL && a.lda == F::LDC ? TA : 0)) * 2);
        }
        __syncwarp();
        produce_tile<DK, F::LDK>(st, a.W + cn * C * a.ldw, a.ldw, lane, 0, &p.full[s]);
        produce_tile<DK, F::LDK>(st + C * F::LDK, a.Kd + cn * C * a.ldw, a.ldw, lane, 1, &p.full[s]);
        if (FULL) {
            produce_tile<DK, F::LDK>(st + F::QD, a.Qd + cn * C * a.ldw, a.ldw, lane, 2, &p.full[s]);
            produce_tile<C, F::LDC>(st + F::AQ, a.A + cn * C * a.lda, a.lda, lane, 3, &p.full[s]);
        }
        warp_tile<DVS, F::LDV>(xt, x + (long long)n * C * xs_t, xs_t, x_rows - n * C, lane);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" :: "r"(smem_u32(&p.full[s])) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}
// Barrier of the NT threads that multiply; false for all of them if it is for one.
__device__ __forceinline__ bool all_of(bool ok) {
    int r;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 q, %1, 0;\nbarrier.cta.red.and.pred p, 1, %2, q;\nselp.b32 %0, 1, 0, p;\n}"
                 : "=r"(r) : "r"((int)ok), "n"(NT) : "memory");
    return r != 0;
}
__device__ __forceinline__ void sync_workers() { asm volatile("barrier.cta.sync 1, %0;" :: "n"(NT) : "memory"); }

// write a [rows x DVS] bf16 tile held in shared memory (row stride LDV) to global rows of stride `gld`
template <int LDV>
__device__ __forceinline__ void store_rows(const bf16* s, bf16* g, int rows, long long gld) {
    for (int i = threadIdx.x; i < rows * (DVS / 8); i += NT) {
        const int r = i / (DVS / 8), c = (i % (DVS / 8)) * 8;
        *reinterpret_cast<uint4*>(g + (long long)r * gld + c) = *reinterpret_cast<const uint4*>(s + r * LDV + c);
    }
}

// this warp's tile of an fp32 state [dk][dv] (null: zeros), to registers and in bf16 to shared memory; and back
template <int SN>
__device__ __forceinline__ void load_state(float (&S)[SN][4], const float* src, int dv, int col0, bf16* Sb, int ldv, int m0, int n0) {
    const int l = threadIdx.x & 31, r = m0 + (l >> 2);
#pragma unroll
    for (int nt = 0; nt < SN; ++nt) {
        const int c = col0 + n0 + nt * 8 + (l & 3) * 2;
        if (src != nullptr) {
            const float* p = src + (long long)r * dv + c;
            S[nt][0] = p[0]; S[nt][1] = p[1];
            S[nt][2] = p[8 * dv]; S[nt][3] = p[8 * dv + 1];
        } else {
            S[nt][0] = S[nt][1] = S[nt][2] = S[nt][3] = 0.f;
        }
    }
    store_acc_bf16<SN>(S, Sb, ldv, m0, n0);
}
template <int SN>
__device__ __forceinline__ void save_state(const float (&S)[SN][4], float* dst, int dv, int col0, int m0, int n0) {
    const int l = threadIdx.x & 31, r = m0 + (l >> 2);
#pragma unroll
    for (int nt = 0; nt < SN; ++nt) {
        float* p = dst + (long long)r * dv + col0 + n0 + nt * 8 + (l & 3) * 2;
        p[0] = S[nt][0]; p[1] = S[nt][1];
        p[8 * dv] = S[nt][2]; p[8 * dv + 1] = S[nt][3];
    }
}

// OUT: the outputs O are wanted (the forward pass); without: Vn and the entering states only (what the backward pass rebuilds).
// Eight warps multiply: 16 x 16 of Vn = U - W S each, a barrier, their part of the next state and 16 x 16 of O = Qd S + A Vn, which the next
// step does not wait for any longer than for the state (two copies of the state, so that Qd S may still read the old one).
template <int DK, bool OUT>
__global__ void __launch_bounds__(NT + 32, DK == 128 && OUT ? 1 : 2) delta_scan_fwd_kernel(Args a) {
    using F = Cfg<DK>;
    constexpr int STAGES = F::stages(OUT), STAGE = OUT ? F::FULL : F::QD;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ Pipe pipe;
    bf16* stage = reinterpret_cast<bf16*>(smem_raw);
    bf16* Sb = stage + STAGES * STAGE;               // [2][DK][LDV]
    bf16* Vb = Sb + 2 * DK * F::LDV;                 // [C][LDV]  Vn of the chunk
    bf16* Ob = Vb + C * F::LDV;                      // [C][LDV]  output staging
    const int col0 = blockIdx.x * DVS;
    const long long bh = blockIdx.y;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int s_m0 = DK == 128 ? 16 * w : 16 * (w & 3), s_n0 = DK == 128 ? 0 : 16 * (w >> 2);
    const int m0 = 16 * (w & 3), v_n0 = 16 * (w >> 2);
    init_pipe<STAGES>(pipe);
    if (w == NT / 32) {
        produce<DK, OUT, STAGES, false>(stage, a, pipe, a.U + (bh * a.N) * C * a.dv + col0, a.dv, a.N * C, bh);
        return;
    }
    bf16* og = OUT ? a.O + (bh / a.H) * a.os_b + (bh % a.H) * a.os_h + col0 : nullptr;
    float S[F::SN][4];
    load_state<F::SN>(S, a.S0 == nullptr ? nullptr : a.S0 + bh * DK * a.dv, a.dv, col0, Sb, F::LDV, s_m0, s_n0);
    for (int n = 0; n < a.N; ++n) {
        const float gamma = a.gamma[bh * a.N + n];
        const bf16* Wt = stage + (n % STAGES) * STAGE;
        const bf16* Kt = Wt + C * F::LDK;
        const bf16* Ut = Wt + 2 * C * F::LDK;
        const bf16* Qt = Wt + F::QD;
        const bf16* At = Wt + F::AQ;
        const bf16* So = Sb + (n & 1) * DK * F::LDV;
        const bool ok = tc::mbar_wait(&pipe.full[n % STAGES], (n / STAGES) & 1, &pipe.aborted, a.err, 0x6b00 | (n % STAGES));
        if (!all_of(ok)) break;                                    // the state in front of the chunk is complete, Vb free
        if (a.Vn != nullptr) store_rows<F::LDV>(So, a.Sn + ((bh * a.N + n) * DK) * a.dv + col0, DK, a.dv);
        float acc[2][4];
        zero_acc<2>(acc);
        warp_gemm<2, DK, false, true>(acc, Wt, F::LDK, m0, So, F::LDV, v_n0);
        const int r0 = m0 + (l >> 2);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const int c = v_n0 + nt * 8 + (l & 3) * 2;
            const __nv_bfloat162 u0 = *reinterpret_cast<const __nv_bfloat162*>(Ut + r0 * F::LDV + c);
            const __nv_bfloat162 u1 = *reinterpret_cast<const __nv_bfloat162*>(Ut + (r0 + 8) * F::LDV + c);
            acc[nt][0] = __bfloat162float(u0.x) - acc[nt][0]; acc[nt][1] = __bfloat162float(u0.y) - acc[nt][1];
            acc[nt][2] = __bfloat162float(u1.x) - acc[nt][2]; acc[nt][3] = __bfloat162float(u1.y) - acc[nt][3];
        }
        store_acc_bf16<2>(acc, Vb, F::LDV, m0, v_n0);
        sync_workers();                                            // Vb complete
        // S <- gamma S + Kd^T Vn
#pragma unroll
        for (int nt = 0; nt < F::SN; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[nt][e] *= gamma;
        warp_gemm<F::SN, C, true, true>(S, Kt, F::LDK, s_m0, Vb, F::LDV, s_n0);
        store_acc_bf16<F::SN>(S, Sb + ((n + 1) & 1) * DK * F::LDV, F::LDV, s_m0, s_n0);
        if (a.Vn != nullptr) store_rows<F::LDV>(Vb, a.Vn + ((bh * a.N + n) * C) * a.dv + col0, C, a.dv);
        if (OUT) {
            zero_acc<2>(acc);
            warp_gemm<2, DK, false, true>(acc, Qt, F::LDK, m0, So, F::LDV, v_n0);
            for (int k0 = 0; k0 <= m0; k0 += 16) warp_gemm<2, 16, false, true>(acc, At + k0, F::LDC, m0, Vb + k0 * F::LDV, F::LDV, v_n0);
            store_acc_bf16<2>(acc, Ob, F::LDV, m0, v_n0);
            __syncwarp();
            const int r = m0 + (l >> 1), c = v_n0 + (l & 1) * 8, t = n * C + r;       // the warp's own 16 x 16
            if (t < a.T) *reinterpret_cast<uint4*>(og + (long long)t * a.os_t + c) = *reinterpret_cast<const uint4*>(Ob + r * F::LDV + c);
        }
        __syncwarp();
        if (l == 0) tc::mbar_arrive(&pipe.empty[n % STAGES]);
    }
    save_state<F::SN>(S, a.Sfinal + bh * DK * a.dv, a.dv, col0, s_m0, s_n0);
}

// Reverse walk: dS' enters from the right (gradient of the state leaving the chunk).
template <int DK>
__global__ void __launch_bounds__(NT + 32, 1) delta_scan_bwd_kernel(Args a) {
    using F = Cfg<DK>;
    constexpr int STAGES = F::stages(true), STAGE = F::FULL;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ Pipe pipe;
    bf16* stage = reinterpret_cast<bf16*>(smem_raw);
    bf16* Sb = stage + STAGES * STAGE;                    // [DK][LDV]  bf16 copy of dS'
    bf16* Vb = Sb + DK * F::LDV;                     // [C][LDV]   dVn of the chunk
    const int col0 = blockIdx.x * DVS;
    const long long bh = blockIdx.y;
    const int w = threadIdx.x >> 5;
    const int s_m0 = DK == 128 ? 16 * w : 16 * (w & 3), s_n0 = DK == 128 ? 0 : 16 * (w >> 2);
    const int m0 = 16 * (w & 3), v_n0 = 16 * (w >> 2);
    init_pipe<STAGES>(pipe);
    if (w == NT / 32) {
        produce<DK, true, STAGES, true>(stage, a, pipe, a.dO + (bh / a.H) * a.gs_b + (bh % a.H) * a.gs_h + col0, a.gs_t, a.T, bh);
        return;
    }
    float S[F::SN][4];
    load_state<F::SN>(S, a.dSfinal == nullptr ? nullptr : a.dSfinal + bh * DK * a.dv, a.dv, col0, Sb, F::LDV, s_m0, s_n0);
    for (int i = 0; i < a.N; ++i) {
        const int n = a.N - 1 - i;
        const float gamma = a.gamma[bh * a.N + n];
        const bf16* Wt = stage + (i % STAGES) * STAGE;
        const bf16* Kt = Wt + C * F::LDK;
        const bf16* Gt = Wt + 2 * C * F::LDK;         // dO slice
        const bf16* Qt = Wt + F::QD;
        const bf16* At = Wt + F::AQ;
        const bool ok = tc::mbar_wait(&pipe.full[i % STAGES], (i / STAGES) & 1, &pipe.aborted, a.err, 0x6b10 | (i % STAGES));
        if (!all_of(ok)) break;                                    // the gradient behind the chunk is complete, Vb free
        store_rows<F::LDV>(Sb, a.dSn + ((bh * a.N + n) * DK) * a.dv + col0, DK, a.dv);
        // dVn = A^T dO + Kd dS'
        float acc[2][4];
        zero_acc<2>(acc);
        for (int k0 = m0; k0 < C; k0 += 16) warp_gemm<2, 16, true, true>(acc, At + k0 * F::LDC, F::LDC, m0, Gt + k0 * F::LDV, F::LDV, v_n0);
        warp_gemm<2, DK, false, true>(acc, Kt, F::LDK, m0, Sb, F::LDV, v_n0);
        store_acc_bf16<2>(acc, Vb, F::LDV, m0, v_n0);
        // dS = gamma dS' + Qd^T dO - W^T dVn; what does not wait for dVn first
#pragma unroll
        for (int nt = 0; nt < F::SN; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[nt][e] *= gamma;
        warp_gemm<F::SN, C, true, true>(S, Qt, F::LDK, s_m0, Gt, F::LDV, s_n0);
        sync_workers();                                            // Vb complete; reads of Sb done
        float t[F::SN][4];
        zero_acc<F::SN>(t);
        warp_gemm<F::SN, C, true, true>(t, Wt, F::LDK, s_m0, Vb, F::LDV, s_n0);
#pragma unroll
        for (int nt = 0; nt < F::SN; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[nt][e] -= t[nt][e];
        store_acc_bf16<F::SN>(S, Sb, F::LDV, s_m0, s_n0);
        store_rows<F::LDV>(Vb, a.dVn + ((bh * a.N + n) * C) * a.dv + col0, C, a.dv);
        __syncwarp();
        if ((threadIdx.x & 31) == 0) tc::mbar_arrive(&pipe.empty[i % STAGES]);
    }
    save_state<F::SN>(S, a.dS0 + bh * DK * a.dv, a.dv, col0, s_m0, s_n0);
}


// ---------------------------------------------------------------------------------------------------------------
// Chunk-parallel construction of the tiles (forward): one CTA per (batch, head, chunk).
//   b_i = inclusive cumulative log decay inside the chunk,  Gamma_ij = e^{b_i - b_j}
//   A   = strictly-lower(diag(beta) (K K^T . Gamma)),   T = (I + A)^{-1}
//   W = T (beta e^{b} K),  U = T (beta V),  Aqk = scale tril((Q K^T) . Gamma),  Qd = scale e^{b} Q,  Kd = e^{b_C - b} K
// The inverse is taken in fp32 by halves: the four 16 x 16 diagonal blocks by substitution, one column per thread, then
// [[T0, 0], [-T1 (A10 T0), T1]] twice, with all threads on the small products.  A substitution over the whole chunk, one
// column per thread, is a chain of 2016 multiply-adds on two warps; it was most of this kernel's time.
// What bounds the kernel is the traffic of its tiles (120 KB in and out per chunk at D = 128); three CTAs of eight warps per SM
// overlap one chunk's loads with another's products.  2 x 4096 tokens, 16 heads of 128: 110 -> 84 us (floor 37).
// ---------------------------------------------------------------------------------------------------------------
struct PrepArgs {
    const bf16 *q, *k, *v;             // [B,T,H,D] with the strides below (elements)
    long long qs_b, qs_t, qs_h, ks_b, ks_t, ks_h, vs_b, vs_t, vs_h;
    const float* beta;                 // [B,T,H]
    const float* g;                    // [B,T,H] log decay, or null
    bf16 *W, *U, *Qd, *Kd, *A;         // outputs: U [BH, N, C, D]; W, Qd, Kd with rows of D + 8, A with rows of C + 8 (as the scans stage them)
    float* gamma;                      // [BH, N]
    int B, T, H, N;
    float scale;
    bf16* Tinv;                        // [BH, N, C, C] the inverse, or null
};

constexpr int NTP = 256;               // threads of the chunk-parallel tile kernel
constexpr int LDF = C + 4;             // row stride of the fp32 matrix (16-byte rows)

// X = A B for fp32 matrices of N x N (N = 16 or 32) inside arrays of row stride LDF; NTP threads, `sign` on the result.
// Four neighbouring columns per thread; `count` independent products, `step` elements apart.
template <int N>
__device__ __forceinline__ void small_product(const float* A, const float* B, float* X, float sign, int count, int step) {
    constexpr int PER = N * N / 4;                            // threads of one product
    for (int i = threadIdx.x; i < PER * count; i += NTP) {
        const int m = i / PER, r = (i % PER) / (N / 4), c = (i % (N / 4)) * 4;
        const float *a = A + m * step + r * LDF, *b = B + m * step + c;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < N; k += 4) {
            const float4 av = *reinterpret_cast<const float4*>(a + k);
            const float* ap = reinterpret_cast<const float*>(&av);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float4 bv = *reinterpret_cast<const float4*>(b + (k + e) * LDF);
                x.x += ap[e] * bv.x; x.y += ap[e] * bv.y; x.z += ap[e] * bv.z; x.w += ap[e] * bv.w;
            }
        }
        *reinterpret_cast<float4*>(X + m * step + r * LDF + c) = make_float4(sign * x.x, sign * x.y, sign * x.z, sign * x.w);
    }
}

// F holds a strictly lower triangular A (zeros elsewhere); on return its lower blocks hold T = (I + A)^{-1}.  The blocks above the
// diagonal are scratch.  Called by all NTP threads with A visible; ends with a barrier.
__device__ __forceinline__ void unit_lower_inverse(float* F) {
    if (threadIdx.x < C) {
        const int blk = threadIdx.x >> 4, c = threadIdx.x & 15;
        float* D = F + (blk * 16) * LDF + blk * 16;
        float t[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float acc = (i == c) ? 1.f : 0.f;
#pragma unroll
            for (int j = 0; j < i; ++j) acc -= D[i * LDF + j] * t[j];
            t[i] = acc;
        }
        __syncwarp();                                        // both blocks of this warp have been read
#pragma unroll
        for (int i = 0; i < 16; ++i) D[i * LDF + c] = t[i];
    }
    __syncthreads();
    constexpr int S2 = 32 * LDF + 32;                        // from one half of the diagonal to the other
    // the (1,0) and (3,2) blocks
    small_product<16>(F + 16 * LDF, F, F + 16, 1.f, 2, S2);                       // A10 T0 -> above the diagonal
    __syncthreads();
    small_product<16>(F + 16 * LDF + 16, F + 16, F + 16 * LDF, -1.f, 2, S2);      // -T1 (A10 T0)
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * 16 * 4; i += NTP) {                          // the scratch blocks are zeros of T
        const int m = i >> 6, r = (i >> 2) & 15, c = (i & 3) * 4;
        *reinterpret_cast<float4*>(F + m * S2 + r * LDF + 16 + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    // the lower left quarter
    small_product<32>(F + 32 * LDF, F, F + 32, 1.f, 1, 0);
    __syncthreads();
    small_product<32>(F + 32 * LDF + 32, F + 32, F + 32 * LDF, -1.f, 1, 0);
    __syncthreads();
}

template <int D>
__global__ void __launch_bounds__(NTP, 3) delta_prep_fwd_kernel(PrepArgs a) {
    constexpr int LD = D + 8, LDC = C + 8, NH = D / 16;      // NH: n-tiles of a warp's half of D columns
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16* Ks = reinterpret_cast<bf16*>(smem_raw);            // [C][LD]
    bf16* Vs = Ks + C * LD;                                  // [C][LD]  V, then beta V
    bf16* Qs = Vs + C * LD;                                  // [C][LD]  Q, then beta e^b K
    float* F = reinterpret_cast<float*>(Qs + C * LD);        // [C][LDF] strictly lower A, then T
    bf16* Tb = reinterpret_cast<bf16*>(F);                   // [C][LDC] T in bf16 (over F)
    float* bcum = F + C * LDF;                               // [C]
    float* bet = bcum + C;                                   // [C]
    const int n = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int m0 = 16 * (w & 3), half = w >> 2;
    const int t0 = n * C;
    const int valid = min(C, a.T - t0);
    const long long cn = (long long)bh * a.N + n;

    load_tile_async<C, D, LD>(Ks, a.k + b * a.ks_b + h * a.ks_h + (long long)t0 * a.ks_t, a.ks_t, valid);
    load_tile_async<C, D, LD>(Qs, a.q + b * a.qs_b + h * a.qs_h + (long long)t0 * a.qs_t, a.qs_t, valid);
    cp_async_commit();
    load_tile_async<C, D, LD>(Vs, a.v + b * a.vs_b + h * a.vs_h + (long long)t0 * a.vs_t, a.vs_t, valid);
    cp_async_commit();
    if (w == 0) {                                            // decay table: two tokens per lane, warp scan
        const int i0 = 2 * l, i1 = 2 * l + 1;
        float g0 = 0.f, g1 = 0.f, be0 = 0.f, be1 = 0.f;
        if (i0 < valid) {
            const long long o = ((long long)b * a.T + t0 + i0) * a.H + h;
            be0 = a.beta[o];
            if (a.g != nullptr) g0 = a.g[o];
        }
        if (i1 < valid) {
            const long long o = ((long long)b * a.T + t0 + i1) * a.H + h;
            be1 = a.beta[o];
            if (a.g != nullptr) g1 = a.g[o];
        }
        float s = g0 + g1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float x = __shfl_up_sync(0xffffffffu, s, o);
            if (l >= o) s += x;
        }
        bcum[i1] = s;
        bcum[i0] = s - g1;
        bet[i0] = be0;
        bet[i1] = be1;
    }
    cp_async_wait<1>();
    __syncthreads();
    const float btot = bcum[C - 1];
    // ---- K K^T -> A (fp32, strictly lower) and Q K^T -> Aqk (bf16, to global); warp: 16 rows x 32 columns, tiles above the
    //      diagonal are only zeroed
    {
        const int nc = 32 * half;
        float kk[4][4], qk[4][4];
        zero_acc<4>(kk);
        zero_acc<4>(qk);
        if (nc <= m0) {
            warp_gemm<4, D, false, false>(kk, Ks, LD, m0, Ks, LD, nc);
            warp_gemm<4, D, false, false>(qk, Qs, LD, m0, Ks, LD, nc);
        }
        bf16* Ag = a.A + cn * C * LDC;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int i = m0 + (l >> 2) + 8 * hh;
                const int j = nc + nt * 8 + (l & 3) * 2;
                const float bi = bcum[i], be = bet[i];
                const float d0 = __expf(bi - bcum[j]), d1 = __expf(bi - bcum[j + 1]);
                *reinterpret_cast<float2*>(F + i * LDF + j) = make_float2(i > j ? be * d0 * kk[nt][2 * hh] : 0.f,
                                                                          i > j + 1 ? be * d1 * kk[nt][2 * hh + 1] : 0.f);
                const float a0 = i >= j ? a.scale * d0 * qk[nt][2 * hh] : 0.f;
                const float a1 = i >= j + 1 ? a.scale * d1 * qk[nt][2 * hh + 1] : 0.f;
                *reinterpret_cast<__nv_bfloat162*>(Ag + i * LDC + j) = __floats2bfloat162_rn(a0, a1);
            }
    }
    cp_async_wait<0>();
    __syncthreads();
    // ---- the elementwise tiles: Qd and Kd to global, beta e^b K over Q, beta V in place
    for (int x = threadIdx.x; x < C * (D / 8); x += NTP) {
        const int i = x / (D / 8), c = (x % (D / 8)) * 8;
        const float bi = bcum[i], be = bet[i];
        const float fk = be * __expf(bi), fq = a.scale * __expf(bi), fd = __expf(btot - bi);
        Vec<bf16> kx, vx, qx, o1, o2, o3, o4;
        kx.load(Ks + i * LD + c);
        vx.load(Vs + i * LD + c);
        qx.load(Qs + i * LD + c);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            o1.set(e, kx.get(e) * fk);
            o2.set(e, vx.get(e) * be);
            o3.set(e, qx.get(e) * fq);
            o4.set(e, kx.get(e) * fd);
        }
        o1.store(Qs + i * LD + c);
        o2.store(Vs + i * LD + c);
        o3.store(a.Qd + (cn * C + i) * LD + c);
        o4.store(a.Kd + (cn * C + i) * LD + c);
    }
    if (threadIdx.x == 0) a.gamma[cn] = __expf(btot);
    unit_lower_inverse(F);
    {                                                        // T to bf16: read everything, then write over it
        const int i = threadIdx.x >> 2, c = (threadIdx.x & 3) * 16;
        float t[16];
#pragma unroll
        for (int e = 0; e < 16; e += 4) *reinterpret_cast<float4*>(t + e) = *reinterpret_cast<const float4*>(F + i * LDF + c + e);
        __syncthreads();
        Vec<bf16> lo, hi;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            lo.set(e, c + e <= i ? t[e] : 0.f);              // above the diagonal is scratch
            hi.set(e, c + 8 + e <= i ? t[8 + e] : 0.f);
        }
        lo.store(Tb + i * LDC + c);
        hi.store(Tb + i * LDC + c + 8);
        if (a.Tinv != nullptr) {
            lo.store(a.Tinv + (cn * C + i) * C + c);
            hi.store(a.Tinv + (cn * C + i) * C + c + 8);
        }
    }
    __syncthreads();
    // ---- W = T Kb, U = T (beta V): warp -> 16 rows, half of the columns; T is lower triangular
#pragma unroll
    for (int which = 0; which < 2; ++which) {
        const bf16* X = which == 0 ? Qs : Vs;
        const int ld = which == 0 ? LD : D;
        bf16* Y = (which == 0 ? a.W : a.U) + cn * C * ld + half * (D / 2);
        float acc[NH][4];
        zero_acc<NH>(acc);
        for (int k0 = 0; k0 <= m0; k0 += 16) warp_gemm<NH, 16, false, true>(acc, Tb + k0, LDC, m0, X + k0 * LD, LD, half * (D / 2));
        const int r = m0 + (l >> 2), cc = (l & 3) * 2;
#pragma unroll
        for (int nt = 0; nt < NH; ++nt) {
            *reinterpret_cast<__nv_bfloat162*>(Y + r * ld + cc + nt * 8) = __floats2bfloat162_rn(acc[nt][0], acc[nt][1]);
            *reinterpret_cast<__nv_bfloat162*>(Y + (r + 8) * ld + cc + nt * 8) = __floats2bfloat162_rn(acc[nt][2], acc[nt][3]);
        }
    }
}


// ---------------------------------------------------------------------------------------------------------------
// Chunk-parallel backward of everything that is not the state recurrence: one CTA per (batch, head, chunk).
// Inputs: q, k, v, beta, g (to rebuild the tiles), the entering state S_n and the gradient dS'_n of the leaving state,
// Vn, dVn (= dU) and dO of the chunk (written by the two scan kernels), T from the tile kernel.  The gradient of the chunk's total
// decay, dgamma_n = <dS'_n, S_n> (gated case), is formed here too.
//
//   through the scan equations      dW = -dVn S^T,  dQd = dO S^T,  dKd = Vn dS'^T,  dAqk = tril(dO Vn^T)
//   through W = T Kb, U = T Vb      dKb = T^T dW,  dVb = T^T dU,  dT = dW Kb^T + dU Vb^T,  dA = -strict_lower(T^T dT T^T)
//   through the tiles               dq = s e^b dQd + P K                         P = s Gamma . dAqk
//                                   dk = e^{b_C-b} dKd + P^T Q + beta e^b dKb + M K + M^T K          M = beta_i Gamma . dA
//                                   dv = beta dVb
//                                   dbeta_i = e^{b_i} <dKb_i, k_i> + <dVb_i, v_i> + sum_j dA_ij Gamma_ij (k_i.k_j)
//                                   db_i (gradient of the cumulative log decay) from every e^{b}: rows minus columns of
//                                   dAqk . Aqk and dA . A, +<dQd_i, Qd_i>, -<dKd_j, Kd_j> (and their sum on b_C),
//                                   +beta_i e^{b_i} <dKb_i, k_i>, + dgamma gamma on b_C;   dg_s = sum_{i >= s} db_i
// The products are mma.sync tiles on bf16 copies in shared memory with fp32 accumulation; dk accumulates in registers
// across the phases, every other output is finished inside one phase.
// ---------------------------------------------------------------------------------------------------------------
struct PrepBwdArgs {
    const bf16 *q, *k, *v;
    long long qs_b, qs_t, qs_h, ks_b, ks_t, ks_h, vs_b, vs_t, vs_h;
    const float* beta;
    const float* g;                    // or null
    const bf16 *Sn, *dSn;              // [BH, N, D, D]
    const bf16 *Vn, *dVn;              // [BH, N, C, D]
    const bf16* dO;                    // strides below (elements; batch, token, head)
    long long gs_b, gs_t, gs_h;
    const bf16* Tinv;                  // [BH, N, C, C] from the tile kernel
    bf16 *dq, *dk, *dv;                // contiguous [B, T, H, D]
    float *dbeta, *dg;                 // [B, T, H]
    int B, T, H, N;
    float scale;
};

// lo / hi += sum over the thread's columns of acc[row][col] * tile[row][col] for its two rows (r, r + 8)
template <int NTL>
__device__ __forceinline__ void row_dot(const float (&acc)[NTL][4], const bf16* tile, int ld, int m0, float& lo, float& hi) {
    const int l = threadIdx.x & 31;
    const int r = m0 + (l >> 2), c = (l & 3) * 2;
#pragma unroll
    for (int nt = 0; nt < NTL; ++nt) {
        const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(tile + r * ld + c + nt * 8);
        const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(tile + (r + 8) * ld + c + nt * 8);
        lo += acc[nt][0] * __bfloat162float(a.x) + acc[nt][1] * __bfloat162float(a.y);
        hi += acc[nt][2] * __bfloat162float(b.x) + acc[nt][3] * __bfloat162float(b.y);
    }
}

template <int NTL>
__device__ __forceinline__ void scale_rows(float (&acc)[NTL][4], float lo, float hi) {
#pragma unroll
    for (int nt = 0; nt < NTL; ++nt) { acc[nt][0] *= lo; acc[nt][1] *= lo; acc[nt][2] *= hi; acc[nt][3] *= hi; }
}

// write a warp's [16 x 8 NTL] accumulator rows to global rows (bf16), rows >= valid skipped
template <int NTL>
__device__ __forceinline__ void store_rows_global(const float (&acc)[NTL][4], bf16* g, long long row_stride, int m0, int valid) {
    const int l = threadIdx.x & 31;
    const int r = m0 + (l >> 2), c = (l & 3) * 2;
#pragma unroll
    for (int nt = 0; nt < NTL; ++nt) {
        if (r < valid) *reinterpret_cast<__nv_bfloat162*>(g + r * row_stride + c + nt * 8) = __floats2bfloat162_rn(acc[nt][0], acc[nt][1]);
        if (r + 8 < valid) *reinterpret_cast<__nv_bfloat162*>(g + (r + 8) * row_stride + c + nt * 8) = __floats2bfloat162_rn(acc[nt][2], acc[nt][3]);
    }
}

// 512 threads: warp w works on rows 16 (w & 3) .. +15 and on column quarter (w >> 2) of every product (the tiles allow one CTA
// per SM only, so sixteen warps hide each other's shared-memory and tensor-pipe latencies).  Of the C x C products only
// the blocks on and below the diagonal are computed or read.  Sums over rows and columns stay in registers until the end: a
// shared atomic per element and the substitution for T were two thirds of this kernel's time, T now comes from the tile kernel
// that has just run.  Tiles arrive in the order they are needed.  Bound by shared-memory reads of the fragments (about 3 cycles per
// 2 cycles of tensor pipe); a CTA goes on to the next chunk, whose tiles load while it works on this one.  2 x 4096 tokens, 16 heads of 128: 580 -> 224 us,
// and with the loads ahead 213.
constexpr int NTB = 512;

template <int D>
__global__ void __launch_bounds__(NTB, 1) delta_prep_bwd_kernel(PrepBwdArgs a) {
    constexpr int LD = D + 8, LDC = C + 8, NQ = D / 32, QD = D / 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16* K2 = reinterpret_cast<bf16*>(smem_raw);            // [2][C][LD] of this chunk and the next
    bf16* Qs = K2 + 2 * C * LD;                              // [C][LD]
    bf16* Vs = Qs + C * LD;                                  // [C][LD]
    bf16* Gs = Vs + C * LD;                                  // [C][LD]  dO, later dW
    bf16* Ns = Gs + C * LD;                                  // [C][LD]  Vn
    bf16* Us = Ns + C * LD;                                  // [C][LD]  dVn = dU
    bf16* Sb = Us + C * LD;                                  // [D][LD]  S_n
    bf16* Db = Sb + D * LD;                                  // [D][LD]  dS'_n
    bf16* Tb = Db + D * LD;                                  // [C][LDC] T
    bf16* Ps = Tb + C * LDC;                                 // [C][LDC] P, later M
    bf16* X1 = Ps + C * LDC;                                 // [C][LDC] dT
    bf16* X2 = X1 + C * LDC;                                 // [C][LDC] T^T dT
    float* bcum = reinterpret_cast<float*>(X2 + C * LDC);    // [C]
    float* bet = bcum + C;                                   // [C]
    float* rdb = bet + C;                                    // [4][C] row sums of the decay gradient, by column quarter
    float* rbe = rdb + 4 * C;                                // [4][C] ... of the gradient of beta
    float* cdb = rbe + 4 * C;                                // [4][C] column sums, by row block
    float* tot = cdb + 4 * C;                                // [2][16] per warp: <dS'_n, S_n>, sum of <dKd_j, Kd_j>
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int qd = w >> 2, m0 = 16 * (w & 3), r0 = m0 + (l >> 2), c0 = (l & 3) * 2;
    const bool gated = a.g != nullptr;
    const int nd = qd * QD;                                  // first column of this warp's quarter of a D-wide product
    const int nc = qd * 16;                                  // ... of a C-wide product
    const bool lower = nc <= m0;                             // does the warp's C x C block touch the lower triangle?

    // A CTA goes through its chunks, and the next chunk's tiles come in as soon as this one's are done with, in four groups: (K, Q), (Vn, S_n, dS'_n),
    // (dO, dVn, V), T.
    const int total = a.N * a.B * a.H;
    struct At { int b, h, t0, valid; long long cn; };
    auto place = [&](int idx) -> At {
        const int bh = idx / a.N, n = idx % a.N;
        return {bh / a.H, bh % a.H, n * C, min(C, a.T - n * C), (long long)idx};
    };
    auto load_kq = [&](const At& x, bf16* Kd) {
        load_tile_async<C, D, LD>(Kd, a.k + x.b * a.ks_b + x.h * a.ks_h + (long long)x.t0 * a.ks_t, a.ks_t, x.valid);
        load_tile_async<C, D, LD>(Qs, a.q + x.b * a.qs_b + x.h * a.qs_h + (long long)x.t0 * a.qs_t, a.qs_t, x.valid);
    };
    auto load_states = [&](const At& x) {
        load_tile_async<C, D, LD>(Ns, a.Vn + x.cn * C * D, D, C);
        load_tile_async<D, D, LD>(Sb, a.Sn + x.cn * D * D, D, D);
        load_tile_async<D, D, LD>(Db, a.dSn + x.cn * D * D, D, D);
    };
    auto load_grads = [&](const At& x) {
        load_tile_async<C, D, LD>(Gs, a.dO + x.b * a.gs_b + x.h * a.gs_h + (long long)x.t0 * a.gs_t, a.gs_t, x.valid);
        load_tile_async<C, D, LD>(Us, a.dVn + x.cn * C * D, D, C);
        load_tile_async<C, D, LD>(Vs, a.v + x.b * a.vs_b + x.h * a.vs_h + (long long)x.t0 * a.vs_t, a.vs_t, x.valid);
    };
    auto load_t = [&](const At& x) { load_tile_async<C, C, LDC>(Tb, a.Tinv + x.cn * C * C, C, C); };
    const int i0 = 2 * l, i1 = 2 * l + 1;
    float g0 = 0.f, g1 = 0.f, be0 = 0.f, be1 = 0.f;                    // warp 0: decays and betas of two tokens, a chunk ahead
    auto load_scalars = [&](const At& x) {
        const long long o = ((long long)x.b * a.T + x.t0 + i0) * a.H + x.h;
        const bool v0 = i0 < x.valid, v1 = i1 < x.valid;
        be0 = v0 ? a.beta[o] : 0.f; be1 = v1 ? a.beta[o + a.H] : 0.f;
        g0 = v0 && a.g != nullptr ? a.g[o] : 0.f; g1 = v1 && a.g != nullptr ? a.g[o + a.H] : 0.f;
    };
    {
        const At x = place(blockIdx.x);
        load_kq(x, K2); cp_async_commit();
        load_states(x); cp_async_commit();
        load_grads(x); cp_async_commit();
        load_t(x); cp_async_commit();
        if (w == 0) load_scalars(x);
    }
    for (int idx = blockIdx.x, turn = 0; idx < total; idx += gridDim.x, turn ^= 1) {
    const At c = place(idx);
    const int b = c.b, h = c.h, t0 = c.t0, valid = c.valid;
    const bool more = idx + (int)gridDim.x < total;
    const At nx = place(more ? idx + (int)gridDim.x : idx);
    bf16 *Ks = K2 + turn * C * LD, *Kn = K2 + (turn ^ 1) * C * LD;
    if (w == 0) {
        float s = g0 + g1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const float x = __shfl_up_sync(0xffffffffu, s, o); if (l >= o) s += x; }
        bcum[i1] = s; bcum[i0] = s - g1; bet[i0] = be0; bet[i1] = be1;
        if (more) load_scalars(nx);
    }
    cp_async_wait<3>();
    __syncthreads();
    const float btot = bcum[C - 1];
    const float b_lo = bcum[r0], b_hi = bcum[r0 + 8], be_lo = bet[r0], be_hi = bet[r0 + 8];
    // this thread's sums: rows r0 and r0 + 8 over its columns, its four columns over its rows
    float db_lo = 0.f, db_hi = 0.f, dbe_lo = 0.f, dbe_hi = 0.f, kd = 0.f, col[4] = {0.f, 0.f, 0.f, 0.f};

    // ---- (1) K K^T and Q K^T, kept in registers ------------------------------------------------------------------
    float kk[2][4], qk[2][4], gam[2][4];
    zero_acc<2>(kk);
    zero_acc<2>(qk);
    if (lower) {
        warp_gemm<2, D, false, false>(kk, Ks, LD, m0, Ks, LD, nc);
        warp_gemm<2, D, false, false>(qk, Qs, LD, m0, Ks, LD, nc);
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = r0 + 8 * (e >> 1), j = nc + nt * 8 + c0 + (e & 1);
            gam[nt][e] = i >= j ? __expf(((e >> 1) ? b_hi : b_lo) - bcum[j]) : 0.f;             // Gamma_ij
        }
    cp_async_wait<1>();
    __syncthreads();
    // ---- (2) dAqk = tril(dO Vn^T); P = scale Gamma . dAqk; decay gradients of Aqk ------------------------------------
    if (lower) {
        float da[2][4];
        zero_acc<2>(da);
        warp_gemm<2, D, false, false>(da, Gs, LD, m0, Ns, LD, nc);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            float pv[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                pv[e] = a.scale * gam[nt][e] * da[nt][e];             // P_ij
                const float t_ = pv[e] * qk[nt][e];                   // dAqk_ij Aqk_ij
                if (e >> 1) db_hi += t_; else db_lo += t_;
                col[2 * nt + (e & 1)] -= t_;
            }
            *reinterpret_cast<__nv_bfloat162*>(Ps + r0 * LDC + nc + nt * 8 + c0) = __floats2bfloat162_rn(pv[0], pv[1]);
            *reinterpret_cast<__nv_bfloat162*>(Ps + (r0 + 8) * LDC + nc + nt * 8 + c0) = __floats2bfloat162_rn(pv[2], pv[3]);
        }
    }
    __syncthreads();                                                   // Ps
    // ---- (3) dq = scale e^b (dO S^T) + P K; its decay gradient <dQd_i, Qd_i>; dk += P^T Q -----------------------------
    float acc_dk[NQ][4], acc[NQ][4];
    zero_acc<NQ>(acc_dk);
    zero_acc<NQ>(acc);
    warp_gemm<NQ, D, false, false>(acc, Gs, LD, m0, Sb, LD, nd);      // dQd = dO S^T  (S stored [dk][dv] = [n][k])
    scale_rows<NQ>(acc, a.scale * __expf(b_lo), a.scale * __expf(b_hi));
    row_dot<NQ>(acc, Qs + nd, LD, m0, db_lo, db_hi);                  // <dQd_i, Qd_i> over this thread's columns
    for (int k0 = 0; k0 <= m0; k0 += 16) warp_gemm<NQ, 16, false, true>(acc, Ps + k0, LDC, m0, Ks + k0 * LD, LD, nd);
    store_rows_global<NQ>(acc, a.dq + (((long long)b * a.T + t0) * a.H + h) * D + nd, (long long)a.H * D, m0, valid);
    for (int k0 = m0; k0 < C; k0 += 16) warp_gemm<NQ, 16, true, true>(acc_dk, Ps + k0 * LDC, LDC, m0, Qs + k0 * LD, LD, nd);
    // ---- (4) dW = -dVn S^T -> shared, in dO's buffer once every warp is done with dO ---------------------------------
    zero_acc<NQ>(acc);
    warp_gemm<NQ, D, false, false>(acc, Us, LD, m0, Sb, LD, nd);
    scale_rows<NQ>(acc, -1.f, -1.f);
    cp_async_wait<0>();
    __syncthreads();                                                   // dO and Q are free; T is here
    if (more) load_kq(nx, Kn);
    cp_async_commit();
    store_acc_bf16<NQ>(acc, Gs, LD, m0, nd);                           // Gs now holds dW
    // ---- (5) dgamma = <dS'_n, S_n>; dKd = Vn dS'^T -------------------------------------------------------------------
    float dgam = 0.f;
    if (gated) {
        for (int i = threadIdx.x; i < D * D / 8; i += NTB) {
            const int o = (i / (D / 8)) * LD + (i % (D / 8)) * 8;
            const uint4 x4 = *reinterpret_cast<const uint4*>(Sb + o), y4 = *reinterpret_cast<const uint4*>(Db + o);
            const __nv_bfloat162 *x = reinterpret_cast<const __nv_bfloat162*>(&x4), *y = reinterpret_cast<const __nv_bfloat162*>(&y4);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 fx = __bfloat1622float2(x[e]), fy = __bfloat1622float2(y[e]);
                dgam += fx.x * fy.x + fx.y * fy.y;
            }
        }
    }
    zero_acc<NQ>(acc);
    warp_gemm<NQ, D, false, false>(acc, Ns, LD, m0, Db, LD, nd);      // dKd_j = Vn_j dS'^T
    scale_rows<NQ>(acc, __expf(btot - b_lo), __expf(btot - b_hi));
    {
        float d_lo = 0.f, d_hi = 0.f;
        row_dot<NQ>(acc, Ks + nd, LD, m0, d_lo, d_hi);                // <dKd_j, Kd_j>
        db_lo -= d_lo; db_hi -= d_hi;
        kd = d_lo + d_hi;
    }
#pragma unroll
    for (int nt = 0; nt < NQ; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc_dk[nt][e] += acc[nt][e];
    // ---- (6) dVb = T^T dU: dv, dbeta --------------------------------------------------------------------------------
    zero_acc<NQ>(acc);
    for (int k0 = m0; k0 < C; k0 += 16) warp_gemm<NQ, 16, true, true>(acc, Tb + k0 * LDC, LDC, m0, Us + k0 * LD, LD, nd);
    row_dot<NQ>(acc, Vs + nd, LD, m0, dbe_lo, dbe_hi);                // <dVb_i, v_i>
    scale_rows<NQ>(acc, be_lo, be_hi);
    store_rows_global<NQ>(acc, a.dv + (((long long)b * a.T + t0) * a.H + h) * D + nd, (long long)a.H * D, m0, valid);
    __syncthreads();                                                   // dW complete; Vn, S_n and dS'_n are free
    if (more) load_states(nx);
    cp_async_commit();
    // ---- (7) dKb = T^T dW: its part of dk, dbeta and db -------------------------------------------------------------
    zero_acc<NQ>(acc);
    for (int k0 = m0; k0 < C; k0 += 16) warp_gemm<NQ, 16, true, true>(acc, Tb + k0 * LDC, LDC, m0, Gs + k0 * LD, LD, nd);
    {
        float d_lo = 0.f, d_hi = 0.f;
        row_dot<NQ>(acc, Ks + nd, LD, m0, d_lo, d_hi);                // <dKb_i, k_i>
        const float e_lo = __expf(b_lo), e_hi = __expf(b_hi), f_lo = be_lo * e_lo, f_hi = be_hi * e_hi;
        dbe_lo += e_lo * d_lo; dbe_hi += e_hi * d_hi;
        db_lo += f_lo * d_lo; db_hi += f_hi * d_hi;
#pragma unroll
        for (int nt = 0; nt < NQ; ++nt) {
            acc_dk[nt][0] += f_lo * acc[nt][0]; acc_dk[nt][1] += f_lo * acc[nt][1];
            acc_dk[nt][2] += f_hi * acc[nt][2]; acc_dk[nt][3] += f_hi * acc[nt][3];
        }
    }
    // ---- (8) dT_ij = beta_j e^{b_j} (dW_i . k_j) + beta_j (dU_i . v_j) -> X1;  X2 = T^T dT;  dA = -(X2 T^T), strictly lower
    if (lower) {
        float x[2][4], y[2][4];
        zero_acc<2>(x);
        zero_acc<2>(y);
        warp_gemm<2, D, false, false>(x, Gs, LD, m0, Ks, LD, nc);
        warp_gemm<2, D, false, false>(y, Us, LD, m0, Vs, LD, nc);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int j = nc + nt * 8 + c0 + (e & 1);
                x[nt][e] = bet[j] * (__expf(bcum[j]) * x[nt][e] + y[nt][e]);
            }
        store_acc_bf16<2>(x, X1, LDC, m0, nc);
    }
    __syncthreads();
    if (more) load_grads(nx);                                          // dW, dVn and V have been read
    cp_async_commit();
    if (lower) {
        float x[2][4];
        zero_acc<2>(x);
        for (int k0 = m0; k0 < C; k0 += 16) warp_gemm<2, 16, true, true>(x, Tb + k0 * LDC, LDC, m0, X1 + k0 * LDC, LDC, nc);
        store_acc_bf16<2>(x, X2, LDC, m0, nc);
    }
    __syncthreads();
    if (lower) {
        float x[2][4];
        zero_acc<2>(x);
        for (int k0 = 0; k0 <= nc; k0 += 16) warp_gemm<2, 16, false, false>(x, X2 + k0, LDC, m0, Tb + k0, LDC, nc);   // (X2 T^T)_ij = sum_k X2_ik T_jk
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            float mv[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = r0 + 8 * (e >> 1), j = nc + nt * 8 + c0 + (e & 1);
                const float dA = i > j ? -x[nt][e] : 0.f;
                const float be = (e >> 1) ? be_hi : be_lo;
                const float t1 = dA * gam[nt][e] * kk[nt][e];          // dA_ij Gamma_ij (k_i.k_j) -> dbeta_i
                const float t2 = t1 * be;                              // dA_ij A_ij -> db_i, -db_j
                if (e >> 1) { dbe_hi += t1; db_hi += t2; } else { dbe_lo += t1; db_lo += t2; }
                col[2 * nt + (e & 1)] -= t2;
                mv[e] = dA * be * gam[nt][e];                          // M_ij
            }
            *reinterpret_cast<__nv_bfloat162*>(Ps + r0 * LDC + nc + nt * 8 + c0) = __floats2bfloat162_rn(mv[0], mv[1]);
            *reinterpret_cast<__nv_bfloat162*>(Ps + (r0 + 8) * LDC + nc + nt * 8 + c0) = __floats2bfloat162_rn(mv[2], mv[3]);
        }
    }
    // the sums of this warp: rows over the four lanes that share them, columns over the eight
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
        db_lo += __shfl_xor_sync(0xffffffffu, db_lo, o); db_hi += __shfl_xor_sync(0xffffffffu, db_hi, o);
        dbe_lo += __shfl_xor_sync(0xffffffffu, dbe_lo, o); dbe_hi += __shfl_xor_sync(0xffffffffu, dbe_hi, o);
    }
#pragma unroll
    for (int o = 4; o <= 16; o <<= 1)
#pragma unroll
        for (int i = 0; i < 4; ++i) col[i] += __shfl_xor_sync(0xffffffffu, col[i], o);
    kd = warp_sum(kd);
    dgam = warp_sum(dgam);
    if ((l & 3) == 0) {
        rdb[qd * C + r0] = db_lo; rdb[qd * C + r0 + 8] = db_hi;
        rbe[qd * C + r0] = dbe_lo; rbe[qd * C + r0 + 8] = dbe_hi;
    }
    if (l < 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) cdb[(w & 3) * C + nc + (i >> 1) * 8 + c0 + (i & 1)] = col[i];
    }
    if (l == 0) { tot[w] = dgam; tot[16 + w] = kd; }
    __syncthreads();                                                   // Ps holds M; the sums are in; T has been read
    if (more) load_t(nx);
    cp_async_commit();
    // ---- (9) dk += M K + M^T K; store ---------------------------------------------------------------------------------
    for (int k0 = 0; k0 <= m0; k0 += 16) warp_gemm<NQ, 16, false, true>(acc_dk, Ps + k0, LDC, m0, Ks + k0 * LD, LD, nd);
    for (int k0 = m0; k0 < C; k0 += 16) warp_gemm<NQ, 16, true, true>(acc_dk, Ps + k0 * LDC, LDC, m0, Ks + k0 * LD, LD, nd);
    store_rows_global<NQ>(acc_dk, a.dk + (((long long)b * a.T + t0) * a.H + h) * D + nd, (long long)a.H * D, m0, valid);
    // ---- (10) dbeta; dg_s = sum_{i >= s} db_i (b_C also gets the sum of <dKd_j, Kd_j> and dgamma gamma) -------------------
    if (w == 0) {
        float x0 = 0.f, x1 = 0.f, e0 = 0.f, e1 = 0.f, last = 0.f;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            x0 += rdb[p * C + i0] + cdb[p * C + i0]; x1 += rdb[p * C + i1] + cdb[p * C + i1];
            e0 += rbe[p * C + i0]; e1 += rbe[p * C + i1];
        }
        if (l == 31) {
            const float gamma = __expf(btot);                          // gamma = e^{b_C}: d b_C += dgamma gamma
            for (int p = 0; p < NTB / 32; ++p) last += tot[p] * gamma + tot[16 + p];
            x1 += last;
        }
        float s = x0 + x1;                                             // suffix sums over lane pairs
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const float y = __shfl_down_sync(0xffffffffu, s, o); if (l + o < 32) s += y; }
        const long long o0 = ((long long)b * a.T + t0 + i0) * a.H + h, o1 = o0 + a.H;
        if (i0 < valid) { a.dbeta[o0] = e0; if (a.dg != nullptr) a.dg[o0] = s; }
        if (i1 < valid) { a.dbeta[o1] = e1; if (a.dg != nullptr) a.dg[o1] = s - x0; }
    }
    }
}

template <int D> constexpr size_t prep_bwd_smem() {
    return (size_t)(7 * C * (D + 8) + 2 * D * (D + 8) + 4 * C * (C + 8)) * 2 + (size_t)(14 * C + 32) * 4;
}

template <int D> constexpr size_t prep_smem() { return (size_t)3 * C * (D + 8) * 2 + (size_t)(C * LDF + 2 * C) * 4; }

}  // namespace dr
}  // namespace lmoe

using namespace lmoe;

// dir 0: forward, dir 1: backward.  dk in {64, 128}; dv a multiple of 32.  Grid = (dv / 32, B*H).
LMOE_API int lmoe_delta_scan(int dir, int dk, int BH, const dr::Args* ap, cudaStream_t st) {
    const dr::Args a = *ap;
    if (a.dv % dr::DVS || (dk != 64 && dk != 128) || BH <= 0 || a.H <= 0 || a.err == nullptr) return -1;
    if (!(a.ldw == dk && a.lda == dr::C) && !(a.ldw == dk + 8 && a.lda == dr::C + 8)) return -1;
    // The kernels of lsm_delta_tc.cu have half as many CTAs.  Where the CTAs here are more than SMs, that alone decides; sequences x chunks, here and there in us:
    // outputs 64 x 26 82 and 42, 38 x 8 28 and 16, 256 x 2 38 and 28; Vn and the states only (the backward pass rebuilds them) 55 and 37, 19 and 14, 24 and 22;
    // reverse 80 and 42, 28 and 16, 38 and 26.  With an SM for every CTA it is the latency of a step: theirs is shorter with outputs (2 x 32 49.7 and 46.2, 2 x 128
    // 189 and 170, 32 x 64 97 and 90) and in the reverse scan (48.9 and 46.1, 186 and 169, 95 and 89), enough from 32 chunks on for their later start and the
    // host's time for their tensor maps (37 x 8 15.4 and 16.0, 15.2 and 16.2), and longer where Vn and the states are all that is wanted
    // (37.0 and 42.7, 138 and 159, 82 and 82).
    const bool out = dir != 0 || a.O != nullptr;
    const bool shared = (long long)BH * (a.dv / dr::DVS) > sm_count();
    if (dk == dr::TC_DK && a.dv % dr::TC_DV == 0 && (shared || (out && a.N >= 32))) return dr::scan_tc(dir, BH, a, st);
    dim3 grid(a.dv / dr::DVS, BH);
#define LMOE_DR_LAUNCH(KERNEL, DK)                                                                                     \
    do {                                                                                                               \
        auto kernel = KERNEL;                                                                                          \
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dr::Cfg<DK>::smem(out)); \
        if (e != cudaSuccess) return (int)e;                                                                           \
        kernel<<<grid, dr::NT + 32, dr::Cfg<DK>::smem(out), st>>>(a);                                                      \
    } while (0)
    if (dir != 0) { if (dk == 128) LMOE_DR_LAUNCH(dr::delta_scan_bwd_kernel<128>, 128); else LMOE_DR_LAUNCH(dr::delta_scan_bwd_kernel<64>, 64); }
    else if (out) { if (dk == 128) LMOE_DR_LAUNCH((dr::delta_scan_fwd_kernel<128, true>), 128); else LMOE_DR_LAUNCH((dr::delta_scan_fwd_kernel<64, true>), 64); }
    else { if (dk == 128) LMOE_DR_LAUNCH((dr::delta_scan_fwd_kernel<128, false>), 128); else LMOE_DR_LAUNCH((dr::delta_scan_fwd_kernel<64, false>), 64); }
#undef LMOE_DR_LAUNCH
    return (int)cudaGetLastError();
}

// Tiles of the chunked (gated) delta rule for every chunk of every (batch, head): grid (N, B*H).  dk = dv = D in {64, 128}.
LMOE_API int lmoe_delta_prepare(int D, const dr::PrepArgs* ap, cudaStream_t st) {
    const dr::PrepArgs a = *ap;
    if (a.N <= 0 || a.B * a.H <= 0) return -1;
    dim3 grid(a.N, a.B * a.H);
    if (D == 128) {
        cudaError_t e = cudaFuncSetAttribute(dr::delta_prep_fwd_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dr::prep_smem<128>());
        if (e != cudaSuccess) return (int)e;
        dr::delta_prep_fwd_kernel<128><<<grid, dr::NTP, dr::prep_smem<128>(), st>>>(a);
    } else if (D == 64) {
        cudaError_t e = cudaFuncSetAttribute(dr::delta_prep_fwd_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dr::prep_smem<64>());
        if (e != cudaSuccess) return (int)e;
        dr::delta_prep_fwd_kernel<64><<<grid, dr::NTP, dr::prep_smem<64>(), st>>>(a);
    } else return -2;
    return (int)cudaGetLastError();
}

// Chunk-parallel backward of the tile construction and of the chunk-local scan equations: grid (N, B*H).
LMOE_API int lmoe_delta_prepare_bwd(int D, const dr::PrepBwdArgs* ap, cudaStream_t st) {
    const dr::PrepBwdArgs a = *ap;
    if (a.N <= 0 || a.B * a.H <= 0) return -1;
    const int grid = (int)std::min<long long>((long long)a.N * a.B * a.H, sm_count());
    if (D == 128) {
        cudaError_t e = cudaFuncSetAttribute(dr::delta_prep_bwd_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dr::prep_bwd_smem<128>());
        if (e != cudaSuccess) return (int)e;
        dr::delta_prep_bwd_kernel<128><<<grid, dr::NTB, dr::prep_bwd_smem<128>(), st>>>(a);
    } else if (D == 64) {
        cudaError_t e = cudaFuncSetAttribute(dr::delta_prep_bwd_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dr::prep_bwd_smem<64>());
        if (e != cudaSuccess) return (int)e;
        dr::delta_prep_bwd_kernel<64><<<grid, dr::NTB, dr::prep_bwd_smem<64>(), st>>>(a);
    } else return -2;
    return (int)cudaGetLastError();
}
