// y[M, N] = x[M, K] W[N, K]^T for M <= 16: the linears of one-token decode steps.
//
// With a handful of rows the product is bound by reading W once (2 N K bytes); a 256 x 256 tensor-core tile would spend
// its time on rows that do not exist.  Here a CTA owns 16 rows of W at a time and its eight warps split K.  Every lane brings
// 16-byte pieces of two W rows (into slots of shared memory of its own, or registers) and, with one x row, on into mma.sync.m16n8k16
// fragments: the sum over k does not care about the order of k, so the eight consecutive elements a lane loads are used as the
// k slots that lane owns in two MMA steps (the same assignment for the W and the x fragment), and nothing is transposed or
// exchanged.  The eight partial tiles are added through shared memory.  No atomics: results are deterministic.
// Two kernels differ in how W arrives, and give the same bits:
//   gemm_skinny_kernel        two CTAs per SM walk the row blocks with 64 KB of copies in flight each, over the ends of row blocks too.
//                             For many row blocks of short rows: a CTA per row block drains the memory system at every block's end.
//                             (W of 128256 x 2048 96 us with a CTA per block, 91 so; 16384 x 2048 16.4 and 13.5.)
//   gemm_skinny_block_kernel  a CTA (or cluster) per row block, its loads in registers.  For long rows, where the loop over K is what counts
//                             (W of 32000 x 4096 50 us on the first kernel, 43 so; 8192 x 8192 27.9 and 23.8), and for few row blocks, where
//                             there is no next block to copy for (2560 x 1024 behind a norm kernel 8.4 and 7.4).
// use_ring below has the rule.  Both are launched with programmatic stream serialization: their first eight steps of W are in flight
// before they wait for the kernel that produces x, so consecutive linears of a decode step keep HBM busy across the kernel
// boundaries (the small kernels in between call griddepcontrol.launch_dependents at their start).
#include <cstdlib>

#include "common.cuh"
#include "mma_utils.cuh"

namespace lmoe {
namespace sk {

__device__ __forceinline__ uint4 ld_stream(const bf16* p) { return __ldcs(reinterpret_cast<const uint4*>(p)); }
// 16 bytes of global memory to shared memory, zeros where `ok` is false
__device__ __forceinline__ void copy16(uint32_t dst, const bf16* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

__device__ __forceinline__ uint32_t sk_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void sk_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// store a float into the shared memory of CTA `rank` of the cluster, at the address `p` has in this CTA
__device__ __forceinline__ void st_cluster_f32(float* p, uint32_t rank, float v) {
    uint32_t local = (uint32_t)__cvta_generic_to_shared(p), remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(remote), "f"(v) : "memory");
}

// NTILES 1: M <= 8, 2: M <= 16.  KS: CTAs of a cluster that split K between them (for matrices with few rows, so that
// every SM streams a piece of W); their partial tiles meet in the shared memory of the cluster's first CTA.
// OUT: bf16 result, fp32 result, fp32 added to what y holds (the residual stream of a decode step), or bf16 silu(gate) * up
// for W = [gate | up] [2 N, K], where a CTA's 16 rows of W are eight of gate and the eight of up that go with them.
enum { OUT_BF16 = 0, OUT_F32 = 1, OUT_F32_ADD = 2, OUT_SWIGLU = 3 };
template <int OUT> constexpr int ROWS = OUT == OUT_SWIGLU ? 8 : 16;      // columns of y per row block
template <int OUT>
__device__ __forceinline__ void put(void* y, long long i, float v) {
    if (OUT == OUT_BF16) reinterpret_cast<bf16*>(y)[i] = __float2bfloat16(v);
    else if (OUT == OUT_F32) reinterpret_cast<float*>(y)[i] = v;
    else reinterpret_cast<float*>(y)[i] += v;
}

constexpr int PF = 8, STEP = 256;                                        // steps in flight; elements of K per step of the eight warps
__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16(v)); }

// The eight warps' partial tiles of a row block, added up and stored.
template <int NTILES, int KS, int OUT>
__device__ __forceinline__ void finish_block(const float (&acc)[NTILES][4], float (*red)[NTILES][32][4], float (*cred)[NTILES][32][4], uint32_t crank,
                                             int row_lo, void* y, long long ldy, int M, int N) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, q = l & 3;
    const int row_hi = row_lo + 8;
    const bool lo_ok = row_lo < N, hi_ok = row_hi < N;
#pragma unroll
    for (int t = 0; t < NTILES; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) red[w][t][l][e] = acc[t][e];
    __syncthreads();
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    if (w < NTILES) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[e] += red[i][w][l][e];
    }
    if (KS > 1) {
        // the CTA's partial tile goes to slot `crank` of the first CTA; it adds the slots in rank order (deterministic)
        if (w < NTILES) {
#pragma unroll
            for (int e = 0; e < 4; ++e) st_cluster_f32(&cred[crank][w][l][e], 0, s[e]);
        }
        sk_cluster_sync();
        if (crank != 0) return;
        if (w < NTILES) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s[e] = 0.f;
#pragma unroll
                for (int i = 0; i < KS; ++i) s[e] += cred[i][w][l][e];
            }
        }
    }
    if (w < NTILES) {
        const int n0 = 8 * w + 2 * q;                                   // batch rows n0, n0 + 1
        if (OUT == OUT_SWIGLU) {                                        // of gate and up in bf16, as where they pass through memory
            if (lo_ok && n0 < M) put<OUT_BF16>(y, (long long)n0 * ldy + row_lo, silu_f(bf16_round(s[0])) * bf16_round(s[2]));
            if (lo_ok && n0 + 1 < M) put<OUT_BF16>(y, (long long)(n0 + 1) * ldy + row_lo, silu_f(bf16_round(s[1])) * bf16_round(s[3]));
            return;
        }
        if (n0 < M) {
            if (lo_ok) put<OUT>(y, (long long)n0 * ldy + row_lo, s[0]);
            if (hi_ok) put<OUT>(y, (long long)n0 * ldy + row_hi, s[2]);
        }
        if (n0 + 1 < M) {
            if (lo_ok) put<OUT>(y, (long long)(n0 + 1) * ldy + row_lo, s[1]);
            if (hi_ok) put<OUT>(y, (long long)(n0 + 1) * ldy + row_hi, s[3]);
        }
    }
}

// A CTA, or a cluster of KS that split K, takes row blocks blockIdx.x / KS, + gridDim.x / KS, ...  A lane's pieces of W go through PF slots of
// shared memory that only this lane writes and reads, so nothing but its own copies is waited for, and the next steps' copies stay
// in flight over the reduction and the store of a row block.
// ONE: a lane's piece of x (K / KS at most PF steps) stays in registers.

template <int NTILES, int KS, int OUT, bool ONE>
__global__ void __launch_bounds__(256, 2) gemm_skinny_kernel(const bf16* x, long long ldx, const bf16* W,
                                                             long long ldw, void* y, long long ldy, int M, int N, int K) {
    extern __shared__ __align__(16) uint4 slots[];                       // [PF][2][256]
    __shared__ float red[2][8][NTILES][32][4];
    __shared__ float cred[2][KS][NTILES][32][4];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int g = l >> 2, q = l & 3;
    const uint32_t crank = KS > 1 ? sk_cluster_rank() : 0;
    const bf16* xr[NTILES];
    bool x_ok[NTILES];
#pragma unroll
    for (int t = 0; t < NTILES; ++t) {
        x_ok[t] = g + 8 * t < M;
        xr[t] = x + (long long)(x_ok[t] ? g + 8 * t : 0) * ldx + q * 8;
    }
    const uint4 zero = make_uint4(0, 0, 0, 0);
    const int kslice = K / KS;                                           // a multiple of 32 (checked by the launcher)
    const int k_beg = (int)crank * kslice + w * 32, k_end = (int)(crank + 1) * kslice;
    const int steps = (kslice + STEP - 1) / STEP, blocks = (N + ROWS<OUT> - 1) / ROWS<OUT>, stride = gridDim.x / KS;
    const uint32_t my = (uint32_t)__cvta_generic_to_shared(slots) + threadIdx.x * 16;
    int c_block = blockIdx.x / KS, c_k = k_beg, c_step = 0;              // the next step to copy
    auto copy = [&](int slot) {
        const int r = c_block * ROWS<OUT> + g, r_hi = OUT == OUT_SWIGLU ? r + N : r + 8;
        const bool in = c_block < blocks && c_k < k_end, lo = in && r < N, hi = in && (OUT == OUT_SWIGLU ? r : r_hi) < N;
        copy16(my + slot * 8192, W + (lo ? (long long)r * ldw + c_k + q * 8 : 0), lo);
        copy16(my + slot * 8192 + 4096, W + (hi ? (long long)r_hi * ldw + c_k + q * 8 : 0), hi);
        asm volatile("cp.async.commit_group;" ::: "memory");
        c_k += STEP;
        if (++c_step == steps) {
            c_step = 0;
            c_k = k_beg;
            c_block += stride;
        }
    };
    // The weights do not depend on the kernel before this one: the first steps of W are requested before waiting for
    // it (programmatic dependent launch), so the weight stream of one linear overlaps the tail of whatever produced x.
#pragma unroll
    for (int i = 0; i < PF; ++i) copy(i);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");     // the next kernel may start its own copies
    // x is complete and visible from here on.  (No pointer of this kernel is __restrict__: loads through those may move ahead of the wait.)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint4 xk[ONE ? NTILES : 1][PF];
    if (ONE) {
#pragma unroll
        for (int i = 0; i < PF; ++i)
#pragma unroll
            for (int t = 0; t < NTILES; ++t) {
                const int k = k_beg + i * STEP;
                xk[ONE ? t : 0][i] = x_ok[t] && k < k_end ? *reinterpret_cast<const uint4*>(xr[t] + k) : zero;
            }
    }
    int slot = 0, buf = 0;
    for (int block = blockIdx.x / KS; block < blocks; block += stride, buf ^= 1) {
        const int row_lo = block * ROWS<OUT> + g;
        float acc[NTILES][4];
#pragma unroll
        for (int t = 0; t < NTILES; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
        auto use = [&](const uint4 (&b)[NTILES]) {
            asm volatile("cp.async.wait_group %0;" :: "n"(PF - 1) : "memory");
            const uint4 a_lo = slots[slot * 512 + threadIdx.x], a_hi = slots[slot * 512 + 256 + threadIdx.x];
            const uint32_t f1[4] = {a_lo.x, a_hi.x, a_lo.y, a_hi.y};
            const uint32_t f2[4] = {a_lo.z, a_hi.z, a_lo.w, a_hi.w};
#pragma unroll
            for (int t = 0; t < NTILES; ++t) {
                mma16816(acc[t], f1, b[t].x, b[t].y);
                mma16816(acc[t], f2, b[t].z, b[t].w);
            }
            copy(slot);                                                  // behind the use of what the slot held
            slot = (slot + 1) % PF;
        };
        if (ONE) {
#pragma unroll
            for (int i = 0; i < PF; ++i)
                if (i < steps) {
                    uint4 b[NTILES];
#pragma unroll
                    for (int t = 0; t < NTILES; ++t) b[t] = xk[ONE ? t : 0][i];
                    use(b);
                }
        } else {
#pragma unroll 4
            for (int i = 0; i < steps; ++i) {
                const int k = k_beg + i * STEP;
                uint4 b[NTILES];
#pragma unroll
                for (int t = 0; t < NTILES; ++t) b[t] = x_ok[t] && k < k_end ? *reinterpret_cast<const uint4*>(xr[t] + k) : zero;
                use(b);
            }
        }
        finish_block<NTILES, KS, OUT>(acc, red[buf], cred[buf], crank, row_lo, y, ldy, M, N);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// A CTA, or a cluster of KS that split K, per row block.  The first PF steps of W are requested ahead of the wait for x.
template <int NTILES, int KS, int OUT>
__global__ void __launch_bounds__(256) gemm_skinny_block_kernel(const bf16* x, long long ldx, const bf16* W, long long ldw, void* y, long long ldy,
                                                                int M, int N, int K) {
    __shared__ float red[8][NTILES][32][4];
    __shared__ float cred[KS][NTILES][32][4];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int g = l >> 2, q = l & 3;
    const uint32_t crank = KS > 1 ? sk_cluster_rank() : 0;
    const int row_lo = (blockIdx.x / KS) * ROWS<OUT> + g, row_hi = OUT == OUT_SWIGLU ? row_lo + N : row_lo + 8;
    const bool lo_ok = row_lo < N, hi_ok = OUT == OUT_SWIGLU ? lo_ok : row_hi < N;
    const bf16* w_lo = W + (long long)(lo_ok ? row_lo : 0) * ldw + q * 8;
    const bf16* w_hi = W + (long long)(hi_ok ? row_hi : 0) * ldw + q * 8;
    const bf16* xr[NTILES];
    bool x_ok[NTILES];
#pragma unroll
    for (int t = 0; t < NTILES; ++t) {
        x_ok[t] = g + 8 * t < M;
        xr[t] = x + (long long)(x_ok[t] ? g + 8 * t : 0) * ldx + q * 8;
    }
    float acc[NTILES][4];
#pragma unroll
    for (int t = 0; t < NTILES; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    const int kslice = K / KS;                                           // a multiple of 32 (checked by the launcher)
    const int k_beg = (int)crank * kslice + w * 32, k_end = (int)(crank + 1) * kslice;
    uint4 a_lo[PF], a_hi[PF];
#pragma unroll
    for (int i = 0; i < PF; ++i) {
        const int k = k_beg + i * STEP;
        a_lo[i] = lo_ok && k < k_end ? ld_stream(w_lo + k) : zero;
        a_hi[i] = hi_ok && k < k_end ? ld_stream(w_hi + k) : zero;
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");     // the next kernel may start its own loads
    // x is complete and visible from here on.  (No pointer of this kernel is __restrict__: loads through those may move ahead of the wait.)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    auto use = [&](const uint4& lo, const uint4& hi, int k) {
        const uint32_t f1[4] = {lo.x, hi.x, lo.y, hi.y};
        const uint32_t f2[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
        for (int t = 0; t < NTILES; ++t) {
            const uint4 b = x_ok[t] ? *reinterpret_cast<const uint4*>(xr[t] + k) : zero;
            mma16816(acc[t], f1, b.x, b.y);
            mma16816(acc[t], f2, b.z, b.w);
        }
    };
#pragma unroll
    for (int i = 0; i < PF; ++i)
        if (k_beg + i * STEP < k_end) use(a_lo[i], a_hi[i], k_beg + i * STEP);
#pragma unroll 4
    for (int k = k_beg + PF * STEP; k < k_end; k += STEP)
        use(lo_ok ? ld_stream(w_lo + k) : zero, hi_ok ? ld_stream(w_hi + k) : zero, k);
    finish_block<NTILES, KS, OUT>(acc, red, cred, crank, row_lo, y, ldy, M, N);
}

template <int NTILES, int KS, int OUT>
static int launch_skinny(const bf16* x, long long ldx, const bf16* W, long long ldw, void* y, long long ldy, int M, int N, int K,
                         int sms, bool ring, cudaStream_t st) {
    const int row_blocks = (N + ROWS<OUT> - 1) / ROWS<OUT>;
    auto kernel = gemm_skinny_block_kernel<NTILES, KS, OUT>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(row_blocks * KS);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    if (ring) {
        kernel = K / KS <= PF * STEP ? gemm_skinny_kernel<NTILES, KS, OUT, true> : gemm_skinny_kernel<NTILES, KS, OUT, false>;
        cfg.gridDim = dim3(min(row_blocks, 2 * sms / KS) * KS);          // two CTAs per SM
        cfg.dynamicSmemBytes = PF * 8192;
        const int rc = (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PF * 8192);
        if (rc) return rc;
    }
    cudaLaunchAttribute attr[2];
    int na = 0;
    // the kernel may start while its predecessor in the stream is still running; it waits (griddepcontrol.wait) before it
    // reads x
    static const bool pdl = [] { const char* e = getenv("LMOE_SKINNY_PDL"); return e == nullptr || e[0] != '0'; }();
    if (pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    if (KS > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = KS;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return (int)cudaLaunchKernelEx(&cfg, kernel, x, ldx, W, ldw, y, ldy, M, N, K);
}

// Copies across row blocks (gemm_skinny_kernel) or a CTA per row block (gemm_skinny_block_kernel)?  Times in us, block / ring, of a small norm kernel
// and the product that follows it, W from memory, as decode steps have them:
//   K not split: the ring from the second wave of row blocks on while rows are short.  8 rows of x, 32000 of W: K = 1024 17.6 / 13.5, 2048 28.1 /
//     23.8, 3072 41.0 / 44.2, 4096 49.7 / 56.9; 8192 of W: K = 2048 11.9 / 9.1, 3072 15.7 / 15.0, 4096 18.3 / 18.3, 8192 29.9 / 32.9, 14336 46.8 / 55.7;
//     16 rows of x, 32000 of W: K = 3072 46.7 / 43.3, 4096 56.7 / 55.0.  One wave (4736 of W): K = 1024 4.9 / 5.2, 4096 12.2 / 13.7.
//   K over a cluster: the ring where a CTA's slice of K is worth its slots, and while that fits them or clusters have two row blocks at most.  8 rows of x,
//     2560 of W: K = 1024 7.4 / 8.4, 2048 8.7 / 9.7, 3072 10.8 / 10.3, 8192 18.3 / 15.3, 11008 25.8 / 29.1; 512 of W: K = 1024 3.5 / 3.5, 2048 4.0 /
//     3.6; 2048 of W: K = 1024 5.9 / 6.0, 2048 6.8 / 7.0 (but a decode step of four 2048-wide layers 321 / 317), 8192 15.5 / 11.8, 14336 23.2 / 20.4.
static bool use_ring(int M, int K, int row_blocks, int sms, bool split) {
    if (split) return row_blocks <= sms ? K >= 2048 : K > 2560 && K <= 4 * PF * STEP;
    return row_blocks > 2 * sms && (K <= 2560 || (K <= 4096 && (M > 8 || row_blocks <= 4 * sms)) || (K <= 5120 && row_blocks <= 3 * sms));
}

template <int OUT>
static int dispatch(const bf16* x, long long ldx, const bf16* W, long long ldw, void* y, long long ldy, int M, int N, int K,
                    cudaStream_t st) {
    static const int sms = sm_count();
    // few row blocks: the four CTAs of a cluster split K so that the whole GPU streams W
    const int row_blocks = (N + ROWS<OUT> - 1) / ROWS<OUT>;
    const bool split = row_blocks < 2 * sms && K % 128 == 0;
    const bool ring = use_ring(M, K, row_blocks, sms, split);
    if (M <= 8) return split ? launch_skinny<1, 4, OUT>(x, ldx, W, ldw, y, ldy, M, N, K, sms, ring, st)
                             : launch_skinny<1, 1, OUT>(x, ldx, W, ldw, y, ldy, M, N, K, sms, ring, st);
    return split ? launch_skinny<2, 4, OUT>(x, ldx, W, ldw, y, ldy, M, N, K, sms, ring, st)
                 : launch_skinny<2, 1, OUT>(x, ldx, W, ldw, y, ldy, M, N, K, sms, ring, st);
}

}  // namespace sk
}  // namespace lmoe

static int skinny_shape_ok(const void* x, long long ldx, const void* W, long long ldw, int M, int N, int K) {
    if (M <= 0 || M > 16 || N <= 0 || K <= 0 || K % 32 != 0 || ldx % 8 != 0 || ldw % 8 != 0) return 0;
    return ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
}

// x [M, K] (row pitch ldx), W [N, K] (row pitch ldw), y [M, N] (row pitch ldy), all bf16; M <= 16, K a multiple of 32,
// pitches multiples of 8 elements and bases 16-byte aligned.  Returns -1 for shapes it does not take.
LMOE_API int lmoe_gemm_skinny(const void* x, long long ldx, const void* W, long long ldw, void* y, long long ldy, int M, int N,
                              int K, cudaStream_t st) {
    using namespace lmoe;
    if (!skinny_shape_ok(x, ldx, W, ldw, M, N, K)) return -1;
    return sk::dispatch<sk::OUT_BF16>((const bf16*)x, ldx, (const bf16*)W, ldw, y, ldy, M, N, K, st);
}

// The same product in fp32: y [M, N] floats, overwritten or (accumulate != 0) added to.
LMOE_API int lmoe_gemm_skinny_f32(const void* x, long long ldx, const void* W, long long ldw, float* y, long long ldy, int M, int N,
                                  int K, int accumulate, cudaStream_t st) {
    using namespace lmoe;
    if (!skinny_shape_ok(x, ldx, W, ldw, M, N, K)) return -1;
    return accumulate ? sk::dispatch<sk::OUT_F32_ADD>((const bf16*)x, ldx, (const bf16*)W, ldw, y, ldy, M, N, K, st)
                      : sk::dispatch<sk::OUT_F32>((const bf16*)x, ldx, (const bf16*)W, ldw, y, ldy, M, N, K, st);
}

// y [M, F] = silu(gate) * up for [gate | up] = x W^T, W [2 F, K]; the bits of lmoe_gemm_skinny followed by the SwiGLU kernel.
LMOE_API int lmoe_gemm_skinny_swiglu(const void* x, long long ldx, const void* W, long long ldw, void* y, long long ldy, int M, int F,
                                     int K, cudaStream_t st) {
    using namespace lmoe;
    if (!skinny_shape_ok(x, ldx, W, ldw, M, F, K)) return -1;
    return sk::dispatch<sk::OUT_SWIGLU>((const bf16*)x, ldx, (const bf16*)W, ldw, y, ldy, M, F, K, st);
}
