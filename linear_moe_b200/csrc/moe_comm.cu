// Expert-parallel token exchange of the MoE layer over NVLink peer memory: no NCCL all-to-all, no host sync.
//
// Replaces the reference's permute -> all_to_all -> permute ... unpermute -> all_to_all -> unpermute chain
// (moe/token_dispatcher.py:412-548, whose split sizes are read back by the host with .tolist()) with
//
//   moe_exchange_kernel   sums the chunk histograms; every rank stores its per-expert token counts into every peer's count matrix, releases a
//                         flag, waits (bounded) for the peers' rows and derives, on the device: the padded row
//                         offsets of its local experts in its receive buffer (the grouped GEMM's problem sizes) and,
//                         for every global expert, the row in the owner's receive buffer where THIS rank's tokens
//                         for that expert start.
//   moe_count_kernel      per-chunk histograms of the (token, slot) -> expert assignments (chunks of 4096 assignments).
//   moe_assign_kernel     destination (rank, row) of every (token, slot) pair: a counting sort that is stable in the
//                         assignment index (deterministic row order), without any library sort.
//   moe_push_kernel       dispatch: every (token, slot) row is written straight into the owner rank's receive buffer
//                         with 16-byte peer stores (optionally scaled, which is the backward of the combine); the
//                         last CTA to finish releases a flag on every peer and waits for theirs.
//   moe_zero_pads_kernel  clears the padding rows behind every expert segment so that the weight-gradient GEMMs,
//                         which contract over the padded rows, see zeros.
//   moe_signal_kernel     "my expert outputs are complete" flag to every peer.
//   moe_pull_kernel       combine: waits for the owners' flags, then every token gathers its k expert outputs from
//                         the owners' result buffers with 16-byte peer loads, weights them by the routing
//                         probabilities and sums them in fp32 (un-permute + weighted sum + all-to-all in one pass).
//
// Buffers are symmetric allocations shared by all MoE layers; a push/pull pair of one layer is ordered against the
// next layer's by the flags themselves (a rank starts its next push only after its pull, which waited for every owner's
// compute; an owner overwrites its result buffer only after every peer's next push).  Flags carry monotonically
// increasing epochs.  Every spin is bounded: on expiry the kernel records {kernel, peer} in the status word and goes
// on (results are then wrong but finite, every address stays in bounds) and the host raises after the step.
#include "common.cuh"

namespace lmoe {

__device__ __forceinline__ void moe_st_rel(int* p, int v) {
    asm volatile("st.release.sys.global.s32 [%0], %1;\n" :: "l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int moe_ld_acq(const int* p) {
    int v;
    asm volatile("ld.acquire.sys.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}

struct MoeArgs {
    int* const* peer_cnt;       // [W] count matrices, int32 [W(src)][E]
    int* const* peer_flags;     // [W] flag arrays, int32 [3][W(src)]: counts ready / push done / outputs ready
    bf16* const* peer_x;        // [W] receive buffers [cap][h]
    bf16* const* peer_y;        // [W] result buffers [cap][h]
    int* status;
    unsigned int* done_ctr;
    int rank, world, E, El, cap, h;
    int epoch;
    long long spin_limit;
    // exchange
    int* offs;                  // [El+1] out: padded row offsets of the local experts
    int* real;                  // [El]   out: tokens received per local expert
    int* send_base;             // [E]    out: first row of this rank's tokens in the owner's buffer, -1 = do not send
    // count / assign
    const long long* idx;       // [n_assign] expert id of every (token, slot) pair, -1 = dropped
    int* blockhist;             // [nchunks][E] assignments per chunk and expert
    int* blockbase;             // [nchunks][E] exclusive prefix of blockhist over the chunks
    int nchunks;
    int* dest_rank;             // [n_assign]
    int* dest_row;              // [n_assign]
    // push / pull
    const bf16* src;            // [T][h]
    const float* w;             // [n_assign] or null
    bf16* out;                  // [T][h]
    bf16* rows;                 // [n_assign][h] or null: the gathered rows, unweighted
    int n_assign, k;
    int pad;                    // expert segments in the receive buffer start at multiples of `pad` rows
};

// wait until flags[phase][j] >= epoch for every peer j; one thread per peer.  Returns through smem `fail`.
__device__ __forceinline__ void moe_wait_all(const MoeArgs& a, int phase, int code, int* fail) {
    if ((int)threadIdx.x < a.world) {
        const int* f = a.peer_flags[a.rank] + phase * a.world + threadIdx.x;
        long long spins = 0;
        while (moe_ld_acq(f) < a.epoch) {
            if (++spins > a.spin_limit) {
                atomicCAS(a.status, 0, (9 << 24) | ((int)threadIdx.x << 16) | code);
                *fail = 1;
                break;
            }
            __nanosleep(64);
        }
    }
}

__global__ void moe_exchange_kernel(MoeArgs a) {
    extern __shared__ int sm[];
    int* tot = sm;                 // [E]
    int* prior = sm + a.E;         // [E]
    int* over = sm + 2 * a.E;      // [W]
    __shared__ int fail;
    if (threadIdx.x == 0) fail = 0;
    for (int e = threadIdx.x; e < a.E; e += blockDim.x) {
        int c = 0;
        for (int ch = 0; ch < a.nchunks; ++ch) {                     // exclusive prefix over the chunks, total = this rank's count
            a.blockbase[ch * a.E + e] = c;
            c += a.blockhist[ch * a.E + e];
        }
        for (int j = 0; j < a.world; ++j) a.peer_cnt[j][a.rank * a.E + e] = c;
    }
    __threadfence_system();
    __syncthreads();
    if ((int)threadIdx.x < a.world) moe_st_rel(a.peer_flags[threadIdx.x] + 0 * a.world + a.rank, a.epoch);
    moe_wait_all(a, 0, 1, &fail);
    __syncthreads();
    const int* cnt = a.peer_cnt[a.rank];
    for (int e = threadIdx.x; e < a.E; e += blockDim.x) {
        int t = 0, p = 0;
        for (int s = 0; s < a.world; ++s) {
            const int c = fail ? 0 : max(__ldcg(cnt + s * a.E + e), 0);
            if (s < a.rank) p += c;
            t += c;
        }
        tot[e] = t;
        prior[e] = p;
    }
    __syncthreads();
    if ((int)threadIdx.x < a.world) {
        const int d = threadIdx.x;
        long long run = 0;
        for (int el = 0; el < a.El; ++el) run += (tot[d * a.El + el] + a.pad - 1) / a.pad * a.pad;
        over[d] = run > a.cap;
        if (run > a.cap) atomicCAS(a.status, 0, (9 << 24) | (d << 16) | 7);        // receive buffer of rank d too small
    }
    __syncthreads();
    if ((int)threadIdx.x < a.world) {
        const int d = threadIdx.x;
        int run = 0;
        for (int el = 0; el < a.El; ++el) {
            const int e = d * a.El + el;
            a.send_base[e] = over[d] ? -1 : run + prior[e];
            if (d == a.rank) { a.offs[el] = over[d] ? 0 : run; a.real[el] = over[d] ? 0 : tot[e]; }
            run += (tot[e] + a.pad - 1) / a.pad * a.pad;
        }
        if (d == a.rank) a.offs[a.El] = over[d] ? 0 : run;
    }
}

constexpr int ASSIGN_CHUNK = 4096, ASSIGN_PER_THREAD = 16;          // 256 threads x 16 consecutive assignments

// grid = nchunks: histogram of one chunk of assignments
__global__ void moe_count_kernel(MoeArgs a) {
    extern __shared__ int hist[];
    for (int e = threadIdx.x; e < a.E; e += blockDim.x) hist[e] = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * ASSIGN_CHUNK;
    for (int i = threadIdx.x; i < ASSIGN_CHUNK; i += blockDim.x) {
        const long long p = base + i;
        if (p < a.n_assign) {
            const long long e = a.idx[p];
            if (e >= 0 && e < a.E) atomicAdd(&hist[e], 1);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < a.E; e += blockDim.x) a.blockhist[blockIdx.x * a.E + e] = hist[e];
}

// grid = nchunks, 256 threads, dynamic smem 256 * E * 2 bytes: thread t owns assignments [16 t, 16 t + 16) of the chunk
__global__ void moe_assign_kernel(MoeArgs a) {
    extern __shared__ unsigned short cnt[];                          // [256][E] -> exclusive prefix over the threads
    const int t = threadIdx.x;
    unsigned short* mine = cnt + t * a.E;
    for (int e = 0; e < a.E; ++e) mine[e] = 0;
    const long long base = (long long)blockIdx.x * ASSIGN_CHUNK + (long long)t * ASSIGN_PER_THREAD;
    long long ev[ASSIGN_PER_THREAD];
#pragma unroll
    for (int i = 0; i < ASSIGN_PER_THREAD; ++i) {
        const long long p = base + i;
        long long e = p < a.n_assign ? a.idx[p] : -1;
        if (e >= a.E) e = -1;
        ev[i] = e;
        if (e >= 0) mine[e]++;
    }
    __syncthreads();
    for (int e = t; e < a.E; e += blockDim.x) {
        unsigned int run = 0;
        for (int r = 0; r < (int)blockDim.x; ++r) {
            const unsigned short c = cnt[r * a.E + e];
            cnt[r * a.E + e] = (unsigned short)run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ASSIGN_PER_THREAD; ++i) {
        const long long p = base + i;
        if (p >= a.n_assign) break;
        const long long e = ev[i];
        int dr = -1, row = -1;
        if (e >= 0) {
            const int pos = mine[e]++;
            const int sb = a.send_base[e];
            if (sb >= 0) { dr = (int)e / a.El; row = sb + a.blockbase[blockIdx.x * a.E + e] + pos; }
            if (row >= a.cap) { dr = -1; row = -1; }
        }
        a.dest_rank[p] = dr;
        a.dest_row[p] = row;
    }
}

__global__ void moe_push_kernel(MoeArgs a) {
    __shared__ int fail, last;
    const int wpb = blockDim.x >> 5, l = threadIdx.x & 31;
    const int vecs = a.h / 8;
    for (long long as = (long long)blockIdx.x * wpb + (threadIdx.x >> 5); as < a.n_assign; as += (long long)gridDim.x * wpb) {
        const int dr = a.dest_rank[as];
        if (dr < 0) continue;
        const uint4* s = reinterpret_cast<const uint4*>(a.src + (as / a.k) * a.h);
        uint4* d = reinterpret_cast<uint4*>(a.peer_x[dr] + (long long)a.dest_row[as] * a.h);
        if (a.w == nullptr) {
            for (int c = l; c < vecs; c += 32) d[c] = s[c];
        } else {
            const float wt = a.w[as];
            for (int c = l; c < vecs; c += 32) {
                uint4 v = s[c];
                __nv_bfloat162* hv = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float2 f = __bfloat1622float2(hv[i]);
                    hv[i] = __floats2bfloat162_rn(f.x * wt, f.y * wt);
                }
                d[c] = v;
            }
        }
    }
    // grid-wide completion -> flag to every peer -> wait for every peer's flag
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
        fail = 0;
        last = atomicAdd(a.done_ctr, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence_system();
    if ((int)threadIdx.x < a.world) moe_st_rel(a.peer_flags[threadIdx.x] + 1 * a.world + a.rank, a.epoch);
    moe_wait_all(a, 1, 2, &fail);
    if (threadIdx.x == 0) *a.done_ctr = 0;
}

// grid (El, chunks): zero rows [offs[el] + real[el], offs[el+1]) of the local receive buffer
__global__ void moe_zero_pads_kernel(MoeArgs a) {
    const int el = blockIdx.x;
    const int lo = a.offs[el] + a.real[el], hi = min(a.offs[el + 1], a.cap);
    const int vecs = a.h / 8;
    uint4* x = reinterpret_cast<uint4*>(a.peer_x[a.rank]);
    const long long n = (long long)max(hi - lo, 0) * vecs;
    for (long long i = (long long)blockIdx.y * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.y * blockDim.x)
        x[(long long)lo * vecs + i] = make_uint4(0, 0, 0, 0);
}

__global__ void moe_signal_kernel(MoeArgs a) {
    __threadfence_system();
    if ((int)threadIdx.x < a.world) moe_st_rel(a.peer_flags[threadIdx.x] + 2 * a.world + a.rank, a.epoch);
}

template <int KMAX>
__global__ void moe_pull_kernel(MoeArgs a) {
    __shared__ int fail;
    if (threadIdx.x == 0) fail = 0;
    __syncthreads();
    moe_wait_all(a, 2, 3, &fail);
    __syncthreads();
    const int wpb = blockDim.x >> 5, l = threadIdx.x & 31;
    const int vecs = a.h / 8;
    const int T = a.n_assign / a.k;
    for (long long t = (long long)blockIdx.x * wpb + (threadIdx.x >> 5); t < T; t += (long long)gridDim.x * wpb) {
        const uint4* rp[KMAX];
        float wt[KMAX];
#pragma unroll
        for (int j = 0; j < KMAX; ++j) {
            rp[j] = nullptr;
            wt[j] = 0.f;
            if (j < a.k) {
                const int dr = a.dest_rank[t * a.k + j];
                if (dr >= 0) {
                    rp[j] = reinterpret_cast<const uint4*>(a.peer_y[dr] + (long long)a.dest_row[t * a.k + j] * a.h);
                    wt[j] = a.w != nullptr ? a.w[t * a.k + j] : 1.f;
                }
            }
        }
        for (int c = l; c < vecs; c += 32) {
            uint4 v[KMAX];
#pragma unroll
            for (int j = 0; j < KMAX; ++j) v[j] = rp[j] != nullptr ? __ldcg(rp[j] + c) : make_uint4(0, 0, 0, 0);
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < KMAX; ++j) {
                const __nv_bfloat162* hv = reinterpret_cast<const __nv_bfloat162*>(&v[j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float2 f = __bfloat1622float2(hv[i]);
                    acc[2 * i] += wt[j] * f.x;
                    acc[2 * i + 1] += wt[j] * f.y;
                }
                if (a.rows != nullptr && j < a.k)
                    reinterpret_cast<uint4*>(a.rows + (t * a.k + j) * a.h)[c] = v[j];
            }
            uint4 o;
            __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
            for (int i = 0; i < 4; ++i) ho[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
            reinterpret_cast<uint4*>(a.out + t * a.h)[c] = o;
        }
    }
}

// Gradient of the routing probabilities in the combine: d_probs[t, j] = <rows[t * k + j, :], d_out[t, :]> (zero for a
// dropped assignment).  One warp per token: the token's output gradient is read once per 256-element piece and reused
// for its k gathered rows.  (A batched matrix product with one output column per batch runs this at a fraction of the
// memory bandwidth.)
template <int KMAX>
__global__ void moe_dprobs_kernel(const bf16* __restrict__ rows, const bf16* __restrict__ d_out, const int* __restrict__ dest_rank,
                                  float* __restrict__ d_probs, int T, int k, int h) {
    const int wpb = blockDim.x >> 5, l = threadIdx.x & 31;
    for (long long t = (long long)blockIdx.x * wpb + (threadIdx.x >> 5); t < T; t += (long long)gridDim.x * wpb) {
        float acc[KMAX];
#pragma unroll
        for (int j = 0; j < KMAX; ++j) acc[j] = 0.f;
        const uint4* dp = reinterpret_cast<const uint4*>(d_out + t * h);
        for (int c = l; c < h / 8; c += 32) {
            const uint4 dv = __ldg(dp + c);
            const __nv_bfloat162* d2 = reinterpret_cast<const __nv_bfloat162*>(&dv);
            float2 df[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) df[i] = __bfloat1622float2(d2[i]);
#pragma unroll
            for (int j = 0; j < KMAX; ++j) {
                if (j < k) {
                    const uint4 rv = __ldcs(reinterpret_cast<const uint4*>(rows + (t * k + j) * h) + c);
                    const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rv);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 rf = __bfloat1622float2(r2[i]);
                        acc[j] += rf.x * df[i].x + rf.y * df[i].y;
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < KMAX; ++j) {
            if (j < k) {
                float v = acc[j];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (l == 0) d_probs[t * k + j] = dest_rank[t * k + j] >= 0 ? v : 0.f;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// One rank: the same routing and exchange with plain pointers, without counts matrices, flags and waits.  Two launches build the routing
// record (three and a fence between them before), one brings the rows, with the padding rows' zeros, and one takes the results; the gradient of
// the combine forms the routing weights' gradient from the same rows of d_out that it sends, and reads the experts' results where they are
// (a copy of them in token order was written by the forward pass for that: 134 MB at 8192 tokens x 8 of width 1024).
// The three exchange kernels are bound by memory: a warp takes a token, reads its row once for all k destinations and has all its pieces in flight.
// 8192 tokens x 8 of 64 experts, width 1024, in us: routing 57 -> 17, push 53 -> 28, combine 55 -> 30, its gradients 100 -> 74.
// ---------------------------------------------------------------------------------------------------------------------
struct MoeLocalArgs {
    const long long* idx;       // [T * k] expert of every (token, slot) pair, outside [0, E) = dropped
    int *hist;                  // [E][nchunks] scratch
    int *offs, *real;           // [E + 1], [E] out
    int *dest_rank, *dest_row;  // [T * k] out: 0 and the row, or -1 and -1
    int* status;
    const bf16* src;            // [T][h] rows to send
    bf16* x;                    // [rows][h] where they go
    const bf16* y;              // [rows][h] the experts' results
    const float* w;             // [T * k] or null
    bf16* out;                  // [T][h]
    float* d_probs;             // [T * k]
    int T, k, E, cap, h, pad, nchunks;
};
constexpr int LOCAL_CHUNK = 1024;                                    // assignments of a block: eight warps x four rounds of 32

__global__ void __launch_bounds__(256) moe_local_count_kernel(MoeLocalArgs a) {
    extern __shared__ int sh[];
    for (int e = threadIdx.x; e < a.E; e += 256) sh[e] = 0;
    __syncthreads();
    const long long n = (long long)a.T * a.k, base = (long long)blockIdx.x * LOCAL_CHUNK;
    long long e[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long p = base + i * 256 + threadIdx.x;
        e[i] = p < n ? a.idx[p] : -1;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (e[i] >= 0 && e[i] < a.E) atomicAdd(&sh[e[i]], 1);
    __syncthreads();
    for (int x = threadIdx.x; x < a.E; x += 256) a.hist[(long long)x * a.nchunks + blockIdx.x] = sh[x];
}

// Rows in the order of the assignments inside every expert's segment (a stable counting sort).  Every block sums the histograms itself.
__global__ void __launch_bounds__(256) moe_local_assign_kernel(MoeLocalArgs a) {
    extern __shared__ int sh[];
    int *tot = sh, *base = sh + a.E, *cnt = sh + 2 * a.E;             // [E] rows of an expert, [E] first row of this block's, [8][E]
    __shared__ int over;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    for (int e = w; e < a.E; e += 8) {
        int all = 0, before = 0;
        for (int c = l; c < a.nchunks; c += 32) {
            const int x = a.hist[(long long)e * a.nchunks + c];
            all += x;
            if (c < (int)blockIdx.x) before += x;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { all += __shfl_xor_sync(0xffffffffu, all, o); before += __shfl_xor_sync(0xffffffffu, before, o); }
        if (l == 0) { tot[e] = all; base[e] = before; }
    }
    for (int i = threadIdx.x; i < 8 * a.E; i += 256) cnt[i] = 0;
    __syncthreads();
    if (w == 0) {                                                    // segments start at multiples of `pad` rows
        long long run = 0;
        for (int e0 = 0; e0 < a.E; e0 += 32) {
            const int e = e0 + l, n = e < a.E ? tot[e] : 0;
            const long long padded = ((long long)n + a.pad - 1) / a.pad * a.pad;
            long long s = padded;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const long long x = __shfl_up_sync(0xffffffffu, s, o);
                if (l >= o) s += x;
            }
            const long long first = run + s - padded;                // past the capacity the numbers are not used
            if (e < a.E) {
                base[e] += (int)min(first, (long long)a.cap);
                if (blockIdx.x == 0) { a.offs[e] = (int)min(first, (long long)a.cap); a.real[e] = n; }
            }
            run += __shfl_sync(0xffffffffu, s, 31);
        }
        if (l == 0) {
            over = run > a.cap;
            if (blockIdx.x == 0) a.offs[a.E] = (int)min(run, (long long)a.cap);
            if (run > a.cap) atomicCAS(a.status, 0, (9 << 24) | 7);  // receive buffer too small
        }
    }
    __syncthreads();
    if (over && blockIdx.x == 0) {
        for (int e = threadIdx.x; e <= a.E; e += 256) { a.offs[e] = 0; if (e < a.E) a.real[e] = 0; }
    }
    const long long n = (long long)a.T * a.k, p0 = (long long)blockIdx.x * LOCAL_CHUNK + w * 128 + l;
    int ev[4], pos[4], *mine = cnt + w * a.E;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long p = p0 + i * 32, e = p < n ? a.idx[p] : -1;
        ev[i] = e >= 0 && e < a.E ? (int)e : -1;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t same = __match_any_sync(0xffffffffu, ev[i]);
        const int rank = __popc(same & ((1u << l) - 1));
        pos[i] = ev[i] >= 0 ? mine[ev[i]] + rank : 0;
        __syncwarp();
        if (ev[i] >= 0 && rank == 0) mine[ev[i]] += __popc(same);
        __syncwarp();
    }
    __syncthreads();
    for (int e = threadIdx.x; e < a.E; e += 256) {
        int run = base[e];
#pragma unroll
        for (int r = 0; r < 8; ++r) { const int c = cnt[r * a.E + e]; cnt[r * a.E + e] = run; run += c; }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long p = p0 + i * 32;
        if (p >= n) break;
        const bool sent = ev[i] >= 0 && !over;
        a.dest_rank[p] = sent ? 0 : -1;
        a.dest_row[p] = sent ? mine[ev[i]] + pos[i] : -1;
    }
}

__device__ __forceinline__ uint4 times(uint4 v, float w) {
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        h[i] = __floats2bfloat162_rn(f.x * w, f.y * w);
    }
    return v;
}
__device__ __forceinline__ void add_dot(float& s, uint4 x, uint4 y) {
    const __nv_bfloat162 *a = reinterpret_cast<const __nv_bfloat162*>(&x), *b = reinterpret_cast<const __nv_bfloat162*>(&y);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(a[i]), g = __bfloat1622float2(b[i]);
        s += f.x * g.x + f.y * g.y;
    }
}

// Rows of src (times w) to their segments; DOT: also d_probs[t, j] = <y[row of (t, j)], src[t]> (zero for a dropped pair).  Then the padding rows.
template <int KMAX, bool DOT>
__global__ void __launch_bounds__(256) moe_local_push_kernel(MoeLocalArgs a) {
    const int wpb = blockDim.x >> 5, l = threadIdx.x & 31, vecs = a.h / 8;
    const long long warp = (long long)blockIdx.x * wpb + (threadIdx.x >> 5), warps = (long long)gridDim.x * wpb;
    uint4* x = reinterpret_cast<uint4*>(a.x);
    const uint4 *src = reinterpret_cast<const uint4*>(a.src), *y = reinterpret_cast<const uint4*>(a.y);
    for (long long t = warp; t < a.T; t += warps) {
        for (int j0 = 0; j0 < a.k; j0 += KMAX) {
            const int kj = min(KMAX, a.k - j0);
            const int my_row = l < kj ? a.dest_row[t * a.k + j0 + l] : -1;
            const float my_w = a.w != nullptr && l < kj ? a.w[t * a.k + j0 + l] : 1.f;
            int row[KMAX];
            float wt[KMAX], dot[KMAX];
#pragma unroll
            for (int j = 0; j < KMAX; ++j) { row[j] = __shfl_sync(0xffffffffu, my_row, j); wt[j] = __shfl_sync(0xffffffffu, my_w, j); dot[j] = 0.f; }
            constexpr int U = DOT ? 1 : 4;                            // pieces of the row in flight (DOT: with KMAX rows of y each)
            for (int c0 = l; c0 < vecs; c0 += 32 * U) {
                uint4 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = c0 + 32 * u < vecs ? __ldg(src + t * vecs + c0 + 32 * u) : make_uint4(0, 0, 0, 0);
                if (DOT) {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        uint4 r[KMAX];
                        const int c = c0 + 32 * u;
#pragma unroll
                        for (int j = 0; j < KMAX; ++j) r[j] = row[j] >= 0 && c < vecs ? __ldcs(y + (long long)row[j] * vecs + c) : make_uint4(0, 0, 0, 0);
#pragma unroll
                        for (int j = 0; j < KMAX; ++j) add_dot(dot[j], r[j], v[u]);
                    }
                }
#pragma unroll
                for (int j = 0; j < KMAX; ++j)
                    if (row[j] >= 0) {
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            if (c0 + 32 * u < vecs) x[(long long)row[j] * vecs + c0 + 32 * u] = a.w != nullptr ? times(v[u], wt[j]) : v[u];
                    }
            }
            if (DOT) {
#pragma unroll
                for (int j = 0; j < KMAX; ++j) {
                    const float s = warp_sum(dot[j]);
                    if (l == 0 && j < kj) a.d_probs[t * a.k + j0 + j] = row[j] >= 0 ? s : 0.f;
                }
            }
        }
    }
    constexpr int ROWS = 8;                                          // padding rows of a warp at a time
    const int per = (a.pad + ROWS - 1) / ROWS;
    for (long long u = warp; u < (long long)a.E * per; u += warps) {
        const int e = (int)(u / per), lo = a.offs[e] + a.real[e] + (int)(u % per) * ROWS, hi = min(a.offs[e + 1], lo + ROWS);
        for (long long i = (long long)lo * vecs + l; i < (long long)hi * vecs; i += 32) x[i] = make_uint4(0, 0, 0, 0);
    }
}

// out[t] = sum_j w[t, j] y[row of (t, j)] in fp32
constexpr int PULL_SEG = 64;                                         // 16-byte pieces
template <int KMAX>
__global__ void __launch_bounds__(256) moe_local_pull_kernel(MoeLocalArgs a) {
    const int wpb = blockDim.x >> 5, l = threadIdx.x & 31, vecs = a.h / 8;
    const uint4* y = reinterpret_cast<const uint4*>(a.y);
    const int segs = (vecs + PULL_SEG - 1) / PULL_SEG;               // a warp takes a piece of a token: the last round of warps is short
    for (long long at = (long long)blockIdx.x * wpb + (threadIdx.x >> 5); at < (long long)a.T * segs; at += (long long)gridDim.x * wpb) {
        const long long t = at / segs;
        const int c_lo = (int)(at % segs) * PULL_SEG, c_hi = min(vecs, c_lo + PULL_SEG);
        const int my_row = l < a.k ? a.dest_row[t * a.k + l] : -1;
        const float my_w = l < a.k ? (a.w != nullptr ? a.w[t * a.k + l] : 1.f) : 0.f;
        int row[KMAX];
        float wt[KMAX];
#pragma unroll
        for (int j = 0; j < KMAX; ++j) {
            row[j] = __shfl_sync(0xffffffffu, my_row, j);
            wt[j] = row[j] >= 0 ? __shfl_sync(0xffffffffu, my_w, j) : 0.f;
        }
        for (int c = c_lo + l; c < c_hi; c += 32) {
            uint4 v[KMAX];
#pragma unroll
            for (int j = 0; j < KMAX; ++j) v[j] = row[j] >= 0 ? __ldcg(y + (long long)row[j] * vecs + c) : make_uint4(0, 0, 0, 0);
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < KMAX; ++j) {
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = __bfloat1622float2(h[i]);
                    acc[2 * i] += wt[j] * f.x;
                    acc[2 * i + 1] += wt[j] * f.y;
                }
            }
            uint4 o;
            __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
            for (int i = 0; i < 4; ++i) ho[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
            reinterpret_cast<uint4*>(a.out)[t * vecs + c] = o;
        }
    }
}

}  // namespace lmoe

using namespace lmoe;

// The exchange of one rank.  which: 0 route, 1 push (with a.d_probs: and the routing weights' gradient), 2 pull.  h a multiple of 8, rows
// 16-byte aligned.
LMOE_API int lmoe_moe_local(int which, const MoeLocalArgs* ap, int num_sms, cudaStream_t st) {
    const MoeLocalArgs a = *ap;
    if (a.h % 8 != 0) return -2;
    const long long warps = which == 2 ? (long long)a.T * ((a.h / 8 + PULL_SEG - 1) / PULL_SEG) : a.T;
    const int grid = (int)std::min<long long>(std::max<long long>((warps + 7) / 8, 1), (long long)num_sms * 8);
    if (which == 0) {
        if ((size_t)256 * a.E * sizeof(unsigned short) > 200 * 1024) return -4;      // the limit of moe_assign_kernel
        if (a.nchunks > 0) moe_local_count_kernel<<<a.nchunks, 256, a.E * sizeof(int), st>>>(a);
        moe_local_assign_kernel<<<std::max(a.nchunks, 1), 256, 10 * a.E * sizeof(int), st>>>(a);
    } else if (which == 1) {
        if (a.d_probs != nullptr) {
            if (a.k <= 2) moe_local_push_kernel<2, true><<<grid, 256, 0, st>>>(a);
            else if (a.k <= 4) moe_local_push_kernel<4, true><<<grid, 256, 0, st>>>(a);
            else moe_local_push_kernel<8, true><<<grid, 256, 0, st>>>(a);
        } else {
            if (a.k <= 2) moe_local_push_kernel<2, false><<<grid, 256, 0, st>>>(a);
            else if (a.k <= 4) moe_local_push_kernel<4, false><<<grid, 256, 0, st>>>(a);
            else moe_local_push_kernel<8, false><<<grid, 256, 0, st>>>(a);
        }
    } else if (which == 2) {
        if (a.k <= 2) moe_local_pull_kernel<2><<<grid, 256, 0, st>>>(a);
        else if (a.k <= 4) moe_local_pull_kernel<4><<<grid, 256, 0, st>>>(a);
        else if (a.k <= 8) moe_local_pull_kernel<8><<<grid, 256, 0, st>>>(a);
        else if (a.k <= 16) moe_local_pull_kernel<16><<<grid, 256, 0, st>>>(a);
        else return -3;
    } else return -1;
    return (int)cudaGetLastError();
}

// which: 0 exchange, 1 assign, 2 push, 3 zero pads, 4 signal, 5 pull, 6 count
LMOE_API int lmoe_moe_comm(int which, const MoeArgs* ap, int num_sms, cudaStream_t st) {
    const MoeArgs a = *ap;
    if (a.h % 8 != 0 || a.world > 32) return -2;
    const int T = a.k > 0 ? a.n_assign / a.k : 0;
    switch (which) {
    case 0:
        moe_exchange_kernel<<<1, 256, (2 * a.E + a.world) * sizeof(int), st>>>(a);
        break;
    case 1:
        if (a.nchunks > 0) {
            const size_t sm = (size_t)256 * a.E * sizeof(unsigned short);
            if (sm > 200 * 1024) return -4;
            cudaFuncSetAttribute(moe_assign_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
            moe_assign_kernel<<<a.nchunks, 256, sm, st>>>(a);
        }
        break;
    case 6:
        if (a.nchunks > 0) moe_count_kernel<<<a.nchunks, 256, a.E * sizeof(int), st>>>(a);
        break;
    case 2: {
        int grid = (int)std::min<long long>(std::max<long long>((a.n_assign + 7) / 8, 1), (long long)num_sms * 8);
        moe_push_kernel<<<grid, 256, 0, st>>>(a);
        break;
    }
    case 3:
        moe_zero_pads_kernel<<<dim3(a.El, 8), 256, 0, st>>>(a);
        break;
    case 4:
        moe_signal_kernel<<<1, 32, 0, st>>>(a);
        break;
    case 5: {
        int grid = (int)std::min<long long>(std::max<long long>((T + 7) / 8, 1), (long long)num_sms * 8);
        if (a.k <= 2) moe_pull_kernel<2><<<grid, 256, 0, st>>>(a);
        else if (a.k <= 4) moe_pull_kernel<4><<<grid, 256, 0, st>>>(a);
        else if (a.k <= 8) moe_pull_kernel<8><<<grid, 256, 0, st>>>(a);
        else if (a.k <= 16) moe_pull_kernel<16><<<grid, 256, 0, st>>>(a);
        else return -3;
        break;
    }
    default:
        return -1;
    }
    return (int)cudaGetLastError();
}

// d_probs [T, k] fp32 from the gathered expert outputs rows [T * k, h] (bf16) and the combine's output gradient
// d_out [T, h] (bf16); h a multiple of 8, k <= 16.
LMOE_API int lmoe_moe_dprobs(const void* rows, const void* d_out, const int* dest_rank, float* d_probs, int T, int k, int h,
                             int num_sms, cudaStream_t st) {
    if (T <= 0) return 0;
    if (h % 8 != 0 || k <= 0 || k > 16) return -1;
    const int grid = (int)std::min<long long>(((long long)T + 7) / 8, (long long)num_sms * 8);
    const bf16* r = (const bf16*)rows;
    const bf16* d = (const bf16*)d_out;
    if (k <= 2) moe_dprobs_kernel<2><<<grid, 256, 0, st>>>(r, d, dest_rank, d_probs, T, k, h);
    else if (k <= 4) moe_dprobs_kernel<4><<<grid, 256, 0, st>>>(r, d, dest_rank, d_probs, T, k, h);
    else if (k <= 8) moe_dprobs_kernel<8><<<grid, 256, 0, st>>>(r, d, dest_rank, d_probs, T, k, h);
    else moe_dprobs_kernel<16><<<grid, 256, 0, st>>>(r, d, dest_rank, d_probs, T, k, h);
    return (int)cudaGetLastError();
}
