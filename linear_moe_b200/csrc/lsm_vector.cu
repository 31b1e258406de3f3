// Chunked linear attention with a log decay per key channel (GLA, HGRN2), forward and backward, bf16 in / fp32 state.
//
//   S_t = diag(e^{g_t}) S_{t-1} + k_t^T v_t,   o_t = scale * q_t S_t,     g_t in R^{dk} (<= 0)
//
// Replaces fla's chunk_gla Triton kernels that the reference calls (gla/gla.py:94, hgrn2/hgrn2.py:76).  Same
// three-step structure as lsm_scalar.cu (group summaries -> combine -> sweep; no chunk state in HBM).
//
// Per chunk, with b_i the inclusive in-chunk cumulative log decay (a vector per token) and b_m its value at the
// middle token, the operands are rescaled around the middle so that neither factor can overflow:
//   q~_i = q_i e^{b_i - b_m},  k~_j = k_j e^{b_m - b_j}          (q~_i . k~_j = q_i . k_j e^{b_i - b_j} for j <= i)
//   O    = scale [ (q~ k~^T . mask) V + q~ (diag(e^{b_m}) S) ]
//   S   <- diag(e^{b_C - b_m}) [ diag(e^{b_m}) S + k~^T V ]
// The backward uses the same rescaled tiles:
//   dq = e^{b_i - b_m} . scale [ (dO V^T . mask) k~ + dO (diag(e^{b_m}) S)^T ]
//   dk = e^{b_m - b_j} . [ (scale dO V^T . mask)^T q~ + V (diag(e^{b_C - b_m}) dS)^T ]
//   dv = (scale q~ k~^T . mask)^T dO + k~ (diag(e^{b_C - b_m}) dS)
//   dS <- diag(e^{b_m}) [ diag(e^{b_C - b_m}) dS + scale q~^T dO ]
// The gate gradient is d g = reverse-cumsum_t (q . dq - k . dk) per channel (the kernels at the end of this file).
//
// These kernels take 64-wide heads, and 128-wide ones where a group has one chunk; the others are in lsm_vector_tc.cu.
//
// 512 threads, one CTA per SM (two where 64-wide heads have more CTAs than SMs): a warp owns 16 rows of every product and a quarter of its columns (of the state: half or a quarter).  For the
// gates a thread owns two channels and VCH / GR consecutive tokens: running sums stay in registers, the GR groups of tokens meet in one
// small table, and the next chunk's gates and tiles are on their way while this one is worked on.  (With eight warps, single buffers and a
// 64-step running sum in 128 threads the chunks were bound by latency.)
#include "lsm_vector.cuh"
#include "mma_utils.cuh"

namespace lmoe {

constexpr int VCH = 64;
constexpr int VTHREADS = 512;

template <int D> struct VCfg {
    static constexpr int LD = D + 8, PLD = VCH + 8, TILE = VCH * LD;
    static constexpr int S_RB = D / 16, S_CB = 16 / S_RB, S_NT = D / (8 * S_CB);      // the state: row blocks, column blocks, n-tiles per warp
    static constexpr int O_NT = D / 32;                                               // n-tiles of a [VCH x D] product per warp
    static constexpr int PAIRS = D / 2, GR = VTHREADS / PAIRS, RPG = VCH / GR;        // gates: channel pairs, groups of tokens, tokens per group
};

// A thread's place for the gates: channels 2 * pair and 2 * pair + 1 of tokens grp * RPG ..
template <int D> struct Place {
    int pair, grp, row0;
    __device__ __forceinline__ Place() : pair(threadIdx.x % VCfg<D>::PAIRS), grp(threadIdx.x / VCfg<D>::PAIRS) { row0 = grp * VCfg<D>::RPG; }
};
template <int D>
__device__ __forceinline__ void load_gates(const GlaArgs& a, int b, int h, int c, const Place<D>& at, float2 (&g)[VCfg<D>::RPG]) {
    const float* p = a.gk + (((int64_t)b * a.T + (int64_t)c * VCH + at.row0) * a.H + h) * D + 2 * at.pair;
    const int valid = a.T - c * VCH - at.row0;
#pragma unroll
    for (int i = 0; i < VCfg<D>::RPG; ++i)
        g[i] = i < valid ? __ldg(reinterpret_cast<const float2*>(p + (int64_t)i * a.H * D)) : make_float2(0.f, 0.f);
}
template <int D>
__device__ __forceinline__ void save_group_sum(float* sums, const Place<D>& at, const float2 (&g)[VCfg<D>::RPG]) {
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < VCfg<D>::RPG; ++i) { s.x += g[i].x; s.y += g[i].y; }
    *reinterpret_cast<float2*>(sums + at.grp * D + 2 * at.pair) = s;
}
// of groups lo .. hi - 1, this thread's channels
template <int D>
__device__ __forceinline__ float2 groups_sum(const float* sums, const Place<D>& at, int lo, int hi) {
    float2 s = make_float2(0.f, 0.f);
    for (int j = lo; j < hi; ++j) {
        const float2 x = *reinterpret_cast<const float2*>(sums + j * D + 2 * at.pair);
        s.x += x.x; s.y += x.y;
    }
    return s;
}
// g[i] <- b_i - b_m (m: the chunk's middle token), from the gates of the chunk
template <int D>
__device__ __forceinline__ void about_middle(float2 (&g)[VCfg<D>::RPG], const float* sums, const Place<D>& at) {
    constexpr int GR = VCfg<D>::GR, RPG = VCfg<D>::RPG;
    if (at.grp < GR / 2) {
        float2 s = groups_sum<D>(sums, at, at.grp + 1, GR / 2);
#pragma unroll
        for (int i = RPG - 1; i >= 0; --i) {
            const float2 x = g[i];
            g[i] = make_float2(-s.x, -s.y);
            s.x += x.x; s.y += x.y;
        }
    } else {
        float2 s = groups_sum<D>(sums, at, GR / 2, at.grp);
#pragma unroll
        for (int i = 0; i < RPG; ++i) { s.x += g[i].x; s.y += g[i].y; g[i] = s; }
    }
}
// tab[0][d] = e^{b_m}, tab[1][d] = e^{b_C - b_m}
template <int D>
__device__ __forceinline__ void half_decays(float* tab, const float* sums) {
    constexpr int GR = VCfg<D>::GR;
    if (threadIdx.x < 2 * D) {
        const int d = threadIdx.x % D, half = threadIdx.x / D;
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < GR / 2; ++j) s += sums[(half * (GR / 2) + j) * D + d];
        tab[half * D + d] = __expf(s);
    }
}
__device__ __forceinline__ void mul2(bf16* p, float fx, float fy) {
    __nv_bfloat162* x = reinterpret_cast<__nv_bfloat162*>(p);
    const float2 v = __bfloat1622float2(*x);
    *x = __floats2bfloat162_rn(v.x * fx, v.y * fy);
}

template <int NT>
__device__ __forceinline__ void rowscale_acc(float (&acc)[NT][4], float f0, float f1) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) { acc[nt][0] *= f0; acc[nt][1] *= f0; acc[nt][2] *= f1; acc[nt][3] *= f1; }
}
// mask only (no decay): keep (row >= col) if LOWER else (row <= col); multiply by scale; store bf16
template <int LOWER>
__device__ __forceinline__ void mask_store_plain(const float (&acc)[2][4], bf16* P, int pld, int m0, int n0, float scale) {
    const int l = threadIdx.x & 31;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            int r = m0 + (l >> 2) + 8 * hh, c = n0 + nt * 8 + (l & 3) * 2;
            bool k0 = LOWER ? r >= c : r <= c, k1 = LOWER ? r >= c + 1 : r <= c + 1;
            *reinterpret_cast<__nv_bfloat162*>(P + r * pld + c) =
                __floats2bfloat162_rn(k0 ? acc[nt][2 * hh] * scale : 0.f, k1 ? acc[nt][2 * hh + 1] * scale : 0.f);
        }
}
// this warp's [16 x D / 4] block of a tile to global rows
template <int D, int LD>
__device__ __forceinline__ void store_block(const bf16* tile, int m0, int n0, bf16* g, int64_t row_stride, int valid) {
    constexpr int VPR = D / 32;
    const int l = threadIdx.x & 31;
#pragma unroll
    for (int i = l; i < 16 * VPR; i += 32) {
        const int r = m0 + i / VPR, c = n0 + (i % VPR) * 8;
        if (r < valid) *reinterpret_cast<uint4*>(g + (int64_t)r * row_stride + c) = *reinterpret_cast<const uint4*>(tile + r * LD + c);
    }
}
// Write diag(f) * S (registers, rows r and r + 8) as bf16 into Sb.
template <int D>
__device__ __forceinline__ void store_state_scaled(const float (&acc)[VCfg<D>::S_NT][4], bf16* Sb, int s_m0, int s_n0, float f0, float f1) {
    using C = VCfg<D>;
    const int l = threadIdx.x & 31;
    const int r = s_m0 + (l >> 2), c = s_n0 + (l & 3) * 2;
#pragma unroll
    for (int nt = 0; nt < C::S_NT; ++nt) {
        *reinterpret_cast<__nv_bfloat162*>(Sb + r * C::LD + c + nt * 8) = __floats2bfloat162_rn(acc[nt][0] * f0, acc[nt][1] * f0);
        *reinterpret_cast<__nv_bfloat162*>(Sb + (r + 8) * C::LD + c + nt * 8) = __floats2bfloat162_rn(acc[nt][2] * f1, acc[nt][3] * f1);
    }
}
template <int D>
__device__ __forceinline__ void load_state_regs(const float* src, float (&acc)[VCfg<D>::S_NT][4], int s_m0, int s_n0) {
    using C = VCfg<D>;
    const int l = threadIdx.x & 31;
    const int r = s_m0 + (l >> 2), cc = s_n0 + (l & 3) * 2;
#pragma unroll
    for (int nt = 0; nt < C::S_NT; ++nt) {
        float2 x = *reinterpret_cast<const float2*>(src + (int64_t)r * D + cc + nt * 8);
        float2 y = *reinterpret_cast<const float2*>(src + (int64_t)(r + 8) * D + cc + nt * 8);
        acc[nt][0] = x.x; acc[nt][1] = x.y; acc[nt][2] = y.x; acc[nt][3] = y.y;
    }
}

// ---------------------------------------------------------------------------------------------
// 1. group summaries.  REV = 0: S <- diag(e^{b_C}) S + (K e^{b_C - b})^T V (ascending chunks)
//                      REV = 1: dS <- diag(e^{b_C}) dS + (Q e^{b} scale)^T dO (descending chunks)
// ---------------------------------------------------------------------------------------------
template <int D, int REV, int CTAS>
__global__ void __launch_bounds__(VTHREADS, CTAS) gla_state_scan_kernel(GlaArgs a) {
    using C = VCfg<D>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16* Xs = reinterpret_cast<bf16*>(smem_raw);                  // [2][VCH][LD]
    bf16* Ys = Xs + 2 * C::TILE;                                   // [2][VCH][LD]
    float* sums = reinterpret_cast<float*>(Ys + 2 * C::TILE);      // [2][GR][D]
    const int grp = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int nchunks = (a.T + VCH - 1) / VCH;
    const int c_lo = grp * a.cpg, c_hi = min(nchunks, c_lo + a.cpg), n = c_hi - c_lo;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int s_m0 = 16 * (w % C::S_RB), s_n0 = (w / C::S_RB) * (C::S_NT * 8);
    const int r = s_m0 + (l >> 2);
    const Place<D> at;
    const bf16* xg = REV ? a.q + b * a.qs_b + h * a.qs_h : a.k + b * a.ks_b + h * a.ks_h;
    const int64_t xs_t = REV ? a.qs_t : a.ks_t;
    const bf16* yg = REV ? a.d_o + ((int64_t)b * a.T * a.H + h) * D : a.v + b * a.vs_b + h * a.vs_h;
    const int64_t ys_t = REV ? (int64_t)a.H * D : a.vs_t;
    auto chunk_at = [&](int i) { return REV ? c_hi - 1 - i : c_lo + i; };
    auto issue = [&](int i) {
        const int c = chunk_at(i);
        load_tile_async<VCH, D, C::LD>(Xs + (i & 1) * C::TILE, xg + (int64_t)c * VCH * xs_t, xs_t, a.T - c * VCH);
        load_tile_async<VCH, D, C::LD>(Ys + (i & 1) * C::TILE, yg + (int64_t)c * VCH * ys_t, ys_t, a.T - c * VCH);
    };
    float acc[C::S_NT][4];
    zero_acc<C::S_NT>(acc);
    float gs0 = 0.f, gs1 = 0.f;                                    // running group decay of rows r, r + 8
    float2 g[C::RPG];
    if (n > 0) { issue(0); load_gates<D>(a, b, h, chunk_at(0), at, g); save_group_sum<D>(sums, at, g); }
    cp_async_commit();
    for (int i = 0; i < n; ++i) {
        bf16 *X = Xs + (i & 1) * C::TILE, *Y = Ys + (i & 1) * C::TILE;
        float* sm = sums + (i & 1) * C::GR * D;
        cp_async_wait<0>();
        __syncthreads();                                           // tiles and group sums of this chunk visible; the other stage is free
        if (i + 1 < n) issue(i + 1);
        cp_async_commit();
        if (REV) {                                                 // q e^{b} scale
            float2 s = groups_sum<D>(sm, at, 0, at.grp);
#pragma unroll
            for (int e = 0; e < C::RPG; ++e) {
                s.x += g[e].x; s.y += g[e].y;
                mul2(X + (at.row0 + e) * C::LD + 2 * at.pair, __expf(s.x) * a.scale, __expf(s.y) * a.scale);
            }
        } else {                                                   // k e^{b_C - b}
            float2 s = groups_sum<D>(sm, at, at.grp + 1, C::GR);
#pragma unroll
            for (int e = C::RPG - 1; e >= 0; --e) {
                mul2(X + (at.row0 + e) * C::LD + 2 * at.pair, __expf(s.x), __expf(s.y));
                s.x += g[e].x; s.y += g[e].y;
            }
        }
        if (i + 1 < n) load_gates<D>(a, b, h, chunk_at(i + 1), at, g);
        float t0 = 0.f, t1 = 0.f;
#pragma unroll
        for (int j = 0; j < C::GR; ++j) { t0 += sm[j * D + r]; t1 += sm[j * D + r + 8]; }
        rowscale_acc<C::S_NT>(acc, __expf(t0), __expf(t1));
        gs0 += t0; gs1 += t1;
        __syncthreads();
        warp_gemm<C::S_NT, VCH, true, true>(acc, X, C::LD, s_m0, Y, C::LD, s_n0);
        if (i + 1 < n) save_group_sum<D>(sums + ((i + 1) & 1) * C::GR * D, at, g);
    }
    float* out = a.states + ((int64_t)bh * a.G + grp) * D * D;
    const int cc = s_n0 + (l & 3) * 2;
#pragma unroll
    for (int nt = 0; nt < C::S_NT; ++nt) {
        *reinterpret_cast<float2*>(out + (int64_t)r * D + cc + nt * 8) = make_float2(acc[nt][0], acc[nt][1]);
        *reinterpret_cast<float2*>(out + (int64_t)(r + 8) * D + cc + nt * 8) = make_float2(acc[nt][2], acc[nt][3]);
    }
    if (a.gdecay != nullptr && s_n0 == 0 && (l & 3) == 0) {
        float* gd = a.gdecay + ((int64_t)bh * a.G + grp) * D;
        gd[r] = gs0;
        gd[r + 8] = gs1;
    }
}

// 2. combine with a per-row (key channel) decay; a thread owns V consecutive values of the state
template <int REV, int V>
__global__ void __launch_bounds__(256) gla_combine_kernel(float* __restrict__ states, const float* __restrict__ gdecay, const float* __restrict__ seed,
                                                          float* __restrict__ final_out, int G, int D) {
    const int bh = blockIdx.y;
    const int e = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    const int DD = D * D;
    if (e >= DD) return;
    const int row = e / D;
    Values<V> carry;
    if (seed != nullptr) carry = load_values<V>(seed + (int64_t)bh * DD + e);
    else
#pragma unroll
        for (int c = 0; c < V; ++c) carry.x[c] = 0.f;
    // batches of loads in flight together (a load per group that waits for the previous store is bound by memory latency)
    constexpr int NB = 8;
    for (int i0 = 0; i0 < G; i0 += NB) {
        Values<V> m[NB];
        float dec[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j)
            if (i0 + j < G) {
                const int g = REV ? G - 1 - (i0 + j) : i0 + j;
                m[j] = load_values<V>(states + ((int64_t)bh * G + g) * DD + e);
                dec[j] = __expf(gdecay[((int64_t)bh * G + g) * D + row]);
            }
#pragma unroll
        for (int j = 0; j < NB; ++j)
            if (i0 + j < G) {
                const int g = REV ? G - 1 - (i0 + j) : i0 + j;
                *reinterpret_cast<Values<V>*>(states + ((int64_t)bh * G + g) * DD + e) = carry;
#pragma unroll
                for (int c = 0; c < V; ++c) carry.x[c] = dec[j] * carry.x[c] + m[j].x[c];
            }
    }
    if (final_out != nullptr) *reinterpret_cast<Values<V>*>(final_out + (int64_t)bh * DD + e) = carry;
}

// ---------------------------------------------------------------------------------------------
// 3a. forward output (MODE 0) / backward dq (MODE 1): forward sweep carrying S.
// ---------------------------------------------------------------------------------------------
template <int D, int MODE, int CTAS>
__global__ void __launch_bounds__(VTHREADS, CTAS) gla_fwd_sweep_kernel(GlaArgs a) {
    using C = VCfg<D>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16* tiles = reinterpret_cast<bf16*>(smem_raw);               // [2] x { q (mode 0) | dO (mode 1), k, v }
    bf16* Sb = tiles + 6 * C::TILE;
    bf16* P = Sb + D * C::LD;
    float* sums = reinterpret_cast<float*>(P + VCH * C::PLD);      // [2][GR][D]
    float* tabs = sums + 2 * C::GR * D;                            // [2][2][D]
    const int grp = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int nchunks = (a.T + VCH - 1) / VCH;
    const int c_lo = grp * a.cpg, c_hi = min(nchunks, c_lo + a.cpg);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int s_m0 = 16 * (w % C::S_RB), s_n0 = (w / C::S_RB) * (C::S_NT * 8), sr = s_m0 + (l >> 2);
    const int m0 = 16 * (w & 3), o_n0 = (w >> 2) * (D / 4), a_n0 = (w >> 2) * 16;
    const Place<D> at;
    const bf16* qg = MODE == 0 ? a.q + b * a.qs_b + h * a.qs_h : a.d_o + ((int64_t)b * a.T * a.H + h) * D;
    const int64_t qst = MODE == 0 ? a.qs_t : (int64_t)a.H * D;
    const bf16* kg = a.k + b * a.ks_b + h * a.ks_h;
    const bf16* vg = a.v + b * a.vs_b + h * a.vs_h;
    bf16* og; int64_t ost;
    if (MODE == 0) { og = a.o + ((int64_t)b * a.T * a.H + h) * D; ost = (int64_t)a.H * D; }
    else { og = a.dq + b * a.dqs_b + h * a.dqs_h; ost = a.dqs_t; }
    auto issue = [&](int c) {
        const int valid = a.T - c * VCH;
        bf16* t = tiles + ((c - c_lo) & 1) * 3 * C::TILE;
        load_tile_async<VCH, D, C::LD>(t, qg + (int64_t)c * VCH * qst, qst, valid);
        load_tile_async<VCH, D, C::LD>(t + C::TILE, kg + (int64_t)c * VCH * a.ks_t, a.ks_t, valid);
        load_tile_async<VCH, D, C::LD>(t + 2 * C::TILE, vg + (int64_t)c * VCH * a.vs_t, a.vs_t, valid);
    };
    float acc_s[C::S_NT][4];
    load_state_regs<D>(a.states + ((int64_t)bh * a.G + grp) * D * D, acc_s, s_m0, s_n0);
    float2 g[C::RPG], up[MODE == 1 ? C::RPG : 1];                  // up: e^{b_i - b_m} for dq's epilogue
    if (c_lo < c_hi) { issue(c_lo); load_gates<D>(a, b, h, c_lo, at, g); save_group_sum<D>(sums, at, g); }
    cp_async_commit();
    __syncthreads();
    if (c_lo < c_hi) half_decays<D>(tabs, sums);
    for (int c = c_lo; c < c_hi; ++c) {
        const int s = (c - c_lo) & 1, valid = a.T - c * VCH;
        bf16 *Tq = tiles + s * 3 * C::TILE, *Tk = Tq + C::TILE, *Tv = Tk + C::TILE;
        const float *sm = sums + s * C::GR * D, *tab = tabs + s * 2 * D;
        float *sm_next = sums + (s ^ 1) * C::GR * D, *tab_next = tabs + (s ^ 1) * 2 * D;
        cp_async_wait<0>();
        __syncthreads();                                            // tiles and tables of this chunk visible; the other stage is free
        if (c + 1 < c_hi) issue(c + 1);
        cp_async_commit();
        about_middle<D>(g, sm, at);
#pragma unroll
        for (int i = 0; i < C::RPG; ++i) {
            const int o = (at.row0 + i) * C::LD + 2 * at.pair;
            if (MODE == 0) mul2(Tq + o, __expf(g[i].x), __expf(g[i].y));            // q~ (in mode 1 the tile is dO, unscaled)
            else up[i] = make_float2(__expf(g[i].x), __expf(g[i].y));
            mul2(Tk + o, __expf(-g[i].x), __expf(-g[i].y));                         // k~
        }
        const float em0 = tab[sr], em1 = tab[sr + 8], ee0 = tab[D + sr], ee1 = tab[D + sr + 8];
        rowscale_acc<C::S_NT>(acc_s, em0, em1);                                     // e^{b_m} S
        store_state_scaled<D>(acc_s, Sb, s_m0, s_n0, 1.f, 1.f);
        if (c + 1 < c_hi) load_gates<D>(a, b, h, c + 1, at, g);
        __syncthreads();
        float acc_o[C::O_NT][4];
        zero_acc<C::O_NT>(acc_o);
        {
            float acc_a[2][4];
            zero_acc<2>(acc_a);
            if (MODE == 0) {
                warp_gemm<C::O_NT, D, false, true>(acc_o, Tq, C::LD, m0, Sb, C::LD, o_n0);          // q~ (e^{b_m} S)
                if (a_n0 <= m0) warp_gemm<2, D, false, false>(acc_a, Tq, C::LD, m0, Tk, C::LD, a_n0);     // q~ k~^T
            } else {
                warp_gemm<C::O_NT, D, false, false>(acc_o, Tq, C::LD, m0, Sb, C::LD, o_n0);         // dO (e^{b_m} S)^T
                if (a_n0 <= m0) warp_gemm<2, D, false, false>(acc_a, Tq, C::LD, m0, Tv, C::LD, a_n0);     // dO V^T
            }
            rowscale_acc<C::O_NT>(acc_o, a.scale, a.scale);
            if (a_n0 <= m0) mask_store_plain<1>(acc_a, P, C::PLD, m0, a_n0, a.scale);               // (the blocks above are never read)
        }
        if (c + 1 < c_hi) save_group_sum<D>(sm_next, at, g);
        __syncthreads();
        if (c + 1 < c_hi) half_decays<D>(tab_next, sm_next);
        const bf16* X = MODE == 0 ? Tv : Tk;
        for (int k0 = 0; k0 <= m0; k0 += 16) warp_gemm<C::O_NT, 16, false, true>(acc_o, P + k0, C::PLD, m0, X + k0 * C::LD, C::LD, o_n0);   // A V | dA k~
        store_acc_bf16<C::O_NT>(acc_o, Tq, C::LD, m0, o_n0);                        // (nobody reads Tq any more)
        // state: S <- e^{b_C - b_m} [ e^{b_m} S + k~^T V ]
        warp_gemm<C::S_NT, VCH, true, true>(acc_s, Tk, C::LD, s_m0, Tv, C::LD, s_n0);
        rowscale_acc<C::S_NT>(acc_s, ee0, ee1);
        if (MODE == 0) {
            __syncwarp();
            store_block<D, C::LD>(Tq, m0, o_n0, og + (int64_t)c * VCH * ost, ost, valid);
        } else {
            __syncthreads();                                        // dq = e^{b_i - b_m} . (...), by the threads that have the factors
#pragma unroll
            for (int i = 0; i < C::RPG; ++i) {
                const int row = at.row0 + i;
                const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(Tq + row * C::LD + 2 * at.pair));
                if (row < valid)
                    *reinterpret_cast<__nv_bfloat162*>(og + ((int64_t)c * VCH + row) * ost + 2 * at.pair) = __floats2bfloat162_rn(x.x * up[i].x, x.y * up[i].y);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// 3b. backward dk, dv: reverse sweep carrying dS.
// ---------------------------------------------------------------------------------------------
template <int D, int CTAS>
__global__ void __launch_bounds__(VTHREADS, CTAS) gla_bwd_dkv_kernel(GlaArgs a) {
    using C = VCfg<D>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16* tiles = reinterpret_cast<bf16*>(smem_raw);                // [2] x { q, k, v, dO }
    bf16* Sb = tiles + 8 * C::TILE;                                 // diag(e^{b_C - b_m}) dS
    bf16* P1 = Sb + D * C::LD;
    bf16* P2 = P1 + VCH * C::PLD;
    float* sums = reinterpret_cast<float*>(P2 + VCH * C::PLD);      // [2][GR][D]
    float* tabs = sums + 2 * C::GR * D;                             // [2][2][D]
    const int grp = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int nchunks = (a.T + VCH - 1) / VCH;
    const int c_lo = grp * a.cpg, c_hi = min(nchunks, c_lo + a.cpg);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int s_m0 = 16 * (w % C::S_RB), s_n0 = (w / C::S_RB) * (C::S_NT * 8), sr = s_m0 + (l >> 2);
    const int m0 = 16 * (w & 3), o_n0 = (w >> 2) * (D / 4), a_n0 = (w >> 2) * 16;
    const Place<D> at;
    const bf16* qg = a.q + b * a.qs_b + h * a.qs_h;
    const bf16* kg = a.k + b * a.ks_b + h * a.ks_h;
    const bf16* vg = a.v + b * a.vs_b + h * a.vs_h;
    const bf16* gg = a.d_o + ((int64_t)b * a.T * a.H + h) * D;
    const int64_t gst = (int64_t)a.H * D;
    bf16* dkg = a.dk + b * a.dks_b + h * a.dks_h;
    bf16* dvg = a.dv + b * a.dvs_b + h * a.dvs_h;
    auto issue = [&](int c) {
        const int valid = a.T - c * VCH;
        bf16* t = tiles + ((c_hi - 1 - c) & 1) * 4 * C::TILE;
        load_tile_async<VCH, D, C::LD>(t, qg + (int64_t)c * VCH * a.qs_t, a.qs_t, valid);
        load_tile_async<VCH, D, C::LD>(t + C::TILE, kg + (int64_t)c * VCH * a.ks_t, a.ks_t, valid);
        load_tile_async<VCH, D, C::LD>(t + 2 * C::TILE, vg + (int64_t)c * VCH * a.vs_t, a.vs_t, valid);
        load_tile_async<VCH, D, C::LD>(t + 3 * C::TILE, gg + (int64_t)c * VCH * gst, gst, valid);
    };
    float acc_s[C::S_NT][4];
    load_state_regs<D>(a.states + ((int64_t)bh * a.G + grp) * D * D, acc_s, s_m0, s_n0);
    float2 g[C::RPG], dn[C::RPG];                                   // dn: e^{b_m - b_j} for dk's epilogue
    if (c_lo < c_hi) { issue(c_hi - 1); load_gates<D>(a, b, h, c_hi - 1, at, g); save_group_sum<D>(sums, at, g); }
    cp_async_commit();
    __syncthreads();
    if (c_lo < c_hi) half_decays<D>(tabs, sums);
    for (int c = c_hi - 1; c >= c_lo; --c) {
        const int s = (c_hi - 1 - c) & 1, valid = a.T - c * VCH;
        bf16 *Tq = tiles + s * 4 * C::TILE, *Tk = Tq + C::TILE, *Tv = Tk + C::TILE, *Tg = Tv + C::TILE;
        const float *sm = sums + s * C::GR * D, *tab = tabs + s * 2 * D;
        float *sm_next = sums + (s ^ 1) * C::GR * D, *tab_next = tabs + (s ^ 1) * 2 * D;
        cp_async_wait<0>();
        __syncthreads();
        if (c > c_lo) issue(c - 1);
        cp_async_commit();
        about_middle<D>(g, sm, at);
#pragma unroll
        for (int i = 0; i < C::RPG; ++i) {
            const int o = (at.row0 + i) * C::LD + 2 * at.pair;
            mul2(Tq + o, __expf(g[i].x), __expf(g[i].y));
            dn[i] = make_float2(__expf(-g[i].x), __expf(-g[i].y));
            mul2(Tk + o, dn[i].x, dn[i].y);
        }
        const float em0 = tab[sr], em1 = tab[sr + 8], ee0 = tab[D + sr], ee1 = tab[D + sr + 8];
        store_state_scaled<D>(acc_s, Sb, s_m0, s_n0, ee0, ee1);
        __syncthreads();
        float acc_dv[C::O_NT][4], acc_dk[C::O_NT][4];
        zero_acc<C::O_NT>(acc_dv);
        zero_acc<C::O_NT>(acc_dk);
        if (a_n0 >= m0) {
            float acc_a[2][4];
            zero_acc<2>(acc_a);
            warp_gemm<2, D, false, false>(acc_a, Tk, C::LD, m0, Tq, C::LD, a_n0);             // k~ q~^T
            mask_store_plain<0>(acc_a, P1, C::PLD, m0, a_n0, a.scale);
            zero_acc<2>(acc_a);
            warp_gemm<2, D, false, false>(acc_a, Tv, C::LD, m0, Tg, C::LD, a_n0);             // V dO^T
            mask_store_plain<0>(acc_a, P2, C::PLD, m0, a_n0, a.scale);
        }
        warp_gemm<C::O_NT, D, false, true>(acc_dv, Tk, C::LD, m0, Sb, C::LD, o_n0);           // k~ (e^{b_C-b_m} dS)
        warp_gemm<C::O_NT, D, false, false>(acc_dk, Tv, C::LD, m0, Sb, C::LD, o_n0);          // V (e^{b_C-b_m} dS)^T
        if (c > c_lo) { load_gates<D>(a, b, h, c - 1, at, g); save_group_sum<D>(sm_next, at, g); }
        __syncthreads();
        if (c > c_lo) half_decays<D>(tab_next, sm_next);
        for (int k0 = m0; k0 < VCH; k0 += 16) {
            warp_gemm<C::O_NT, 16, false, true>(acc_dv, P1 + k0, C::PLD, m0, Tg + k0 * C::LD, C::LD, o_n0);      // Abar dO
            warp_gemm<C::O_NT, 16, false, true>(acc_dk, P2 + k0, C::PLD, m0, Tq + k0 * C::LD, C::LD, o_n0);      // Bbar q~
        }
        store_acc_bf16<C::O_NT>(acc_dv, Tv, C::LD, m0, o_n0);                                 // (K and V have been read)
        store_acc_bf16<C::O_NT>(acc_dk, Tk, C::LD, m0, o_n0);
        // dS <- e^{b_m} [ e^{b_C - b_m} dS + scale q~^T dO ]: fold `scale` by scaling around the product
        rowscale_acc<C::S_NT>(acc_s, ee0 / a.scale, ee1 / a.scale);
        warp_gemm<C::S_NT, VCH, true, true>(acc_s, Tq, C::LD, s_m0, Tg, C::LD, s_n0);
        rowscale_acc<C::S_NT>(acc_s, em0 * a.scale, em1 * a.scale);
        __syncwarp();
        store_block<D, C::LD>(Tv, m0, o_n0, dvg + (int64_t)c * VCH * a.dvs_t, a.dvs_t, valid);
        __syncthreads();                                            // dk = e^{b_m - b_j} . (...), by the threads that have the factors
#pragma unroll
        for (int i = 0; i < C::RPG; ++i) {
            const int row = at.row0 + i;
            const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(Tk + row * C::LD + 2 * at.pair));
            if (row < valid)
                *reinterpret_cast<__nv_bfloat162*>(dkg + ((int64_t)c * VCH + row) * a.dks_t + 2 * at.pair) = __floats2bfloat162_rn(x.x * dn[i].x, x.y * dn[i].y);
        }
    }
}

template <int D> constexpr size_t gla_smem_scan() { return (size_t)4 * VCfg<D>::TILE * 2 + (size_t)2 * VCfg<D>::GR * D * 4; }
template <int D> constexpr size_t gla_smem_sweep() {
    return (size_t)6 * VCfg<D>::TILE * 2 + (size_t)D * VCfg<D>::LD * 2 + (size_t)VCH * VCfg<D>::PLD * 2 + (size_t)(2 * VCfg<D>::GR + 4) * D * 4;
}
template <int D> constexpr size_t gla_smem_dkv() {
    return (size_t)8 * VCfg<D>::TILE * 2 + (size_t)D * VCfg<D>::LD * 2 + (size_t)2 * VCH * VCfg<D>::PLD * 2 + (size_t)(2 * VCfg<D>::GR + 4) * D * 4;
}

}  // namespace lmoe

using namespace lmoe;

template <int D, int CTAS>
static int gla_launch(int which, const GlaArgs& a, cudaStream_t st) {
    dim3 grid(a.G, a.B * a.H);
#define GLAUNCH(KERNEL, SMEM)                                                                              \
    do {                                                                                                   \
        int rc = (int)cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(SMEM)); \
        if (rc) return rc;                                                                                 \
        KERNEL<<<grid, VTHREADS, SMEM, st>>>(a);                                                           \
    } while (0)
    if (which == 0) GLAUNCH((gla_state_scan_kernel<D, 0, CTAS>), gla_smem_scan<D>());
    else if (which == 1) GLAUNCH((gla_state_scan_kernel<D, 1, CTAS>), gla_smem_scan<D>());
    else if (which == 2) GLAUNCH((gla_fwd_sweep_kernel<D, 0, CTAS>), gla_smem_sweep<D>());
    else if (which == 3) GLAUNCH((gla_fwd_sweep_kernel<D, 1, CTAS>), gla_smem_sweep<D>());
    else if (which == 4) GLAUNCH((gla_bwd_dkv_kernel<D, CTAS>), gla_smem_dkv<D>());
    else return -1;
#undef GLAUNCH
    return (int)cudaGetLastError();
}

static int gla_launch(int which, int D, const GlaArgs& a, lvt::Maps& maps, cudaStream_t st) {
    if (D == 128) return a.wide ? lvt::launch(which, a, maps, st) : gla_launch<128, 1>(which, a, st);
    if (D != 64) return -2;
    // 64-wide heads, more CTAs than SMs: two per SM with 64 registers a thread overlap each other's steps.  Outputs, one and two per SM:
    // 64 x 256 tokens of 16 heads 216 and 185 us, 64 x 128 144 and 123, 32 x 64 56 and 50; where every CTA has an SM to itself the
    // registers are worth more (8 x 2048 of 8 heads, 128 CTAs: 81 and 91).
    return (long long)a.G * a.B * a.H > sm_count() ? gla_launch<64, 2>(which, a, st) : gla_launch<64, 1>(which, a, st);
}

// which: 0 forward state scan, 1 reverse state scan, 2 forward output, 3 backward dq, 4 backward dk/dv
LMOE_API int lmoe_gla_launch(int which, int D, const GlaArgs* ap, cudaStream_t st) {
    lvt::Maps maps;
    return gla_launch(which, D, *ap, maps, st);
}

LMOE_API int lmoe_gla_combine(int rev, float* states, const float* gdecay, const float* seed, float* final_out, int BH,
                              int G, int D, cudaStream_t st) {
    // Four values a thread once that leaves a block for every SM.  Pairs x groups, forward, one and four values: 64 x 2 16.5 and 8.3 us, 32 x 4 10.4 and
    // 6.3, 16 x 9 9.0 and 6.3, 9 x 16 8.5 and 8.4, 4 x 37 8.7 and 8.9 (reverse 8.4 and 12.4), 1 x 148 12.6 and 25.4.
    const int v = (long long)BH * (D * D / 1024) >= sm_count() ? 4 : 1;
    dim3 grid((D * D / v + 255) / 256, BH);
    if (rev) {
        if (v == 4) gla_combine_kernel<1, 4><<<grid, 256, 0, st>>>(states, gdecay, seed, final_out, G, D);
        else gla_combine_kernel<1, 1><<<grid, 256, 0, st>>>(states, gdecay, seed, final_out, G, D);
    } else {
        if (v == 4) gla_combine_kernel<0, 4><<<grid, 256, 0, st>>>(states, gdecay, seed, final_out, G, D);
        else gla_combine_kernel<0, 1><<<grid, 256, 0, st>>>(states, gdecay, seed, final_out, G, D);
    }
    return (int)cudaGetLastError();
}

// Summaries, combine and outputs of a forward call: the three launches behind one host call.
LMOE_API int lmoe_gla_forward(int D, const GlaArgs* ap, const float* seed, float* final_out, cudaStream_t st) {
    lvt::Maps maps;
    int rc = gla_launch(0, D, *ap, maps, st);
    if (rc) return rc;
    rc = lmoe_gla_combine(0, ap->states, ap->gdecay, seed, final_out, ap->B * ap->H, ap->G, D, st);
    if (rc) return rc;
    return gla_launch(2, D, *ap, maps, st);
}

// dq (of `ap`, with the entering states), summaries of the state's gradient, combine, dk and dv (of `bp`, whose states are the gradient's): four launches
// behind one host call.  gdecay: of the forward call.
LMOE_API int lmoe_gla_backward(int D, const GlaArgs* ap, const GlaArgs* bp, const float* gdecay, const float* seed, float* dinit, cudaStream_t st) {
    lvt::Maps maps;
    int rc = gla_launch(3, D, *ap, maps, st);
    if (rc) return rc;
    rc = gla_launch(1, D, *bp, maps, st);
    if (rc) return rc;
    rc = lmoe_gla_combine(1, bp->states, gdecay, seed, dinit, bp->B * bp->H, bp->G, D, st);
    if (rc) return rc;
    return gla_launch(4, D, *bp, maps, st);
}

// ---------------------------------------------------------------------------------------------------------------
// Gradient of the vector log-gates: dg[b,t,h,d] = sum_{i >= t} (q . dq - k . dk)[b,i,h,d]  (reverse cumulative sum
// over time per channel).  One launch, 12 bytes of traffic per element, where a cluster of CTAs per head covers the tokens
// (gla_dg_kernel); otherwise two launches over segments of 256 tokens: per-segment channel sums, then every segment walks its tokens
// backwards starting from the sum of the later segments, 20 bytes per element.
// ---------------------------------------------------------------------------------------------------------------
namespace lmoe {
constexpr int DG_SEG = 256;
struct DgArgs {
    const bf16 *q, *k, *dq, *dk;
    int64_t qs_b, qs_t, qs_h, ks_b, ks_t, ks_h, dqs_b, dqs_t, dqs_h, dks_b, dks_t, dks_h;
    float* dg;            // [B,T,H,D] contiguous
    float* segsum;        // [B*H, nseg, D]
    int B, T, H, D, nseg; // nseg 0: gla_dg_kernel
};
// q*dq - k*dk for eight consecutive channels of one token (16-byte loads; the pitches are multiples of 8 elements)
__device__ __forceinline__ void dg_term8(const DgArgs& a, int b, int t, int h, int d, float (&o)[8]) {
    const uint4 q4 = __ldg(reinterpret_cast<const uint4*>(a.q + b * a.qs_b + (int64_t)t * a.qs_t + h * a.qs_h + d));
    const uint4 k4 = __ldg(reinterpret_cast<const uint4*>(a.k + b * a.ks_b + (int64_t)t * a.ks_t + h * a.ks_h + d));
    const uint4 dq4 = __ldg(reinterpret_cast<const uint4*>(a.dq + b * a.dqs_b + (int64_t)t * a.dqs_t + h * a.dqs_h + d));
    const uint4 dk4 = __ldg(reinterpret_cast<const uint4*>(a.dk + b * a.dks_b + (int64_t)t * a.dks_t + h * a.dks_h + d));
    const __nv_bfloat162* q2 = reinterpret_cast<const __nv_bfloat162*>(&q4);
    const __nv_bfloat162* k2 = reinterpret_cast<const __nv_bfloat162*>(&k4);
    const __nv_bfloat162* dq2 = reinterpret_cast<const __nv_bfloat162*>(&dq4);
    const __nv_bfloat162* dk2 = reinterpret_cast<const __nv_bfloat162*>(&dk4);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 fq = __bfloat1622float2(q2[i]), fk = __bfloat1622float2(k2[i]);
        const float2 fdq = __bfloat1622float2(dq2[i]), fdk = __bfloat1622float2(dk2[i]);
        o[2 * i] = fq.x * fdq.x - fk.x * fdk.x;
        o[2 * i + 1] = fq.y * fdq.y - fk.y * fdk.y;
    }
}

// The two launches: grid (nseg, B*H), 256 threads.  D / 8 threads cover the channels of one token with 16-byte accesses;
// the 256 / (D / 8) thread groups each own a contiguous run of DG_SEG / groups tokens of the segment.
// 1. per-segment sums of the terms
__global__ void __launch_bounds__(256) gla_dg_segsum_kernel(DgArgs a) {
    __shared__ float part[32][129];                                    // [group][channel], D <= 128
    const int seg = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int tpr = a.D / 8, groups = 256 / tpr, L = DG_SEG / groups;
    const int grp = threadIdx.x / tpr, d = (threadIdx.x % tpr) * 8;
    const int t0 = seg * DG_SEG + grp * L, t1 = min(a.T, t0 + L);
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int t = t0; t < t1; ++t) {
        float o[8];
        dg_term8(a, b, t, h, d, o);
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] += o[i];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) part[grp][d + i] = s[i];
    __syncthreads();
    if (threadIdx.x < a.D) {
        float tot = 0.f;
        for (int g2 = 0; g2 < groups; ++g2) tot += part[g2][threadIdx.x];
        a.segsum[((int64_t)bh * a.nseg + seg) * a.D + threadIdx.x] = tot;
    }
}
// 2. running suffix sums: later segments from the table, later token runs of this segment through shared memory, then
//    the run's own tokens from last to first (re-read; they are in L2 from the first pass of this CTA)
__global__ void __launch_bounds__(256) gla_dg_scan_kernel(DgArgs a) {
    __shared__ float part[32][129];
    const int seg = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int tpr = a.D / 8, groups = 256 / tpr, L = DG_SEG / groups;
    const int grp = threadIdx.x / tpr, d = (threadIdx.x % tpr) * 8;
    const int t0 = seg * DG_SEG + grp * L, t1 = min(a.T, t0 + L);
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int t = t0; t < t1; ++t) {
        float o[8];
        dg_term8(a, b, t, h, d, o);
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] += o[i];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) part[grp][d + i] = s[i];
    __syncthreads();
    float run[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float r = 0.f;
        for (int s2 = a.nseg - 1; s2 > seg; --s2) r += a.segsum[((int64_t)bh * a.nseg + s2) * a.D + d + i];
        for (int g2 = groups - 1; g2 > grp; --g2) r += part[g2][d + i];
        run[i] = r;
    }
    for (int t = t1 - 1; t >= t0; --t) {
        float o[8];
        dg_term8(a, b, t, h, d, o);
#pragma unroll
        for (int i = 0; i < 8; ++i) run[i] += o[i];
        float4* dst = reinterpret_cast<float4*>(a.dg + (((int64_t)b * a.T + t) * a.H + h) * a.D + d);
        dst[0] = make_float4(run[0], run[1], run[2], run[3]);
        dst[1] = make_float4(run[4], run[5], run[6], run[7]);
    }
}

// In one launch: a cluster of up to eight CTAs per (batch, head), a CTA DGC tokens of every round, rounds from the last tokens to the first.  D / 4 threads cover
// the channels of a token, and every group of them keeps the terms of L consecutive tokens in registers, so nothing is read twice: sums of
// the groups meet in shared memory, sums of the CTAs through distributed shared memory, and the rounds behind in a register.  Bound by memory, two
// CTAs per SM; 8 x 2048 tokens of 8 heads of 128 (201 MB, 31 us at the copy rate): 51 us, the two launches 35 + 54.
constexpr int DGC = 128;
template <int D>
__global__ void __launch_bounds__(256, 2) gla_dg_kernel(DgArgs a) {
    constexpr int TPR = D / 4, GROUPS = 256 / TPR, L = DGC / GROUPS;
    __shared__ float part[2][GROUPS][D], total[2][D], behind[D];
    const int tid = threadIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int rank = blockIdx.x, ctas = gridDim.x;                      // the cluster is a row of the grid
    const int grp = tid / TPR, d = (tid % TPR) * 4;
    const bf16 *q = a.q + b * a.qs_b + h * a.qs_h + d, *k = a.k + b * a.ks_b + h * a.ks_h + d;
    const bf16 *dq = a.dq + b * a.dqs_b + h * a.dqs_h + d, *dk = a.dk + b * a.dks_b + h * a.dks_h + d;
    float* dg = a.dg + ((int64_t)b * a.T * a.H + h) * D + d;
    const int rounds = (a.T + ctas * DGC - 1) / (ctas * DGC);
    float carry = 0.f;                                                  // the rounds behind; threads tid < D: of channel tid
    for (int r = rounds - 1, turn = 0; r >= 0; --r, turn ^= 1) {
        const int t0 = (r * ctas + rank) * DGC + grp * L;
        float x[L][4];
#pragma unroll
        for (int i0 = 0; i0 < L; i0 += 4) {
            uint2 v[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t t = t0 + i0 + i;
                const bool in = t < a.T;
                const uint2 none = make_uint2(0u, 0u);
                v[i][0] = in ? __ldg(reinterpret_cast<const uint2*>(q + t * a.qs_t)) : none;
                v[i][1] = in ? __ldg(reinterpret_cast<const uint2*>(dq + t * a.dqs_t)) : none;
                v[i][2] = in ? __ldg(reinterpret_cast<const uint2*>(k + t * a.ks_t)) : none;
                v[i][3] = in ? __ldg(reinterpret_cast<const uint2*>(dk + t * a.dks_t)) : none;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                auto at = [](const uint2& u, int c) -> float {
                    const uint32_t w = c < 2 ? u.x : u.y;
                    return __uint_as_float(c & 1 ? w & 0xffff0000u : w << 16);
                };
#pragma unroll
                for (int c = 0; c < 4; ++c) x[i0 + i][c] = at(v[i][0], c) * at(v[i][1], c) - at(v[i][2], c) * at(v[i][3], c);
            }
        }
        // sums from a token to the end of its group's run
#pragma unroll
        for (int i = L - 2; i >= 0; --i)
#pragma unroll
            for (int c = 0; c < 4; ++c) x[i][c] += x[i + 1][c];
        *reinterpret_cast<float4*>(&part[turn][grp][d]) = make_float4(x[0][0], x[0][1], x[0][2], x[0][3]);
        __syncthreads();
        if (tid < D) {
            float s = 0.f;
#pragma unroll
            for (int g = GROUPS - 1; g >= 0; --g) s += part[turn][g][tid];
            total[turn][tid] = s;
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (tid < D) {
            float all = carry;
            for (int c = ctas - 1; c >= 0; --c) {
                if (c == rank) behind[tid] = all;
                uint32_t p;
                float v;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p) : "r"((uint32_t)__cvta_generic_to_shared(&total[turn][tid])), "r"(c));
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(p) : "memory");
                all += v;
            }
            carry = all;
        }
        __syncthreads();
        float4 run = *reinterpret_cast<const float4*>(&behind[d]);
        for (int g = GROUPS - 1; g > grp; --g) {
            const float4 y = *reinterpret_cast<const float4*>(&part[turn][g][d]);
            run.x += y.x; run.y += y.y; run.z += y.z; run.w += y.w;
        }
#pragma unroll
        for (int i = 0; i < L; ++i)
            if (t0 + i < a.T) *reinterpret_cast<float4*>(dg + (int64_t)(t0 + i) * a.H * D) = make_float4(run.x + x[i][0], run.y + x[i][1], run.z + x[i][2], run.w + x[i][3]);
    }
    // a CTA's totals stay until every other one has read them
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <int D>
static int dg_launch(const DgArgs& a, cudaStream_t st) {
    int ctas = 1;
    while (ctas < 8 && ctas * DGC < a.T) ctas *= 2;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(ctas, a.B * a.H); cfg.blockDim = dim3(256); cfg.stream = st; cfg.attrs = at; cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, gla_dg_kernel<D>, a);
}
}  // namespace lmoe

LMOE_API int lmoe_gla_dg(const lmoe::DgArgs* ap, cudaStream_t st) {
    lmoe::DgArgs a = *ap;
    if ((a.D != 64 && a.D != 128) || a.T <= 0) return -1;
    if ((a.qs_t | a.qs_h | a.qs_b | a.ks_t | a.ks_h | a.ks_b | a.dqs_t | a.dqs_h | a.dqs_b | a.dks_t | a.dks_h | a.dks_b) % 8) return -1;
    if (((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.dq | (uintptr_t)a.dk) & 15) return -1;
    if (a.nseg == 0) return a.D == 128 ? lmoe::dg_launch<128>(a, st) : lmoe::dg_launch<64>(a, st);
    if (a.nseg != (a.T + lmoe::DG_SEG - 1) / lmoe::DG_SEG) return -1;
    dim3 grid(a.nseg, a.B * a.H);
    lmoe::gla_dg_segsum_kernel<<<grid, 256, 0, st>>>(a);
    lmoe::gla_dg_scan_kernel<<<grid, 256, 0, st>>>(a);
    return (int)cudaGetLastError();
}
