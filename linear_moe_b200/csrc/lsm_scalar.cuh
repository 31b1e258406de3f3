// Arguments of the scalar-decay linear attention kernels (lsm_scalar.cu, lsm_scalar_tc.cu).
#pragma once
#include "common.cuh"

namespace lmoe {

struct LsmArgs {
    const bf16 *q, *k, *v, *d_o;   // d_o: contiguous [B,T,H,D] (backward only)
    int64_t qs_b, qs_t, qs_h, ks_b, ks_t, ks_h, vs_b, vs_t, vs_h;
    bf16 *o, *dq, *dk, *dv;        // outputs (o contiguous; dq/dk/dv with the strides below)
    int64_t dqs_b, dqs_t, dqs_h, dks_b, dks_t, dks_h, dvs_b, dvs_t, dvs_h;
    const float* g;                // gmode 1: [H]; gmode 2: [B,T,H]
    int gmode;
    float scale;
    int B, T, H, G, cpg;           // G groups of cpg chunks
    float* states;                 // [B,H,G,D,D]
    float* gdecay;                 // [B,H,G] total log decay per group (gmode 2)
    int* err;                      // error word of the bounded waits (chunk 128)
    int chunk;                     // 64: kernels of lsm_scalar.cu; 128: of lsm_scalar_tc.cu (128-wide heads).  Groups count 64-token chunks in both.
};

namespace lst {
// the launches of lmoe_lsm_scalar_launch for 128-wide heads
int launch(int which, const LsmArgs& a, cudaStream_t st);
}  // namespace lst

}  // namespace lmoe
