// Arguments of the kernels for linear attention with a decay per key channel (lsm_vector.cu, lsm_vector_tc.cu).
#pragma once
#include <cuda.h>
#include "common.cuh"

namespace lmoe {

struct GlaArgs {
    const bf16 *q, *k, *v, *d_o;
    int64_t qs_b, qs_t, qs_h, ks_b, ks_t, ks_h, vs_b, vs_t, vs_h;
    bf16 *o, *dq, *dk, *dv;
    int64_t dqs_b, dqs_t, dqs_h, dks_b, dks_t, dks_h, dvs_b, dvs_t, dvs_h;
    const float* gk;               // [B,T,H,D] fp32 log decay
    float scale;
    int B, T, H, G, cpg;           // G groups of cpg 64-token chunks
    float* states;                 // [B,H,G,D,D]
    float* gdecay;                 // [B,H,G,D] total log decay of each group per channel
    int* err;                      // error word of the bounded waits (lsm_vector_tc.cu)
    int wide;                      // 128-wide heads: the kernels of lsm_vector_tc.cu
};

namespace lvt {
// The tensor maps of a call's inputs, made when a launch first wants them
struct Maps { CUtensorMap q, k, v, g, gk; unsigned made = 0; };
// lmoe_gla_launch for `wide`; the launches that share `m` have the same inputs
int launch(int which, const GlaArgs& a, Maps& m, cudaStream_t st);
}  // namespace lvt

}  // namespace lmoe
