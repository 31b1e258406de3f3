// Arguments of the kernels that walk the chunks of the (gated) delta rule (lsm_delta.cu, lsm_delta_tc.cu).
#pragma once
#include "common.cuh"

namespace lmoe {
namespace dr {

constexpr int C = 64;            // chunk length

struct Args {
    const bf16 *W, *U, *Qd, *Kd, *A;   // [BH, N, C, dk] / [BH, N, C, dv] / [BH, N, C, C]
    const float* gamma;                // [BH, N]
    const float* S0;                   // [BH, dk, dv] or null
    const bf16* dO;                    // backward: [B, T, H, dv] with the strides gs_*
    const float* dSfinal;              // backward: [BH, dk, dv] or null
    bf16* O;                           // forward: [B, T, H, dv] with the strides os_*, or null (not wanted)
    bf16* Vn;                          // forward out: [BH, N, C, dv], or null (neither Vn nor Sn is kept)
    bf16* Sn;                          // forward out: state entering chunk n, [BH, N, dk, dv]
    float* Sfinal;                     // forward out: [BH, dk, dv]
    bf16* dVn;                         // backward out: [BH, N, C, dv]
    bf16* dSn;                         // backward out: gradient of the state leaving chunk n, [BH, N, dk, dv]
    float* dS0;                        // backward out: [BH, dk, dv]
    long long os_b, os_t, os_h, gs_b, gs_t, gs_h;
    int N, dv, T, H;
    int ldw, lda;                      // row strides of W, Qd, Kd and of A in memory: dk + 8 and C + 8, or dk and C
    int* err;                          // error word of the bounded waits
};

constexpr int TC_DK = 128, TC_DV = 64;
// The scans for dk = TC_DK and dv a multiple of TC_DV (lsm_delta_tc.cu); dir as in lmoe_delta_scan
int scan_tc(int dir, int BH, const Args& a, cudaStream_t st);

}  // namespace dr
}  // namespace lmoe
