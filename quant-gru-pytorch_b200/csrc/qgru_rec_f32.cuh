// qgru_rec_f32.cuh - launch interface of the fp32 recurrences (qgru_rec_f32.cu): the float forward and
// the chain of state gradients of the backward pass, all T steps in one launch.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

struct qgru_handle;

namespace qgru {

// How a sequence is cut: clusters of P CTAs own Bt batch rows, each CTA U hidden units (a multiple of
// 32); KG = P * U / 32 slices of 32 units; U * KG <= 512 threads.
struct F32RecPlan {
    int H = 0, B = 0, sms = 0;      // what the plan was made for
    bool ok = false;
    int P = 1, U = 32, KG = 1, Bt = 1, G = 1, D = 1;
    size_t smem = 0;
};

// Clamp masks of a quantized training forward, one word per (timestep, row, unit): bit g (z, r, n)
// W*x + bw, 3 + g R*h + br, 6 + g gate input, 9 + g gate output, 12 the new state; 1 = not clamped.
constexpr int PM_IH = 0, PM_HH = 3, PM_IN = 6, PM_OUT = 9, PM_H = 12;

struct FloatFwdArgs {
    int T, B, H;
    const float *R, *wx, *bw, *br;    // R [H][3H]; wx = W*x of all steps [T*B][3H]
    float *h;                         // [(T+1)][B][H], slot 0 holds the initial state
    float *v;                         // [T*B][v_stride * H] or null
    int v_stride;
    int U, P, KG, Bt, D;              // set by the launcher
};
// False: no plan for this shape (H > 512), the caller runs step by step.
bool float_chain_fits(qgru_handle *h, int B);
int float_chain_launch(qgru_handle *h, FloatFwdArgs a, cudaStream_t st);

struct BwdChainArgs {
    int T, B, H;
    const float *R;                   // [H][3H], or its transpose [3H][H] with r_trans
    int r_trans;
    const float *h, *v, *dh_new;      // [(T+1)][B][H], [T*B][4H], [(T+1)][B][H]
    float *dh;                        // [B][H] in / out
    const uint16_t *pm;               // packed clamp masks [T*B][H] or null
    float *dp, *dq;                   // [T*B][3H]: gradients of W*x + bw (masked) and of R*h + br
    float *bias_part;                 // [G][6][H]: column sums of dp (before the W*x + bw mask) and of dq
    int U, P, KG, Bt, D;              // set by the launcher
};
bool bwd_chain_fits(qgru_handle *h, int B, int *groups);
int bwd_chain_launch(qgru_handle *h, BwdChainArgs a, cudaStream_t st);

}  // namespace qgru
