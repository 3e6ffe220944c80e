// qgru_rec_f32.cuh - launch interface of the fp32 recurrences (qgru_rec_f32.cu): the float forward and
// the chain of state gradients of the backward pass, all T steps in one launch.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "qgru_internal.h"

struct qgru_handle;

namespace qgru {

// How a sequence is cut: clusters of P CTAs own Bt batch rows, each CTA U hidden units (a multiple of
// 32); KG = P * U / 32 slices of 32 units; U * KG <= 512 threads.
struct F32RecPlan {
    int H = 0, B = 0, sms = 0, directions = 0;      // what the plan was made for
    bool ok = false;
    int P = 1, U = 32, KG = 1, Bt = 1, G = 1, D = 1;
    int waves = 1;                  // clusters one after the other
    double us = 0;                  // estimate of a step, all waves
    size_t smem = 0;
};

// Weights come in one of two layouts: R [H][3H] with the gates in the order of v (z, r, n), or the module's own
// (torch): R [3H][H], gates in the order r, z, n.  In the second, W*x and the gradients dp, dq have
// that gate order as well, so that no weight and no gradient is transposed or reordered anywhere.
struct FloatFwdArgs {
    int T, B, H;
    const float *R, *wx, *bw, *br;    // wx = W*x of all steps [T*B][3H]; biases may be null
    float *h;                         // [(T+1)][B][H], slot 0 (in reverse slot T) holds the initial state
    float *v;                         // [T*B][v_stride * H] or null
    int v_stride;
    int torch, reverse;               // weight layout; reverse: step s consumes time T - 1 - s
    OutView out;                      // further copies of the states: hf, hn_f
    int U, P, KG, Bt, D;              // set by the launcher
};
// Whether there is a form for the layer (H <= 512); else the caller runs step by step.
bool float_chain_exists(qgru_handle *h);
// The form for B rows, into the handle's plan_fwd; directions: 2 where another one of the same size runs beside it, each
// within its handle's sm_limit.
bool float_chain_plan(qgru_handle *h, int B, int directions);
// Whether T steps of it, with the whole chip to itself, take no longer than a tiled product and a pointwise launch a step.
bool float_chain_is_faster(qgru_handle *h, int T, int B);
int float_chain_launch(qgru_handle *h, FloatFwdArgs a, cudaStream_t st);

struct BwdChainArgs {
    int T, B, H;
    const float *R;                   // [H][3H]; its transpose [3H][H] with r_trans; [3H][H] in the module's gate order with torch
    int r_trans, torch, reverse;
    const float *h, *v;               // [(T+1)][B][H], [T*B][4H]
    const float *dh_new;              // gradient of the state after the step at time t, row b: dh_new + t * dn_ts + b * dn_bs
    long long dn_ts, dn_bs;
    const float *dh_in;               // [B][H] gradient of the last state, or null
    float *dh_out;                    // [B][H] gradient of the initial state, times h0_mask where there is one
    const uint8_t *h0_mask;
    const uint16_t *pm;               // packed clamp masks [T*B][H] or null
    float *dp, *dq;                   // [T*B][3H]: gradients of W*x + bw (masked) and of R*h + br
    float *bias_part;                 // [G][6][H]: sums of dp (before its mask) and of dq over the group's rows
    const int8_t *r8;                 // where R is a quantized weight: its integers [3H][H], gates z, r, n, and the scale of each row
    const float *r_scale;
    int U, P, KG, Bt, D;              // set by the launcher
};
bool bwd_chain_exists(qgru_handle *h);
bool bwd_chain_plan(qgru_handle *h, int B, int directions);     // into plan_bwd
int bwd_chain_launch(qgru_handle *h, BwdChainArgs a, cudaStream_t st);

// The same on the tensor cores, for a quantized R (r8, r_scale and pm are set; qgru_bwd_tc.cu).  The plan is kept in *pl for its
// sizes; false: none.  bwd_chain_tc_is_faster plans into the handle's plan_bwd_tc.
bool bwd_chain_tc_plan(qgru_handle *h, int B, int sms, F32RecPlan *pl);
bool bwd_chain_tc_is_faster(qgru_handle *h, int B);
int bwd_chain_tc_launch(qgru_handle *h, const F32RecPlan &pl, const BwdChainArgs &a, cudaStream_t st);

// Bias gradients from bias_part; masks and either output may be null.
void bwd_bias_launch(qgru_handle *h, const float *part, int G, const uint8_t *m_bw, const uint8_t *m_br, float *dbw, float *dbr, int accumulate,
                     cudaStream_t st);

}  // namespace qgru
