// qgru_internal.h - declarations shared by the host set-up code and the CUDA translation
// units of libqgru_b200.  Nothing here is part of the public ABI (include/qgru.h).
#pragma once
#include <math.h>
#include <stdint.h>

#include <string>

#include "qgru.h"
#include "qgru_math.h"

namespace qgru {

// ---- host helpers implemented in qgru_host.cc
bool encode_mshift(float scale, Rescale *out);
int pot2_shift(float scale);
bool to_fixed_scale(float scale, bool pot2, Rescale *out);
float decode_scale(Rescale r);
bool make_rescale(float src, float dst, bool pot2, Rescale *out);
bool make_rescale_product(float a, float b, float dst, bool pot2, Rescale *out);
bool make_rescale_to_product(float src, float a, float b, bool pot2, Rescale *out);
// One histogram -> op->scale / op->zero_point by Percentile or SQNR (qgru_host.cc), in pieces.
// The SQNR search's candidates: delta and offset of number c come from these scalars.
struct SqnrSearch {
    float hmin, bw;                       // histogram: value of bin i = hmin + (i + 0.5) * bw
    float tiny, steps, max_delta, offset; // symmetric: delta = max(max_delta * (c + 1) / 100, tiny)
    float obs_off, obs_min, obs_max, off_step;
    int sym, n, n_off;
};
// Both sides round every product (no fused multiply-add): a candidate that differs in its last bit would move the
// small errors of a histogram with few values by more than any margin.
QG_HD float sqnr_mul(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
QG_HD void sqnr_candidate(const SqnrSearch &q, int c, float *delta, float *offset) {
    if (q.sym) {
        const float d = sqnr_mul(q.max_delta, (float)(c + 1)) / 100.0f;
        *delta = d > q.tiny ? d : q.tiny;
        *offset = q.offset;
        return;
    }
    const int d = c / q.n_off + 1, o = c % q.n_off;
    float dl = sqnr_mul(q.max_delta, (float)d) / 16.0f;
    dl = dl > q.tiny ? dl : q.tiny;
    const float off = o == q.n_off - 1 ? q.obs_off : rintf(-q.steps + sqnr_mul((float)o, q.off_step));
    float t_min = sqnr_mul(dl, off);
    float t_max = t_min + sqnr_mul(dl, q.steps);
    t_min = q.obs_min > t_min ? q.obs_min : t_min;
    t_max = q.obs_max < t_max ? q.obs_max : t_max;
    float cd = (t_max - t_min) / q.steps;
    cd = cd > q.tiny ? cd : q.tiny;
    *delta = cd;
    *offset = rintf(t_min / cd);
}
SqnrSearch hist_sqnr_search(int bins, float min_val, float max_val, const qgru_op &op);
int hist_sqnr_best(const float *counts, int bins, const SqnrSearch &q, const qgru_op &op, const int *list, int n_list);
int hist_sqnr_finish(const SqnrSearch &q, int best, bool pot2, qgru_op *op);
int hist_percentile_finish(int bins, float min_val, float max_val, bool whole_range, int lo_i, int hi_i, bool pot2, qgru_op *op);
int32_t op_qmin(const qgru_op &o);
int32_t op_qmax(const qgru_op &o);
int32_t lut_eval(const qgru_lut &lut, int32_t q_x, const qgru_op &in_bw, const qgru_op &out_bw);

// ---- device-visible constants of the gate datapath: the scalar part of
// GateQuantParamsT<R> (include/quantize_param_types.h:148-193), derived once per
// set_params instead of being passed by value (968 bytes) on every launch.
enum { ACT_Z = 0, ACT_R = 1, ACT_N = 2 };

struct GateConsts {
    int32_t zp_ih, zp_hh, zp_h;
    int32_t zp_in[3], zp_out[3];          // gate input / output zero points (z, r, n)
    int32_t one_q;                        // round(1/s_z) + zp_z
    Rescale ih_to[3];                     // weight_ih_linear -> gate input (z, r, n)
    Rescale hh_to[2];                     // weight_hh_linear -> gate input (z, r)
    Rescale rh_to_n;                      // (r - zp)(hh_n - zp) -> new gate input
    Rescale n_to_h;                       // new gate output -> h
    Rescale uh_to_h;                      // s_z * s_h -> h
    int32_t in_lo[3], in_hi[3], out_lo[3], out_hi[3];
    int32_t h_lo, h_hi, ih_lo, ih_hi, hh_lo, hh_hi;
    int32_t table_size[3];                // > 0: direct table over the clamped input range
    int32_t table_off[3];                 // offset of that table in the table array (ints)
    int32_t narrow;                       // 1: every gate rescale fits the 32-bit fast form
    float h_scale;                        // decode_scale(toFixedScale(h)) for the float output
    // "fused" form of the cell used by the tensor-core recurrence when every gate input and
    // the R*h+br output are narrow enough to tabulate (see build_fused_tables in qgru_api.cu)
    int32_t fused_ok;
    int32_t k1;                           // one_q - 2*zp_z : (1 - z) numerator minus z_d
    int32_t ft_off[5];                    // offsets of TZ, TR, TN, THZ, THR in the fused table block
    int32_t ih_pre_bytes;                 // storage width (2 or 4) of the pre-rescaled W*x+bw values
    int32_t ft_ih_off, ft_ih_n;           // table of the GEMM-side pre-rescale in the same block (n per gate, 0: none)
    // Index arithmetic of the five fused-cell lookups with the zero points, the clamp and the
    // table offset folded: entry = table[min(max(v + fi_c[k], fi_lo[k]), fi_hi[k])], k = TZ, TR,
    // TN (v = gate input before its clamp) or THZ, THR (v = requantized R*h row before its zero
    // point).  hn_clo/hn_chi clamp the new gate's R*h row in the same zero-point-free domain.
    int32_t fi_c[5], fi_lo[5], fi_hi[5];
    int32_t hn_clo, hn_chi;
    int32_t cell_notie;                   // 1: neither rescale of the fused cell can meet an exact tie (rescale_can_tie)
    qgru_lut lut[3];
};

// What the input-projection GEMM applies after the requantization when the recurrence runs the
// fused cell: out = rescale(ih - zp_ih -> gate input scale of the channel's gate) + zp_in[gate].
struct PreScale {
    int32_t enabled, zp_ih;
    int32_t H;              // hidden size: channel m belongs to gate m / H
    int32_t slice;          // hidden units per slice of the stored tensor [H / slice][N][3][slice]; 0: H, i.e. [N][3H]
    Rescale to[3];
    int32_t zp_in[3];
    unsigned long long *stamp;   // the product's start time, or null (set by the launcher)
    // optional table of that function over the clamped W*x+bw range (gate-major, n entries per
    // gate, index = value - lo); null when the range is too wide to tabulate
    const int32_t *table;
    int32_t table_n, lo;
};

// GateQuantParamsFP + the scalar part of LinearRescaleParamsFP
// (ForwardPassQuantFP::setRescaleParam, src/gru_forward_gpu_quant_fp.cu:821-1003).
struct FsConsts {
    float zp_x, zp_h, zp_ih, zp_hh;
    float zp_in[3], zp_out[3];      // gate inputs / outputs: z, r, n
    float s_in[3], s_out[3];
    float ih_to[3];                 // weight_ih_linear -> gate input
    float hh_to[2];                 // weight_hh_linear -> z, r input
    float rh_to_n;                  // (r * hh_n) -> new gate input
    float n_to_h, uh_to_h, one_q;
    float ih_lo, ih_hi, hh_lo, hh_hi, h_lo, h_hi;
    float in_lo[3], in_hi[3], out_lo[3], out_hi[3];
    float h_scale;                  // decoded scale of h, for the dequantized output
    int h_bits;                     // 8: signed state bytes, 9: unsigned
    // Gate outputs tabulated over the clamped gate input (built on the device by the very code
    // that evaluates a gate directly): entry tab_off[g] + (input - in_lo[g]) of a float table the
    // kernel holds in shared memory.  tab_on = 0: evaluate sigmoid / tanh per cell.
    int tab_on;
    int tab_off[3];
};

// Clamp masks of a quantized training forward, one word per (timestep, row, unit): bit g (z, r, n)
// W*x + bw, 3 + g R*h + br, 6 + g gate input, 9 + g gate output, 12 the new state; 1 = not clamped.
constexpr int PM_IH = 0, PM_HH = 3, PM_IN = 6, PM_OUT = 9, PM_H = 12;

// Dequantization constants of the four slots of v (dequantificationVFPInplace,
// src/quantize_ops.cu:368-397): update, reset, new gate outputs, R*h + br row of the new gate.
struct FsTrainConsts {
    float scale[4], zp[4];
};

// Per output channel constants of one fused linear layer:
//   out = clamp( int32( rescale( acc + corr[m], rs[m] ) ) + zp_out )
// with corr[m] = rescale(bias_q[m], bias_rs[m]) - zp_in * sum_k W_q[k][m]
// (src/gru_forward_cpu_quant.cc:92-99,125-138).
struct LinearConsts {
    const int64_t *corr;  // [3H] device
    const Rescale *rs;    // [3H] device
    const FastLin *fl;    // [3H] device: rs and corr in the folded shift-free form (mq == 0: none)
    int32_t zp_out, lo, hi;
    int32_t fits32;       // 1: acc + corr fits int32 for every channel (one widening multiply)
    // float-storage forward: [3][fs_C] floats (offset, bias term, scale ratio per channel); when
    // set, the epilogue is the reference's float requantization instead of the integer one
    const float *fs = nullptr;
    int32_t fs_C = 0;
};

// Where a recurrence writes its states: element (slot, row b, unit j) at slot * ts + b * bs + j of whichever
// outputs are set (slot s + 1 of step s, T - 1 - s in reverse), and the state after the last step, rows
// dense, at hn_*.
struct OutView {
    float *hf = nullptr;       // dequantized
    int32_t *hq = nullptr;     // int32 containers
    uint8_t *h8 = nullptr;     // 8-bit containers
    size_t ts = 0, bs = 0;
    float *hn_f = nullptr;     // [B][H]
    int32_t *hn_q = nullptr;   // [B][H]
    OutView shifted(size_t slots) const {
        OutView o = *this;
        if (hf) o.hf += slots * ts;
        if (hq) o.hq += slots * ts;
        if (h8) o.h8 += slots * ts;
        return o;
    }
};

}  // namespace qgru
