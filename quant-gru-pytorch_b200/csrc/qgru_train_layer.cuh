// Training of a whole layer as a module calls it: one forward and one backward call for one or both directions, weights
// and gradients in the module's own layout ([3H][I], [3H][H], gates r, z, n), strided tensors, no host
// synchronisation.
//
// A quantized forward is four launches a direction: the weights of this step (quantized, packed, summed, their masks
// and dequantized values in one pass), the prologue, the W*x product and the recurrence, which keeps the gate
// buffer and one word of clamp masks per cell.  A backward is the chain of state gradients, the bias sums
// and three products.  The reverse direction runs on a stream of its own beside the forward one.
// What the backward needs is written to a block of the caller's (qgru_train_saved_bytes), so that several forwards may
// be alive at once; mode 0 is the fp32 GRU, 1 the float-storage path, 2 the integer path.
//
// Included at the end of qgru_api.cu, after qgru_train.cuh.
#pragma once
#include "qgru_gemm_f32.cuh"
#include "qgru_layer.cuh"
#include "qgru_train.cuh"

namespace qgru {

// One row of W (blocks 0 .. 3H - 1) or R (3H .. 6H - 1) per block, rows in the module's order.
struct TrainWeightsArgs {
    const float *w[2], *bias[2];       // [3H][K], [3H] or null (zeros)
    const float *wscale[2], *bscale[2];   // per channel, order z, r, n
    const Rescale *rs[2], *brs[2];
    int8_t *w8[2];                     // [3H][Kpad]
    int32_t *wsum[2], *bias_q[2];
    int64_t *corr[2];
    FastLin *fl[2];
    float *deq[2];                     // [3H][K]
    int8_t *q8;                        // R's integers [3H][H] and scales [3H], channels z, r, n, for the backward
    float *qscale;
    uint8_t *keep[2], *bias_keep[2];
    int K[2], Kpad[2], H;
    int32_t zp_in[2], lo[2], hi[2], b_lo[2], b_hi[2];
    FsChannels ch;                     // float-storage path
    float *chan;                       // [6][3H] or null
};

__global__ void __launch_bounds__(128) k_train_weights(const TrainWeightsArgs a) {
    const int C = 3 * a.H, side = blockIdx.x >= C, row = blockIdx.x - side * C, gt = row / a.H;
    const int c = (gt < 2 ? 1 - gt : gt) * a.H + row % a.H;      // channel of the library: z, r, n
    const int K = a.K[side], Kpad = a.Kpad[side];
    const float scale = a.wscale[side][c], lo = (float)a.lo[side], hi = (float)a.hi[side];
    const float *src = a.w[side] + (size_t)row * K;
    int local = 0;
    for (int k = threadIdx.x; k < Kpad; k += 128) {
        int32_t q = 0;
        if (k < K) {
            const float w = src[k], raw = rintf(w / scale);
            q = quantize_one(w, scale, 0, a.lo[side], a.hi[side]);
            local += q;
            a.deq[side][(size_t)row * K + k] = (float)q * scale;
            a.keep[side][(size_t)row * K + k] = (raw < lo || raw > hi) ? 0 : 1;
        }
        a.w8[side][(size_t)c * Kpad + k] = (int8_t)q;
        if (side && k < K) a.q8[(size_t)c * K + k] = (int8_t)q;
    }
    __shared__ int red[4];
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x) return;
    const int32_t sum = red[0] + red[1] + red[2] + red[3];
    const float b = a.bias[side] ? a.bias[side][row] : 0.f, bs = a.bscale[side][c], b_raw = rintf(b / bs);
    const int32_t bq = quantize_one(b, bs, 0, a.b_lo[side], a.b_hi[side]);
    a.bias_keep[side][row] = (b_raw < (float)a.b_lo[side] || b_raw > (float)a.b_hi[side]) ? 0 : 1;
    a.bias_q[side][c] = bq;
    a.wsum[side][c] = sum;
    if (side) a.qscale[c] = scale;
    const int64_t corr = rescale64((int64_t)bq, a.brs[side][c]) - (int64_t)a.zp_in[side] * (int64_t)sum;
    a.corr[side][c] = corr;
    a.fl[side][c] = make_fast_lin(a.rs[side][c], corr);
    if (a.chan) {
        float *ch = a.chan + (size_t)side * 3 * C;
        ch[c] = fs_offset(sum, (float)a.zp_in[side]);
        ch[C + c] = fs_bias_term(bq, side ? a.ch.inv_br[c] : a.ch.inv_bw[c]);
        ch[2 * C + c] = side ? a.ch.inv_gemm_h[c] : a.ch.inv_gemm_x[c];
    }
}

namespace {

// The caller's block of one direction.  R is in it also where the chain of state gradients reads r8: the backward takes the fp32
// chain if the handle's sm_limit has changed to one that leaves no cluster to the other.
struct TrainSaved {
    float *h, *v, *xd, *W, *R, *r_scale;
    int8_t *r8;
    uint16_t *pm;
    uint8_t *mx, *mh0, *mW, *mR, *mbw, *mbr;
    size_t bytes;
};
TrainSaved train_saved(const qgru_handle *h, int mode, int T, int B, void *base) {
    const size_t N = (size_t)T * B, H = h->H, C = h->C, I = h->I, q = mode ? 1 : 0;
    TrainSaved s{};
    size_t at = 0;
    const auto take = [&](size_t bytes) {
        void *p = base ? static_cast<char *>(base) + at : nullptr;
        at += (bytes + 255) & ~size_t(255);
        return p;
    };
    s.h = (float *)take((N + B) * H * 4);
    s.v = (float *)take(N * 4 * H * 4);
    s.W = (float *)take(C * I * 4);
    s.R = (float *)take(C * H * 4);
    s.xd = (float *)take(q * N * I * 4);
    s.pm = (uint16_t *)take(q * (N * H * 2 + 4));
    s.mx = (uint8_t *)take(q * N * I);
    s.mh0 = (uint8_t *)take(q * B * H);
    s.mW = (uint8_t *)take(q * C * I);
    s.mR = (uint8_t *)take(q * C * H);
    s.mbw = (uint8_t *)take(q * C);
    s.mbr = (uint8_t *)take(q * C);
    s.r8 = (int8_t *)take(q * C * H);
    s.r_scale = (float *)take(q * C * 4);
    s.bytes = at;
    return s;
}

// Width of the stored W*x + bw: the operator's range and one step beyond it on either side.
int train_ih_bytes(const qgru_handle *h) {
    const qgru_op &o = h->p.op[QGRU_OP_IH_LINEAR];
    return op_qmin(o) > -32768 && op_qmax(o) < 32767 ? 2 : 4;
}

// Whether this direction has the one-launch forms of both recurrences (mode 1 needs fs_setup's table size).
int train_plan(qgru_handle *h, int mode, int B, int n_tab, bool *ok) {
    const int sms = h->opt_sm_limit > 0 ? std::min(h->opt_sm_limit, h->sm_count) : h->sm_count;
    *ok = bwd_chain_exists(h);
    if (mode == 0) *ok = *ok && float_chain_exists(h);
    else *ok = *ok && h->fast && h->opt_gemm != 1 && (h->opt_rec == 0 || h->opt_rec >= 5) &&
               rec_reg_plan(h, B, sms, train_ih_bytes(h), mode == 1 ? CELL_FS_TRAIN : CELL_INT_TRAIN, n_tab, &h->plan_train);
    return QGRU_OK;
}

int train_forward_dir(qgru_handle *h, int mode, int T, int B, const void *x, long long x_ts, long long x_bs, const float *h0,
                      const qgru_train_dir &d, OutView out, bool rev, int directions, cudaStream_t st, const uint8_t *x8_shared,
                      cudaEvent_t after_prologue) {
    const int H = h->H, I = h->I, C = h->C;
    const long long N = (long long)T * B;
    const TrainSaved s = train_saved(h, mode, T, B, d.saved);
    float *h_init = s.h + (rev ? (size_t)N * H : 0);
    int rc;
    if (mode == 0) {
        if ((rc = ensure(h, h->f_wx, (size_t)N * C * 4))) return rc;
        if (h0) CK(cudaMemcpyAsync(h_init, h0, (size_t)B * H * 4, cudaMemcpyDeviceToDevice, st));
        else CK(cudaMemsetAsync(h_init, 0, (size_t)B * H * 4, st));
        // (the parameters may change before the backward runs)
        CK(cudaMemcpyAsync(s.W, d.W, (size_t)C * I * 4, cudaMemcpyDeviceToDevice, st));
        CK(cudaMemcpyAsync(s.R, d.R, (size_t)C * H * 4, cudaMemcpyDeviceToDevice, st));
        if ((rc = gemm_f32(h, GemmF32{(const float *)x, false, d.W, true, (float *)h->f_wx.p, N, I, C}, st))) return rc;
        bool ok;
        if ((rc = train_plan(h, mode, B, 0, &ok))) return rc;
        if (!ok || !float_chain_plan(h, B, directions)) return fail(h, QGRU_ERR_UNSUPPORTED, "no one-launch recurrence for this layer");
        return float_chain_launch(h, FloatFwdArgs{T, B, H, d.R, (const float *)h->f_wx.p, d.bw, d.br, s.h, s.v, 4, 1, rev ? 1 : 0, out}, st);
    }
    const qgru_params &p = h->p;
    FsSetup fs;
    if (mode == 1 && (rc = fs_setup(h, fs, st))) return rc;
    const int n_tab = mode == 1 ? fs.n_train_tab : h->n_ttable;
    bool ok;
    if ((rc = train_plan(h, mode, B, n_tab, &ok))) return rc;
    if (!ok) return fail(h, QGRU_ERR_UNSUPPORTED, "no one-launch recurrence for this layer");
    const RecRegPlan &pl = h->plan_train;
    if ((rc = alloc_packed(h, st))) return rc;
    for (int k = 2; k < 4; ++k)
        if ((rc = alloc_once(h, &h->d_wq[k], (size_t)C))) return rc;
    TrainWeightsArgs w{};
    for (int k = 0; k < 2; ++k) {
        const qgru_op &wo = p.op[k ? QGRU_OP_R : QGRU_OP_W], &bo = p.op[k ? QGRU_OP_BR : QGRU_OP_BW];
        w.w[k] = k ? d.R : d.W;
        w.bias[k] = k ? d.br : d.bw;
        w.wscale[k] = h->d_wscale[k];
        w.bscale[k] = h->d_wscale[2 + k];
        w.rs[k] = h->d_rs[k];
        w.brs[k] = h->d_brs[k];
        w.w8[k] = h->d_w8[k];
        w.wsum[k] = h->d_wsum[k];
        w.bias_q[k] = h->d_wq[2 + k];
        w.corr[k] = h->d_corr[k];
        w.fl[k] = h->d_fl[k];
        w.deq[k] = k ? s.R : s.W;
        w.keep[k] = k ? s.mR : s.mW;
        w.bias_keep[k] = k ? s.mbr : s.mbw;
        w.K[k] = k ? H : I;
        w.Kpad[k] = k ? h->Hpad : h->Ipad;
        w.zp_in[k] = p.op[k ? QGRU_OP_H : QGRU_OP_X].zero_point;
        w.lo[k] = op_qmin(wo);
        w.hi[k] = op_qmax(wo);
        w.b_lo[k] = op_qmin(bo);
        w.b_hi[k] = op_qmax(bo);
    }
    w.H = H;
    w.q8 = s.r8;
    w.qscale = s.r_scale;
    if (mode == 1) {
        w.ch = fs.ch;
        w.chan = fs.chan;
    }
    h->weights_set = h->fs_ready = false;       // of the packed forms only those of this path are current
    k_train_weights<<<2 * C, 128, 0, st>>>(w);
    h->launches++;

    const uint8_t *x8 = x8_shared;
    if (!x8) {
        if ((rc = ensure(h, h->x8, (size_t)((N + 127) / 128 * 128) * h->Ipad))) return rc;
        x8 = (const uint8_t *)h->x8.p;
    }
    if ((rc = ensure(h, h->h8, (size_t)(2 * B + 256) * h->Hpad))) return rc;
    const int ih_bytes = train_ih_bytes(h);
    if ((rc = ensure(h, h->ih, pl.ih_elements(N) * ih_bytes))) return rc;
    FwdInput in{mode == 1 ? 1 : 0, x, x_ts, x_bs, h0};
    in.x_keep = s.mx;
    in.h0_keep = s.mh0;
    in.xd = s.xd;
    OutView slot;
    slot.hf = h_init;
    slot.bs = H;
    if ((rc = launch_prologue(h, T, B, in, x8_shared ? nullptr : (uint8_t *)h->x8.p, (uint8_t *)h->h8.p, slot, st))) return rc;
    if (after_prologue) CK(cudaEventRecord(after_prologue, st));
    const int sms = h->opt_sm_limit > 0 ? std::min(h->opt_sm_limit, h->sm_count) : h->sm_count;
    LinearConsts lcx = linear_consts(h, 0);
    lcx.fits32 = 0;
    lcx.lo -= 1;
    lcx.hi += 1;
    if (mode == 1) {
        lcx.fs = fs.chan;
        lcx.fs_C = C;
    }
    PreScale ps{};
    ps.H = H;
    ps.slice = pl.U;
    h->tc.pdl = true;             // (dependent launches: nothing is recorded between them here)
    if ((rc = tc_gemm_launch(h->tc, x8, (N + 127) / 128 * 128, h->d_w8[0], h->w8_rows[0], h->ih.p, N, C, h->Ipad, h->x_uns, ih_bytes, lcx, ps,
                             false, false, h->d_flags + 1, sms, st, &h->err)))
        return rc;
    h->launches++;
    RecRegArgs a{};
    a.pdl = true;
    a.T = T;
    a.B = B;
    a.H = H;
    a.Hpad = h->Hpad;
    a.reverse = rev ? 1 : 0;
    a.r8 = h->d_w8[1];
    a.ih = h->ih.p;
    a.h8 = (const uint8_t *)h->h8.p;
    a.out = out;
    a.lc = linear_consts(h, 1);
    a.tables = mode == 1 ? (const int32_t *)fs.train_tab : h->d_ttables;
    a.n_table = n_tab;
    a.abort_flag = h->d_flags + 1;
    if (mode == 1) {
        a.fs_chan = fs.chan + (size_t)3 * C;
        a.fs = fs.fc;
    }
    a.h_all = s.h;
    a.v = s.v;
    a.pm = s.pm;
    const int v_ops[4] = {QGRU_OP_UPDATE_OUT, QGRU_OP_RESET_OUT, QGRU_OP_NEW_OUT, QGRU_OP_HH_LINEAR};
    for (int k = 0; k < 4; ++k) {
        Rescale f;
        if (!to_fixed_scale(p.op[v_ops[k]].scale, p.use_pot2 != 0, &f)) return fail(h, QGRU_ERR_RANGE, "scale cannot be encoded");
        a.tc.scale[k] = decode_scale(f);
        a.tc.zp[k] = (float)p.op[v_ops[k]].zero_point;
    }
    return rec_reg_launch(h, pl, a, mode == 1 ? CELL_FS_TRAIN : CELL_INT_TRAIN, ih_bytes, st);
}

// The chain of state gradients, the bias gradients and those of W and R; dx is the caller's (two directions add up).
int train_backward_dir(qgru_handle *h, int mode, int T, int B, const float *x, const float *dout, long long do_ts, long long do_bs,
                       const float *dhn, float *dh0, const qgru_train_dir &d, const TrainSaved &s, const float *xd, bool rev, int directions, cudaStream_t st) {
    const int H = h->H, I = h->I, C = h->C;
    const long long N = (long long)T * B;
    int rc;
    const bool tc = mode != 0 && bwd_chain_tc_is_faster(h, B);
    if (!tc && !bwd_chain_plan(h, B, directions)) return fail(h, QGRU_ERR_UNSUPPORTED, "no one-launch recurrence for this layer");
    const int G = tc ? h->plan_bwd_tc.G : h->plan_bwd.G;
    if ((rc = ensure(h, h->bwd_dp, (size_t)N * C * 4))) return rc;
    if ((rc = ensure(h, h->bwd_dq, (size_t)N * C * 4))) return rc;
    if ((rc = ensure(h, h->bwd_bias, ((size_t)G * 2 * C + (size_t)B * H) * 4))) return rc;
    float *dp = (float *)h->bwd_dp.p, *dq = (float *)h->bwd_dq.p, *part = (float *)h->bwd_bias.p;
    if (!dh0) dh0 = part + (size_t)G * 2 * C;
    BwdChainArgs chain{T, B, H, s.R, 1, 1, rev ? 1 : 0, s.h, s.v, dout, do_ts, do_bs, dhn, dh0, mode ? s.mh0 : nullptr, mode ? s.pm : nullptr, dp, dq, part};
    chain.r8 = s.r8;
    chain.r_scale = s.r_scale;
    if ((rc = tc ? bwd_chain_tc_launch(h, h->plan_bwd_tc, chain, st) : bwd_chain_launch(h, chain, st))) return rc;
    if (d.dbw || d.dbr) bwd_bias_launch(h, part, G, mode ? s.mbw : nullptr, mode ? s.mbr : nullptr, d.dbw, d.dbr, 0, st);
    // dW[m][i] = sum_n dp[n][m] * x[n][i];  dR[m][k] = sum_n dq[n][m] * h_{t-1}[n][k]
    if (d.dW && (rc = gemm_f32(h, GemmF32{dp, true, mode ? xd : x, false, d.dW, C, N, I, 0, mode ? s.mW : nullptr}, st))) return rc;
    const float *h_prev = s.h + (rev ? (size_t)B * H : 0);
    if (d.dR && (rc = gemm_f32(h, GemmF32{dq, true, h_prev, false, d.dR, C, N, H, 0, mode ? s.mR : nullptr}, st))) return rc;
    CK(cudaGetLastError());
    return QGRU_OK;
}

int train_check(qgru_handle *h, qgru_handle *rev, int mode, int T, int B) {
    for (qgru_handle *d : {h, rev}) {
        if (!d) continue;
        if (T <= 0 || B <= 0) return fail(h, QGRU_ERR_BAD_ARG, "T and B must be positive");
        if (mode && !d->params_set) return fail(h, QGRU_ERR_NOT_READY, "set_params first");
        if (d->H != h->H || d->I != h->I || d->device != h->device) return fail(h, QGRU_ERR_BAD_ARG, "the two directions differ in device or sizes");
    }
    CK(cudaSetDevice(h->device));
    return layer_streams(h, rev);
}

}  // namespace
}  // namespace qgru

extern "C" {

int qgru_train_saved_bytes(qgru_handle *h, int mode, int T, int B, size_t *bytes) {
    if (!h || !bytes || mode < 0 || mode > 2) return QGRU_ERR_BAD_ARG;
    int rc;
    if ((rc = qgru::train_check(h, nullptr, mode, T, B))) return rc;
    *bytes = 0;
    CK(cudaSetDevice(h->device));
    bool ok = true;
    int n_tab = h->n_ttable;
    if (mode == 1 && h->fast) {
        qgru::FsSetup fs;
        qgru::fs_constants(h, fs);
        n_tab = fs.n_train_tab;
    }
    if ((rc = qgru::train_plan(h, mode, B, n_tab, &ok))) return rc;
    if (ok) *bytes = qgru::train_saved(h, mode, T, B, nullptr).bytes;
    return QGRU_OK;
}

int qgru_train_forward(qgru_handle *h, qgru_handle *rev, int mode, int T, int B, const float *x, long long x_ts, long long x_bs, const float *h0,
                       qgru_train_dir *dirs, float *out, long long out_ts, long long out_bs, float *h_n, void *stream) {
    if (!h || !x || !dirs || !out || !h_n || mode < 0 || mode > 2) return QGRU_ERR_BAD_ARG;
    int rc;
    if ((rc = qgru::train_check(h, rev, mode, T, B))) return rc;
    if ((rc = check_expiry(h, rev))) return rc;
    if (mode == 0 && (x_bs != h->I || x_ts != (long long)B * h->I)) return fail(h, QGRU_ERR_BAD_ARG, "mode 0 needs dense x [T][B][I]");
    CK(cudaSetDevice(h->device));
    cudaStream_t st = (cudaStream_t)stream;
    USE_HANDLE(h, st);
    StreamUse rev_use((rev ? rev : h)->order, (rev ? rev : h)->side);
    if (rev) CK(rev_use.begin(use_.captured()));
    if (rev) rev->captured = use_.captured();
    const size_t BH = (size_t)B * h->H;
    if (rev && mode == 0) CK(cudaEventRecord(rev->ev_split, st));
    for (int k = 0; k < (rev ? 2 : 1); ++k) {
        qgru_handle *d = k ? rev : h;
        OutView o;
        o.ts = (size_t)out_ts;
        o.bs = (size_t)out_bs;
        o.hf = out + (k ? (ptrdiff_t)h->H : -(ptrdiff_t)out_ts);
        o.hn_f = h_n + k * BH;
        cudaStream_t ds = k ? rev->side : st;
        if (k) CK(cudaStreamWaitEvent(ds, rev->ev_split, 0));
        dirs[k].shares_x = k && mode && qgru::same_x_quantization(h, rev);
        const uint8_t *shared = dirs[k].shares_x ? (const uint8_t *)h->x8.p : nullptr;
        rc = qgru::train_forward_dir(d, mode, T, B, x, x_ts, x_bs, h0 ? h0 + k * BH : nullptr, dirs[k], o, k == 1, rev ? 2 : 1, ds, shared,
                                     rev && !k && mode ? rev->ev_split : nullptr);
        if (rc && k) h->err = rev->err;
        if (k) {
            CK(cudaEventRecord(rev->ev_join, ds));
            CK(cudaStreamWaitEvent(st, rev->ev_join, 0));
            rev->order.tail = rev->ev_join;
        }
        if (rc) return rc;
    }
    return QGRU_OK;
}

int qgru_train_backward(qgru_handle *h, qgru_handle *rev, int mode, int T, int B, const float *x, const float *dout, long long do_ts,
                        long long do_bs, const float *dh_n, float *dx, float *dh0, const qgru_train_dir *dirs, void *stream) {
    if (!h || !dout || !dirs || mode < 0 || mode > 2 || (mode == 0 && !x)) return QGRU_ERR_BAD_ARG;
    int rc;
    if ((rc = qgru::train_check(h, rev, mode, T, B))) return rc;
    if ((rc = check_expiry(h, rev))) return rc;
    CK(cudaSetDevice(h->device));
    cudaStream_t st = (cudaStream_t)stream;
    USE_HANDLE(h, st);
    // the reverse direction's buffers are read on `st` last, by the product that adds its share of dx
    StreamUse rev_use((rev ? rev : h)->order, st);
    if (rev) CK(rev_use.begin(use_.captured()));
    const size_t BH = (size_t)B * h->H;
    const bool shared = rev && dirs[1].shares_x;
    qgru::TrainSaved s[2];
    for (int k = 0; k < (rev ? 2 : 1); ++k) s[k] = qgru::train_saved(h, mode, T, B, dirs[k].saved);
    const float *xd[2] = {s[0].xd, shared ? s[0].xd : s[1].xd};
    const uint8_t *mx[2] = {s[0].mx, shared ? s[0].mx : s[1].mx};
    if (rev) {
        CK(cudaEventRecord(rev->ev_split, st));
        CK(cudaStreamWaitEvent(rev->side, rev->ev_split, 0));
    }
    const long long N = (long long)T * B;
    int rc2 = QGRU_OK;
    for (int k = rev ? 1 : 0; k >= 0; --k) {
        qgru_handle *d = k ? rev : h;
        rc = qgru::train_backward_dir(d, mode, T, B, x, dout + k * h->H, do_ts, do_bs, dh_n ? dh_n + k * BH : nullptr, dh0 ? dh0 + k * BH : nullptr,
                                      dirs[k], s[k], xd[k], k == 1, rev ? 2 : 1, k ? rev->side : st);
        if (k) {
            if (rc) h->err = rev->err;
            rc2 = rc;
            CK(cudaEventRecord(rev->ev_join, rev->side));
        }
    }
    // dx[n][i] = sum_m dp[n][m] * W[m][i], the reverse direction's added to the forward one's
    if (!rc && dx) rc = gemm_f32(h, GemmF32{(const float *)h->bwd_dp.p, false, s[0].W, false, dx, N, h->C, h->I, 0, mode ? mx[0] : nullptr}, st);
    if (rev) CK(cudaStreamWaitEvent(st, rev->ev_join, 0));
    if (rc || rc2) return rc ? rc : rc2;
    if (rev && dx)
        return gemm_f32(rev, GemmF32{(const float *)rev->bwd_dp.p, false, s[1].W, false, dx, N, h->C, h->I, 2, mode ? mx[1] : nullptr}, st);
    return QGRU_OK;
}

}  // extern "C"
