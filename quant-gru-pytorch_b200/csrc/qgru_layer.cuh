// The forward of a whole layer as a module calls it: one or both directions in one call, strided input and
// output (batch-first tensors, the two halves of a bidirectional output), no dense intermediate and no
// host synchronisation.
//
// A call is three launches per direction (prologue, W*x product, recurrence) with a timing event before and behind them and,
// where they are not dependent launches (run_reg), one on either side of the product; the
// reverse direction runs on a stream of its own beside the forward one and reads the rows the forward
// direction has quantized where both quantize x the same way.  A call on another stream than the one before waits for
// that one's work on the GPU (StreamUse): calls of one layer never overlap.  A device-side
// wait that runs out is known to the host at once: the first call after that reports it, or qgru_synchronize.
//
// Included at the end of qgru_api.cu, after qgru_fstorage.cuh.
#pragma once
#include "qgru_fstorage.cuh"

namespace qgru {
namespace {

bool same_x_quantization(const qgru_handle *a, const qgru_handle *b) {
    const qgru_op &p = a->p.op[QGRU_OP_X], &q = b->p.op[QGRU_OP_X];
    return a->I == b->I && a->x_scale == b->x_scale && p.zero_point == q.zero_point && op_qmin(p) == op_qmin(q) &&
           op_qmax(p) == op_qmax(q);
}

// The reverse direction's stream and the events that fork and join it.
int layer_streams(qgru_handle *h, qgru_handle *rev) {
    if (!rev || rev->ev_join) return QGRU_OK;
    if (!rev->side) CK(cudaStreamCreateWithFlags(&rev->side, cudaStreamNonBlocking));
    if (!rev->ev_split) CK(cudaEventCreateWithFlags(&rev->ev_split, cudaEventDisableTiming));
    CK(cudaEventCreateWithFlags(&rev->ev_join, cudaEventDisableTiming));
    return QGRU_OK;
}

// x, h0, out, h_n: fp32 (mode 0, 1) or int32 (mode 2).
int layer_forward(qgru_handle *h, qgru_handle *rev, int mode, int T, int B, const void *x, long long x_ts, long long x_bs,
                  const void *h0, void *out, long long out_ts, long long out_bs, void *h_n, cudaStream_t st) {
    int rc;
    for (qgru_handle *d : {h, rev}) {
        if (!d) continue;
        if ((rc = check_forward_args(d, T, B))) return d == h ? rc : fail(h, rc, d->err);
    }
    if ((rc = check_expiry(h, rev))) return rc;
    if (rev && (rev->device != h->device || rev->I != h->I || rev->H != h->H))
        return fail(h, QGRU_ERR_BAD_ARG, "the two directions differ in device or sizes");
    CK(cudaSetDevice(h->device));
    if ((rc = layer_streams(h, rev))) return rc;
    USE_HANDLE(h, st);
    StreamUse rev_use((rev ? rev : h)->order, (rev ? rev : h)->side);
    if (rev) CK(rev_use.begin(use_.captured()));
    if (rev) rev->captured = use_.captured();
    const size_t BH = (size_t)B * h->H;
    // a 32-bit row offset inside a step is what the cluster recurrence has room for
    if (out_bs < 0 || out_ts < 0 || out_bs > (1ll << 25)) return fail(h, QGRU_ERR_UNSUPPORTED, "output stride too large");
    for (int d = 0; d < (rev ? 2 : 1); ++d) {
        qgru_handle *k = d ? rev : h;
        OutView o;
        o.ts = (size_t)out_ts;
        o.bs = (size_t)out_bs;
        // step s writes slot s + 1 (forward) or T - 1 - s (reverse); the output holds slots 1..T or 0..T-1
        const ptrdiff_t off = d ? (ptrdiff_t)h->H : -(ptrdiff_t)out_ts;
        if (mode == 2) {
            o.hq = (int32_t *)out + off;
            o.hn_q = (int32_t *)h_n + d * BH;
        } else {
            o.hf = (float *)out + off;
            o.hn_f = (float *)h_n + d * BH;
        }
        FwdInput in{mode, x, x_ts, x_bs, h0 ? (const char *)h0 + d * BH * 4 : nullptr};
        const uint8_t *shared = nullptr;
        cudaStream_t ds = st;
        const bool generic = mode != 1 && use_generic(k);
        if (d) {
            ds = rev->side;
            CK(cudaStreamWaitEvent(ds, rev->ev_split, 0));
            if (!generic && !(mode != 1 && use_generic(h)) && same_x_quantization(h, rev)) shared = (const uint8_t *)h->x8.p;
        }
        cudaEvent_t after = rev && !d ? rev->ev_split : nullptr;
        const unsigned fl = d ? QGRU_FLAG_REVERSE : 0;
        rc = mode == 1 ? fstorage_forward(k, T, B, in, o, false, fl, ds, shared, after)
                       : forward_dir(k, T, B, in, o, false, fl, ds, shared, after);
        if (rc && d) h->err = k->err;
        if (d) {   // (a direction that failed may have queued some of its work)
            CK(cudaEventRecord(rev->ev_join, ds));
            CK(cudaStreamWaitEvent(st, rev->ev_join, 0));
            rev->order.tail = rev->ev_join;
            h->order.tail = nullptr;            // x8 is read until the directions have joined
        }
        if (rc) return rc;
    }
    return QGRU_OK;
}

}  // namespace
}  // namespace qgru

extern "C" {

int qgru_layer_forward(qgru_handle *h, qgru_handle *rev, int float_storage, int T, int B, const float *x, long long x_ts,
                       long long x_bs, const float *h0, float *out, long long out_ts, long long out_bs, float *h_n,
                       void *stream) {
    if (!h || !x || !out || !h_n) return QGRU_ERR_BAD_ARG;
    return qgru::layer_forward(h, rev, float_storage ? 1 : 0, T, B, x, x_ts, x_bs, h0, out, out_ts, out_bs, h_n, (cudaStream_t)stream);
}

int qgru_layer_forward_i32(qgru_handle *h, qgru_handle *rev, int T, int B, const int32_t *x_q, long long x_ts, long long x_bs,
                           const int32_t *h0_q, int32_t *out_q, long long out_ts, long long out_bs, int32_t *h_n_q, void *stream) {
    if (!h || !x_q || !out_q || !h_n_q) return QGRU_ERR_BAD_ARG;
    return qgru::layer_forward(h, rev, 2, T, B, x_q, x_ts, x_bs, h0_q, out_q, out_ts, out_bs, h_n_q, (cudaStream_t)stream);
}

}  // extern "C"
