// qgru_backward.cu - backward pass of the GRU: hasteGRUBackward (src/gru_interface.cc:215-240,
// src/gru_backward_gpu.cu) and quantGRUBackward with the straight-through masks of QAT
// (src/gru_interface.cc:246-290, src/gru_backward_gpu_quant.cu).  One implementation: the float
// backward is the masked one with every mask absent.
//
// Per timestep, last to first: dh becomes the gradients of the two linear layers' outputs (dp for
// W*x + bw, dq for R*h + br) and the part of dh that flows through the update gate; dh += dq * R^T.
// All steps in one launch (k_bwd_chain, qgru_rec_f32.cu), which also sums dp and dq over the rows for
// the bias gradients in a fixed order (the reference adds them with atomics, in arbitrary order).
// Then dx = dp * W^T, dR += h^T * dq, dW += x^T * dp (k_gemm_f32; the reference calls cuBLAS SGEMM,
// fp32 without tensor-op math in this pass).
#include "qgru_gemm_f32.cuh"
#include "qgru_handle.h"
#include "qgru_rec_f32.cuh"

using namespace qgru;

namespace {

// The clamp masks of a step's cells in one word each (PM_* bits): the recurrence reads two bytes per cell
// and step instead of ten or thirteen.  Absent masks keep everything.
__global__ void k_bwd_pack_masks(uint16_t *__restrict__ pm, long long N, int H, const uint8_t *__restrict__ ih,
                                 const uint8_t *__restrict__ hh, const uint8_t *__restrict__ gin,
                                 const uint8_t *__restrict__ gout, const uint8_t *__restrict__ hm) {
    const long long total = N * H;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long n = i / H;
        const long long at = n * 3 * H + (i - n * H);
        unsigned m = 0;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            const long long k = at + (long long)g * H;
            m |= (unsigned)(!ih || ih[k]) << (PM_IH + g) | (unsigned)(!hh || hh[k]) << (PM_HH + g) |
                 (unsigned)(!gin || gin[k]) << (PM_IN + g) | (unsigned)(!gout || gout[k]) << (PM_OUT + g);
        }
        m |= (unsigned)(!hm || hm[i]) << PM_H;
        pm[i] = (uint16_t)m;
    }
}

// The pointwise part of one timestep (kernel::PointwiseOperations, src/gru_backward_gpu.cu:26-88;
// with masks kernel::PointwiseOperationsQuant, src/gru_backward_gpu_quant.cu:72-250, zoneout
// off).  h: h_{t-1} [B][H]; v: (z, r, g, R*h_g + br_g) [B][4H]; dh_new: gradient arriving at
// h_t from outside; dh: in: gradient arriving from step t+1, out: its part through the update
// gate (the R^T part is added by the GEMM that follows).  pm: packed masks of the step or null; 1 keeps
// the gradient, 0 (the forward clamped there) drops it.
__global__ void __launch_bounds__(256)
k_bwd_pointwise(int B, int H, const float *__restrict__ h, const float *__restrict__ v,
                const float *__restrict__ dh_new, float *__restrict__ dh, float *__restrict__ dp,
                float *__restrict__ dq, const uint16_t *__restrict__ pm) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (j >= H || b >= B) return;
    const size_t base = (size_t)b * H + j;
    float dh_total = dh_new[base] + dh[base];
    const unsigned m = pm ? pm[base] : 0xffffu;
    if (!(m >> PM_H & 1)) dh_total *= 0.f;
    const float *vb = v + (size_t)b * 4 * H + j;
    const float z = vb[0], r = vb[H], g = vb[2 * H], q_g = vb[3 * H];
    dh[base] = z * dh_total;
    const float dg = (1.0f - z) * dh_total;
    const float dz = (h[base] - g) * dh_total;
    const float dp_g = (1.0f - g * g) * dg;            // d_tanh(g) * dg
    const float dq_g = dp_g * r;
    const float dr = dp_g * q_g;
    const float dp_r = (r * (1.0f - r)) * dr;          // d_sigmoid(r) * dr
    const float dp_z = (z * (1.0f - z)) * dz;
    float p[3] = {dp_z, dp_r, dp_g};
    float q[3] = {dp_z, dp_r, dq_g};
    const size_t idx = (size_t)b * 3 * H + j;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const size_t at = idx + (size_t)k * H;
        const float keep = (m >> (PM_OUT + k) & 1) && (m >> (PM_IN + k) & 1) ? 1.f : 0.f;
        p[k] *= keep;
        q[k] *= keep;
        if (!(m >> (PM_HH + k) & 1)) q[k] *= 0.f;
        dp[at] = p[k];
        dq[at] = q[k];
    }
}

// out[c] += mask[c] * sum_n a[n][c]: the bias gradients.  One block of 256 threads per 32
// columns; rows are added in a fixed order (8 row lanes, then a tree over them).
__global__ void __launch_bounds__(256)
k_bwd_colsum(const float *__restrict__ a, long long N, int M, const uint8_t *__restrict__ mask,
             float *__restrict__ out) {
    __shared__ float part[8][32];
    const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + cx;
    float s = 0.f;
    if (c < M)
        for (long long n = ry; n < N; n += 8) s += a[n * M + c];
    part[ry][cx] = s;
    __syncthreads();
    if (ry == 0 && c < M) {
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) t += part[k][cx];
        if (mask) t *= (float)mask[c];
        out[c] += t;
    }
}

// ApplyMaskKernel (src/gru_backward_gpu_quant.cu:37-42)
__global__ void k_bwd_apply_mask(float *__restrict__ data, const uint8_t *__restrict__ mask, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        data[i] *= (float)mask[i];
}

// The bias gradients from the sums the recurrence leaves per group of batch rows: part [G][6][H] (z, r, n of
// dp, then of dq), added in group order.
__global__ void k_bwd_bias(const float *__restrict__ part, int G, int H, const uint8_t *__restrict__ m_bw,
                           const uint8_t *__restrict__ m_br, float *__restrict__ dbw, float *__restrict__ dbr, int accumulate) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, C = 3 * H;
    if (c >= 2 * C) return;
    float s = 0.f;
    for (int g = 0; g < G; ++g) s += part[(size_t)g * 2 * C + c];
    const bool x_side = c < C;
    const int k = x_side ? c : c - C;
    const uint8_t *mask = x_side ? m_bw : m_br;
    float *out = x_side ? dbw : dbr;
    if (!out) return;
    if (mask) s *= (float)mask[k];
    out[k] = accumulate ? out[k] + s : s;
}

}  // namespace

namespace qgru {

void bwd_bias_launch(qgru_handle *h, const float *part, int G, const uint8_t *m_bw, const uint8_t *m_br, float *dbw, float *dbr, int accumulate,
                     cudaStream_t st) {
    k_bwd_bias<<<(2 * h->C + 127) / 128, 128, 0, st>>>(part, G, h->H, m_bw, m_br, dbw, dbr, accumulate);
    h->launches++;
}

}  // namespace qgru

extern "C" {

int qgru_backward(qgru_handle *h, int T, int B, const float *W_t, const float *R_t, const float *x_t,
                  const float *dh_new, const float *h_all, const float *v, float *dx, float *dW,
                  float *dR, float *dbw, float *dbr, float *dh, const qgru_bwd_masks *mk, void *stream) {
    if (!h || !W_t || !R_t || !x_t || !dh_new || !h_all || !v || !dx || !dW || !dR || !dbw || !dbr || !dh)
        return QGRU_ERR_BAD_ARG;
    if (T <= 0 || B <= 0) return fail(h, QGRU_ERR_BAD_ARG, "T and B must be positive");
    CK(cudaSetDevice(h->device));
    cudaStream_t st = (cudaStream_t)stream;
    USE_HANDLE(h, st);
    const int H = h->H, I = h->I, C = h->C;
    const long long N = (long long)T * B;
    const size_t NH = (size_t)B * H, NH3 = (size_t)B * C;
    int rc;
    if ((rc = ensure(h, h->bwd_dp, (size_t)N * C * sizeof(float)))) return rc;
    if ((rc = ensure(h, h->bwd_dq, (size_t)N * C * sizeof(float)))) return rc;
    float *dp = (float *)h->bwd_dp.p, *dq = (float *)h->bwd_dq.p;
    const qgru_bwd_masks none{};
    const qgru_bwd_masks &m = mk ? *mk : none;
    uint16_t *pm = nullptr;
    if (m.ih_linear || m.hh_linear || m.gate_input || m.gate_output || m.h) {
        if ((rc = ensure(h, h->bwd_pm, (size_t)N * H * sizeof(uint16_t) + 4))) return rc;
        pm = (uint16_t *)h->bwd_pm.p;
        k_bwd_pack_masks<<<grid_for(N * H, 256, h->sm_count), 256, 0, st>>>(pm, N, H, m.ih_linear, m.hh_linear, m.gate_input,
                                                                            m.gate_output, m.h);
        h->launches++;
    }

    if (bwd_chain_plan(h, B, 1)) {
        const int G = h->plan_bwd.G;
        if ((rc = ensure(h, h->bwd_bias, (size_t)G * 2 * C * sizeof(float)))) return rc;
        float *part = (float *)h->bwd_bias.p;
        if ((rc = bwd_chain_launch(h, BwdChainArgs{T, B, H, R_t, 1, 0, 0, h_all, v, dh_new + NH, (long long)NH, H, dh, dh, m.h0, pm, dp, dq, part}, st)))
            return rc;
        bwd_bias_launch(h, part, G, m.bw, m.br, dbw, dbr, 1, st);
    } else {
        // wide layers, step by step: the pointwise part, then dh[b][k] += sum_m dq[b][m] * R_t[m][k]
        const dim3 pw_grid((H + 255) / 256, B);
        for (int i = T - 1; i >= 0; --i) {
            k_bwd_pointwise<<<pw_grid, 256, 0, st>>>(
                B, H, h_all + (size_t)i * NH, v + (size_t)i * NH * 4, dh_new + (size_t)(i + 1) * NH, dh,
                dp + (size_t)i * NH3, dq + (size_t)i * NH3, pm ? pm + (size_t)i * NH : nullptr);
            if ((rc = gemm_f32(h, GemmF32{dq + (size_t)i * NH3, false, R_t, false, dh, B, C, H, true}, st))) return rc;
        }
        // bias gradients: column sums of dp / dq before the W*x + bw mask is applied to dp
        k_bwd_colsum<<<(C + 31) / 32, 256, 0, st>>>(dp, N, C, m.bw, dbw);
        k_bwd_colsum<<<(C + 31) / 32, 256, 0, st>>>(dq, N, C, m.br, dbr);
        if (m.ih_linear)
            k_bwd_apply_mask<<<grid_for(N * C, 256, h->sm_count), 256, 0, st>>>(dp, m.ih_linear, N * C);
        if (m.h0) k_bwd_apply_mask<<<grid_for((long long)NH, 256, h->sm_count), 256, 0, st>>>(dh, m.h0, (long long)NH);
        h->launches += T + 2 + (m.ih_linear ? 1 : 0) + (m.h0 ? 1 : 0);
    }
    // dx[n][i] = sum_m dp[n][m] * W_t[m][i]
    if ((rc = gemm_f32(h, GemmF32{dp, false, W_t, false, dx, N, C, I, false, m.x}, st))) return rc;
    // dR[k][m] += sum_n h[n][k] * dq[n][m]   (h_all's first T slots: h_{t-1} of every step)
    if ((rc = gemm_f32(h, GemmF32{h_all, true, dq, false, dR, H, N, C, true, m.R}, st))) return rc;
    // dW[i][m] += sum_n x_t[i][n] * dp[n][m]
    if ((rc = gemm_f32(h, GemmF32{x_t, false, dp, false, dW, I, N, C, true, m.W}, st))) return rc;
    CK(cudaGetLastError());
    return QGRU_OK;
}

}  // extern "C"
