// qgru_float.cu - the unquantized fp32 GRU ("float mode") and the MinMax calibration pass.
//
// Float mode follows hasteGRUForward / ForwardPass<float> of the reference
// (src/gru_interface.cc:173-207, src/gru_forward_gpu.cu:23-125, 342-414): one product for W*x
// over all timesteps, then the recurrence in one launch (qgru_rec_f32.cu; wider layers than its
// registers hold, and more rows than pay there, run step by step).  Calibration runs the same forward with the gate buffer kept and
// folds the min/max of every operator in one pass over it - the reference
// materialises five capture tensors and seven temporaries of T*B*H floats and reduces each in
// its own pass (src/calibration_gpu.cu:1776-1953).
#include <cfloat>

#include "qgru_gemm_f32.cuh"
#include "qgru_handle.h"
#include "qgru_rec_f32.cuh"

using namespace qgru;

namespace {

// ---- order-preserving float <-> uint mapping so min/max can use integer atomics
__device__ __forceinline__ unsigned f2key(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
inline float key2f(unsigned k) {
    const unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    float f;
    memcpy(&f, &u, 4);
    return f;
}
constexpr unsigned KEY_EMPTY_MIN = 0xffffffffu;  // larger than every finite key
constexpr unsigned KEY_EMPTY_MAX = 0u;

struct MinMax {
    float mn, mx;
    __device__ __forceinline__ void init() { mn = FLT_MAX; mx = -FLT_MAX; }
    // NaN and Inf are skipped, as the reference's reductions do (src/calibration_gpu.cu:254-259)
    __device__ __forceinline__ void add(float v) {
        if (isfinite(v)) { mn = fminf(mn, v); mx = fmaxf(mx, v); }
    }
};

__device__ __forceinline__ void warp_fold(MinMax m, unsigned *acc_min, unsigned *acc_max, int slot,
                                          bool any) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m.mn = fminf(m.mn, __shfl_xor_sync(0xffffffffu, m.mn, o));
        m.mx = fmaxf(m.mx, __shfl_xor_sync(0xffffffffu, m.mx, o));
    }
    if (any && (threadIdx.x & 31) == 0 && m.mn <= m.mx) {
        atomicMin(acc_min + slot, f2key(m.mn));
        atomicMax(acc_max + slot, f2key(m.mx));
    }
}

// ---- one timestep after R*h has been multiplied (wide layers): the float gates of
// src/gru_forward_gpu.cu:23-125 for (b, j).  rh [B][3H] holds R*h without its bias.
__global__ void __launch_bounds__(256)
k_float_step(const float *__restrict__ wx, const float *__restrict__ rh, const float *__restrict__ bw,
             const float *__restrict__ br, const float *__restrict__ h_in, float *__restrict__ h_out,
             float *__restrict__ v, int v_stride, int B, int H) {
    const int j = blockIdx.x * 128 + (threadIdx.x & 127);
    const int b = blockIdx.y * 2 + (threadIdx.x >> 7);
    if (j >= H || b >= B) return;
    const int Cn = 3 * H;
    const float *rhr = rh + (size_t)b * Cn + j;
    const float *wxr = wx + (size_t)b * Cn + j;
    const float rz = rhr[0] + br[j], rr = rhr[H] + br[H + j], rg = rhr[2 * H] + br[2 * H + j];
    const float z = 1.0f / (1.0f + expf(-((wxr[0] + bw[j]) + rz)));
    const float r = 1.0f / (1.0f + expf(-((wxr[H] + bw[H + j]) + rr)));
    const float g = tanhf((wxr[2 * H] + bw[2 * H + j]) + r * rg);
    h_out[(size_t)b * H + j] = z * h_in[(size_t)b * H + j] + (1.0f - z) * g;
    if (v) {
        // 4 slots per row: the reference's training buffer (z, r, n, Rh_n + br_n); 6 slots:
        // all three R*h + br rows as well (z, r, n, Rh_z+br_z, Rh_r+br_r, Rh_n+br_n)
        float *vb = v + (size_t)b * v_stride * H + j;
        vb[0] = z; vb[H] = r; vb[2 * H] = g;
        if (v_stride == 6) { vb[3 * H] = rz; vb[4 * H] = rr; vb[5 * H] = rg; }
        else vb[3 * H] = rg;
    }
}

// ---- min/max of the twelve operators of the cell over a whole sequence, from the forward's buffers: wx
// (W*x) [N][3H], v with six slots, h [N + B][H].  One pass at memory speed (ten reads per cell) instead of
// reductions inside the recurrence, whose registers hold R.  A thread walks rows of one unit.
__global__ void __launch_bounds__(128)
k_minmax_cell(const float *__restrict__ wx, const float *__restrict__ v, const float *__restrict__ h,
              const float *__restrict__ bw, long long N, int B, int H, unsigned *acc_min, unsigned *acc_max) {
    const int j = blockIdx.x * 128 + threadIdx.x;
    constexpr int OPS[12] = {QGRU_OP_H, QGRU_OP_IH_LINEAR, QGRU_OP_HH_LINEAR, QGRU_OP_UPDATE_IN, QGRU_OP_RESET_IN, QGRU_OP_NEW_IN,
                             QGRU_OP_UPDATE_OUT, QGRU_OP_RESET_OUT, QGRU_OP_NEW_OUT, QGRU_OP_MUL_RESET_HIDDEN,
                             QGRU_OP_MUL_NEW_CONTRIB, QGRU_OP_MUL_OLD_CONTRIB};
    MinMax m[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) m[k].init();
    if (j < H) {
        const float bz = bw[j], brr = bw[H + j], bg = bw[2 * H + j];
#pragma unroll 2
        for (long long n = blockIdx.y; n < N; n += gridDim.y) {
            const float *w = wx + n * 3 * H + j, *q = v + n * 6 * H + j;
            const float wz = w[0] + bz, wr = w[H] + brr, wg = w[2 * H] + bg;
            const float z = q[0], r = q[H], g = q[2 * H], rz = q[3 * H], rr = q[4 * H], rg = q[5 * H];
            const float h_old = h[n * H + j], hn = h[(n + B) * H + j];
            m[0].add(hn);
            m[1].add(wz); m[1].add(wr); m[1].add(wg);
            m[2].add(rz); m[2].add(rr); m[2].add(rg);
            m[3].add(wz + rz);
            m[4].add(wr + rr);
            m[5].add(wg + r * rg);
            m[6].add(z); m[7].add(r); m[8].add(g);
            m[9].add(r * rg);
            m[10].add((1.0f - z) * g);
            m[11].add(z * h_old);
        }
    }
#pragma unroll
    for (int k = 0; k < 12; ++k) warp_fold(m[k], acc_min, acc_max, OPS[k], true);
}

// min/max of a whole tensor into slot `slot` (warp shuffles, one atomic pair per warp)
__global__ void k_minmax_tensor(const float *__restrict__ x, long long n, unsigned *acc_min,
                                unsigned *acc_max, int slot) {
    MinMax m;
    m.init();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        m.add(x[i]);
    warp_fold(m, acc_min, acc_max, slot, true);
}

// per-channel min/max of a [K][Cn] matrix: one warp per 32 channels, coalesced over channels
__global__ void k_minmax_channels(const float *__restrict__ w, int K, int Cn, unsigned *cmin,
                                  unsigned *cmax) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= Cn) return;
    MinMax m;
    m.init();
    for (int k = 0; k < K; ++k) m.add(w[(size_t)k * Cn + c]);
    if (m.mn <= m.mx) {
        cmin[c] = f2key(m.mn);
        cmax[c] = f2key(m.mx);
    } else {
        cmin[c] = KEY_EMPTY_MIN;
        cmax[c] = KEY_EMPTY_MAX;
    }
}

__global__ void k_fill_u32(unsigned *p, int n, unsigned v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

__global__ void k_init_h_float(const float *__restrict__ h0, float *__restrict__ h, long long n) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) h[i] = h0 ? h0[i] : 0.f;
}

}  // namespace

namespace qgru {

int float_forward(qgru_handle *h, int T, int B, const float *W, const float *R, const float *bw,
                  const float *br, const float *x, const float *h0, float *h_out, float *v_out,
                  int v_stride, cudaStream_t st) {
    const int H = h->H, Cn = h->C, I = h->I;
    const long long N = (long long)T * B;
    int rc;
    if ((rc = ensure(h, h->f_wx, (size_t)N * Cn * 4))) return rc;
    float *wx = (float *)h->f_wx.p;
    const long long NH = (long long)B * H;
    k_init_h_float<<<(unsigned)((NH + 255) / 256), 256, 0, st>>>(h0, h_out, NH);
    h->launches++;
    if ((rc = gemm_f32(h, GemmF32{x, false, W, false, wx, N, I, Cn}, st))) return rc;
    if (float_chain_is_faster(h, T, B))
        return float_chain_launch(h, FloatFwdArgs{T, B, H, R, wx, bw, br, h_out, v_out, v_stride, 0, 0, OutView()}, st);
    // wide layers, very many rows or a step or two, step by step: R*h as a tiled product, then the pointwise gates
    if ((rc = ensure(h, h->f_acc2, (size_t)B * Cn * 4))) return rc;
    float *rh = (float *)h->f_acc2.p;
    dim3 grid((H + 127) / 128, (B + 1) / 2);
    for (int t = 0; t < T; ++t) {
        const float *hin = h_out + (size_t)t * NH;
        float *hout = h_out + (size_t)(t + 1) * NH;
        float *vt = v_out ? v_out + (size_t)t * B * v_stride * H : nullptr;
        if ((rc = gemm_f32(h, GemmF32{hin, false, R, false, rh, B, H, Cn}, st))) return rc;
        k_float_step<<<grid, 256, 0, st>>>(wx + (size_t)t * B * Cn, rh, bw, br, hin, hout, vt, v_stride, B, H);
        h->launches++;
    }
    CK(cudaGetLastError());
    return QGRU_OK;
}

}  // namespace qgru

extern "C" {

int qgru_forward_float(qgru_handle *h, int T, int B, const float *W, const float *R, const float *bw,
                       const float *br, const float *x, const float *h0, float *h_out, float *v_out,
                       void *stream) {
    if (!h || !W || !R || !bw || !br || !x || !h_out) return QGRU_ERR_BAD_ARG;
    if (T <= 0 || B <= 0) return fail(h, QGRU_ERR_BAD_ARG, "T and B must be positive");
    CK(cudaSetDevice(h->device));
    USE_HANDLE(h, (cudaStream_t)stream);
    return float_forward(h, T, B, W, R, bw, br, x, h0, h_out, v_out, 4, (cudaStream_t)stream);
}

int qgru_calibrate_minmax(qgru_handle *h, int T, int B, const float *W, const float *R,
                          const float *bw, const float *br, const float *x, const float *h0,
                          qgru_ranges *ranges, float *h_out, void *stream) {
    if (!h || !W || !R || !bw || !br || !x || !ranges) return QGRU_ERR_BAD_ARG;
    if (T <= 0 || B <= 0) return fail(h, QGRU_ERR_BAD_ARG, "T and B must be positive");
    if (ranges->hidden != h->H) return fail(h, QGRU_ERR_BAD_ARG, "ranges.hidden != handle hidden_size");
    if (!ranges->min_W || !ranges->max_W || !ranges->min_R || !ranges->max_R || !ranges->min_bw ||
        !ranges->max_bw || !ranges->min_br || !ranges->max_br)
        return fail(h, QGRU_ERR_BAD_ARG, "ranges: per-channel arrays missing");
    CK(cudaSetDevice(h->device));
    cudaStream_t st = (cudaStream_t)stream;
    USE_HANDLE(h, st);
    const int H = h->H, Cn = h->C;
    const size_t nh = (size_t)(T + 1) * B * H;
    int rc;
    float *hbuf = h_out;
    if (!hbuf) {
        if ((rc = ensure(h, h->f_h, nh * 4))) return rc;
        hbuf = (float *)h->f_h.p;
    }
    // accumulators: [0,17) scalar min keys, [17,34) scalar max keys, then 4 x (min[3H], max[3H])
    const int n_acc = 2 * QGRU_NUM_OPS + 8 * Cn;
    if ((rc = ensure(h, h->f_acc, (size_t)n_acc * 4))) return rc;
    unsigned *acc = (unsigned *)h->f_acc.p;
    unsigned *acc_min = acc, *acc_max = acc + QGRU_NUM_OPS, *ch = acc + 2 * QGRU_NUM_OPS;
    k_fill_u32<<<1, 32, 0, st>>>(acc_min, QGRU_NUM_OPS, KEY_EMPTY_MIN);
    k_fill_u32<<<1, 32, 0, st>>>(acc_max, QGRU_NUM_OPS, KEY_EMPTY_MAX);
    const long long nx = (long long)T * B * h->I;
    k_minmax_tensor<<<grid_for(nx, 256, h->sm_count), 256, 0, st>>>(x, nx, acc_min, acc_max, QGRU_OP_X);
    const float *mats[4] = {W, R, bw, br};
    const int rows[4] = {h->I, H, 1, 1};
    for (int k = 0; k < 4; ++k)
        k_minmax_channels<<<(Cn + 127) / 128, 128, 0, st>>>(mats[k], rows[k], Cn, ch + (2 * k) * Cn, ch + (2 * k + 1) * Cn);
    h->launches += 7;
    const long long N = (long long)T * B;
    if ((rc = ensure(h, h->f_v, (size_t)N * 6 * H * 4))) return rc;
    if ((rc = float_forward(h, T, B, W, R, bw, br, x, h0, hbuf, (float *)h->f_v.p, 6, st))) return rc;
    const dim3 mg((H + 127) / 128, (unsigned)std::min<long long>(N, std::max(1, 8 * h->sm_count / ((H + 127) / 128))));
    k_minmax_cell<<<mg, 128, 0, st>>>((const float *)h->f_wx.p, (const float *)h->f_v.p, hbuf, bw, N, B, H, acc_min, acc_max);
    h->launches++;
    CK(cudaGetLastError());
    std::vector<unsigned> host(n_acc);
    CK(cudaMemcpyAsync(host.data(), acc, (size_t)n_acc * 4, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    for (int i = 0; i < QGRU_NUM_OPS; ++i) {
        if (host[i] == KEY_EMPTY_MIN && host[QGRU_NUM_OPS + i] == KEY_EMPTY_MAX) continue;
        ranges->min_v[i] = std::min(ranges->min_v[i], key2f(host[i]));
        ranges->max_v[i] = std::max(ranges->max_v[i], key2f(host[QGRU_NUM_OPS + i]));
    }
    float *mins[4] = {ranges->min_W, ranges->min_R, ranges->min_bw, ranges->min_br};
    float *maxs[4] = {ranges->max_W, ranges->max_R, ranges->max_bw, ranges->max_br};
    for (int k = 0; k < 4; ++k) {
        const unsigned *kmin = host.data() + 2 * QGRU_NUM_OPS + (2 * k) * Cn, *kmax = kmin + Cn;
        for (int c = 0; c < Cn; ++c) {
            if (kmin[c] == KEY_EMPTY_MIN && kmax[c] == KEY_EMPTY_MAX) continue;
            mins[k][c] = std::min(mins[k][c], key2f(kmin[c]));
            maxs[k][c] = std::max(maxs[k][c], key2f(kmax[c]));
        }
    }
    return QGRU_OK;
}

}  // extern "C"
