// qgru_hist.cu - histogram calibration: 2048-bin histograms with range growth of every operator
// of the float GRU, collected on the GPU, and the Percentile / SQNR parameter derivation.
//
// Follows the reference's GPU collector (GPUHistogramCollector::collect,
// src/calibration_gpu.cu:820-876; build_histogram :499-522; redistribute_histogram :524-540;
// kernels :66-158) and its driver collectAllHistogramsGPU
// (src/histogram_calibration_utils.cu:18-123): per tensor and per batch a min/max pass over the
// finite values, the host range rules (first batch fixes the range limit, later batches grow
// the range inside it), a proportional redistribution of the old counts when the range
// changes, and the binning pass.  Differences in how the work is done, not in what is counted:
// the gate tensors are not materialised - one pass over the float forward's buffers takes the ranges of
// all twelve operators of the cell, a second one bins them (each value is computed in registers and
// counted in the block's own twelve histograms) - and a batch is two such passes with ONE host
// synchronisation between them, where all ranges come back at once; the per-channel weight
// histograms are built by one block per channel.  The SQNR search over the candidates of every
// histogram and the percentile scan run on the GPU; what decides a result is re-evaluated by the host
// functions that define it (see k_sqnr_search).
//
// Float expressions that decide a bin keep the reference kernels' operand order, with explicit
// round-to-nearest multiplies and adds so that no fused multiply-add changes a boundary case.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include "qgru_handle.h"

using namespace qgru;

namespace qgru {
int float_forward(qgru_handle *h, int T, int B, const float *W, const float *R, const float *bw,
                  const float *br, const float *x, const float *h0, float *h_out, float *v_out,
                  int v_stride, cudaStream_t st);
}  // namespace qgru

// One collector: counts live on the device, range and bookkeeping on the host.
struct HistMeta {
    float min_val = FLT_MAX, max_val = -FLT_MAX;
    long long total = 0;
    bool valid = false;
    bool stored = false;           // the counts hold something (else they read as zeros)
    bool limit_set = false;
    float limit_min = 0.f, limit_max = 0.f;
};

struct qgru_hist {
    int device = 0, H = 0, bins = 0, n = 0;
    void *own = nullptr;           // storage, where it was allocated here
    float *d_counts = nullptr;     // [n][bins]; a histogram that holds nothing yet is not cleared
    float *d_tmp = nullptr;        // [bins] redistribution target
    unsigned *d_keys = nullptr;    // [MAX_JOBS][2] min / max keys of one batch's collections
    float *d_mm = nullptr;         // [4][2][3H] per-channel minima and maxima of W, R, bw, br
    char *d_scratch = nullptr;     // parameter derivation: per histogram an index, a search job and its result
    float *d_gather = nullptr;     // [GATHER][bins] histograms on their way to the host
    std::vector<HistMeta> meta;
    StreamOrder order;
    bool channels_done[4] = {false, false, false, false};
    std::string err;
};

namespace {

constexpr int GATHER = 128;
constexpr size_t DERIVE_BYTES = 144;   // of scratch per histogram
constexpr int MAX_JOBS = 32;     // collections of one batch: x, twelve operators of the cell, at most twelve weight tensors

// ---- a tensor, or a column block of a [K][ld] matrix
struct Gen {
    const float *p0;
    int ld, c0, width;   // width 0: p0[i]; else p0[k * ld + c0 + j], i = k * width + j
    long long n;         // number of elements
};

__device__ __forceinline__ float gen_value(const Gen &g, long long i) {
    if (g.width == 0) return g.p0[i];
    const long long k = i / g.width;
    return g.p0[k * g.ld + g.c0 + (int)(i - k * g.width)];
}

// ---- the cell's twelve operators from the float forward's buffers: wx (W*x), v (z, r, n, R*h + br) with six slots
// per row, h with the initial state in front.  CELL_SLOT: the operator each value counts for.
constexpr int CELL_VALUES = 16;   // h; three of W*x + bw; three of R*h + br; gate inputs; gate outputs; three products
constexpr int CELL_COUNT = 12;
__device__ constexpr int CELL_SLOT[CELL_VALUES] = {0, 1, 1, 1, 2, 2, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11};
constexpr int CELL_OPS[CELL_COUNT] = {QGRU_OP_H, QGRU_OP_IH_LINEAR, QGRU_OP_HH_LINEAR, QGRU_OP_UPDATE_IN, QGRU_OP_RESET_IN,
                                      QGRU_OP_NEW_IN, QGRU_OP_UPDATE_OUT, QGRU_OP_RESET_OUT, QGRU_OP_NEW_OUT,
                                      QGRU_OP_MUL_RESET_HIDDEN, QGRU_OP_MUL_NEW_CONTRIB, QGRU_OP_MUL_OLD_CONTRIB};
struct CellSrc {
    const float *wx, *v, *h, *bw;
    long long N;
    int B, H;
};
__device__ __forceinline__ void cell_values(const CellSrc &c, long long n, int j, float bz, float br, float bn, float (&x)[CELL_VALUES]) {
    const int H = c.H;
    const float *w = c.wx + n * 3 * H + j, *q = c.v + n * 6 * H + j;
    const float z = q[0], r = q[H], g = q[2 * H], rz = q[3 * H], rr = q[4 * H], rg = q[5 * H];
    const float h_old = c.h[n * H + j];
    x[0] = c.h[(n + c.B) * H + j];
    x[1] = w[0] + bz;
    x[2] = w[H] + br;
    x[3] = w[2 * H] + bn;
    x[4] = rz;
    x[5] = rr;
    x[6] = rg;
    x[7] = x[1] + rz;
    x[8] = x[2] + rr;
    x[13] = __fmul_rn(r, rg);
    x[9] = x[3] + x[13];
    x[10] = z;
    x[11] = r;
    x[12] = g;
    x[14] = __fmul_rn(1.0f - z, g);
    x[15] = __fmul_rn(z, h_old);
}

// ordered-integer keys so that float min/max can use integer atomics
__device__ __forceinline__ unsigned fkey(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
inline float key_to_float(unsigned k) {
    const unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
constexpr unsigned KEY_MIN_EMPTY = 0xffffffffu, KEY_MAX_EMPTY = 0u;

// min / max of the finite values (compute_minmax of the reference filters inf and NaN)
__global__ void __launch_bounds__(256) k_hist_minmax(Gen g, unsigned *mm) {
    float mn = FLT_MAX, mx = -FLT_MAX;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < g.n;
         i += (long long)gridDim.x * blockDim.x) {
        const float v = gen_value(g, i);
        if (isfinite(v)) {
            mn = fminf(mn, v);
            mx = fmaxf(mx, v);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0 && mn <= mx) {
        atomicMin(mm, fkey(mn));
        atomicMax(mm + 1, fkey(mx));
    }
}

// keys of a batch's collections before the range pass
__global__ void k_hist_clear_keys(unsigned *keys) {
    if (threadIdx.x < MAX_JOBS * 2) keys[threadIdx.x] = threadIdx.x & 1 ? KEY_MAX_EMPTY : KEY_MIN_EMPTY;
}

// ranges of the cell's operators: a thread walks rows of one unit
__global__ void __launch_bounds__(128) k_hist_cell_minmax(CellSrc c, unsigned *keys) {
    const int j = blockIdx.x * 128 + threadIdx.x;
    float mn[CELL_COUNT], mx[CELL_COUNT];
#pragma unroll
    for (int k = 0; k < CELL_COUNT; ++k) {
        mn[k] = FLT_MAX;
        mx[k] = -FLT_MAX;
    }
    if (j < c.H) {
        const float bz = c.bw[j], br = c.bw[c.H + j], bn = c.bw[2 * c.H + j];
        // two rows at a time (the second may be the first again): twenty loads in flight per thread
        for (long long n = blockIdx.y; n < c.N; n += 2ll * gridDim.y) {
            float x[CELL_VALUES], x2[CELL_VALUES];
            cell_values(c, n, j, bz, br, bn, x);
            cell_values(c, n + gridDim.y < c.N ? n + gridDim.y : n, j, bz, br, bn, x2);
#pragma unroll
            for (int k = 0; k < CELL_VALUES; ++k)
                if (isfinite(x2[k])) {
                    mn[CELL_SLOT[k]] = fminf(mn[CELL_SLOT[k]], x2[k]);
                    mx[CELL_SLOT[k]] = fmaxf(mx[CELL_SLOT[k]], x2[k]);
                }
#pragma unroll
            for (int k = 0; k < CELL_VALUES; ++k)
                if (isfinite(x[k])) {
                    mn[CELL_SLOT[k]] = fminf(mn[CELL_SLOT[k]], x[k]);
                    mx[CELL_SLOT[k]] = fmaxf(mx[CELL_SLOT[k]], x[k]);
                }
        }
    }
#pragma unroll
    for (int k = 0; k < CELL_COUNT; ++k) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
            mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
        }
    }
    // one pair of atomics per operator and block: they all go to 24 words
    __shared__ float red[2][CELL_COUNT][4];
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int k = 0; k < CELL_COUNT; ++k) {
            red[0][k][threadIdx.x >> 5] = mn[k];
            red[1][k][threadIdx.x >> 5] = mx[k];
        }
    __syncthreads();
    if (threadIdx.x < CELL_COUNT) {
        const int k = threadIdx.x;
        const float lo = fminf(fminf(red[0][k][0], red[0][k][1]), fminf(red[0][k][2], red[0][k][3]));
        const float hi = fmaxf(fmaxf(red[1][k][0], red[1][k][1]), fmaxf(red[1][k][2], red[1][k][3]));
        if (lo <= hi) {
            atomicMin(keys + 2 * k, fkey(lo));
            atomicMax(keys + 2 * k + 1, fkey(hi));
        }
    }
}

// histogram_kernel_shared (src/calibration_gpu.cu:66-104): values below / above the range go to
// the first / last bin, non-finite values are skipped; counts are whole numbers held as float.  The block
// counts in integers (native shared-memory atomics; a float add there is a compare-and-swap loop).
struct BinRange {
    float min_val, max_val, inv_bw;
    float *counts;
};
__device__ __forceinline__ void bin_value(float v, const BinRange &r, int bins, unsigned *sh) {
    if (!isfinite(v)) return;
    int b;
    if (v < r.min_val) b = 0;
    else if (v > r.max_val) b = bins - 1;
    else b = min((int)__fmul_rn(v - r.min_val, r.inv_bw), bins - 1);
    atomicAdd(&sh[b], 1u);
}

__global__ void __launch_bounds__(256) k_hist_add(Gen g, BinRange r, int bins) {
    extern __shared__ unsigned sh[];
    for (int i = threadIdx.x; i < bins; i += blockDim.x) sh[i] = 0u;
    __syncthreads();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < g.n;
         i += (long long)gridDim.x * blockDim.x)
        bin_value(gen_value(g, i), r, bins, sh);
    __syncthreads();
    for (int i = threadIdx.x; i < bins; i += blockDim.x)
        if (sh[i]) atomicAdd(&r.counts[i], (float)sh[i]);
}

struct CellRanges {
    BinRange r[CELL_COUNT];
};
// The twelve operators of the cell in one pass: twelve histograms per block (98 KB at 2048 bins, two
// blocks per SM).  Bound by the shared-memory atomics, 16 per cell.
__global__ void __launch_bounds__(512) k_hist_cell_add(CellSrc c, const __grid_constant__ CellRanges rg, int bins) {
    extern __shared__ unsigned sh[];
    for (int i = threadIdx.x; i < CELL_COUNT * bins; i += blockDim.x) sh[i] = 0u;
    __syncthreads();
    const long long total = c.N * c.H;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long n = i / c.H;
        const int j = (int)(i - n * c.H);
        float x[CELL_VALUES];
        cell_values(c, n, j, c.bw[j], c.bw[c.H + j], c.bw[2 * c.H + j], x);
#pragma unroll
        for (int k = 0; k < CELL_VALUES; ++k) bin_value(x[k], rg.r[CELL_SLOT[k]], bins, sh + CELL_SLOT[k] * bins);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < CELL_COUNT * bins; i += blockDim.x)
        if (sh[i]) atomicAdd(&rg.r[i / bins].counts[i % bins], (float)sh[i]);
}

// redistribute_histogram_kernel (src/calibration_gpu.cu:116-158): each source bin goes to the
// destination bin holding its left edge; the share beyond that bin's right edge goes to the
// bin one destination width further.
__global__ void k_hist_redistribute(const float *__restrict__ src, float src_min, float src_bw,
                                    float *__restrict__ dst, float dst_min, float dst_bw, int bins) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= bins) return;
    const float count = src[i];
    if (count <= 0) return;
    const float inv = 1.0f / dst_bw;
    const float start = __fmaf_rn((float)i, src_bw, src_min);   // fused, as the reference's kernel compiles
    int d = (int)__fmul_rn(start - dst_min, inv);
    d = min(d, bins - 1);
    const float end = __fmaf_rn(dst_bw, (float)(d + 1), dst_min);
    const float split = rintf(__fmul_rn((end - start) / src_bw, count));
    const float first = fminf(split, count);
    atomicAdd(&dst[d], first);
    const float rest = count - first;
    if (rest > 0) {
        int o = (int)__fmul_rn(__fadd_rn(start, dst_bw) - dst_min, inv);
        o = min(o, bins - 1);
        atomicAdd(&dst[o], rest);
    }
}

// per-channel ranges of a [K][C] matrix (compute_per_channel_minmax_kernel, :232-275; degenerate ranges widened
// as collect_per_channel_histograms_batch does on the host, :600-620).  32 channels x 8 row lanes a block.
__global__ void __launch_bounds__(256) k_channel_range(const float *__restrict__ w, int K, int C, float tiny_range, float *mins, float *maxs) {
    __shared__ float smn[8][32], smx[8][32];
    const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5, c = blockIdx.x * 32 + cx;
    float mn = FLT_MAX, mx = -FLT_MAX;
    if (c < C)
        for (int k = ry; k < K; k += 8) {
            const float v = w[(size_t)k * C + c];
            if (isfinite(v)) {
                mn = fminf(mn, v);
                mx = fmaxf(mx, v);
            }
        }
    smn[ry][cx] = mn;
    smx[ry][cx] = mx;
    __syncthreads();
    if (ry || c >= C) return;
    for (int k = 1; k < 8; ++k) {
        mn = fminf(mn, smn[k][cx]);
        mx = fmaxf(mx, smx[k][cx]);
    }
    if (mn > mx) mn = mx = 0.0f;
    if (mn == mx) {
        mn -= 0.5f;
        mx += 0.5f;
    }
    const float range = mx - mn;
    if (range < tiny_range || isnan(range) || isinf(range)) {
        mn = fminf(mn, 0.0f);
        mx = mn + tiny_range;
    }
    mins[c] = mn;
    maxs[c] = mx;
}

// build_per_channel_histogram_kernel (:389-440): one block per channel, ranges prepared on the host
__global__ void __launch_bounds__(128) k_channel_hist(const float *__restrict__ w, int K, int C,
                                                      const float *__restrict__ mins,
                                                      const float *__restrict__ maxs, float *counts, int bins) {
    extern __shared__ unsigned sh[];
    const int c = blockIdx.x;
    for (int i = threadIdx.x; i < bins; i += blockDim.x) sh[i] = 0u;
    __syncthreads();
    const float mn = mins[c], mx = maxs[c];
    float bw = (mx - mn) / bins;
    if (bw < 1e-9f) bw = 1e-9f;
    const BinRange r{mn, mx, 1.0f / bw, nullptr};
    for (int k = threadIdx.x; k < K; k += blockDim.x) bin_value(w[(size_t)k * C + c], r, bins, sh);
    __syncthreads();
    float *out = counts + (size_t)c * bins;
    for (int i = threadIdx.x; i < bins; i += blockDim.x) out[i] = (float)sh[i];
}

// ---- parameter derivation
// Which candidates of a histogram's SQNR search can be the best: noise of every candidate, over
// the histogram's occupied bins; then the candidates within `margin` of the smallest, as a bit mask.  The
// result is defined by the host's sums, whose terms come from the C library's powf and may differ from
// a product in the last bit.  Two fp32 sums of n such terms in the same order differ by less than
// (2 n + 16) * 2^-24 of themselves, so with a margin of twice that the host's winner is always in the
// mask, and where the mask holds one candidate (nearly always: the candidates' noises differ by far
// more) nothing is left to compute.
// (That bound does not ask for the order: a sum of n non-negative terms is within n * 2^-24 of the exact one in any.)
// One block per histogram, as many neighbouring lanes to a candidate as 1024 threads have for all of them: an operator of 2048
// occupied bins and 357 candidates is the longest chain (about 110 cycles a term, a division among them), and with a thread a
// candidate, three in turn, it was the whole launch.  3101 histograms (H = 256, per-channel weights), 101 or 357
// candidates: 128 threads 0.37 ms, 1024 threads 0.08 ms; the whole derivation took 61 ms on 16 host threads.
constexpr int SQNR_WORDS = 12;   // at most 17 * 21 = 357 candidates
constexpr int SQNR_THREADS = 1024;
__global__ void __launch_bounds__(SQNR_THREADS) k_sqnr_search(const float *__restrict__ counts, const int *__restrict__ index,
                                                              const SqnrSearch *__restrict__ jobs, int bins,
                                                              unsigned *__restrict__ mask) {
    __shared__ float val[2048], cnt[2048];
    __shared__ float noise_s[SQNR_WORDS * 32];
    __shared__ unsigned err_s[SQNR_WORDS * 32];   // one occupied bin: the candidate's error and clip flag
    __shared__ int warp_n[SQNR_THREADS / 32], base;
    __shared__ unsigned best_key;
    const SqnrSearch q = jobs[blockIdx.x];
    const float *src = counts + (size_t)index[blockIdx.x] * bins;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        base = 0;
        best_key = 0xffffffffu;
    }
    __syncthreads();
    for (int i0 = 0; i0 < bins; i0 += SQNR_THREADS) {   // occupied bins, in order
        const int i = i0 + tid;
        const float c = i < bins ? src[i] : 0.f;
        const bool on = i < bins && !(c < 1e-6f);
        const unsigned b = __ballot_sync(0xffffffffu, on);
        if (lane == 0) warp_n[warp] = __popc(b);
        __syncthreads();
        if (warp == 0) {                                // where each warp's bins go
            const int mine = warp_n[lane];
            int sum = mine;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += y;
            }
            warp_n[lane] = base + sum - mine;
            __syncwarp();
            if (lane == 31) base += sum;
        }
        __syncthreads();
        if (on) {
            const int at = warp_n[warp] + __popc(b & ((1u << lane) - 1u));
            val[at] = __fadd_rn(q.hmin, __fmul_rn((float)i + 0.5f, q.bw));
            cnt[at] = c;
        }
        __syncthreads();
    }
    const int n = base;
    int lanes = 32;                                     // per candidate
    while (lanes > 1 && q.n * lanes > SQNR_THREADS) lanes >>= 1;
    for (int c0 = 0; c0 < q.n; c0 += SQNR_THREADS / lanes) {
        const int c = c0 + tid / lanes;
        float delta = 0.f, offset = 0.f;
        if (c < q.n) sqnr_candidate(q, c, &delta, &offset);
        float noise = 0.f;
        unsigned err_bits = 0;
        if (delta > 0) {
#pragma unroll 4
            for (int i = tid % lanes; i < n; i += lanes) {
                const float x = val[i];
                float t = rintf(__fsub_rn(__fdiv_rn(x, delta), offset));
                const bool clipped = t < 0 || t > q.steps;
                t = fmaxf(0.0f, fminf(q.steps, t));
                const float e = __fsub_rn(__fmul_rn(__fadd_rn(t, offset), delta), x);
                err_bits = (__float_as_uint(e) & 0x7fffffffu) | (clipped ? 0x80000000u : 0u);
                float err = __fmul_rn(e, e);
                if (clipped) err = __fmul_rn(err, 3.0f);
                noise = __fadd_rn(noise, __fmul_rn(err, cnt[i]));
            }
        }
        for (int o = 1; o < lanes; o <<= 1) noise += __shfl_xor_sync(0xffffffffu, noise, o);
        if (c < q.n && tid % lanes == 0) {
            if (!(delta > 0)) noise = FLT_MAX;
            noise_s[c] = noise;
            err_s[c] = err_bits;
            if (noise < FLT_MAX) atomicMin(&best_key, __float_as_uint(noise));   // non-negative: ordered as integers
        }
    }
    __syncthreads();
    if (best_key == 0xffffffffu) {
        if (tid < SQNR_WORDS) mask[blockIdx.x * SQNR_WORDS + tid] = 0u;
        return;
    }
    const float limit = __uint_as_float(best_key) * (1.0f + (float)(4 * n + 32) * 0x1p-24f);
    if (warp < SQNR_WORDS) {
        const int c = warp * 32 + lane;
        bool in = c < q.n && noise_s[c] <= limit;
        // a bias: one value, and the same error from candidates that are multiples of each other; the first wins
        if (in && n == 1)
            for (int k = 0; k < c && in; ++k) in = err_s[k] != err_s[c] || noise_s[k] > limit;
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (lane == 0) mask[blockIdx.x * SQNR_WORDS + warp] = b;
    }
}

// Histogram::getPercentileRange's two bins (include/histogram_collector.h:105-165): the cumulative counts are
// summed one after another in fp32, as the reference does (above 2^24 the order matters).  One warp per
// histogram.  out: first bin at or above each threshold, or -1, -1 where the whole range is taken.
__global__ void __launch_bounds__(32) k_percentile_bins(const float *__restrict__ counts, const int *__restrict__ index, int bins,
                                                        float clip, int2 *__restrict__ out) {
    __shared__ float cum[2048];
    const float *src = counts + (size_t)index[blockIdx.x] * bins;
    for (int i = threadIdx.x; i < bins; i += 32) cum[i] = src[i];
    __syncwarp();
    if (threadIdx.x != 0) return;
    float s = cum[0];
#pragma unroll 8
    for (int i = 1; i < bins; ++i) {
        s = __fadd_rn(s, cum[i]);
        cum[i] = s;
    }
    int lo = 0, hi = bins - 1;
    if (s < 1e-6f) {
        lo = hi = -1;
    } else {
        // (the sums do not decrease: binary search)
        const auto first = [&](float thr, int none) {
            int a = 0, b = bins;
            while (a < b) {
                const int m = (a + b) / 2;
                if (cum[m] >= thr) b = m;
                else a = m + 1;
            }
            return a < bins ? a : none;
        };
        lo = first(__fmul_rn(s, clip), 0);
        hi = first(__fmul_rn(s, 1.0f - clip), bins - 1);
    }
    out[blockIdx.x] = make_int2(lo, hi);
}

__global__ void k_gather_hist(const float *__restrict__ counts, const int *__restrict__ index, int bins, float *__restrict__ out) {
    const float *src = counts + (size_t)index[blockIdx.x] * bins;
    for (int i = threadIdx.x; i < bins; i += blockDim.x) out[(size_t)blockIdx.x * bins + i] = src[i];
}

int hfail(qgru_hist *hs, int code, const std::string &msg) {
    hs->err = msg;
    return code;
}
#define HCK(call)                                                                       \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess) {                                                        \
            cudaGetLastError();                                                         \
            return hfail(hs, QGRU_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
        }                                                                               \
    } while (0)

float min_scale_bins(int bins) { return std::min(1.19209290e-07f, 0.01f / static_cast<float>(bins)); }

int blocks_for(long long n) { return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 1184)); }

BinRange bin_range(const qgru_hist *hs, float *counts, float min_val, float max_val) {
    float bw = (max_val - min_val) / hs->bins;                  // build_histogram, :503-505
    if (bw < 1e-9f) bw = 1e-9f;
    return BinRange{min_val, max_val, 1.0f / bw, counts};
}

// The host rules of GPUHistogramCollector::collect for collector `idx` and a batch of n values whose range keys
// are `keys`: new range, old counts moved into it, and where the new values are to be counted.
int begin_collect(qgru_hist *hs, int idx, const unsigned *keys, long long n, BinRange *out, cudaStream_t st) {
    HistMeta &m = hs->meta[idx];
    float *counts = hs->d_counts + (size_t)idx * hs->bins;
    float dmin, dmax;
    if (keys[0] == KEY_MIN_EMPTY && keys[1] == KEY_MAX_EMPTY) {
        dmin = dmax = 0.0f;                                     // nothing finite
    } else {
        dmin = key_to_float(keys[0]);
        dmax = key_to_float(keys[1]);
    }
    if (dmin == dmax) {                                         // :829-832
        dmin -= 0.5f;
        dmax += 0.5f;
    }
    const float tiny_range = min_scale_bins(hs->bins) * hs->bins;
    float range = dmax - dmin;
    if (range < tiny_range || std::isnan(range) || std::isinf(range)) {   // :839-844
        dmin = std::min(dmin, 0.0f);
        dmax = std::max(dmax, 0.0f);
        range = tiny_range;
        dmax = dmin + tiny_range;
    }
    if (!m.valid) {
        HCK(cudaMemsetAsync(counts, 0, (size_t)hs->bins * 4, st));
        m.min_val = dmin;
        m.max_val = dmax;
        m.total = n;
        m.valid = m.stored = true;
        // growth limit is infinite (HistogramCollector::Config), as in the reference's default
        m.limit_min = dmin - range * INFINITY / 2.0f;
        m.limit_max = dmax + range * INFINITY / 2.0f;
        m.limit_set = true;
    } else {
        float new_min, new_max;
        if (m.limit_set) {
            new_min = std::max(m.limit_min, std::min(dmin, m.min_val));
            new_max = std::min(m.limit_max, std::max(dmax, m.max_val));
        } else {
            new_min = std::min(dmin, m.min_val);
            new_max = std::max(dmax, m.max_val);
        }
        if (new_min != m.min_val || new_max != m.max_val) {
            // _merge_with_extended_range_gpu, :924-955
            HCK(cudaMemsetAsync(hs->d_tmp, 0, (size_t)hs->bins * 4, st));
            const float src_bw = (hs->bins <= 0 || m.max_val <= m.min_val) ? 1.0f : (m.max_val - m.min_val) / hs->bins;
            if (std::fabs(src_bw) >= min_scale_bins(hs->bins) && !std::isnan(src_bw) && !std::isinf(src_bw)) {
                const float s_bw = (m.max_val - m.min_val) / hs->bins;      // redistribute_histogram, :528-530
                float d_bw = (new_max - new_min) / hs->bins;
                if (d_bw < 1e-9f) d_bw = 1e-9f;
                k_hist_redistribute<<<(hs->bins + 255) / 256, 256, 0, st>>>(counts, m.min_val, s_bw, hs->d_tmp,
                                                                            new_min, d_bw, hs->bins);
            }
            HCK(cudaMemcpyAsync(counts, hs->d_tmp, (size_t)hs->bins * 4, cudaMemcpyDeviceToDevice, st));
            m.min_val = new_min;
            m.max_val = new_max;
        }
        m.total += n;
    }
    *out = bin_range(hs, counts, m.min_val, m.max_val);
    return QGRU_OK;
}

Gen plain(const float *p, long long n) {
    Gen g{};
    g.p0 = p;
    g.n = n;
    return g;
}

struct Job {
    int idx;
    Gen g;
};

// One batch: the ranges of every tensor (and of the cell's operators), one synchronisation, then the counts.
// chan: per-channel histograms to build (matrix, rows), null where not asked for.
int collect_batch(qgru_hist *hs, const std::vector<Job> &jobs, const CellSrc *cell, const float *const chan[4], const int chan_rows[4],
                  cudaStream_t st) {
    const int C = 3 * hs->H, bins = hs->bins, base_job = cell ? CELL_COUNT : 0;
    if (base_job + (int)jobs.size() > MAX_JOBS) return hfail(hs, QGRU_ERR_BAD_ARG, "too many collections in one batch");
    StreamUse use(hs->order, st);
    HCK(use.begin());
    k_hist_clear_keys<<<1, 2 * MAX_JOBS, 0, st>>>(hs->d_keys);
    const float tiny_range = min_scale_bins(bins) * bins;
    std::vector<float> mm;
    for (int k = 0; k < 4 && chan; ++k)
        if (chan[k]) {
            k_channel_range<<<(C + 31) / 32, 256, 0, st>>>(chan[k], chan_rows[k], C, tiny_range, hs->d_mm + (size_t)2 * k * C,
                                                          hs->d_mm + (size_t)(2 * k + 1) * C);
            k_channel_hist<<<C, 128, (size_t)bins * 4, st>>>(chan[k], chan_rows[k], C, hs->d_mm + (size_t)2 * k * C,
                                                            hs->d_mm + (size_t)(2 * k + 1) * C,
                                                            hs->d_counts + (size_t)(QGRU_HIST_CHANNEL0 + k * C) * bins, bins);
            mm.resize((size_t)8 * C);
        }
    if (cell) {
        const int bx = (cell->H + 127) / 128;
        const dim3 grid(bx, (unsigned)std::min<long long>(cell->N, std::max(1, 1184 / bx)));
        k_hist_cell_minmax<<<grid, 128, 0, st>>>(*cell, hs->d_keys);
    }
    for (size_t i = 0; i < jobs.size(); ++i)
        if (jobs[i].g.n > 0)
            k_hist_minmax<<<blocks_for(jobs[i].g.n), 256, 0, st>>>(jobs[i].g, hs->d_keys + 2 * (base_job + i));
    unsigned keys[2 * MAX_JOBS];
    HCK(cudaMemcpyAsync(keys, hs->d_keys, sizeof(keys), cudaMemcpyDeviceToHost, st));
    if (!mm.empty()) HCK(cudaMemcpyAsync(mm.data(), hs->d_mm, mm.size() * 4, cudaMemcpyDeviceToHost, st));
    HCK(cudaStreamSynchronize(st));
    int rc;
    if (cell) {
        CellRanges rg;
        for (int k = 0; k < CELL_COUNT; ++k) {
            const int op = CELL_OPS[k];
            const long long n = cell->N * cell->H * (op == QGRU_OP_IH_LINEAR || op == QGRU_OP_HH_LINEAR ? 3 : 1);
            if ((rc = begin_collect(hs, op, keys + 2 * k, n, &rg.r[k], st))) return rc;
        }
        const size_t smem = (size_t)CELL_COUNT * bins * 4;
        HCK(cudaFuncSetAttribute(k_hist_cell_add, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        const long long blocks = std::max<long long>(1, std::min<long long>((cell->N * cell->H + 8191) / 8192, 296));
        k_hist_cell_add<<<(unsigned)blocks, 512, smem, st>>>(*cell, rg, bins);
    }
    for (size_t i = 0; i < jobs.size(); ++i) {
        if (jobs[i].g.n <= 0) continue;
        BinRange r;
        if ((rc = begin_collect(hs, jobs[i].idx, keys + 2 * (base_job + i), jobs[i].g.n, &r, st))) return rc;
        k_hist_add<<<blocks_for(jobs[i].g.n), 256, (size_t)bins * 4, st>>>(jobs[i].g, r, bins);
    }
    HCK(cudaGetLastError());
    for (int k = 0; k < 4 && chan; ++k)
        if (chan[k]) {
            for (int c = 0; c < C; ++c) {
                HistMeta &m = hs->meta[QGRU_HIST_CHANNEL0 + k * C + c];
                m.min_val = mm[(size_t)2 * k * C + c];
                m.max_val = mm[(size_t)(2 * k + 1) * C + c];
                m.total = chan_rows[k];
                m.valid = m.stored = true;
            }
            hs->channels_done[k] = true;
        }
    return QGRU_OK;
}

size_t hist_storage(int H, int bins) {
    const size_t n = QGRU_HIST_CHANNEL0 + (size_t)4 * 3 * H;
    return ((n + 1 + GATHER) * bins + (size_t)8 * 3 * H + 2 * MAX_JOBS) * 4 + 64 + n * DERIVE_BYTES;
}

}  // namespace

extern "C" {

size_t qgru_hist_bytes(int hidden_size, int num_bins) {
    return hidden_size > 0 && num_bins > 0 && num_bins <= 2048 ? hist_storage(hidden_size, num_bins) : 0;
}

int qgru_hist_create_in(qgru_hist **out, int device, int hidden_size, int num_bins, void *storage, size_t bytes) {
    if (!out || hidden_size <= 0 || num_bins <= 0 || num_bins > 2048 || !storage || bytes < hist_storage(hidden_size, num_bins))
        return QGRU_ERR_BAD_ARG;
    *out = nullptr;
    qgru_hist *hs = new qgru_hist();
    hs->device = device;
    hs->H = hidden_size;
    hs->bins = num_bins;
    hs->n = QGRU_HIST_CHANNEL0 + 4 * 3 * hidden_size;
    hs->meta.resize(hs->n);
    float *p = (float *)storage;
    hs->d_counts = p;
    hs->d_tmp = p += (size_t)hs->n * num_bins;
    hs->d_mm = p += num_bins;
    hs->d_gather = p += (size_t)8 * 3 * hidden_size;
    hs->d_keys = (unsigned *)(p += (size_t)GATHER * num_bins);
    hs->d_scratch = (char *)(((uintptr_t)(p + 2 * MAX_JOBS) + 63) & ~(uintptr_t)63);
    *out = hs;
    return QGRU_OK;
}

int qgru_hist_create(qgru_hist **out, int device, int hidden_size, int num_bins) {
    if (!out || hidden_size <= 0 || num_bins <= 0 || num_bins > 2048) return QGRU_ERR_BAD_ARG;
    *out = nullptr;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) {
        cudaGetLastError();
        return QGRU_ERR_CUDA;
    }
    void *p = nullptr;
    const size_t bytes = hist_storage(hidden_size, num_bins);
    if (cudaSetDevice(device) != cudaSuccess || cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        return QGRU_ERR_NOMEM;
    }
    const int rc = qgru_hist_create_in(out, device, hidden_size, num_bins, p, bytes);
    if (rc == QGRU_OK) (*out)->own = p;
    else cudaFree(p);
    return rc;
}

void qgru_hist_destroy(qgru_hist *hs) {
    if (!hs) return;
    if (hs->own) {
        cudaSetDevice(hs->device);
        cudaFree(hs->own);
        cudaGetLastError();
    }
    hs->order.destroy();
    delete hs;
}

const char *qgru_hist_last_error(const qgru_hist *hs) { return hs ? hs->err.c_str() : "null histogram set"; }

int qgru_hist_count(const qgru_hist *hs) { return hs ? hs->n : 0; }

int qgru_hist_reset(qgru_hist *hs) {
    if (!hs) return QGRU_ERR_BAD_ARG;
    for (HistMeta &m : hs->meta) m = HistMeta();
    for (bool &b : hs->channels_done) b = false;
    return QGRU_OK;
}

int qgru_hist_collect(qgru_hist *hs, int index, const float *data, long long n, void *stream) {
    if (!hs || !data || index < 0 || index >= hs->n || n < 0) return QGRU_ERR_BAD_ARG;
    HCK(cudaSetDevice(hs->device));
    if (n == 0) return QGRU_OK;
    return collect_batch(hs, {Job{index, plain(data, n)}}, nullptr, nullptr, nullptr, (cudaStream_t)stream);
}

int qgru_hist_export(const qgru_hist *hs_c, int index, float *counts, float *min_val, float *max_val,
                     int64_t *total_count) {
    qgru_hist *hs = const_cast<qgru_hist *>(hs_c);
    if (!hs || index < 0 || index >= hs->n) return QGRU_ERR_BAD_ARG;
    const HistMeta &m = hs->meta[index];
    if (min_val) *min_val = m.min_val;
    if (max_val) *max_val = m.max_val;
    if (total_count) *total_count = m.valid ? m.total : 0;
    if (counts && !m.stored) {
        std::fill(counts, counts + hs->bins, 0.0f);
    } else if (counts) {
        HCK(cudaSetDevice(hs->device));
        HCK(cudaDeviceSynchronize());   // the last batch's counts may still be on their way, on any stream
        HCK(cudaMemcpy(counts, hs->d_counts + (size_t)index * hs->bins, (size_t)hs->bins * 4, cudaMemcpyDeviceToHost));
    }
    return QGRU_OK;
}

int qgru_hist_import(qgru_hist *hs, int index, const float *counts, float min_val, float max_val,
                     int64_t total_count) {
    if (!hs || !counts || index < 0 || index >= hs->n || total_count < 0) return QGRU_ERR_BAD_ARG;
    HCK(cudaSetDevice(hs->device));
    HCK(cudaDeviceSynchronize());   // counts may be on their way, on any stream, and so may the work of whoever had this memory before
    HCK(cudaMemcpy(hs->d_counts + (size_t)index * hs->bins, counts, (size_t)hs->bins * 4, cudaMemcpyHostToDevice));
    HistMeta &m = hs->meta[index];
    m = HistMeta();
    m.min_val = min_val;
    m.max_val = max_val;
    m.total = total_count;
    m.valid = total_count > 0;
    m.stored = true;
    // GPUHistogramCollector::merge into an empty collector, src/calibration_gpu.cu:961-979
    const float tiny_range = min_scale_bins(hs->bins) * hs->bins;
    float range = max_val - min_val;
    if (range < tiny_range) range = tiny_range;
    m.limit_min = min_val - range * INFINITY / 2.0f;
    m.limit_max = max_val + range * INFINITY / 2.0f;
    m.limit_set = true;
    if (index >= QGRU_HIST_CHANNEL0) hs->channels_done[(index - QGRU_HIST_CHANNEL0) / (3 * hs->H)] = true;
    return QGRU_OK;
}

int qgru_calibrate_hist(qgru_handle *h, qgru_hist *hs, int T, int B, const float *W, const float *R,
                        const float *bw, const float *br, const float *x, const float *h0,
                        const int32_t *granularity, void *stream) {
    return qgru_calibrate_hist_h(h, hs, T, B, W, R, bw, br, x, h0, granularity, nullptr, stream);
}

int qgru_calibrate_hist_h(qgru_handle *h, qgru_hist *hs, int T, int B, const float *W, const float *R,
                          const float *bw, const float *br, const float *x, const float *h0,
                          const int32_t *granularity, float *h_out, void *stream) {
    if (!h || !hs || !W || !R || !bw || !br || !x || !granularity) return QGRU_ERR_BAD_ARG;
    if (T <= 0 || B <= 0) return fail(h, QGRU_ERR_BAD_ARG, "T and B must be positive");
    if (hs->H != h->H || hs->device != h->device)
        return fail(h, QGRU_ERR_BAD_ARG, "histogram set belongs to another hidden size or device");
    CK(cudaSetDevice(h->device));
    cudaStream_t st = (cudaStream_t)stream;
    USE_HANDLE(h, st);
    const int H = h->H, C = h->C, I = h->I;
    const long long N = (long long)T * B;
    int rc;
    float *hbuf = h_out;
    if (!hbuf) {
        if ((rc = ensure(h, h->f_h, (size_t)(T + 1) * B * H * 4))) return rc;
        hbuf = (float *)h->f_h.p;
    }
    if ((rc = ensure(h, h->f_v, (size_t)N * 6 * H * 4))) return rc;
    float *v = (float *)h->f_v.p;
    if ((rc = float_forward(h, T, B, W, R, bw, br, x, h0, hbuf, v, 6, st))) return rc;
    // the cell's operators: h (without the initial state), W*x + bw, R*h + br, gate inputs and outputs, products
    // (collectAllHistogramsGPU, :27-48, :109-117; collect_gate_histograms, src/calibration_gpu.cu:542-574)
    const CellSrc cell{(const float *)h->f_wx.p, v, hbuf, bw, N, B, H};
    std::vector<Job> jobs{Job{QGRU_OP_X, plain(x, N * I)}};
    // weights and biases by granularity (:50-97): per tensor and per gate every batch, per channel once
    const float *mats[4] = {W, R, bw, br}, *chan[4] = {};
    const int rows[4] = {I, H, 1, 1};
    static const int tensor_idx[4] = {QGRU_OP_W, QGRU_OP_R, QGRU_OP_BW, QGRU_OP_BR};
    for (int k = 0; k < 4; ++k) {
        if (granularity[k] == QGRU_PER_TENSOR) {
            jobs.push_back(Job{tensor_idx[k], plain(mats[k], (long long)rows[k] * C)});
        } else if (granularity[k] == QGRU_PER_GATE) {
            for (int g3 = 0; g3 < 3; ++g3) jobs.push_back(Job{QGRU_HIST_GATE0 + 3 * k + g3, Gen{mats[k], C, g3 * H, H, (long long)rows[k] * H}});
        } else if (!hs->channels_done[k]) {
            chan[k] = mats[k];
        }
    }
    if ((rc = collect_batch(hs, jobs, &cell, chan, rows, st))) {
        h->err = "histogram collection: " + hs->err;
        return rc;
    }
    h->launches += 4 + 2 * jobs.size();
    return QGRU_OK;
}

int qgru_calc_params_from_hist(const qgru_hist *hs_c, int use_percentile, float percentile, qgru_params *p,
                               float *scale_W, float *scale_R, float *scale_bw, float *scale_br) {
    qgru_hist *hs = const_cast<qgru_hist *>(hs_c);
    if (!hs || !p || !scale_W || !scale_R || !scale_bw || !scale_br) return QGRU_ERR_BAD_ARG;
    // ensureSymmetricWeightBiasConfig, src/gru_interface.cc:26-32
    if (!p->op[QGRU_OP_W].symmetric || !p->op[QGRU_OP_R].symmetric || !p->op[QGRU_OP_BW].symmetric ||
        !p->op[QGRU_OP_BR].symmetric)
        return QGRU_ERR_UNSUPPORTED;
    HCK(cudaSetDevice(hs->device));
    HCK(cudaDeviceSynchronize());   // the last batch's counts may still be on their way, on any stream
    const int H = hs->H, C = 3 * H, bins = hs->bins;
    const bool pot2 = p->use_pot2 != 0;
    p->hidden = H;
    // every histogram that is needed, and the operator it derives a scale for
    // (calculateGRUQuantitativeParametersFromHistograms, src/gru_interface.cc:1079-1153)
    static const int scalar_ops[] = {QGRU_OP_X, QGRU_OP_H, QGRU_OP_IH_LINEAR, QGRU_OP_HH_LINEAR,
                                     QGRU_OP_UPDATE_IN, QGRU_OP_RESET_IN, QGRU_OP_NEW_IN,
                                     QGRU_OP_UPDATE_OUT, QGRU_OP_RESET_OUT, QGRU_OP_NEW_OUT,
                                     QGRU_OP_MUL_RESET_HIDDEN, QGRU_OP_MUL_NEW_CONTRIB, QGRU_OP_MUL_OLD_CONTRIB};
    static const int tensor_idx[4] = {QGRU_OP_W, QGRU_OP_R, QGRU_OP_BW, QGRU_OP_BR};
    std::vector<int> index;
    std::vector<qgru_op> ops;
    for (int k : scalar_ops) {
        index.push_back(k);
        ops.push_back(p->op[k]);
    }
    for (int k = 0; k < 4; ++k) {
        const int n = p->granularity[k] == QGRU_PER_TENSOR ? 1 : p->granularity[k] == QGRU_PER_GATE ? 3 : C;
        const int first = p->granularity[k] == QGRU_PER_TENSOR ? tensor_idx[k]
                          : p->granularity[k] == QGRU_PER_GATE ? QGRU_HIST_GATE0 + 3 * k : QGRU_HIST_CHANNEL0 + k * C;
        for (int i = 0; i < n; ++i) {
            index.push_back(first + i);
            ops.push_back(p->op[tensor_idx[k]]);
        }
    }
    const int n = (int)index.size();
    for (int i = 0; i < n; ++i) {
        const HistMeta &m = hs->meta[index[i]];
        if (!m.valid || m.total <= 0) return hfail(hs, QGRU_ERR_NOT_READY, "histogram " + std::to_string(index[i]) + " is empty");
        if ((int64_t)op_qmax(ops[i]) - op_qmin(ops[i]) <= 0) return hfail(hs, QGRU_ERR_BAD_ARG, "operator without a range");
    }
    std::vector<SqnrSearch> search(use_percentile ? 0 : n);
    for (size_t i = 0; i < search.size(); ++i) {
        const HistMeta &m = hs->meta[index[i]];
        search[i] = hist_sqnr_search(bins, m.min_val, m.max_val, ops[i]);
    }
    // device scratch: indices, then search jobs and masks, or percentile bins
    const size_t idx_b = ((size_t)n * 4 + 15) & ~size_t(15), job_b = (search.size() * sizeof(SqnrSearch) + 15) & ~size_t(15);
    static_assert(sizeof(SqnrSearch) + SQNR_WORDS * 4 + 4 + 32 <= DERIVE_BYTES, "scratch per histogram (each part rounded up)");
    HCK(cudaMemcpyAsync(hs->d_scratch, index.data(), (size_t)n * 4, cudaMemcpyHostToDevice, 0));
    const int *d_index = (const int *)hs->d_scratch;
    int rc = QGRU_OK;
    if (use_percentile) {
        const float clip = (100.0f - percentile) / 100.0f;
        std::vector<int2> found(n, make_int2(-1, -1));
        if (clip > 0.0f) {
            int2 *d_out = (int2 *)(hs->d_scratch + idx_b);
            k_percentile_bins<<<n, 32, 0, 0>>>(hs->d_counts, d_index, bins, clip, d_out);
            HCK(cudaGetLastError());
            HCK(cudaMemcpyAsync(found.data(), d_out, (size_t)n * sizeof(int2), cudaMemcpyDeviceToHost, 0));
        }
        HCK(cudaStreamSynchronize(0));
        for (int i = 0; i < n && rc == QGRU_OK; ++i) {
            const HistMeta &m = hs->meta[index[i]];
            rc = hist_percentile_finish(bins, m.min_val, m.max_val, found[i].x < 0, found[i].x, found[i].y, pot2, &ops[i]);
        }
    } else {
        SqnrSearch *d_jobs = (SqnrSearch *)(hs->d_scratch + idx_b);
        unsigned *d_mask = (unsigned *)(hs->d_scratch + idx_b + job_b);
        HCK(cudaMemcpyAsync(d_jobs, search.data(), search.size() * sizeof(SqnrSearch), cudaMemcpyHostToDevice, 0));
        k_sqnr_search<<<n, SQNR_THREADS, 0, 0>>>(hs->d_counts, d_index, d_jobs, bins, d_mask);
        HCK(cudaGetLastError());
        std::vector<unsigned> mask((size_t)n * SQNR_WORDS);
        HCK(cudaMemcpyAsync(mask.data(), d_mask, mask.size() * 4, cudaMemcpyDeviceToHost, 0));
        HCK(cudaStreamSynchronize(0));
        // histograms with more than one candidate left: their counts come to the host, GATHER at a time
        std::vector<int> open, best(n, -1);
        for (int i = 0; i < n; ++i) {
            int left = 0;
            for (int w = 0; w < SQNR_WORDS; ++w) {
                const unsigned b = mask[(size_t)i * SQNR_WORDS + w];
                left += __builtin_popcount(b);
                if (b && best[i] < 0) best[i] = w * 32 + __builtin_ctz(b);
            }
            if (left > 1) open.push_back(i);
        }
        std::vector<float> counts(std::min<size_t>(open.size(), GATHER) * bins);
        for (size_t o = 0; o < open.size(); o += GATHER) {
            const int no = (int)std::min<size_t>(GATHER, open.size() - o);
            std::vector<int> which(no);
            for (int i = 0; i < no; ++i) which[i] = index[open[o + i]];
            HCK(cudaMemcpyAsync(hs->d_scratch, which.data(), (size_t)no * 4, cudaMemcpyHostToDevice, 0));
            k_gather_hist<<<no, 256, 0, 0>>>(hs->d_counts, d_index, bins, hs->d_gather);
            HCK(cudaMemcpyAsync(counts.data(), hs->d_gather, (size_t)no * bins * 4, cudaMemcpyDeviceToHost, 0));
            HCK(cudaStreamSynchronize(0));
            const auto settle = [&](int k) {
                const int i = open[o + k];
                std::vector<int> list;
                for (int c = 0; c < SQNR_WORDS * 32; ++c)
                    if (mask[(size_t)i * SQNR_WORDS + c / 32] >> (c & 31) & 1) list.push_back(c);
                best[i] = hist_sqnr_best(counts.data() + (size_t)k * bins, bins, search[i], ops[i], list.data(), (int)list.size());
            };
            const unsigned nt = no < 32 ? 1u : std::max(1u, std::min(8u, std::thread::hardware_concurrency()));
            std::vector<std::thread> pool;
            for (unsigned w = 1; w < nt; ++w)
                pool.emplace_back([&, w]() { for (int k = (int)w; k < no; k += (int)nt) settle(k); });
            for (int k = 0; k < no; k += (int)nt) settle(k);
            for (std::thread &t : pool) t.join();
        }
        for (int i = 0; i < n && rc == QGRU_OK; ++i) rc = hist_sqnr_finish(search[i], best[i], pot2, &ops[i]);
    }
    if (rc) return hfail(hs, rc, "histogram calibration failed");
    int at = 0;
    for (int k : scalar_ops) p->op[k] = ops[at++];
    float *scales[4] = {scale_W, scale_R, scale_bw, scale_br};
    for (int k = 0; k < 4; ++k) {
        if (p->granularity[k] == QGRU_PER_TENSOR) {
            std::fill(scales[k], scales[k] + C, ops[at++].scale);
        } else if (p->granularity[k] == QGRU_PER_GATE) {
            for (int g = 0; g < 3; ++g) std::fill(scales[k] + g * H, scales[k] + (g + 1) * H, ops[at++].scale);
        } else {
            for (int c = 0; c < C; ++c) scales[k][c] = ops[at++].scale;
        }
        p->op[tensor_idx[k]].scale = scales[k][0];
        p->op[tensor_idx[k]].zero_point = 0;
    }
    return qgru_generate_luts(p);
}

}  // extern "C"
