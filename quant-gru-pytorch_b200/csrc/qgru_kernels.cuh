// qgru_kernels.cuh - device code of the integer GRU forward: boundary quantize kernels,
// the SIMT input-projection GEMM, the persistent recurrence kernel and the generic
// (any bit width) fallback kernels.  Include from ONE translation unit only (it defines
// non-template __global__ functions).  Written for sm_100a; one CTA per SM is assumed for the
// persistent kernel (it claims most of the 227 KB of shared memory).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "qgru_device.cuh"
#include "qgru_internal.h"

namespace qgru {

// --------------------------------------------------------- boundary kernels (a12, a13)

// quantize(float, FixedPointScale, zp, bw) (include/quantize_ops_helper.h:528-533): IEEE
// division by the decoded 16-bit-mantissa scale, round half to even, add zp in float.
__device__ __forceinline__ int32_t quantize_one(float x, float scale, int32_t zp, int32_t lo,
                                                int32_t hi) {
    const float q = rintf(__fdiv_rn(x, scale)) + (float)zp;
    return clampi((int32_t)q, lo, hi);
}

// quantize_f of the float-storage path (include/quantize_ops_helper.h:514-519): the zero point is added before
// rounding, and the value stays a float.
__device__ __forceinline__ float fs_quantize_raw(float x, float scale, int32_t zp) { return rintf(x / scale + (float)zp); }

// What every forward does before its first product, in ONE launch: activations to 8-bit rows padded to
// Kpad (zeros), the initial state to its 8-bit rows and, for the slot layouts, to the outputs' first slot.
// The status words of the call before are cleared.
// Mode 0: fp32 in, integer quantize; 1: fp32 in, float-storage quantize; 2: int32 containers (values
// outside the operator's range, which the reference's quantize step would have clamped, raise bit 0
// of flags[0]; the caller clears the flags beforehand).
struct PrologueArgs {
    const void *x;               // row n = t * B + b at x + t * x_ts + b * x_bs; null: only the state
    long long x_ts, x_bs, N;
    int B, K, Kpad;
    uint8_t *x8;
    void *xq;                    // optional dense copy of the quantized values: int32 (mode 0) or float (mode 1)
    float *xd;                   // optional dense copy of what the quantized values stand for: (q - zp) * scale (modes 0, 1)
    uint8_t *keep;               // optional mask, 1 = the value was not clamped (modes 0, 1)
    float x_scale;
    int32_t x_zp, x_lo, x_hi;
    const void *h0;              // [B][H] fp32 (modes 0, 1) or int32 (mode 2); null: the zero point
    uint8_t *h8;                 // [B][Hpad]
    int H, Hpad;
    OutView slot;                // outputs of the initial slot (slot 0), each may be null
    float h_scale;
    int32_t h_zp, h_lo, h_hi;
    uint8_t *h0_keep;            // optional mask of the initial state (modes 0, 1)
    int *flags;                  // [2]
    int clear;                   // clear the flags
    int q_blocks;                // blocks that quantize x; the rest write the state
    unsigned long long *stamp;   // start time, or null
};

template <int Mode>
__device__ __forceinline__ int32_t prologue_quantize(const void *src, long long i, float scale, int32_t zp, int32_t lo, int32_t hi,
                                                     uint8_t &keep, int *flags) {
    keep = 1;
    if constexpr (Mode == 0) {
        // (quantize_one with its flag: quantize<true>, include/quantize_ops_helper.h:528-533)
        const int32_t q = (int32_t)(rintf(__fdiv_rn(static_cast<const float *>(src)[i], scale)) + (float)zp);
        keep = (q < lo || q > hi) ? 0 : 1;
        return clampi(q, lo, hi);
    } else if constexpr (Mode == 1) {
        const float raw = fs_quantize_raw(static_cast<const float *>(src)[i], scale, zp);
        keep = (raw < (float)lo || raw > (float)hi) ? 0 : 1;
        return (int32_t)fmaxf((float)lo, fminf(raw, (float)hi));
    } else {
        const int32_t q = static_cast<const int32_t *>(src)[i];
        if (q < lo || q > hi) atomicOr(flags, 1);
        return q;
    }
}

// prologue_quantize of four values without division or conversions.  t = x * (1 / scale), in mode 1 with the zero point, differs from what
// is rounded there by less than 2^-22 (|t| + |zp|), and the two round to different integers only if a half lies between them.  t + MAGIC
// (in mode 0 with the zero point: a whole number) is the rounded value in the low bits of a float, where also the limits are.
// Where a half is within 2^-21 (|t| + |zp|), or t is no number below 2^20, the four are divided: one lane in some hundreds.
constexpr float PROLOGUE_MAGIC = 12582912.0f;        // 2^23 + 2^22
struct PrologueNear {
    float inv, base, zp, limit, lo, hi;
    template <int Mode>
    static __device__ __forceinline__ PrologueNear make(const PrologueArgs &a) {
        PrologueNear n;
        n.zp = (float)a.x_zp;
        n.inv = a.x_zp > -(1 << 20) && a.x_zp < (1 << 20) ? __frcp_rn(a.x_scale) : __int_as_float(0x7fffffff);
        n.base = PROLOGUE_MAGIC + (Mode == 0 ? n.zp : 0.f);
        n.limit = 0.5f - (Mode == 0 ? 0.f : fabsf(n.zp) * 0x1p-21f);
        n.lo = PROLOGUE_MAGIC + (float)a.x_lo;
        n.hi = PROLOGUE_MAGIC + (float)a.x_hi;
        return n;
    }
};

// q[v] + MAGIC, clamped, in q and before the clamp in raw (different from q is all that counts)
template <int Mode>
__device__ __forceinline__ void prologue_quantize4(const PrologueArgs &a, const PrologueNear &n, const float4 &x, float (&q)[4], float (&raw)[4]) {
    const float f[4] = {x.x, x.y, x.z, x.w};
    float worst = 0.f;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const float t = Mode == 0 ? __fmul_rn(f[v], n.inv) : __fmaf_rn(f[v], n.inv, n.zp);
        raw[v] = __fadd_rn(t, n.base);
        const float near = __fmaf_rn(fabsf(t), 0x1p-21f, fabsf(__fsub_rn(t, __fsub_rn(raw[v], n.base))));
        asm("max.NaN.f32 %0, %0, %1;" : "+f"(worst) : "f"(near));
        q[v] = fminf(fmaxf(raw[v], n.lo), n.hi);
    }
    if (worst < n.limit) return;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        uint8_t keep;
        q[v] = PROLOGUE_MAGIC + (float)prologue_quantize<Mode>(f, v, a.x_scale, a.x_zp, a.x_lo, a.x_hi, keep, nullptr);
        raw[v] = keep ? q[v] : 0.f;
    }
}

__device__ __forceinline__ void put4(float *p, const float4 &y, bool wide) {
    if (wide) *reinterpret_cast<float4 *>(p) = y;
    else p[0] = y.x, p[1] = y.y, p[2] = y.z, p[3] = y.w;
}

// Vec (rows and base aligned, K a multiple of 4): a warp takes four neighbouring units of 128 columns, a lane four columns of each:
// one 128-bit load and one store of each kind, whole lines.  Memory-bound: 409600 x 128 fp32 60 us, 51200 x 256 with the training
// outputs 22 us (16 columns a thread and a division a value: 77 and 92; conversions and no division: 77 and 26).
// Else a thread takes 16 columns with scalar loads.
template <int Mode, bool Vec>
__global__ void __launch_bounds__(256) k_prologue(const PrologueArgs a) {
    pdl_trigger();
    put_stamp(a.stamp);
    if (blockIdx.x == 0 && threadIdx.x == 0 && a.clear) {
        a.flags[0] = 0;
        a.flags[1] = 0;
    }
    if ((int)blockIdx.x < a.q_blocks) {
        if constexpr (Vec) {
            const int nch = a.Kpad >> 7, lane = threadIdx.x & 31;
            const unsigned units = (unsigned)(a.N * nch), stride = a.q_blocks * 32u;   // (2^32 units would be 512 GB of bytes in x8)
            const PrologueNear near = PrologueNear::make<Mode>(a);
            const int im = __float_as_int(PROLOGUE_MAGIC);
            const bool wide = ((reinterpret_cast<uintptr_t>(a.xq) | reinterpret_cast<uintptr_t>(a.xd) | reinterpret_cast<uintptr_t>(a.keep) * 4) & 15u) == 0;
            for (unsigned u = (blockIdx.x * 8u + (threadIdx.x >> 5)) * 4u; u < units; u += stride) {
                // this unit's row and columns; the next three by one step each
                const unsigned row0 = u / (unsigned)nch, t0 = row0 / (unsigned)a.B;
                int ch = (int)(u - row0 * nch), b = (int)(row0 - t0 * a.B);
                unsigned row = row0;
                const float *src = static_cast<const float *>(a.x) + t0 * a.x_ts + b * a.x_bs;
                float4 in[4];
                unsigned rows[4];
                int ks[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int k = ch * 128 + lane * 4;
                    rows[e] = row;
                    ks[e] = u + e < units ? k : 1 << 30;
                    in[e] = u + e < units && k < a.K ? *reinterpret_cast<const float4 *>(src + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                    if (++ch == nch) {
                        ch = 0;
                        ++row;
                        src += a.x_bs;
                        if (++b == a.B) {
                            b = 0;
                            src += a.x_ts - a.B * a.x_bs;
                        }
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int k = ks[e];
                    if (k >= a.Kpad) continue;
                    uint32_t w = 0;
                    if (k < a.K) {
                        float q[4], raw[4];
                        prologue_quantize4<Mode>(a, near, in[e], q, raw);
                        w = __byte_perm(__byte_perm(__float_as_uint(q[0]), __float_as_uint(q[1]), 0x0040),
                                        __byte_perm(__float_as_uint(q[2]), __float_as_uint(q[3]), 0x0040), 0x5410);
                        const long long at = (long long)rows[e] * a.K + k;
                        const int i[4] = {__float_as_int(q[0]) - im, __float_as_int(q[1]) - im, __float_as_int(q[2]) - im, __float_as_int(q[3]) - im};
                        if (a.xq)
                            put4(static_cast<float *>(a.xq) + at,
                                 Mode == 1 ? make_float4((float)i[0], (float)i[1], (float)i[2], (float)i[3])
                                           : make_float4(__int_as_float(i[0]), __int_as_float(i[1]), __int_as_float(i[2]), __int_as_float(i[3])), wide);
                        if (a.xd)
                            put4(a.xd + at, make_float4((float)(i[0] - a.x_zp) * a.x_scale, (float)(i[1] - a.x_zp) * a.x_scale,
                                                        (float)(i[2] - a.x_zp) * a.x_scale, (float)(i[3] - a.x_zp) * a.x_scale), wide);
                        if (a.keep) {
                            const uchar4 y = make_uchar4(raw[0] == q[0], raw[1] == q[1], raw[2] == q[2], raw[3] == q[3]);
                            if (wide) *reinterpret_cast<uchar4 *>(a.keep + at) = y;
                            else a.keep[at] = y.x, a.keep[at + 1] = y.y, a.keep[at + 2] = y.z, a.keep[at + 3] = y.w;
                        }
                    }
                    *reinterpret_cast<uint32_t *>(a.x8 + (long long)rows[e] * a.Kpad + k) = w;
                }
            }
            return;
        }
        const int kw = a.Kpad >> 4;
        const long long total = a.N * kw;
        for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += a.q_blocks * 256ll) {
            const long long row = i / kw;
            const int k0 = (int)(i - row * kw) * 16;
            const long long t = row / a.B, src = t * a.x_ts + (row - t * a.B) * a.x_bs;
            unsigned w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                if (k0 + 4 * g >= a.K) continue;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int k = k0 + 4 * g + u;
                    if (k >= a.K) continue;
                    uint8_t keep;
                    const int32_t q = prologue_quantize<Mode>(a.x, src + k, a.x_scale, a.x_zp, a.x_lo, a.x_hi, keep, a.flags);
                    w[g] |= ((unsigned)q & 0xffu) << (8 * u);
                    if (a.xq) {
                        if constexpr (Mode == 1) static_cast<float *>(a.xq)[row * a.K + k] = (float)q;
                        else static_cast<int32_t *>(a.xq)[row * a.K + k] = q;
                    }
                    if (Mode != 2 && a.xd) a.xd[row * a.K + k] = (float)(q - a.x_zp) * a.x_scale;
                    if (Mode != 2 && a.keep) a.keep[row * a.K + k] = keep;
                }
            }
            reinterpret_cast<uint4 *>(a.x8)[i] = make_uint4(w[0], w[1], w[2], w[3]);
        }
        return;
    }
    // initial state: quantGRUForwardInt32's h_q[0] fill (src/gru_interface.cc:568-574; the float entry point
    // dequantizes that slot like every other, :704); float storage: src/gru_interface.cc:949-961
    const long long total = (long long)a.B * a.Hpad;
    for (long long i = (blockIdx.x - a.q_blocks) * 256ll + threadIdx.x; i < total; i += (long long)(gridDim.x - a.q_blocks) * 256) {
        const int b = (int)(i / a.Hpad), j = (int)(i % a.Hpad);
        int32_t q = 0;
        if (j < a.H) {
            uint8_t keep = 1;
            q = a.h0 ? prologue_quantize<Mode>(a.h0, (long long)b * a.H + j, a.h_scale, a.h_zp, a.h_lo, a.h_hi, keep, a.flags)
                     : (Mode == 1 ? (int32_t)fmaxf((float)a.h_lo, fminf((float)a.h_zp, (float)a.h_hi)) : a.h_zp);
            put_state(a.slot, 0, b, j, a.H, false, q, a.h_zp, a.h_scale);
            if (a.h0_keep) a.h0_keep[(size_t)b * a.H + j] = keep;
        }
        if (a.h8) a.h8[i] = (uint8_t)q;
    }
}

// fp32 -> int32 containers (generic path and x_q_out).
__global__ void k_quantize_f32_i32(const float *__restrict__ x, int32_t *__restrict__ out,
                                   long long n, float scale, int32_t zp, int32_t lo, int32_t hi) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = quantize_one(x[i], scale, zp, lo, hi);
}

// The same for rows at x + t * ts + b * bs, fp32 or (is_int) already int32.
__global__ void k_gather_quantize(const void *__restrict__ x, int is_int, int32_t *__restrict__ out, long long N, int B, int K,
                                  long long ts, long long bs, float scale, int32_t zp, int32_t lo, int32_t hi) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N * K; i += (long long)gridDim.x * blockDim.x) {
        const long long row = i / K, t = row / B, at = t * ts + (row - t * B) * bs + (i - row * K);
        out[i] = is_int ? static_cast<const int32_t *>(x)[at] : quantize_one(static_cast<const float *>(x)[at], scale, zp, lo, hi);
    }
}

// Per-channel weight quantize, zp = 0 (quantificationPerChannelBitwidth,
// src/quantize_ops.cu:313; channel = idx % C).
__global__ void k_quantize_weights(const float *__restrict__ w, int32_t *__restrict__ out,
                                   long long n, int C, const float *__restrict__ scales, int32_t lo,
                                   int32_t hi) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = quantize_one(w[i], scales[i % C], 0, lo, hi);
}

// dequantize (include/quantize_ops_helper.h:504-508).
__global__ void k_dequantize(const int32_t *__restrict__ q, float *__restrict__ out, long long n,
                             float scale, int32_t zp) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = (float)(q[i] - zp) * scale;
}

// Weight repack: int32 [K][C] (haste layout) -> int8 [C][Kpad] (K contiguous, zero padded)
// plus the column sums used by the zero-point correction.  One CTA per channel.
__global__ void k_pack_weights(const int32_t *__restrict__ wq, int8_t *__restrict__ w8,
                               int32_t *__restrict__ wsum, int K, int Kpad, int C, int *err) {
    const int m = blockIdx.x;
    int local = 0;
    for (int k = threadIdx.x; k < Kpad; k += blockDim.x) {
        int32_t v = 0;
        if (k < K) {
            v = wq[(size_t)k * C + m];
            local += v;
            if (w8 && (v < -128 || v > 127)) atomicOr(err, 2);
        }
        if (w8) w8[(size_t)m * Kpad + k] = (int8_t)v;
    }
    __shared__ int red[32];
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int i = 0; i < (int)((blockDim.x + 31) >> 5); ++i) s += red[i];
        wsum[m] = s;
    }
}

// corr[m] = rescale(bias_q[m], bias_rs[m]) - zp_in * sum_k W_q[k][m]
__global__ void k_channel_consts(const int32_t *__restrict__ bias_q,
                                 const Rescale *__restrict__ bias_rs,
                                 const int32_t *__restrict__ wsum, int32_t zp_in,
                                 int64_t *__restrict__ corr, const Rescale *__restrict__ rs,
                                 FastLin *__restrict__ fl, int C, long long acc_bound, int *flags,
                                 int flag_bit) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= C) return;
    const int64_t c = rescale64((int64_t)bias_q[m], bias_rs[m]) - (int64_t)zp_in * (int64_t)wsum[m];
    corr[m] = c;
    fl[m] = make_fast_lin(rs[m], c);
    // acc + corr must stay inside int32 for the one-multiply epilogue
    const int64_t mag = c < 0 ? -c : c;
    if (mag + acc_bound >= 0x7fffffffll) atomicOr(flags, flag_bit);
    // can this channel's requantization meet an exact tie anywhere in its accumulator range?
    if (rescale_can_tie(rs[m].mult, rs[m].shift, c - acc_bound, c + acc_bound)) atomicOr(flags, flag_bit << 2);
}

// ------------------------------------------------ input projection, SIMT dp4a form (a1)

// ih[n][m] = epilogue( sum_k W8[m][k] * x8[n][k] ), n < N tokens, m < C channels.
// 64x64 output tile per CTA, 256 threads, 4x4 outputs per thread, K staged in 64-byte slabs.
// Raw: store the int32 sums themselves (no zero-point compensation, bias or requantization).
template <bool XUnsigned, typename IhT, bool Raw = false>
__global__ void __launch_bounds__(256)
k_gemm_wx_simt(const uint8_t *__restrict__ x8, const int8_t *__restrict__ w8, IhT *__restrict__ ih,
               long long N, int C, int Kpad, LinearConsts lc) {
    __shared__ unsigned xs[64][17];
    __shared__ unsigned ws[64][17];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const long long n0 = (long long)blockIdx.x * 64;
    const int m0 = blockIdx.y * 64;
    int acc[4][4] = {};
    for (int k0 = 0; k0 < Kpad; k0 += 64) {
        for (int i = threadIdx.x; i < 64 * 16; i += 256) {
            const int r = i >> 4, c = i & 15;
            const int kb = k0 + c * 4;
            unsigned xv = 0, wv = 0;
            if (kb < Kpad) {
                if (n0 + r < N) xv = *reinterpret_cast<const unsigned *>(x8 + (n0 + r) * Kpad + kb);
                if (m0 + r < C) wv = *reinterpret_cast<const unsigned *>(w8 + (size_t)(m0 + r) * Kpad + kb);
            }
            xs[r][c] = xv;
            ws[r][c] = wv;
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            unsigned xv[4];
            int wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) xv[i] = xs[ty * 4 + i][c];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = (int)ws[tx + 16 * j][c];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = dp4a_w<XUnsigned>(wv[j], xv[i], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long n = n0 + ty * 4 + i;
        if (n >= N) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int m = m0 + tx + 16 * j;
            if (m >= C) continue;
            if constexpr (Raw) ih[n * C + m] = (IhT)acc[i][j];
            else if (lc.fs != nullptr)
                ih[n * C + m] = (IhT)(int32_t)fs_linear(acc[i][j], lc.fs[m], lc.fs[lc.fs_C + m], lc.fs[2 * lc.fs_C + m],
                                                        (float)lc.zp_out, (float)lc.lo, (float)lc.hi);
            else ih[n * C + m] = (IhT)linear_epilogue(acc[i][j], lc.corr[m], lc.rs[m], lc.zp_out, lc.lo, lc.hi);
        }
    }
}

// Dense states of the step-by-step paths [(T+1)][B][H] to the view a caller asked for (slots 0 .. slots - 1 of
// `src` to slots 0 .. of the view), and the last state.
__global__ void k_scatter_states(const int32_t *__restrict__ src, OutView o, long long slots, long long hn_slot, int B, int H,
                                 int32_t zp_h, float h_scale) {
    const long long BH = (long long)B * H, total = slots * BH;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long slot = i / BH;
        const int r = (int)(i - slot * BH), b = r / H, j = r - b * H;
        put_state(o, slot, b, j, H, slot == hn_slot, src[i], zp_h, h_scale);
    }
}

// ------------------------------------------------ persistent recurrence, dp4a form (a2+a3)

struct RecArgs {
    int T, B, H, Hpad, C;
    int Hs;        // hidden units per CTA (multiple of 32)
    int Bt;        // batch rows per group
    int P;         // CTAs per group (slices of the hidden dimension)
    int reverse;
    const int8_t *r8;      // [3H][Hpad]
    const void *ih;        // [T*B][3H] int8 or int16
    uint8_t *h8;           // [2][B][Hpad] ping-pong state
    OutView out;
    LinearConsts lc;       // R*h + br epilogue
    const GateConsts *gc;  // device copy
    const int32_t *tables; // activation tables, gc->table_off indexes into it
    int n_table;           // ints in tables
    unsigned *bar;         // one counter per group, 32 words apart
    int *abort_flag;       // set when a barrier wait ran out; every CTA then leaves
    unsigned spin_limit;
    int withhold_arrive = 0;   // failure-path test: CTA 0 skips its arrival after step 0, so its group's wait runs out
    // float-storage forward (k_recurrence_gemv with Cell 3): the float cell of the reference's
    // quantGRUForwardFP; fs_chan = [3][C] offset, bias term, scale ratio of R*h + br per channel
    const float *fs_chan = nullptr;
    FsConsts fs{};
    unsigned long long *stamp = nullptr;   // start time (k_recurrence_gemv_reg)
};

// One CTA owns Hs hidden units (all three gates) of one group of Bt batch rows and keeps its
// slice of R in shared memory for all T steps.  Per step: fetch h_{t-1} of the group's rows,
// R*h with dp4a, requantize, gates, write h_t.  Groups never interact; the P CTAs of a group
// meet once per step at a counter in global memory (bounded spin).
template <bool HUnsigned, typename IhT, bool Narrow>
__global__ void __launch_bounds__(256, 1) k_recurrence_dp4a(RecArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int kw = a.Hpad >> 2;  // words per row
    // layout: GateConsts | tables | corr[3*Hs] i64 | rs[3*Hs] | Rs[3][kw][Hs] words | hs[Bt][kw] words
    GateConsts *gc = reinterpret_cast<GateConsts *>(smem_raw);
    size_t off = (sizeof(GateConsts) + 15) & ~size_t(15);
    int32_t *tables = reinterpret_cast<int32_t *>(smem_raw + off);
    off += ((size_t)a.n_table * 4 + 15) & ~size_t(15);
    int64_t *corr = reinterpret_cast<int64_t *>(smem_raw + off);
    off += (size_t)3 * a.Hs * 8;
    Rescale *rs = reinterpret_cast<Rescale *>(smem_raw + off);
    off += (size_t)3 * a.Hs * sizeof(Rescale);
    unsigned *Rs = reinterpret_cast<unsigned *>(smem_raw + off);
    off += (size_t)3 * kw * a.Hs * 4;
    unsigned *hs = reinterpret_cast<unsigned *>(smem_raw + off);

    const int grp = blockIdx.x / a.P, p = blockIdx.x % a.P;
    const int j0 = p * a.Hs, b0 = grp * a.Bt;
    const int nb = min(a.Bt, a.B - b0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    for (int i = tid; i < (int)(sizeof(GateConsts) / 4); i += 256)
        reinterpret_cast<int *>(gc)[i] = reinterpret_cast<const int *>(a.gc)[i];
    for (int i = tid; i < a.n_table; i += 256) tables[i] = a.tables[i];
    for (int i = tid; i < 3 * a.Hs; i += 256) {
        const int g = i / a.Hs, jl = i % a.Hs, j = j0 + jl;
        const bool ok = j < a.H;
        corr[i] = ok ? a.lc.corr[g * a.H + j] : 0;
        rs[i] = ok ? a.lc.rs[g * a.H + j] : Rescale{1, 1, 0, 0, 0, 0, 0, 0};
    }
    {
        const unsigned *r8w = reinterpret_cast<const unsigned *>(a.r8);
        const int total = 3 * a.Hs * kw;
        for (int i = tid; i < total; i += 256) {
            const int k4 = i % kw, gj = i / kw;
            const int g = gj / a.Hs, jl = gj % a.Hs, j = j0 + jl;
            Rs[(g * kw + k4) * a.Hs + jl] = (j < a.H) ? r8w[(size_t)(g * a.H + j) * kw + k4] : 0u;
        }
    }
    __syncthreads();

    const int JW = a.Hs >> 5;        // warps along the hidden dimension
    const int BW = 8 / JW;           // warps along the batch dimension
    const int wj = warp % JW, wb = warp / JW;
    const int jl = wj * 32 + lane, j = j0 + jl;
    const bool j_ok = j < a.H;
    constexpr int NB = 4;
    const IhT *ihp = reinterpret_cast<const IhT *>(a.ih);
    unsigned *bar = a.bar + grp * 32;
    bool dead = false;

    for (int s = 0; s < a.T; ++s) {
        const int t = a.reverse ? (a.T - 1 - s) : s;                  // x / ih time index
        const long long out_slot = a.reverse ? (a.T - 1 - s) : (s + 1);
        const uint8_t *h_cur = a.h8 + (size_t)(s & 1) * a.B * a.Hpad;
        uint8_t *h_nxt = a.h8 + (size_t)((s + 1) & 1) * a.B * a.Hpad;

        if (a.P > 1 && s > 0) {
            if (tid == 0) {
                const unsigned want = (unsigned)a.P * (unsigned)s;
                unsigned it = 0;
                while (ld_acquire(bar) < want) {
                    if (++it > a.spin_limit || (it % 1024 == 0 && *(volatile int *)a.abort_flag)) {
                        raise_abort(a.abort_flag, 1);
                        break;
                    }
                }
            }
            __syncthreads();
            if (tid == 0 && *(volatile int *)a.abort_flag) dead = true;
            if (__syncthreads_or(dead)) break;
        }

        // h_{t-1} rows of this group -> shared (L2 loads: other CTAs wrote them)
        {
            const uint4 *src = reinterpret_cast<const uint4 *>(h_cur + (size_t)b0 * a.Hpad);
            uint4 *dst = reinterpret_cast<uint4 *>(hs);
            const int total = nb * (a.Hpad >> 4);
            for (int i = tid; i < total; i += 256) dst[i] = __ldcg(src + i);
        }
        __syncthreads();

        for (int bb = wb * NB; bb < nb; bb += BW * NB) {
            int acc[NB][3];
#pragma unroll
            for (int u = 0; u < NB; ++u) acc[u][0] = acc[u][1] = acc[u][2] = 0;
            // ih loads are issued first so they fly under the dot products
            int32_t ihv[NB][3];
#pragma unroll
            for (int u = 0; u < NB; ++u) {
                const int b = bb + u;
#pragma unroll
                for (int g = 0; g < 3; ++g)
                    ihv[u][g] = (b < nb && j_ok)
                                    ? (int32_t)ihp[((size_t)t * a.B + b0 + b) * a.C + g * a.H + j]
                                    : 0;
            }
            for (int k4 = 0; k4 < kw; k4 += 4) {
                uint4 hv[NB];
#pragma unroll
                for (int u = 0; u < NB; ++u) {
                    const int b = min(bb + u, nb - 1);
                    hv[u] = *reinterpret_cast<const uint4 *>(hs + (size_t)b * kw + k4);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int wz = (int)Rs[(0 * kw + k4 + q) * a.Hs + jl];
                    const int wr = (int)Rs[(1 * kw + k4 + q) * a.Hs + jl];
                    const int wn = (int)Rs[(2 * kw + k4 + q) * a.Hs + jl];
#pragma unroll
                    for (int u = 0; u < NB; ++u) {
                        const unsigned h4 = q == 0 ? hv[u].x : q == 1 ? hv[u].y : q == 2 ? hv[u].z : hv[u].w;
                        acc[u][0] = dp4a_w<HUnsigned>(wz, h4, acc[u][0]);
                        acc[u][1] = dp4a_w<HUnsigned>(wr, h4, acc[u][1]);
                        acc[u][2] = dp4a_w<HUnsigned>(wn, h4, acc[u][2]);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < NB; ++u) {
                const int b = bb + u;
                if (b >= nb || !j_ok) continue;
                int32_t hh[3];
#pragma unroll
                for (int g = 0; g < 3; ++g)
                    hh[g] = linear_epilogue(acc[u][g], corr[g * a.Hs + jl], rs[g * a.Hs + jl],
                                            a.lc.zp_out, a.lc.lo, a.lc.hi);
                const uint8_t hb = reinterpret_cast<const uint8_t *>(hs)[(size_t)b * a.Hpad + j];
                const int32_t h_old = HUnsigned ? (int32_t)hb : (int32_t)(int8_t)hb;
                const int32_t hn = gru_cell<Narrow>(*gc, tables, ihv[u][0], ihv[u][1], ihv[u][2],
                                                    hh[0], hh[1], hh[2], h_old);
                h_nxt[(size_t)(b0 + b) * a.Hpad + j] = (uint8_t)hn;
                put_state(a.out, out_slot, b0 + b, j, a.H, s + 1 == a.T, hn, gc->zp_h, gc->h_scale);
            }
        }
        __syncthreads();
        if (a.P > 1 && tid == 0 && !(a.withhold_arrive && blockIdx.x == 0 && s == 0)) {
            __threadfence();
            atomicAdd(bar, 1u);
        }
    }
}

// ------------------------------------------- persistent recurrence, small batch (GEMV form)

// One CTA per batch row, the whole R (3H x Hpad int8, H <= 256) in shared memory for all T
// steps: rows never interact, so there is no inter-CTA synchronisation at all and the step is
// as short as one matrix-vector product plus one cell.  A quad of threads owns one hidden unit:
// each lane takes a quarter of K for the unit's three gate rows (dp4a), two shuffles add the
// partial sums, lane 0 of the quad requantizes and runs the cell.  R is stored in the order the
// threads read it ([16-byte chunk][gate][thread]), so every 128-bit load is conflict-free.
// The state h_t stays in shared memory (two buffers, one __syncthreads per step).
// Cell: 0 generic datapath, 1 its 32-bit ("narrow") rescales, 2 the tabulated branch-free cell
// (W*x+bw arrives pre-rescaled from the GEMM; every scale in shift-free form), 3 the float cell
// of the float-storage forward (W*x+bw arrives requantized by the GEMM's float epilogue).
template <bool HUnsigned, typename IhT, int Cell>
__global__ void __launch_bounds__(1024, 1) k_recurrence_gemv(const __grid_constant__ GateConsts gc, RecArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int NT = blockDim.x;             // 4 * units (units rounded up to 32)
    const int Kq = a.Hpad >> 2;            // K bytes per lane of a quad
    const int nch = Kq >> 4;               // 16-byte chunks per lane and gate row (2 or 4)
    // layout: tables | hs[2][Hs] | Rq[nch * 3][NT] uint4.  The four K-quarters of a state buffer
    // are 16 bytes further apart than their length, so that the four 16-byte segments a warp
    // reads at once fall into different banks.
    const int Qs = Kq + 16, Hs = 4 * Qs;
    int32_t *tables = reinterpret_cast<int32_t *>(smem_raw);
    size_t off = ((size_t)a.n_table * 4 + 15) & ~size_t(15);
    unsigned char *hs = smem_raw + off;
    off += (size_t)2 * Hs;
    uint4 *Rq = reinterpret_cast<uint4 *>(smem_raw + off);

    const int tid = threadIdx.x, qd = tid & 3, j = tid >> 2;
    const int b = blockIdx.x;
    const bool j_ok = j < a.H;

    for (int i = tid; i < a.n_table; i += NT) tables[i] = a.tables[i];
    for (int i = tid; i < a.Hpad; i += NT) {
        const int at = (i / Kq) * Qs + (i % Kq);
        hs[at] = a.h8[(size_t)b * a.Hpad + i];      // initial state of this row (buffer 0 of h8)
        hs[Hs + at] = 0;
    }
    const int j_at = (j / Kq) * Qs + (j % Kq);      // where unit j's byte sits in a state buffer
    for (int g = 0; g < 3; ++g)
        for (int c = 0; c < nch; ++c) {
            uint4 w = make_uint4(0u, 0u, 0u, 0u);
            if (j_ok) w = *reinterpret_cast<const uint4 *>(a.r8 + (size_t)(g * a.H + j) * a.Hpad + qd * Kq + 16 * c);
            Rq[(size_t)(c * 3 + g) * NT + tid] = w;
        }
    // per-unit constants of the R*h + br epilogue (used by lane 0 of the quad)
    int64_t corr[3] = {0, 0, 0};
    Rescale rs[3];
    FastLin fl[3];
    bool fast = a.lc.fits32 != 0;
#pragma unroll
    for (int g = 0; g < 3; ++g) {
        rs[g] = Rescale{1, 1, 0, 0, 0, 0, 0, 0};
        fl[g] = FastLin{0, 0, 0, 0, 0, 0};
        if (j_ok) {
            corr[g] = a.lc.corr[g * a.H + j];
            rs[g] = a.lc.rs[g * a.H + j];
            fl[g] = a.lc.fl[g * a.H + j];
        }
        fast = fast && fl[g].mq != 0;
    }
    float fsk[3][3] = {};
    if constexpr (Cell == 3) {
#pragma unroll
        for (int g = 0; g < 3; ++g)
#pragma unroll
            for (int k = 0; k < 3; ++k) fsk[g][k] = j_ok ? a.fs_chan[(size_t)k * a.C + g * a.H + j] : 0.f;
    }
    __syncthreads();

    const IhT *ihp = reinterpret_cast<const IhT *>(a.ih);
    const uint32_t tab = (uint32_t)__cvta_generic_to_shared(tables);
    const bool worker = qd == 0 && j_ok;
    // W*x + bw of this row: loaded one step ahead, so the cell never waits for global memory
    auto load_ih = [&](int s, int32_t (&v)[3]) {
        const int t = a.reverse ? (a.T - 1 - s) : s;
        const IhT *src = ihp + ((size_t)t * a.B + b) * a.C + j;
        v[0] = (int32_t)src[0];
        v[1] = (int32_t)src[a.H];
        v[2] = (int32_t)src[2 * a.H];
    };
    int32_t ihv[3] = {0, 0, 0};
    if (worker) load_ih(0, ihv);
    for (int s = 0; s < a.T; ++s) {
        const long long out_slot = a.reverse ? (a.T - 1 - s) : (s + 1);
        const unsigned char *h_cur = hs + (size_t)(s & 1) * Hs;
        unsigned char *h_nxt = hs + (size_t)((s + 1) & 1) * Hs;
        int32_t ihn[3] = {0, 0, 0};
        if (worker && s + 1 < a.T) load_ih(s + 1, ihn);
        int acc[3] = {0, 0, 0};
        const uint4 *hq4 = reinterpret_cast<const uint4 *>(h_cur + qd * Qs);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (c >= nch) break;
            const uint4 hv = hq4[c];
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                const uint4 w = Rq[(size_t)(c * 3 + g) * NT + tid];
                acc[g] = dp4a_w<HUnsigned>((int)w.x, hv.x, acc[g]);
                acc[g] = dp4a_w<HUnsigned>((int)w.y, hv.y, acc[g]);
                acc[g] = dp4a_w<HUnsigned>((int)w.z, hv.z, acc[g]);
                acc[g] = dp4a_w<HUnsigned>((int)w.w, hv.w, acc[g]);
            }
        }
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            acc[g] += __shfl_xor_sync(0xffffffffu, acc[g], 1);
            acc[g] += __shfl_xor_sync(0xffffffffu, acc[g], 2);
        }
        if (worker) {
            const unsigned char hb = h_cur[j_at];
            const int32_t h_old = HUnsigned ? (int32_t)hb : (int32_t)(int8_t)hb;
            int32_t hn;
            if constexpr (Cell == 2) {
                const int32_t z_d = fused_gate_fast(gc, tab, ACT_Z, ihv[0], lin_round(acc[0], fl[0]));
                const int32_t r_d = fused_gate_fast(gc, tab, ACT_R, ihv[1], lin_round(acc[1], fl[1]));
                hn = fused_finish_fast(gc, tab, ihv[2], lin_round(acc[2], fl[2]), z_d, r_d, h_old);
            } else if constexpr (Cell == 3) {
                // (computing the update and the reset gate on two lanes of the quad measured no faster)
                const float fih[3] = {(float)ihv[0], (float)ihv[1], (float)ihv[2]};
                float fhh[3];
#pragma unroll
                for (int g = 0; g < 3; ++g)
                    fhh[g] = fs_linear(acc[g], fsk[g][0], fsk[g][1], fsk[g][2], a.fs.zp_hh, a.fs.hh_lo, a.fs.hh_hi);
                const float u_g = fs_sigmoid_gate_tab(a.fs, tab, 0, fih[0], fhh[0]);
                const float r_g = fs_sigmoid_gate_tab(a.fs, tab, 1, fih[1], fhh[1]);
                hn = (int32_t)fs_finish_tab(a.fs, tab, u_g, r_g, fih[2], fhh[2], (float)h_old);
            } else {
                int32_t hh[3];
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    if (fast) hh[g] = linear_epilogue_fast(acc[g], fl[g], a.lc.zp_out, a.lc.lo, a.lc.hi);
                    else hh[g] = linear_epilogue(acc[g], corr[g], rs[g], a.lc.zp_out, a.lc.lo, a.lc.hi);
                }
                hn = gru_cell<Cell == 1>(gc, tables, ihv[0], ihv[1], ihv[2], hh[0], hh[1], hh[2], h_old);
            }
            h_nxt[j_at] = (unsigned char)hn;
            put_state(a.out, out_slot, b, j, a.H, s + 1 == a.T, hn, gc.zp_h, gc.h_scale);
        }
        ihv[0] = ihn[0];
        ihv[1] = ihn[1];
        ihv[2] = ihn[2];
        __syncthreads();
    }
}

// The same with R in REGISTERS (the branch-free cells only): two threads own one hidden unit, each
// half of K for the unit's three gate rows, i.e. 3 * KT bytes of R (KT = Hpad / 2 = 64 or 128) held
// in 48 or 96 registers for all T steps.  A step then reads only the state (a few hundred bytes,
// broadcast) from shared memory instead of all of R (196 KB at H = 256, which at 128 bytes per
// clock is 1536 cycles on its own): KT / 4 * 3 dp4a per thread.  The threads of the upper K half
// are the upper half of the CTA's warps: they hand their three partial sums over through shared
// memory (a named barrier they only arrive on), and the lower half's warps run the cell with every
// lane busy.  The per-unit constants of the R*h + br requantization live in shared memory (the
// registers belong to R).  What is no part of the step's chain (W*x + bw of the next steps, the output of the last one) the upper
// half does while the lower one computes the cell.
// H = 256, one row: 0.91 -> 0.82 us a step (about 1150 cycles of dp4a, 400 of cell); H = 128: 0.52 -> 0.43.
// Cell: 2 the tabulated integer cell, 3 the float cell of the float-storage forward (as in k_recurrence_gemv).
template <bool HUnsigned, typename IhT, int KT, int Cell = 2, bool Tie = true>
__global__ void __launch_bounds__(512, 1) k_recurrence_gemv_reg(const __grid_constant__ GateConsts gc, RecArgs a) {
    static_assert(Cell == 2 || Cell == 3, "the branch-free cells only");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    static_assert(KT == 64 || KT == 128, "Hpad = 128 or 256");
    constexpr int QS = KT + 16;            // the two K halves of a state buffer sit 16 bytes further apart than their length
    constexpr int HS = 2 * QS;
    const int NT = blockDim.x;             // 2 * units (units rounded up to 32: whole warps per K half)
    int32_t *tables = reinterpret_cast<int32_t *>(smem_raw);
    size_t off = ((size_t)a.n_table * 4 + 15) & ~size_t(15);
    unsigned char *hs = smem_raw + off;
    off += (size_t)2 * HS;
    int *part = reinterpret_cast<int *>(smem_raw + off);          // [3][units]: the upper K half's partial sums
    off += (size_t)3 * (NT >> 1) * sizeof(int);
    int32_t *ring = reinterpret_cast<int32_t *>(smem_raw + off);  // [2][3][units]: W*x + bw of this and the next step
    off += (size_t)6 * (NT >> 1) * sizeof(int);
    FastLin *fls = reinterpret_cast<FastLin *>(smem_raw + off);   // Cell 2: [3][units]
    float *fsk = reinterpret_cast<float *>(smem_raw + off);       // Cell 3: [3 gates][3 constants][units]

    const int tid = threadIdx.x, units = NT >> 1, half = tid >= units ? 1 : 0, j = tid - half * units;
    const int b = blockIdx.x;
    const bool j_ok = j < a.H;

    for (int i = tid; i < a.n_table; i += NT) tables[i] = a.tables[i];
    if constexpr (Cell == 2) {
        for (int i = tid; i < 3 * units; i += NT) {
            const int g = i / units, u = i % units;
            fls[i] = u < a.H ? a.lc.fl[g * a.H + u] : FastLin{0, 0, 0, 0, 0, 0};
        }
    } else {
        for (int i = tid; i < 9 * units; i += NT) {
            const int gk = i / units, u = i % units, g = gk / 3, k = gk % 3;
            fsk[i] = u < a.H ? a.fs_chan[(size_t)k * a.C + g * a.H + u] : 0.f;
        }
    }
    const int j_at = (j / KT) * QS + (j % KT);      // where unit j's byte sits in a state buffer
    uint32_t R[3][KT / 4];
#pragma unroll
    for (int g = 0; g < 3; ++g)
#pragma unroll
        for (int c = 0; c < KT / 16; ++c) {
            uint4 w = make_uint4(0u, 0u, 0u, 0u);
            if (j_ok) w = *reinterpret_cast<const uint4 *>(a.r8 + (size_t)(g * a.H + j) * a.Hpad + half * KT + 16 * c);
            R[g][4 * c + 0] = w.x;
            R[g][4 * c + 1] = w.y;
            R[g][4 * c + 2] = w.z;
            R[g][4 * c + 3] = w.w;
        }
    // (everything up to here is the handle's own and may run beside the launches before)
    pdl_wait();
    put_stamp(a.stamp);
    for (int i = tid; i < 2 * KT; i += NT) {
        const int at = (i / KT) * QS + (i % KT);
        hs[at] = a.h8[(size_t)b * a.Hpad + i];      // initial state of this row (buffer 0 of h8)
        hs[HS + at] = 0;
    }
    __syncthreads();

    const uint32_t tab = (uint32_t)__cvta_generic_to_shared(tables);
    const auto product = [&](const unsigned char *h, int (&acc)[3]) {
        acc[0] = acc[1] = acc[2] = 0;
        const uint4 *hq4 = reinterpret_cast<const uint4 *>(h);
#pragma unroll
        for (int c = 0; c < KT / 16; ++c) {
            const uint4 hv = hq4[c];
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                acc[g] = dp4a_w<HUnsigned>((int)R[g][4 * c + 0], hv.x, acc[g]);
                acc[g] = dp4a_w<HUnsigned>((int)R[g][4 * c + 1], hv.y, acc[g]);
                acc[g] = dp4a_w<HUnsigned>((int)R[g][4 * c + 2], hv.z, acc[g]);
                acc[g] = dp4a_w<HUnsigned>((int)R[g][4 * c + 3], hv.w, acc[g]);
            }
        }
    };
    // (a thread without a unit reads its neighbour's)
    const IhT *ih_in = reinterpret_cast<const IhT *>(a.ih) + ((size_t)(a.reverse ? a.T - 1 : 0) * a.B + b) * a.C + min(j, a.H - 1);
    const ptrdiff_t ih_step = (a.reverse ? -(ptrdiff_t)a.B : (ptrdiff_t)a.B) * a.C;
    // fp32 output alone, as a module asks for it: a running pointer instead of the address arithmetic of every view
    const bool plain = a.out.hf && !a.out.hq && !a.out.h8;
    float *hf = plain ? a.out.hf + (size_t)(a.reverse ? a.T - 1 : 1) * a.out.ts + (size_t)b * a.out.bs + j : nullptr;
    const long long hf_step = a.reverse ? -(long long)a.out.ts : (long long)a.out.ts;
    const auto emit = [&](int s, int32_t hn) {       // state after step s of unit j
        if (!j_ok) return;
        if (plain) {
            const float f = (float)(hn - gc.zp_h) * gc.h_scale;
            *hf = f;
            if (s + 1 == a.T && a.out.hn_f) a.out.hn_f[(size_t)b * a.H + j] = f;
            hf += hf_step;
        } else {
            put_state(a.out, a.reverse ? (a.T - 1 - s) : (s + 1), b, j, a.H, s + 1 == a.T, hn, gc.zp_h, gc.h_scale);
        }
    };
    if (half) {
        // The upper half hands its partial sums to the lower half's thread of the same unit and has nothing to wait for.  While
        // that computes the cell it stores the state of the step before and fetches W*x + bw two steps ahead, so that the lower
        // half, whose chain of instructions is the step, has neither.  (The loads have no condition: the last steps read their own
        // again.  Under one, what was loaded is copied, and waited for, where the branches meet.)
        int32_t ihn[3];
        const auto load_ih = [&]() {
            ihn[0] = (int32_t)ih_in[0];
            ihn[1] = (int32_t)ih_in[a.H];
            ihn[2] = (int32_t)ih_in[2 * a.H];
        };
        const auto leave_ih = [&](int s) {
#pragma unroll
            for (int g = 0; g < 3; ++g) ring[((s & 1) * 3 + g) * units + j] = ihn[g];
        };
        load_ih();
        leave_ih(0);
        if (a.T > 1) ih_in += ih_step;
        load_ih();
        __syncthreads();
        const auto state = [&](int s) {
            const unsigned char q = hs[(size_t)(s & 1) * HS + j_at];
            return HUnsigned ? (int32_t)q : (int32_t)(int8_t)q;
        };
        for (int s = 0; s < a.T; ++s) {
            int acc[3];
            product(hs + (size_t)(s & 1) * HS + QS, acc);
#pragma unroll
            for (int g = 0; g < 3; ++g) part[g * units + j] = acc[g];
            asm volatile("bar.arrive 1, %0;" ::"r"(NT) : "memory");
            leave_ih(s + 1);
            if (s + 2 < a.T) ih_in += ih_step;
            load_ih();
            if (s > 0) emit(s - 1, state(s));
            __syncthreads();
        }
        emit(a.T - 1, state(a.T));
        return;
    }
    const unsigned char h0 = hs[j_at];
    int32_t h_old = HUnsigned ? (int32_t)h0 : (int32_t)(int8_t)h0;      // this thread's unit, from step to step in a register
    __syncthreads();
    for (int s = 0; s < a.T; ++s) {
        int acc[3];
        product(hs + (size_t)(s & 1) * HS, acc);
        int32_t ih[3];
#pragma unroll
        for (int g = 0; g < 3; ++g) ih[g] = ring[((s & 1) * 3 + g) * units + j];
        int32_t hn;
        if constexpr (Cell == 2) {
            constexpr bool Ahead = KT == 64;         // (where R leaves registers: the constants ahead of the barrier)
            FastLin f[3];
            if constexpr (Ahead)
#pragma unroll
                for (int g = 0; g < 3; ++g) f[g] = fls[g * units + j];
            asm volatile("bar.sync 1, %0;" ::"r"(NT) : "memory");
#pragma unroll
            for (int g = 0; g < 3; ++g) acc[g] += part[g * units + j];
            const auto lin = [&](int g) { return lin_round<Tie>(acc[g], Ahead ? f[g] : fls[g * units + j]); };
            const int32_t z_d = fused_gate_fast(gc, tab, ACT_Z, ih[0], lin(0));
            const int32_t r_d = fused_gate_fast(gc, tab, ACT_R, ih[1], lin(1));
            hn = fused_finish_fast<Tie>(gc, tab, ih[2], lin(2), z_d, r_d, h_old);
        } else {
            asm volatile("bar.sync 1, %0;" ::"r"(NT) : "memory");
#pragma unroll
            for (int g = 0; g < 3; ++g) acc[g] += part[g * units + j];
            const float fih[3] = {(float)ih[0], (float)ih[1], (float)ih[2]};
            float fhh[3];
#pragma unroll
            for (int g = 0; g < 3; ++g)
                fhh[g] = fs_linear(acc[g], fsk[(g * 3 + 0) * units + j], fsk[(g * 3 + 1) * units + j],
                                   fsk[(g * 3 + 2) * units + j], a.fs.zp_hh, a.fs.hh_lo, a.fs.hh_hi);
            const float u_g = fs_sigmoid_gate_tab(a.fs, tab, 0, fih[0], fhh[0]);
            const float r_g = fs_sigmoid_gate_tab(a.fs, tab, 1, fih[1], fhh[1]);
            hn = (int32_t)fs_finish_tab(a.fs, tab, u_g, r_g, fih[2], fhh[2], (float)h_old);
        }
        h_old = hn;
        if (j_ok) hs[(size_t)((s + 1) & 1) * HS + j_at] = (unsigned char)hn;
        __syncthreads();
    }
}

// --------------------------------------------- generic fallback (any bit width, int32 data)

// out[n][m] = epilogue( sum_k W_q[k][m] * in[n][k] ) with 64-bit accumulation
// (quantizedGemmBiasFused's arithmetic, src/gru_forward_gpu_quant.cu:110-180), in two forms.
// One output per thread: bound by the latency of its K dependent steps, whatever the number of outputs, until the
// SMs' resident threads are all in use; from there on by reading W again for every row.
// (unrolled by 4, 8 or 16 with running pointers, or with launch bounds: 3 to 70 % slower at K = 512)
__global__ void k_linear_rows(const int32_t *__restrict__ wq, const int32_t *__restrict__ in, int32_t *__restrict__ out, long long N, int K, int C,
                              LinearConsts lc, uint8_t *__restrict__ keep) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const long long n = blockIdx.y;
    if (m >= C || n >= N) return;
    int64_t acc = 0;
    for (int k = 0; k < K; ++k) acc += (int64_t)wq[(size_t)k * C + m] * (int64_t)in[n * K + k];
    out[n * C + m] = linear_epilogue(acc, lc.corr[m], lc.rs[m], lc.zp_out, lc.lo, lc.hi, keep ? keep + n * C + m : nullptr);
}

// 32 x 64 tiles, 2 x 4 outputs per thread, K in slabs of 32 through shared memory; bound by the widening multiply-adds.
__global__ void __launch_bounds__(256)
k_linear_tiles(const int32_t *__restrict__ wq, const int32_t *__restrict__ in, int32_t *__restrict__ out, long long N, int K, int C,
               LinearConsts lc, uint8_t *__restrict__ keep) {
    __shared__ int32_t xs[32][33];
    __shared__ __align__(16) int32_t ws[32][64];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const long long n0 = (long long)blockIdx.x * 32;
    const int m0 = blockIdx.y * 64;
    int64_t acc[2][4] = {};
    for (int k0 = 0; k0 < K; k0 += 32) {
        for (int i = tid; i < 32 * 32; i += 256) {
            const int r = i >> 5, k = i & 31;
            xs[r][k] = n0 + r < N && k0 + k < K ? in[(n0 + r) * K + k0 + k] : 0;
        }
        for (int i = tid; i < 32 * 64; i += 256) {
            const int k = i >> 6, m = i & 63;
            ws[k][m] = m0 + m < C && k0 + k < K ? wq[(size_t)(k0 + k) * C + m0 + m] : 0;
        }
        __syncthreads();
        const int kn = min(32, K - k0);
        for (int k = 0; k < kn; ++k) {
            const int4 w = *reinterpret_cast<const int4 *>(&ws[k][tx * 4]);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int64_t x = xs[ty * 2 + r][k];
                acc[r][0] += (int64_t)w.x * x;
                acc[r][1] += (int64_t)w.y * x;
                acc[r][2] += (int64_t)w.z * x;
                acc[r][3] += (int64_t)w.w * x;
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const long long n = n0 + ty * 2 + r;
            const int m = m0 + tx * 4 + c;
            if (n < N && m < C) out[n * C + m] = linear_epilogue(acc[r][c], lc.corr[m], lc.rs[m], lc.zp_out, lc.lo, lc.hi, keep ? keep + n * C + m : nullptr);
        }
}

// The recurrence with states of up to 16 bits and 8-bit R, H <= 256, in one launch instead of two per step: one CTA per
// batch row keeps R in shared memory (as k_recurrence_gemv) and the state as two bytes per unit in planes of
// their own, low bytes unsigned, high bytes with the operator's sign, so that both products are dp4a and
// sum = 256 * high + low is exact.  A quad of threads owns a unit: after the shuffles lanes 0, 1, 2 requantize
// the rows of one gate each, lanes 0 and 1 run the update and the reset gate side by side, lane 2 the rest.
// Bound by that chain of 64-bit rescales and segment searches: 21 rows of H = 100, 61 steps, 16-bit operators 122 us
// (two launches per step: 800).
struct WideArgs {
    int T, B, H, Hpad, C, reverse;
    const int8_t *r8;          // [3H][Hpad]
    const int32_t *ih;         // [T*B][3H] W*x + bw
    const int32_t *h0;         // [B][H]
    OutView out;
    LinearConsts lc;           // R*h + br epilogue
    const int32_t *tables;
    int n_table;
};
// shared memory: tables | thresholds [3][16] | segments [3][16] | state [2 buffers][2 planes] | R
__host__ __device__ inline size_t wide_smem(int H, int Hpad, int n_table) {
    const size_t units = (size_t)(H + 31) / 32 * 32;
    return (((size_t)n_table * 4 + 15) & ~size_t(15)) + 3 * 16 * 4 + 3 * 16 * sizeof(qgru_lut_segment) + (size_t)4 * (Hpad + 64) + 3 * units * Hpad;
}

template <bool HUnsigned>
__global__ void __launch_bounds__(1024, 1) k_recurrence_wide(const __grid_constant__ GateConsts gc, const __grid_constant__ WideArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int NT = blockDim.x, Kq = a.Hpad >> 2, nch = Kq >> 4, Qs = Kq + 16, Hs = 4 * Qs;
    int32_t *tables = reinterpret_cast<int32_t *>(smem_raw);
    size_t off = ((size_t)a.n_table * 4 + 15) & ~size_t(15);
    int32_t *thr = reinterpret_cast<int32_t *>(smem_raw + off);
    off += 3 * 16 * 4;
    qgru_lut_segment *seg = reinterpret_cast<qgru_lut_segment *>(smem_raw + off);
    off += 3 * 16 * sizeof(qgru_lut_segment);
    unsigned char *hs = smem_raw + off;                   // [buffer][plane][Hs]
    off += (size_t)4 * Hs;
    uint4 *Rq = reinterpret_cast<uint4 *>(smem_raw + off);
    const int tid = threadIdx.x, qd = tid & 3, j = tid >> 2, b = blockIdx.x;
    const bool j_ok = j < a.H;
    for (int i = tid; i < a.n_table; i += NT) tables[i] = a.tables[i];
    for (int i = tid; i < 48; i += NT) {
        thr[i] = gc.lut[i >> 4].seg[i & 15].threshold;
        seg[i] = gc.lut[i >> 4].seg[i & 15];
    }
    for (int i = tid; i < a.Hpad; i += NT) {
        const int at = (i / Kq) * Qs + (i % Kq);
        const int32_t q = i < a.H ? a.h0[(size_t)b * a.H + i] : 0;
        hs[at] = (unsigned char)q;
        hs[Hs + at] = (unsigned char)(q >> 8);
        hs[2 * Hs + at] = hs[3 * Hs + at] = 0;
    }
    for (int g = 0; g < 3; ++g)
        for (int c = 0; c < nch; ++c) {
            uint4 w = make_uint4(0u, 0u, 0u, 0u);
            if (j_ok) w = *reinterpret_cast<const uint4 *>(a.r8 + (size_t)(g * a.H + j) * a.Hpad + qd * Kq + 16 * c);
            Rq[(size_t)(c * 3 + g) * NT + tid] = w;
        }
    // this lane's gate
    const int g = min(qd, 2), gs = min(qd, 1);
    const int64_t corr = j_ok ? a.lc.corr[g * a.H + j] : 0;
    const Rescale rs = j_ok ? a.lc.rs[g * a.H + j] : Rescale{1, 1, 0, 0, 0, 0, 0, 0};
    const Rescale ih_to = gc.ih_to[g], hh_to = gc.hh_to[gs];
    const int32_t zp_in = gc.zp_in[g], in_lo = gc.in_lo[g], in_hi = gc.in_hi[g], out_lo = gc.out_lo[g], out_hi = gc.out_hi[g];
    const int32_t t_size = gc.table_size[g], t_off = gc.table_off[g], lut_zp = gc.lut[g].zp_x;
    const auto act = [&](int32_t pre) {                   // activation() for this lane's gate
        const int32_t q = clampi(pre, in_lo, in_hi);
        if (t_size > 0) return tables[t_off + (q - in_lo)];
        int sg = QGRU_LUT_SEGMENTS - 1;
#pragma unroll
        for (int i = QGRU_LUT_SEGMENTS - 2; i >= 0; --i)
            if (q < thr[g * 16 + i]) sg = i;
        return clampi(lut_segment(seg[g * 16 + sg], lut_zp, q), out_lo, out_hi);
    };
    const int j_at = (j / Kq) * Qs + (j % Kq);
    const long long dir = a.reverse ? -1 : 1;
    const int32_t *src = a.ih + ((size_t)(a.reverse ? a.T - 1 : 0) * a.B + b) * a.C + g * a.H + j;
    const long long src_step = dir * a.B * a.C;
    int32_t ihv = j_ok ? *src : 0;
    __syncthreads();
    for (int s = 0; s < a.T; ++s) {
        const unsigned char *h_cur = hs + (s & 1) * 2 * Hs;
        unsigned char *h_nxt = hs + ((s + 1) & 1) * 2 * Hs;
        int32_t ihn = 0;
        src += src_step;
        if (j_ok && s + 1 < a.T) ihn = *src;
        int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
        const uint4 *l4 = reinterpret_cast<const uint4 *>(h_cur + qd * Qs), *h4 = reinterpret_cast<const uint4 *>(h_cur + Hs + qd * Qs);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (c >= nch) break;
            const uint4 x = l4[c], y = h4[c];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const uint4 w = Rq[(size_t)(c * 3 + k) * NT + tid];
                lo[k] = dp4a_w<true>((int)w.x, x.x, lo[k]);
                hi[k] = dp4a_w<HUnsigned>((int)w.x, y.x, hi[k]);
                lo[k] = dp4a_w<true>((int)w.y, x.y, lo[k]);
                hi[k] = dp4a_w<HUnsigned>((int)w.y, y.y, hi[k]);
                lo[k] = dp4a_w<true>((int)w.z, x.z, lo[k]);
                hi[k] = dp4a_w<HUnsigned>((int)w.z, y.z, hi[k]);
                lo[k] = dp4a_w<true>((int)w.w, x.w, lo[k]);
                hi[k] = dp4a_w<HUnsigned>((int)w.w, y.w, hi[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] += __shfl_xor_sync(0xffffffffu, lo[k], 1);
            hi[k] += __shfl_xor_sync(0xffffffffu, hi[k], 1);
            lo[k] += __shfl_xor_sync(0xffffffffu, lo[k], 2);
            hi[k] += __shfl_xor_sync(0xffffffffu, hi[k], 2);
        }
        const int my_lo = g == 0 ? lo[0] : g == 1 ? lo[1] : lo[2], my_hi = g == 0 ? hi[0] : g == 1 ? hi[1] : hi[2];
        const int32_t hh = linear_epilogue((int64_t)my_hi * 256 + my_lo, corr, rs, a.lc.zp_out, a.lc.lo, a.lc.hi);
        const int32_t a_ih = rescale_diff<false>(ihv, gc.zp_ih, ih_to);
        // gru_cell<false>, the update and the reset gate in lanes 0 and 1
        const int32_t gate = act(a_ih + rescale_diff<false>(hh, gc.zp_hh, hh_to) + zp_in);
        const int32_t z = __shfl_sync(0xffffffffu, gate, 0, 4), r = __shfl_sync(0xffffffffu, gate, 1, 4);
        if (qd == 2 && j_ok) {
            const int64_t r_hh = ((int64_t)r - gc.zp_out[ACT_R]) * ((int64_t)hh - gc.zp_hh);
            const int32_t n = act(a_ih + (int32_t)rescale64(r_hh, gc.rh_to_n) + zp_in);
            const int32_t n_h = rescale_diff<false>(n, gc.zp_out[ACT_N], gc.n_to_h) + gc.zp_h;
            const int32_t h_old = (HUnsigned ? (int32_t)h_cur[Hs + j_at] : (int32_t)(int8_t)h_cur[Hs + j_at]) * 256 + (int32_t)h_cur[j_at];
            const int64_t z_d = (int64_t)z - gc.zp_out[ACT_Z];
            const int64_t old_c = z_d * ((int64_t)h_old - gc.zp_h);
            const int64_t one_minus = ((int64_t)gc.one_q - z) - gc.zp_out[ACT_Z];
            const int64_t new_c = one_minus * ((int64_t)n_h - gc.zp_h);
            const int32_t hn = clampi((int32_t)rescale64(old_c + new_c, gc.uh_to_h) + gc.zp_h, gc.h_lo, gc.h_hi);
            h_nxt[j_at] = (unsigned char)hn;
            h_nxt[Hs + j_at] = (unsigned char)(hn >> 8);
            put_state(a.out, a.reverse ? (a.T - 1 - s) : (s + 1), b, j, a.H, s + 1 == a.T, hn, gc.zp_h, gc.h_scale);
        }
        ihv = ihn;
        __syncthreads();
    }
}

// v: optional [B][4H] out of this step: update, reset, new gate outputs and the R*h + br row of
// the new gate (the training buffer of the reference).
__global__ void k_gates_generic(const int32_t *__restrict__ ih, const int32_t *__restrict__ hh,
                                const int32_t *__restrict__ h_in, int32_t *__restrict__ h_out,
                                int32_t *__restrict__ v, int B, int H, const GateConsts *__restrict__ gcp,
                                const int32_t *__restrict__ tables) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (j >= H || b >= B) return;
    const size_t w = (size_t)b * 3 * H + j;
    int32_t gates[3];
    h_out[(size_t)b * H + j] = gru_cell<false>(*gcp, tables, ih[w], ih[w + H], ih[w + 2 * H], hh[w],
                                               hh[w + H], hh[w + 2 * H], h_in[(size_t)b * H + j], gates);
    if (v) {
        int32_t *vb = v + (size_t)b * 4 * H + j;
        vb[0] = gates[0];
        vb[H] = gates[1];
        vb[2 * H] = gates[2];
        vb[3 * H] = hh[w + 2 * H];
    }
}

// The training form of k_gates_generic: v as above plus the clamp masks of this step (each may be
// null): gate inputs and gate outputs [B][3H], new state [B][H]; 1 = not clamped.
__global__ void k_gates_train(const int32_t *__restrict__ ih, const int32_t *__restrict__ hh,
                              const int32_t *__restrict__ h_in, int32_t *__restrict__ h_out,
                              int32_t *__restrict__ v, uint8_t *__restrict__ m_in,
                              uint8_t *__restrict__ m_out, uint8_t *__restrict__ m_h, int B, int H,
                              const GateConsts *__restrict__ gcp) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (j >= H || b >= B) return;
    const size_t w = (size_t)b * 3 * H + j;
    int32_t gates[3];
    uint32_t keep = 0;
    h_out[(size_t)b * H + j] = gru_cell_train(*gcp, nullptr, ih[w], ih[w + H], ih[w + 2 * H], hh[w], hh[w + H],
                                              hh[w + 2 * H], h_in[(size_t)b * H + j], gates, keep);
    int32_t *vb = v + (size_t)b * 4 * H + j;
    vb[0] = gates[0];
    vb[H] = gates[1];
    vb[2 * H] = gates[2];
    vb[3 * H] = hh[w + 2 * H];
#pragma unroll
    for (int g = 0; g < 3; ++g) {
        if (m_in) m_in[w + g * H] = keep >> (PM_IN + g) & 1;
        if (m_out) m_out[w + g * H] = keep >> (PM_OUT + g) & 1;
    }
    if (m_h) m_h[(size_t)b * H + j] = keep >> PM_H & 1;
}

}  // namespace qgru
