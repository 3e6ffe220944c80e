// qgru_rec_f32.cu - the two fp32 recurrences as persistent kernels: h_t of the float forward
// (ForwardPass<float> of the reference, src/gru_forward_gpu.cu:23-125, 342-414) and the chain of state
// gradients of the backward pass (src/gru_backward_gpu.cu, src/gru_backward_gpu_quant.cu).
//
// Both are one matrix-vector product with R per batch row and step, 3 H^2 multiply-adds, with a
// dependency from step to step.  A cluster of P CTAs works on Bt batch rows and holds all of R in
// REGISTERS for the whole launch: a thread keeps 96 of its values (3 gates x 32 inputs of one unit
// in the forward, 4 outputs x 24 inputs in the backward), so a step reads only the state (broadcast or
// conflict-free 128-bit loads, a few per 48 packed multiply-adds) and is bound by the fp32 pipe for
// many rows and by its own latency for few.  R in shared memory instead would cost 1600 cycles of
// shared-memory bandwidth per step at 200 KB a CTA.
//
// Between the CTAs of a cluster: every CTA writes its own results of a step into its own shared memory,
// one cluster barrier follows, and the readers PULL what they need with remote loads (the barrier
// then has no remote stores to wait for).  The forward pulls the state, H values per row; the
// backward, whose operand has 3H values per row, multiplies where the operand is produced and pulls
// the partial sums instead, again H values per row.  Sums are added in a fixed order.
//
// Measured on a B200 against the two launches per step (tiled product, pointwise kernel) that it replaces, in us
// per step: backward H = 512, B = 256: 221 -> 22; H = 262, B = 65: 112 -> 3.3; H = 128, B = 32: 48 -> 2.0.
// Forward with gate buffer H = 262, B = 65: 36 -> 3.0; H = 256, B = 64: 31 -> 2.7; H = 128, B = 32: 1.6.
#include "qgru_rec_f32.cuh"

#include "qgru_cluster.cuh"
#include "qgru_gemm_f32.cuh"
#include "qgru_handle.h"

namespace qgru {
using namespace clu;
namespace {

constexpr int MAX_ROWS = 40;                 // batch rows per cluster
constexpr int RB = 8;                        // forward: rows between two block barriers

// block of gate g (z, r, n) in weights, W*x and gradients
__device__ __forceinline__ int gate_block(int torch, int g) { return torch && g < 2 ? 1 - g : g; }

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float4 ld_remote4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float ld_remote(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cp_async4(void *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// wait until at most D - 1 of this thread's copy groups are in flight
__device__ __forceinline__ void cp_async_wait_depth(int D) {
    if (D == 1) cp_async_wait<0>();
    else cp_async_wait<2>();
}

// ------------------------------------------------------------------------------- float forward
// Floats of shared memory: the state of all H units for the rows (two buffers where one CTA owns them
// all: the cell writes the next one directly), this CTA's own units (two buffers, read by the
// peers), the partial sums of the KG input slices for RB rows (two buffers), W*x of the next D steps, the
// gate buffer of the step on its way out, the biases.
__host__ __device__ inline size_t fwd_smem_floats(int P, int U, int KG, int Bt, int D) {
    return (size_t)(P == 1 ? 2 : 1) * Bt * P * U + (P > 1 ? (size_t)2 * Bt * U : 0) +
           (size_t)(Bt > KG && Bt > RB ? 2 : 1) * KG * (Bt > KG && Bt > RB ? RB : Bt) * 3 * U + (size_t)D * Bt * 3 * U + (size_t)6 * Bt * U + (size_t)6 * U;
}

// One: a thread has at most one cell a step (Bt <= KG; all rows are one block): its results stay in registers between the
// cell and the stores, and no loop, staging buffer or 64-bit index is left around them.  A step of few rows
// is a chain of some 900 dependent instructions at about five cycles each, so their number is what counts.
// Alone: one CTA, no cluster.  Beside R, 32 registers are left of 128 where a CTA has 512 threads (97 to 128 units in one CTA), and what the
// cluster needs does not fit: us a step, H = 128, 300 rows 3.6 -> 2.8, 500 rows 4.4 -> 3.3 (240 bytes of spills -> 60).
template <bool One, int MaxThreads, bool Alone>
__global__ void __launch_bounds__(MaxThreads, 1) k_float_chain(const FloatFwdArgs a) {
    extern __shared__ __align__(16) float sm[];
    const int U = a.U, P = Alone ? 1 : a.P, KG = a.KG, Bt = a.Bt, D = a.D, PU = P * U, H = a.H, C = 3 * H;
    const int rb = One ? Bt : RB, rb_max = min(Bt, rb), BtU = Bt * U;
    float *hs = sm;
    float *own = hs + (size_t)(P == 1 ? 2 : 1) * Bt * PU;
    float *part = own + (P > 1 ? 2 * BtU : 0);
    const int part_n = KG * rb_max * 3 * U;
    float *wxs = part + (Bt > rb ? 2 : 1) * part_n;         // [D][Bt][3][U]
    float *vst = wxs + (size_t)D * 3 * BtU;                 // [6][Bt][U]
    float *bias = vst + (size_t)6 * BtU;

    const int tid = threadIdx.x, NT = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int p = P > 1 ? (int)cluster_rank() : 0;
    const int b0 = (blockIdx.x / P) * Bt, nb = min(Bt, a.B - b0);
    // product: this thread multiplies inputs kg * 32 .. + 31 of unit u's three gate rows
    const int UB = U >> 5, kg = warp / UB, u = (warp % UB) * 32 + lane;
    uint64_t R2[3][16];
    {
        const int j = p * U + u;
#pragma unroll
        for (int g = 0; g < 3; ++g)
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int k = kg * 32 + 2 * i;
                const size_t at = a.torch ? ((size_t)gate_block(1, g) * H + j) * H + k : (size_t)k * C + g * H + j;
                const float lo = (j < H && k < H) ? a.R[at] : 0.f;
                const float hi = (j < H && k + 1 < H) ? a.R[at + (a.torch ? 1 : C)] : 0.f;
                R2[g][i] = pack2(lo, hi);
            }
    }
    // cell: unit cu, rows cb, cb + KG, ... of each block of RB rows
    const int cu = tid % U, cb = tid / U, cj = p * U + cu;
    const bool j_ok = cj < H;
    for (int i = tid; i < 6 * U; i += NT) {
        const int g = i / U, j = p * U + i % U;
        const float *src = g < 3 ? a.bw : a.br;
        bias[i] = j < H && src ? src[gate_block(a.torch, g % 3) * H + j] : 0.f;
    }
    // the initial state
    const float *h_init = a.h + (a.reverse ? (size_t)a.T * a.B * H : 0);
    if (P == 1) {
        for (int i = tid; i < 2 * Bt * PU; i += NT) {
            const int b = i / PU, j = i % PU;
            hs[i] = (b < nb && j < H) ? h_init[(size_t)(b0 + b) * H + j] : 0.f;
        }
    } else {
        for (int i = tid; i < 2 * BtU; i += NT) {
            const int b = i / U, j = p * U + i % U;
            own[i] = (b < nb && j < H) ? h_init[(size_t)(b0 + b) * H + j] : 0.f;
        }
    }
    // running pointers of this thread's unit: one add per step instead of 64-bit products per access
    const int vs = a.v_stride * H;
    const long long dir = a.reverse ? -1 : 1;
    const size_t row0 = (size_t)(a.reverse ? a.T - 1 : 0) * a.B + b0;      // first row of the first step
    const float *wx_next = a.wx + row0 * C + cj;
    float *h_out = a.h + (row0 + (a.reverse ? 0 : a.B)) * H + cj;
    float *v_out = a.v ? a.v + row0 * vs + cj : nullptr;
    float *u_out = a.out.hf ? a.out.hf + (size_t)(a.reverse ? a.T - 1 : 1) * a.out.ts + (size_t)b0 * a.out.bs + cj : nullptr;
    const long long wx_step = dir * a.B * C, h_step = dir * a.B * H, v_step = dir * a.B * vs, u_step = dir * (long long)a.out.ts;
    int g_off[3];
#pragma unroll
    for (int g = 0; g < 3; ++g) g_off[g] = gate_block(a.torch, g) * H;
    int slot_in = 0, fetched = 0;
    const bool act = One && j_ok && cb < nb;                 // One: this thread's cell is (row cb, unit cu)
    if constexpr (One) wx_next += (size_t)cb * C;
    long long row = (long long)row0 + cb;                    // One: this cell's row of the step
    auto fetch_wx = [&]() {   // each thread fetches what its own cells will read
        if constexpr (One) {
            if (act && fetched < a.T) {
                float *dst = wxs + (slot_in * Bt + cb) * 3 * U + cu;
#pragma unroll
                for (int g = 0; g < 3; ++g) cp_async4(dst + g * U, wx_next + g_off[g]);
            }
        } else if (fetched < a.T && j_ok) {
            float *dst = wxs + slot_in * 3 * BtU + cu;
            for (int r0 = 0; r0 < nb; r0 += RB)
                for (int b = r0 + cb; b < min(nb, r0 + RB); b += KG) {
                    const float *src = wx_next + b * C;
#pragma unroll
                    for (int g = 0; g < 3; ++g) cp_async4(dst + (b * 3 + g) * U, src + g_off[g]);
                }
        }
        wx_next += wx_step;
        ++fetched;
        slot_in = slot_in + 1 == D ? 0 : slot_in + 1;
        cp_async_commit();
    };
    for (int d = 0; d < D; ++d) fetch_wx();
    if (P > 1) {
        cluster_arrive();
        cluster_wait();
    } else {
        __syncthreads();
    }
    const int u4 = tid % (U >> 2), r4 = tid / (U >> 2), r4_step = NT / (U >> 2);
    const uint32_t own_u32 = smem_addr(own) + (uint32_t)u4 * 16u;
    int slot = 0;

    for (int s = 0; s < a.T; ++s) {
        const float *hcur = hs;
        if (P > 1) {
            // pull the peers' units; four remote loads in flight per thread
            const uint32_t src = own_u32 + (uint32_t)((s & 1) * BtU) * 4u;
            for (int r = r4; r < P * nb; r += 4 * r4_step) {
                float4 x[4];
                float *dst[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int rr = r + k * r4_step, q = rr / nb, b = rr - q * nb;
                    dst[k] = hs + b * PU + q * U + u4 * 4;
                    if (rr < P * nb) x[k] = ld_remote4(map_to_rank(src + (uint32_t)(b * U) * 4u, (uint32_t)q));
                }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (r + k * r4_step < P * nb) *reinterpret_cast<float4 *>(dst[k]) = x[k];
            }
            __syncthreads();
        } else {
            hcur = hs + (s & 1) * BtU;
        }
        const float *hk = hcur + kg * 32;
        const float *wxc = wxs + slot * 3 * BtU + cu;
        float *next = P > 1 ? own + ((s + 1) & 1) * BtU + cu : hs + ((s + 1) & 1) * BtU + cu;
        float o_z = 0.f, o_r = 0.f, o_g = 0.f, o_rz = 0.f, o_rr = 0.f, o_rg = 0.f, o_h = 0.f;   // One: this step's cell
        for (int r0 = 0, pb = 0; r0 < nb; r0 += rb, pb ^= 1) {
            const int r1 = min(nb, r0 + rb);
            float *pk = part + pb * part_n + kg * rb_max * 3 * U + u;
            int b = r0;
            // (two rows at a time where there are registers for it)
            if constexpr (!One || MaxThreads < 512) for (; b + 2 <= r1; b += 2, pk += 6 * U) {
                uint64_t acc[2][3] = {};
                const float *h0 = hk + b * PU, *h1 = h0 + PU;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const ulonglong2 x0 = *reinterpret_cast<const ulonglong2 *>(h0 + 4 * i);
                    const ulonglong2 x1 = *reinterpret_cast<const ulonglong2 *>(h1 + 4 * i);
#pragma unroll
                    for (int g = 0; g < 3; ++g) {
                        acc[0][g] = ffma2(R2[g][2 * i], x0.x, acc[0][g]);
                        acc[1][g] = ffma2(R2[g][2 * i], x1.x, acc[1][g]);
                        acc[0][g] = ffma2(R2[g][2 * i + 1], x0.y, acc[0][g]);
                        acc[1][g] = ffma2(R2[g][2 * i + 1], x1.y, acc[1][g]);
                    }
                }
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int g = 0; g < 3; ++g) {
                        float lo, hi;
                        unpack2(acc[r][g], lo, hi);
                        pk[(r * 3 + g) * U] = lo + hi;
                    }
            }
            for (; b < r1; ++b, pk += 3 * U) {
                uint64_t acc[3] = {};
                const float *h0 = hk + b * PU;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const ulonglong2 x0 = *reinterpret_cast<const ulonglong2 *>(h0 + 4 * i);
#pragma unroll
                    for (int g = 0; g < 3; ++g) {
                        acc[g] = ffma2(R2[g][2 * i], x0.x, acc[g]);
                        acc[g] = ffma2(R2[g][2 * i + 1], x0.y, acc[g]);
                    }
                }
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    float lo, hi;
                    unpack2(acc[g], lo, hi);
                    pk[g * U] = lo + hi;
                }
            }
            if (r0 == 0) cp_async_wait_depth(D);
            __syncthreads();
            if constexpr (One) {
                if (act) {
                    // (loads of several slices in flight, added in slice order)
                    const float *q = part + cb * 3 * U + cu, *w = wxc + cb * 3 * U, *bi = bias + cu;
                    const int step = rb_max * 3 * U;
                    float sum[3] = {0.f, 0.f, 0.f};
                    int k = 0;
                    for (; k + 4 <= KG; k += 4, q += 4 * step) {
                        float y[4][3];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
#pragma unroll
                            for (int g = 0; g < 3; ++g) y[e][g] = q[e * step + g * U];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
#pragma unroll
                            for (int g = 0; g < 3; ++g) sum[g] += y[e][g];
                    }
                    for (; k < KG; ++k, q += step)
#pragma unroll
                        for (int g = 0; g < 3; ++g) sum[g] += q[g * U];
                    o_rz = sum[0] + bi[3 * U];
                    o_rr = sum[1] + bi[4 * U];
                    o_rg = sum[2] + bi[5 * U];
                    o_z = 1.0f / (1.0f + expf(-((w[0] + bi[0]) + o_rz)));
                    o_r = 1.0f / (1.0f + expf(-((w[U] + bi[U]) + o_rr)));
                    o_g = tanhf((w[2 * U] + bi[2 * U]) + o_r * o_rg);
                    o_h = o_z * hcur[cb * PU + cj] + (1.0f - o_z) * o_g;
                    next[cb * U] = o_h;
                }
            } else if (j_ok) {
                for (int c = r0 + cb; c < r1; c += KG) {
                    float sum[3] = {0.f, 0.f, 0.f};
                    const float *q = part + pb * part_n + (c - r0) * 3 * U + cu;
                    for (int k = 0; k < KG; ++k, q += rb_max * 3 * U)
#pragma unroll
                        for (int g = 0; g < 3; ++g) sum[g] += q[g * U];
                    const float *w = wxc + c * 3 * U;
                    const float rz = sum[0] + bias[3 * U + cu], rr = sum[1] + bias[4 * U + cu], rg = sum[2] + bias[5 * U + cu];
                    const float z = 1.0f / (1.0f + expf(-((w[0] + bias[cu]) + rz)));
                    const float r = 1.0f / (1.0f + expf(-((w[U] + bias[U + cu]) + rr)));
                    const float g = tanhf((w[2 * U] + bias[2 * U + cu]) + r * rg);
                    const float h_old = hcur[c * PU + cj];
                    const float hn = z * h_old + (1.0f - z) * g;
                    next[c * U] = hn;
                    if (v_out) {
                        float *t = vst + c * U + cu;
                        t[0] = z;
                        t[BtU] = r;
                        t[2 * BtU] = g;
                        if (a.v_stride == 6) {
                            t[3 * BtU] = rz;
                            t[4 * BtU] = rr;
                            t[5 * BtU] = rg;
                        } else {
                            t[3 * BtU] = rg;
                        }
                    }
                }
            }
        }
        if (P > 1) cluster_arrive();
        else __syncthreads();
        // Results leave for global memory behind the arrive: a cluster barrier's release waits for
        // every store before it, and nothing in the next step waits for these.
        if constexpr (One) {
            if (act) {
                // (addresses from the row index: a pointer per output would not fit beside R)
                a.h[(row + (a.reverse ? 0 : a.B)) * H + cj] = o_h;
                if (a.out.hf) a.out.hf[(size_t)(a.reverse ? a.T - 1 - s : s + 1) * a.out.ts + (size_t)(b0 + cb) * a.out.bs + cj] = o_h;
                if (s + 1 == a.T && a.out.hn_f) a.out.hn_f[(size_t)(b0 + cb) * H + cj] = o_h;
                if (a.v) {
                    float *vb = a.v + row * vs + cj;
                    vb[0] = o_z;
                    vb[H] = o_r;
                    vb[2 * H] = o_g;
                    vb[3 * H] = a.v_stride == 6 ? o_rz : o_rg;
                    if (a.v_stride == 6) {
                        vb[4 * H] = o_rr;
                        vb[5 * H] = o_rg;
                    }
                }
            }
            row += dir * a.B;
        } else if (j_ok)
            for (int r0 = 0; r0 < nb; r0 += RB)
                for (int c = r0 + cb; c < min(nb, r0 + RB); c += KG) {
                    const float hn = next[c * U];
                    h_out[c * H] = hn;
                    if (u_out) u_out[(size_t)c * a.out.bs] = hn;
                    if (s + 1 == a.T && a.out.hn_f) a.out.hn_f[(size_t)(b0 + c) * H + cj] = hn;
                    if (v_out) {
                        const float *t = vst + c * U + cu;
                        float *vb = v_out + c * vs;
#pragma unroll
                        for (int k = 0; k < 4; ++k) vb[k * H] = t[k * BtU];
                        if (a.v_stride == 6) {
                            vb[4 * H] = t[4 * BtU];
                            vb[5 * H] = t[5 * BtU];
                        }
                    }
                }
        if constexpr (!One) {
            h_out += h_step;
            if (v_out) v_out += v_step;
            if (u_out) u_out += u_step;
        }
        slot = slot + 1 == D ? 0 : slot + 1;
        fetch_wx();
        if (P > 1) cluster_wait();
    }
    // (the last barrier follows the last remote load of every peer: a CTA may leave)
}

// --------------------------------------------------------------------------- backward chain
// Floats of shared memory: dq of this CTA's units (the product's operand) and dp beside it, the partial sums
// for every unit (two buffers, read by the peers), seven operands of the cell for D steps, z * dh, six bias
// sums per thread.
__host__ __device__ inline size_t bwd_smem_floats(int P, int U, int KG, int Bt, int D) {
    (void)P;
    return (size_t)2 * Bt * 3 * U + (size_t)2 * KG * Bt * U + (size_t)D * 7 * Bt * U + (size_t)Bt * U + (size_t)6 * U * KG;
}

// One: a thread has at most one cell a step (Bt <= KG), see the forward; its bias sums stay in registers too.
template <bool One, int MaxThreads>
__global__ void __launch_bounds__(MaxThreads, 1) k_bwd_chain(const BwdChainArgs a) {
    extern __shared__ __align__(16) float sm[];
    const int U = a.U, P = a.P, KG = a.KG, Bt = a.Bt, D = a.D, H = a.H, C = 3 * H, BtU = Bt * U;
    float *dqs = sm;                                        // [Bt][3U]
    float *dps = dqs + 3 * BtU;                             // [Bt][3U]
    float *part = dps + 3 * BtU;                            // [2][U / 32][P owners][Bt][U]
    float *stage = part + 2 * KG * BtU;                     // [D][7][Bt][U]
    float *zdh = stage + D * 7 * BtU;                       // [Bt][U]
    float *bsum = zdh + BtU;                                // [6][threads]

    const int tid = threadIdx.x, NT = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int p = P > 1 ? (int)cluster_rank() : 0;
    const int grp = blockIdx.x / P, b0 = grp * Bt, nb = min(Bt, a.B - b0);
    // product: outputs ob * 32 + 4 q .. + 3, inputs sl * 96 + 24 m .. + 23 of this CTA's 3U
    const int ob = warp % KG, sl = warp / KG, q = lane & 7, mg = lane >> 3;
    const int in0 = sl * 96 + mg * 24;
    uint64_t R2[4][12];
#pragma unroll
    for (int o = 0; o < 4; ++o) {
        const int k = ob * 32 + q * 4 + o;
#pragma unroll
        for (int i = 0; i < 12; ++i) {
            float w[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int m = in0 + 2 * i + e, g = m / U, j = p * U + m % U;
                w[e] = (k < H && j < H) ? (a.r_trans ? a.R[((size_t)gate_block(a.torch, g) * H + j) * H + k] : a.R[(size_t)k * C + (size_t)g * H + j]) : 0.f;
            }
            R2[o][i] = pack2(w[0], w[1]);
        }
    }
    // cell: unit cu, rows cb, cb + KG, ...
    const int cu = tid % U, cb = tid / U, cj = p * U + cu;
    const bool j_ok = cj < H;
    for (int i = tid; i < 6 * BtU; i += NT) dqs[i] = 0.f;   // dqs and dps
#pragma unroll
    for (int k = 0; k < 6; ++k) bsum[k * NT + tid] = 0.f;
    // Running pointers, last step first.  The cell's operands of a step, each thread its own: v (4), dh_new,
    // h_{t-1}, the 32-bit word that holds the cell's 16 mask bits.
    const long long dir = a.reverse ? 1 : -1, BH = dir * a.B * H;
    const size_t t_last = a.reverse ? 0 : a.T - 1, last = t_last * a.B + b0;      // first row of the last step
    const float *v_in = a.v + last * 4 * H + cj, *dn_in = a.dh_new + (long long)t_last * a.dn_ts + b0 * a.dn_bs + cj,
                *h_in = a.h + (last + (a.reverse ? a.B : 0)) * H + cj;
    size_t m_at = last * H + cj;
    float *dp_out = a.dp + last * C + cj, *dq_out = a.dq + last * C + cj;
    int g_off[3];
#pragma unroll
    for (int g = 0; g < 3; ++g) g_off[g] = gate_block(a.torch, g) * H;
    const bool act = One && j_ok && cb < nb;                 // One: this thread's cell is (row cb, unit cu)
    if constexpr (One) {
        v_in += (size_t)cb * 4 * H;
        dn_in += cb * a.dn_bs;
        h_in += (size_t)cb * H;
        m_at += (size_t)cb * H;
        dp_out += (size_t)cb * C;
        dq_out += (size_t)cb * C;
    }
    int slot_in = 0, left = a.T;
    auto fetch = [&]() {
        if constexpr (One) {
            if (act && left > 0) {
                float *d = stage + slot_in * 7 * BtU + cb * U + cu;
#pragma unroll
                for (int k = 0; k < 4; ++k) cp_async4(d + k * BtU, v_in + k * H);
                cp_async4(d + 4 * BtU, dn_in);
                cp_async4(d + 5 * BtU, h_in);
                if (a.pm) cp_async4(d + 6 * BtU, reinterpret_cast<const float *>(a.pm + (m_at & ~(size_t)1)));
            }
        } else if (left > 0 && j_ok) {
            float *dst = stage + slot_in * 7 * BtU + cu;
            for (int b = cb; b < nb; b += KG) {
                float *d = dst + b * U;
                const float *vb = v_in + b * 4 * H;
#pragma unroll
                for (int k = 0; k < 4; ++k) cp_async4(d + k * BtU, vb + k * H);
                cp_async4(d + 4 * BtU, dn_in + b * a.dn_bs);
                cp_async4(d + 5 * BtU, h_in + b * H);
                if (a.pm) cp_async4(d + 6 * BtU, reinterpret_cast<const float *>(a.pm + ((m_at + b * H) & ~(size_t)1)));
            }
        }
        v_in += 4 * BH;
        dn_in += dir * a.dn_ts;
        h_in += BH;
        m_at += BH;
        --left;
        slot_in = slot_in + 1 == D ? 0 : slot_in + 1;
        cp_async_commit();
    };
    for (int d = 0; d < D; ++d) fetch();
    size_t m_par = last * H + cj + (One ? (size_t)cb * H : 0);   // parity of the cell's mask index
    const uint32_t part_u32 = smem_addr(part);
    // gradient of the state of (row b, own unit): the part through the update gate plus the KG partial sums,
    // added in a fixed order, eight remote loads in flight
    auto carry = [&](int buf, int b) {
        float s = zdh[b * U + cu];
        const int off = buf * KG * BtU + p * BtU + b * U + cu;
        for (int k = 0; k < U / 32; ++k) {
            if (P == 1) {
                s += part[off + k * BtU];
                continue;
            }
            const uint32_t at = part_u32 + (uint32_t)(off + k * P * BtU) * 4u;
            for (int r = 0; r < P; r += 8) {
                float y[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) y[e] = r + e < P ? ld_remote(map_to_rank(at, (uint32_t)(r + e))) : 0.f;
#pragma unroll
                for (int e = 0; e < 8; ++e) s += y[e];
            }
        }
        return s;
    };
    float o_sum[6] = {}, o_dp[3] = {}, o_dq[3] = {};
    int slot = 0;
    __syncthreads();                                        // the zeros of dqs and dps are complete

    for (int i = a.T - 1; i >= 0; --i) {
        const int buf = i & 1;
        cp_async_wait_depth(D);
        const auto cell = [&](int b) {
                const int at = b * U + cu;
                const float *d = stage + slot * 7 * BtU + at;
                const float z = d[0], r = d[BtU], g = d[2 * BtU], q_g = d[3 * BtU], h_old = d[5 * BtU];
                const float in = i == a.T - 1 ? (a.dh_in ? a.dh_in[(size_t)(b0 + b) * H + cj] : 0.f) : carry(buf ^ 1, b);
                uint32_t m = 0xffffffffu;
                if (a.pm) m = __float_as_uint(d[6 * BtU]) >> ((One ? m_par & 1 : (m_par + b * H) & 1) * 16);
                float dh = d[4 * BtU] + in;
                if (!(m >> PM_H & 1)) dh *= 0.f;
                zdh[at] = z * dh;
                const float dg = (1.0f - z) * dh;
                const float dz = (h_old - g) * dh;
                const float dp_g = (1.0f - g * g) * dg;
                const float dp_r = (r * (1.0f - r)) * (dp_g * q_g);
                const float dp_z = (z * (1.0f - z)) * dz;
                float dp[3] = {dp_z, dp_r, dp_g}, dq[3] = {dp_z, dp_r, dp_g * r};
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    // (a dropped gradient is multiplied by 0, so that what is not finite stays visible)
                    const float keep = (m >> (PM_OUT + k) & 1) && (m >> (PM_IN + k) & 1) ? 1.f : 0.f;
                    dp[k] *= keep;
                    dq[k] *= keep;
                    if (!(m >> (PM_HH + k) & 1)) dq[k] *= 0.f;
                    dqs[b * 3 * U + k * U + cu] = dq[k];
                    if constexpr (One) {
                        o_sum[k] += dp[k];
                        o_sum[3 + k] += dq[k];
                    } else {
                        bsum[k * NT + tid] += dp[k];
                        bsum[(3 + k) * NT + tid] += dq[k];
                    }
                    if (!(m >> (PM_IH + k) & 1)) dp[k] *= 0.f;
                    if constexpr (One) {
                        o_dp[k] = dp[k];
                        o_dq[k] = dq[k];
                    } else {
                        dps[b * 3 * U + k * U + cu] = dp[k];
                    }
                }
        };
        if constexpr (One) {
            if (act) cell(cb);
        } else if (j_ok) {
            for (int b = cb; b < nb; b += KG) cell(b);
        }
        __syncthreads();
        const float *x = dqs + in0;
        const int owner = ob * 32 / U;
        float *po = part + buf * KG * BtU + (sl * P + owner) * BtU + (ob * 32 - owner * U) + q * 4 + (mg >> 1) * 2 + (mg & 1);
        for (int b = 0; b < nb; ++b, x += 3 * U, po += U) {
            uint64_t acc[4] = {};
#pragma unroll
            for (int t = 0; t < 6; ++t) {
                const ulonglong2 xv = *reinterpret_cast<const ulonglong2 *>(x + 4 * t);
#pragma unroll
                for (int o = 0; o < 4; ++o) {
                    acc[o] = ffma2(R2[o][2 * t], xv.x, acc[o]);
                    acc[o] = ffma2(R2[o][2 * t + 1], xv.y, acc[o]);
                }
            }
            float y[4];
#pragma unroll
            for (int o = 0; o < 4; ++o) {
                float lo, hi;
                unpack2(acc[o], lo, hi);
                y[o] = lo + hi;
            }
            // add the four input groups of the warp; lane group mg ends up with output mg of the quad
            const bool up = (mg & 2) != 0;
            const float k0 = up ? y[2] : y[0], k1 = up ? y[3] : y[1];
            const float s0 = __shfl_xor_sync(0xffffffffu, up ? y[0] : y[2], 16);
            const float s1 = __shfl_xor_sync(0xffffffffu, up ? y[1] : y[3], 16);
            const float a0 = k0 + s0, a1 = k1 + s1;
            const bool odd = (mg & 1) != 0;
            const float s2 = __shfl_xor_sync(0xffffffffu, odd ? a0 : a1, 8);
            *po = (odd ? a1 : a0) + s2;
        }
        if (P > 1) cluster_arrive();
        else __syncthreads();
        // (behind the arrive: see the forward)
        if constexpr (One) {
            if (act)
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    dp_out[g_off[k]] = o_dp[k];
                    dq_out[g_off[k]] = o_dq[k];
                }
        } else if (j_ok)
            for (int b = cb; b < nb; b += KG) {
                const float *dpb = dps + b * 3 * U + cu, *dqb = dqs + b * 3 * U + cu;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    dp_out[b * C + g_off[k]] = dpb[k * U];
                    dq_out[b * C + g_off[k]] = dqb[k * U];
                }
            }
        dp_out += 3 * BH;
        dq_out += 3 * BH;
        m_par += BH;
        slot = slot + 1 == D ? 0 : slot + 1;
        fetch();
        if (P > 1) cluster_wait();
    }
    if (j_ok)
        for (int b = cb; b < nb; b += KG) {
            const size_t at = (size_t)(b0 + b) * H + cj;
            const float dh = carry(0, b);
            a.dh_out[at] = a.h0_mask ? dh * (float)a.h0_mask[at] : dh;
        }
    if constexpr (One)
#pragma unroll
        for (int k = 0; k < 6; ++k) bsum[k * NT + tid] = o_sum[k];
    __syncthreads();
    for (int c = tid; c < 6 * U; c += NT) {
        const int k = c / U, uu = c % U;
        if (p * U + uu >= H) continue;
        float s = 0.f;
        for (int t = 0; t < KG; ++t) s += bsum[k * NT + t * U + uu];
        a.bias_part[((size_t)grp * 6 + (k < 3 ? 0 : 3) + gate_block(a.torch, k % 3)) * H + p * U + uu] = s;
    }
    if (P > 1) {   // nobody leaves while a peer may still read its partial sums
        cluster_arrive();
        cluster_wait();
    }
}

template <typename Kern>
int active_clusters(Kern kern, int P, int threads, size_t smem) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)P);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)P;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        (P > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template <typename Kern, typename Args>
cudaError_t launch_chain(Kern kern, const F32RecPlan &pl, Args &a, cudaStream_t st) {
    a.U = pl.U;
    a.P = pl.P;
    a.KG = pl.KG;
    a.Bt = pl.Bt;
    a.D = pl.D;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem);
    if (e != cudaSuccess) return e;
    if (pl.P > 8 && (e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(pl.G * pl.P));
    cfg.blockDim = dim3((unsigned)(pl.U * pl.KG));
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)pl.P;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, a);
}

// A form per cluster size whose registers hold R: 96 values in each of at most 512 threads a CTA.  `kern(threads)`: the kernel that a
// CTA of so many threads runs.  us per step, 32 / 64 units a CTA: forward H = 256: 1 row 1.9 / 3.5, 64 rows (5 a cluster) 2.8 / 3.9,
// 128 rows (9) 5.1 / 4.7; H = 128: 1 row 1.6 / 1.9, 256 rows (7, more than a cell a thread) 4.6 / 2.6; H = 160, 512 rows 10.8 / 7.5; backward
// H = 256: 1 row 2.0 / 2.7, 96 rows 3.6 / 3.9, 128 rows 5.3 / 4.4.  One CTA against clusters: H = 96 1.35 / 1.7, H = 128 (512 threads)
// 2.1 / 1.6.  The cost of a form is fitted to such times (H = 32 .. 512, 1 to 512 rows, one and two directions); that of CTAs of more
// than 384 threads and, backward, of two CTAs of 64 units to every form of 1 to 40 rows (as fitted before, two waves of one cell
// a thread were passed over forward: H = 480, 89 rows in two directions 24.2 us a step, now 16.9; and two CTAs taken for one
// backward: H = 128, 512 rows in two directions 8.9, now 7.8).
template <typename KernOf>
void make_plan(qgru_handle *h, int B, int sms, int directions, bool fwd, KernOf kern, size_t (*floats)(int, int, int, int, int), F32RecPlan *pl) {
    const int H = h->H;
    if (pl->H == H && pl->B == B && pl->sms == sms && pl->directions == directions) return;
    *pl = F32RecPlan{};
    pl->H = H;
    pl->B = B;
    pl->sms = sms;
    pl->directions = directions;
    const int chip = std::min(directions * sms, h->sm_count);   // side by side: as many clusters again, on as many SMs again
    double best = 0;
    for (int P = 1; P <= 16; ++P) {
        const int U = ((H + P - 1) / P + 31) / 32 * 32, KG = P * U / 32, threads = U * KG;
        if (threads > 512 || (P - 1) * U >= H) continue;
        const int active0 = active_clusters(kern(threads), P, threads, floats(P, U, KG, 1, 1) * sizeof(float));
        if (active0 <= 0) continue;
        // Cycles of a step of Bt rows: block barriers, the cell and, in a cluster, its barrier and the remote loads; the product and the
        // partial sums of a row, where a warp of 32 units has fewer neighbours to share the row's state with.  With more than a cell a
        // thread a row costs a block barrier's share at least.  CTAs of more than 384 threads spill.
        const int warps = threads / 32;
        const bool large = threads > 384;
        const double base = P == 1 ? 2050.0 : large ? 6000.0 : U == 32 ? 2950.0 : 3100.0 + 100.0 * (P - 2);
        const auto step = [&](int rows, int sharing) {
            const bool one = rows <= KG;
            if (large && P == 1) return fwd ? (one ? 3000.0 + 50.0 * warps * rows : 1500.0 + 104.0 * warps * rows)
                                            : (one ? 3800.0 + 81.0 * warps * rows : 4950.0 + 86.0 * warps * rows);
            if (large && fwd && one) return 5600.0 + (160.0 + 45.0 * warps) * rows;
            if (P == 2 && U == 64 && !fwd) return one ? 3600.0 + 608.0 * rows : 4220.0 + 838.0 * rows;
            if (one) return base + (U == 32 ? 70.0 : 47.0) * warps * rows * sharing;
            return fwd ? base + 2000.0 + std::max(750.0, (U == 32 ? 80.0 : 66.0) * warps) * rows * sharing
                       : base + 2400.0 + (U == 32 ? std::max(540.0, 65.0 * warps) : 52.0 * warps) * rows * sharing;
        };
        for (int Bt = 1; Bt <= MAX_ROWS && Bt <= B; ++Bt) {
            // operands three steps ahead where a step is shorter than a trip to memory
            const int D = Bt <= std::max(RB, KG) ? 3 : 1;
            const size_t smem = floats(P, U, KG, Bt, D) * sizeof(float);
            if (smem > (size_t)h->smem_optin) break;
            const int per_sm = std::max<int>(1, (int)std::min<size_t>((size_t)(active0 * P / h->sm_count), (size_t)(227 * 1024) / (smem + 1024)));
            const int active = std::max(1, std::min(active0, chip * per_sm / P));
            const int G = (B + Bt - 1) / Bt, waves = (directions * G + active - 1) / active;
            const int sharing = std::max(1, std::min(per_sm, (directions * G * P + chip - 1) / chip));
            double cost = waves * step(Bt, sharing);
            // One cluster too many for the chip: the last one of the second direction starts when the last one of the first, which has the
            // rest of the rows, is done.  us a step of both directions, such a plan / the best of the others: H = 262, 65 rows backward 5.4 /
            // 7.3; H = 320, 51 rows 4.7 / 6.1 forward, 5.5 / 7.1 backward; H = 416, 43 rows 8.6 / 10.7, 7.7 / 10.4.
            if (directions > 1 && directions * G == active + 1) cost = std::min(cost, std::max(step(Bt, sharing), 2.0 * step(B - (G - 1) * Bt, sharing)));
            if (best == 0 || cost < best) {
                best = cost;
                pl->P = P;
                pl->U = U;
                pl->KG = KG;
                pl->Bt = Bt;
                pl->D = D;
                pl->G = G;
                pl->waves = waves;
                pl->us = cost / 1900.0;          // (MHz under such a load)
                pl->smem = smem;
                pl->ok = true;
            }
        }
    }
}

// The kernel whose occupancy a form is planned with: the one for several cells a thread.  That for one cell has the same number of
// registers (168, with more than 384 threads 128).
auto fwd_kernel(int threads) { return threads <= 384 ? k_float_chain<false, 384, false> : k_float_chain<false, 512, false>; }
auto bwd_kernel(int threads) { return threads <= 384 ? k_bwd_chain<false, 384> : k_bwd_chain<false, 512>; }

// Whether one of make_plan's forms runs at all.
template <typename KernOf>
bool any_form(qgru_handle *h, KernOf kern, size_t (*floats)(int, int, int, int, int), int *known) {
    if (*known >= 0) return *known == 1;
    *known = 0;
    for (int P = 1; P <= 16 && *known == 0; ++P) {
        const int U = ((h->H + P - 1) / P + 31) / 32 * 32, KG = P * U / 32, threads = U * KG;
        const size_t smem = floats(P, U, KG, 1, 3) * sizeof(float);
        if (threads <= 512 && (P - 1) * U < h->H && smem <= (size_t)h->smem_optin && active_clusters(kern(threads), P, threads, smem) > 0) *known = 1;
    }
    return *known == 1;
}

// The SMs that this handle's kernels may take.
int side_sms(const qgru_handle *h) { return h->opt_sm_limit > 0 ? std::min(h->opt_sm_limit, h->sm_count) : h->sm_count; }

}  // namespace

bool float_chain_exists(qgru_handle *h) { return any_form(h, fwd_kernel, fwd_smem_floats, &h->f32_fwd_exists); }

bool float_chain_plan(qgru_handle *h, int B, int directions) {
    make_plan(h, B, side_sms(h), directions, true, fwd_kernel, fwd_smem_floats, &h->plan_fwd);
    return h->plan_fwd.ok;
}

// Every wave of clusters loads R first, and thousands of rows make many waves, where the tiled product of a step reads R once
// for 64 or 128 rows.  us per step in calls of 20, chain / step by step: H = 512: 180 rows 18.6 / 22.9, 300 rows 30.9 / 26.7; H = 384: 256
// rows 18.3 / 20.4, 600 rows 40.6 / 29.2; H = 256: 800 rows 20.5 / 27.4, 2048 rows 47.1 / 36.1; H = 128: 4096 rows 22.3 / 32.2, 6000 rows
// 33.4 / 31.1.  The chain as its plan costs it and 8 us a wave for R, the steps as fitted around the line between the two (far
// beyond it the product is on the tensor cores, and the steps cost less than this says).  Over 792 calls of 2, 3, 5 and 20 steps (H = 32 ..
// 512, 1 to 8192 rows) the choice costs 0.3 % in the mean; 15 lose more than 5 %, the worst (H = 96, 8192 rows, 3 steps) 38 %.
bool float_chain_is_faster(qgru_handle *h, int T, int B) {
    // (float inference and calibration run one direction after the other: each has the whole chip)
    make_plan(h, B, h->sm_count, 1, true, fwd_kernel, fwd_smem_floats, &h->plan_fwd);
    const F32RecPlan &pl = h->plan_fwd;
    if (!pl.ok) return false;
    const double H = h->H;
    return 8.0 + 8.0 * pl.waves + T * pl.us <= T * (17.0 + (1.32e-7 * H + 1.0e-5) * H * B);
}

// (forms of at most 384 threads have registers to spare beside R: the backward has no spills there, the forward 48 and 68
// bytes; with 512 threads 228 to 348 bytes, without a cluster 60)
int float_chain_launch(qgru_handle *h, FloatFwdArgs a, cudaStream_t st) {
    const F32RecPlan &pl = h->plan_fwd;
    const bool one = pl.Bt <= pl.KG, small = pl.U * pl.KG <= 384;
    CK(launch_chain(one ? (small ? k_float_chain<true, 384, false> : pl.P == 1 ? k_float_chain<true, 512, true> : k_float_chain<true, 512, false>)
                        : (small ? k_float_chain<false, 384, false> : k_float_chain<false, 512, false>), pl, a, st));
    h->launches++;
    return QGRU_OK;
}

bool bwd_chain_exists(qgru_handle *h) { return any_form(h, bwd_kernel, bwd_smem_floats, &h->f32_bwd_exists); }

bool bwd_chain_plan(qgru_handle *h, int B, int directions) {
    make_plan(h, B, side_sms(h), directions, false, bwd_kernel, bwd_smem_floats, &h->plan_bwd);
    return h->plan_bwd.ok;
}

// us per step in chains of 80, here / on the tensor cores: H = 100: 1 row 1.8 / 1.5, 256 rows 3.1 / 1.9; H = 256: 2.0 / 1.5, 6.0 / 2.9;
// H = 512: 2.8 / 2.0, 21.9 / 5.3.  Up to 96 units one CTA holds R in its registers: 1.2 (H = 64) to 1.45 (H = 96).
bool bwd_chain_tc_is_faster(qgru_handle *h, int B) {
    return h->H > 96 && bwd_chain_tc_plan(h, B, side_sms(h), &h->plan_bwd_tc);
}

int bwd_chain_launch(qgru_handle *h, BwdChainArgs a, cudaStream_t st) {
    const F32RecPlan &pl = h->plan_bwd;
    const bool one = pl.Bt <= pl.KG, small = pl.U * pl.KG <= 384;
    CK(launch_chain(one ? (small ? k_bwd_chain<true, 384> : k_bwd_chain<true, 512>) : (small ? k_bwd_chain<false, 384> : k_bwd_chain<false, 512>),
                    pl, a, st));
    h->launches++;
    return QGRU_OK;
}

}  // namespace qgru
