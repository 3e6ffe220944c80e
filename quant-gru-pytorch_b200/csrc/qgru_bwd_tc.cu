// qgru_bwd_tc.cu - the chain of state gradients of a quantized layer's training step on the tensor cores.
//
// dh_{t-1} = z dh_t + dq_t R: 3 H^2 multiply-adds per batch row and step with a dependency from step to step.  A cluster of
// P = ceil(H / U) CTAs works on a few rows; a CTA owns U units.  It multiplies where the operand is produced: its 3U values of
// dq per row (three gates) times the 3U rows of R they belong to give a partial dh for all H units, 128 units a tile of
// tcgen05.mma kind::f16, fp32 accumulators in tensor memory.  R is the quantized weight: its integers are exact in bf16 and
// stay on chip for the whole launch, in shared memory and, what does not fit there, in tensor memory (196 KB a CTA at
// H = 512, U = 64); its scale, one per channel and therefore per value of dq, is multiplied into dq.  (128ths of the integers and
// 128 times the scale: the products have the size of dq times R, and neither end of fp32's range comes closer.)  dq * scale is
// the exact sum of three bf16 values, which lie side by side as columns of one MMA (3 x rows wide): their products are exact,
// each third has accumulators of its own, and the sums meet in fp32.  The second part is kept 2^8, the third 2^16 times as
// large, so that both are exact down to fp32's smallest numbers (as they are, they fall below bf16's from 2^-110 down).
// The tensor cores add with truncation, over at most 192 products here.  Error of the layer's gradients against float64 (2-norm; H =
// 128 to 512, 1 to 256 rows, 50 to 200 steps, output gradients of one sign and of both) over that of the fp32 chain: dx 0.92 to 1.03,
// dh0 0.76 to 1.05, dR 0.98 to 1.08 (8e-8 to 3e-7 all of them).
//
// A step: cells (a warp per two or four rows and 32 units) add the P partial sums of their units and make dq; one thread a tile
// issues its MMAs; sixteen warps read the accumulators, 32 units each, and store them with 16-byte st.async into the
// CTA that owns the units, counted on its mbarrier.
//
// Every buffer is written again in every step.  What orders the next write after the last read:
//   dq's operand     the cells wait for the MMAs of ALL tiles of the step before (b_free) before they store; that their own
//                    partial sums have come says nothing of the tiles whose units other CTAs own.  (One barrier that every tile
//                    commits to: a wait for each tile's acc_full in turn was 0.35 us a step at H = 512);
//   accumulators     the MMAs of a step wait for an arrival of every warp (b_full): of a warp with cells when its share of dq is
//                    stored, of one without at the head of the step, of both behind their reads of the step before;
//   partial sums     a cluster barrier, arrived on when a warp has read what came for the last step and waited for before the
//                    next ones are sent; it lies behind the MMAs' time;
//   their mbarrier   armed for the next step by a thread that has seen the last one complete, before it arrives on that
//                    cluster barrier.
//
// us a step (80 steps), fp32 pipe / here: H = 512, 256 rows 21.9 / 5.3 (10700 cycles: 1700 cells, 2100 MMAs, 1600 reading the accumulators,
// 3200 until the last partial sum has come; those are 30 KB a CTA and step), 32 rows 4.5 / 2.4; H = 256, 256 rows 6.0 / 2.9; H = 128, 32 rows
// 1.8 / 1.5.  Pulling the partial sums with remote loads behind the barrier instead of st.async: 10900 cycles, and
// 0.2 us a step more at H <= 256.  Operands of the cells are fetched without a condition: under one, each value was copied, and
// waited for, where the branches meet (4700 to 7700 cycles a step).
#include <algorithm>

#include "qgru_cluster.cuh"
#include "qgru_device.cuh"
#include "qgru_handle.h"
#include "qgru_rec_f32.cuh"
#include "qgru_tc.cuh"

namespace qgru {
using namespace clu;
namespace {

constexpr int WARPS = 16, THREADS = 32 * WARPS;
constexpr int MAX_BT = 40;                   // 3 x 40 columns (128 with padding) in each of four tiles: all of tensor memory
constexpr long long WAIT_BUDGET = 2000000000ll;   // about a second of SM clocks
constexpr size_t MIN_SMEM = 116 * 1024;      // one CTA an SM, so that every CTA gets its tensor memory

// Both operands have their rows contiguous (units of R, batch rows of dq): 64 rows x 8 K of 1024 bytes, 128 bytes a K, the
// 16-byte chunk XOR K mod 8; groups of 8 K follow one another, then, `group` bytes on, the next 64 rows.
constexpr uint32_t DESC_HI = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t operand_at(int row, int k, int group) {
    return (uint32_t)((row >> 6) * group + (k >> 3) * 1024 + (k & 7) * 128 + ((((row & 63) >> 3) ^ (k & 7)) << 4) + (row & 7) * 2);
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b64 da, db;\n"
        "mov.b64 da, {%1, %5};\n"
        "mov.b64 db, {%2, %5};\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n"
        "}\n" ::"r"(d),
        "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(DESC_HI)
        : "memory");
}

// The same with A in tensor memory: a lane a unit, a column two K.
__device__ __forceinline__ void mma_bf16_ts(uint32_t d, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b64 db;\n"
        "mov.b64 db, {%2, %5};\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n"
        "}\n" ::"r"(d),
        "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(DESC_HI)
        : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

struct BwdTcArgs : BwdChainArgs {
    int rows;                  // Bt rounded up to four
    int width, tiles, groups;  // columns of an MMA, tiles of 128 units, groups of 64 units
    int nt;                    // how many of the 3U / 16 steps of K have their part of R in tensor memory: the last ones
    size_t smem;
    int *abort_flag;
};

// q / 128 as a bf16 value: exact
__device__ __forceinline__ uint32_t r_operand(int8_t q) { return __float_as_uint((float)q * 0x1p-7f) >> 16; }

// x as w0 + 2^-8 w1 + 2^-16 w2, each a bf16 value in the upper half of a word: exact for finite x, subnormal ones too (w0 leaves a
// multiple of 2^-149 below 2^-8 of x or 2^-133, w1 one below 2^-16 of x or 2^-141); what is not finite (or rounds to infinity)
// is the first part alone, so that its products are those of x
__device__ __forceinline__ void split3(float x, uint32_t (&w)[3]) {
    asm("cvt.rn.bf16x2.f32 %0, %1, 0f00000000;" : "=r"(w[0]) : "f"(x));
    float r = (x - __uint_as_float(w[0])) * 0x1p8f;
    r = fabsf(r) <= 3.0e38f ? r : 0.f;
    asm("cvt.rn.bf16x2.f32 %0, %1, 0f00000000;" : "=r"(w[1]) : "f"(r));
    r = (r - __uint_as_float(w[1])) * 0x1p8f;
    asm("cvt.rn.bf16x2.f32 %0, %1, 0f00000000;" : "=r"(w[2]) : "f"(r));
}

// RPT: rows of a cell thread.
template <int U, int RPT>
__global__ void __launch_bounds__(THREADS, 1) k_bwd_chain_tc(const BwdTcArgs a) {
    static_assert(RPT == 2 || RPT == 4, "rows are padded to four");
    constexpr int K = 3 * U, UW = U / 32, B_GROUP = K * 128;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *ops = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int ks = K / 16 - a.nt, a_group = ks * 16 * 128;                                  // steps of K in shared memory
    unsigned char *b_ops = ops + a.groups * a_group;
    float *recv = reinterpret_cast<float *>(b_ops + (3 * a.rows + 63) / 64 * B_GROUP);      // [P][rows / 4][U][4]
    float *bsum = recv + a.P * U * a.rows;                                                  // [cell warps][6][32]
    uint64_t *bars = reinterpret_cast<uint64_t *>(bsum + WARPS * 6 * 32);
    uint64_t *got = bars, *b_full = bars + 1, *b_free = bars + 2, *acc_full = bars + 3;     // acc_full: one per tile
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 7);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, H = a.H, P = a.P;
    const int p = (int)cluster_rank();
    const int grp = blockIdx.x / P, b0 = grp * a.Bt, nb = min(a.Bt, a.B - b0);
    const int cell_warps = a.rows / RPT * UW;
    const uint32_t recv_bytes = (uint32_t)(P * min(U, (H - p * U + 31) & ~31) * a.rows * 4);
    if (tid == 0) {
        tc::mbar_init(got, 1);
        tc::mbar_init(b_full, WARPS);
        tc::mbar_init(b_free, (uint32_t)a.tiles);
        for (int t = 0; t < 4; ++t) tc::mbar_init(&acc_full[t], 1);
        tc::fence_barrier_init();
        tc::mbar_expect_tx(got, recv_bytes);
    }
    if (warp == WARPS - 1) tc::tmem_alloc(tmem_slot, 512);
    // R: unit j of all, value k = gate * U + u of this CTA's; rows past the matrix are zero
    const auto weight = [&](int j, int k) {
        const int ju = p * U + k % U;
        return j < H && ju < H ? r_operand(a.r8[((size_t)(k / U) * H + ju) * H + j]) : 0u;
    };
    const bool words = H % 4 == 0;       // (the integers start at a 256-byte boundary)
    const int quads = a.groups * 16;
#pragma unroll 4
    for (int i = tid; i < ks * 16 * quads; i += THREADS) {
        const int j = i % quads * 4, k = i / quads, ju = p * U + k % U;
        uint32_t w[4] = {0u, 0u, 0u, 0u};
        if (words) {
            const char4 q = j < H && ju < H ? *reinterpret_cast<const char4 *>(a.r8 + ((size_t)(k / U) * H + ju) * H + j) : make_char4(0, 0, 0, 0);
            w[0] = r_operand(q.x);
            w[1] = r_operand(q.y);
            w[2] = r_operand(q.z);
            w[3] = r_operand(q.w);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = weight(j + e, k);
        }
        *reinterpret_cast<uint2 *>(ops + operand_at(j, k, a_group)) = make_uint2(w[0] | w[1] << 16, w[2] | w[3] << 16);
    }
    for (int i = tid; i < (3 * a.rows + 63) / 64 * B_GROUP / 16; i += THREADS) reinterpret_cast<uint4 *>(b_ops)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const uint32_t tmem = *tmem_slot, tmem_a = tmem + (uint32_t)(a.tiles * a.width);
    const int tile = warp >> 2, quad = warp & 3;             // accumulators: tile, 32 of its units
    if (tile < a.tiles) {
        for (int t = 0; t < a.nt; ++t) {
            uint32_t w[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int j = tile * 128 + quad * 32 + lane, k = (ks + t) * 16 + 2 * c;
                w[c] = weight(j, k) | weight(j, k + 1) << 16;
            }
            tmem_st8(tmem_a + ((uint32_t)(quad * 32) << 16) + (uint32_t)((t * a.tiles + tile) * 8), w);
        }
        tc::tmem_st_wait();
    }
    fence_proxy_async_cta();
    tc::tc_fence_before_sync();
    cluster_arrive();
    cluster_wait();
    tc::tc_fence_after_sync();

    // cells: unit cu of this CTA's, rows r0 .. r0 + RPT - 1
    const bool cells = warp < cell_warps;
    const int r0 = warp / UW * RPT, cu = warp % UW * 32 + lane, cj = p * U + cu;
    bool act[RPT];
#pragma unroll
    for (int e = 0; e < RPT; ++e) act[e] = cells && cj < H && r0 + e < nb;
    const long long dir = a.reverse ? 1 : -1, BH = dir * a.B * H;
    const size_t t_last = a.reverse ? 0 : a.T - 1, last = t_last * a.B + b0;    // first row of the last step
    const int lj = min(cj, H - 1);
    const float *v_in = a.v + last * 4 * H + lj, *dn_in = a.dh_new + (long long)t_last * a.dn_ts + b0 * a.dn_bs + lj,
                *h_in = a.h + (last + (a.reverse ? a.B : 0)) * H + lj;
    const uint16_t *m_in = a.pm + last * H + lj;
    float *dp_out = a.dp + (last + r0) * 3 * H + cj, *dq_out = a.dq + (last + r0) * 3 * H + cj;
    int g_off[3];
    float scale[3];
#pragma unroll
    for (int g = 0; g < 3; ++g) {
        g_off[g] = (a.torch && g < 2 ? 1 - g : g) * H;
        scale[g] = cj < H ? a.r_scale[g * H + cj] * 128.f : 0.f;
    }
    // Operands of the next step: v (4), gradient from outside, state before, masks.  The loads have no condition: a cell that does
    // not exist reads the place of one that does, so that no value waits for its load before it is used, a step later.
    int row[RPT];
#pragma unroll
    for (int e = 0; e < RPT; ++e) row[e] = min(r0 + e, nb - 1);
    float x[RPT][6];
    uint32_t m[RPT];
    const auto fetch = [&]() {
#pragma unroll
        for (int e = 0; e < RPT; ++e) {
#pragma unroll
            for (int k = 0; k < 4; ++k) x[e][k] = v_in[(row[e] * 4 + k) * H];
            x[e][4] = dn_in[row[e] * a.dn_bs];
            x[e][5] = h_in[row[e] * H];
            m[e] = m_in[row[e] * H];
        }
    };
    const auto next = [&]() {
        v_in += 4 * BH;
        dn_in += dir * a.dn_ts;
        h_in += BH;
        m_in += BH;
    };
    float zdh[RPT] = {}, sum[6] = {};
    fetch();
    bool ok = true;
    // what the P CTAs have sent for this thread's cells, added in their order
    const auto carry = [&](float (&y)[RPT]) {
        const float *q = recv + ((r0 >> 2) * U + cu) * 4 + (r0 & 3);
        const int step = U * a.rows;
        const auto add = [&](const float *at, float (&w)[RPT]) {
            if constexpr (RPT == 4) {
                const float4 v = *reinterpret_cast<const float4 *>(at);
                w[0] = v.x;
                w[1] = v.y;
                w[2] = v.z;
                w[3] = v.w;
            } else {
                const float2 v = *reinterpret_cast<const float2 *>(at);
                w[0] = v.x;
                w[1] = v.y;
            }
        };
        int s = 0;
        for (; s + 4 <= P; s += 4, q += 4 * step) {
            float w[4][RPT];
#pragma unroll
            for (int e = 0; e < 4; ++e) add(q + e * step, w[e]);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < RPT; ++i) y[i] += w[e][i];
        }
        for (; s < P; ++s, q += step) {
            float w[RPT];
            add(q, w);
#pragma unroll
            for (int i = 0; i < RPT; ++i) y[i] += w[i];
        }
    };
    const int unit0 = tile * 128 + quad * 32;
    const bool drains = tile < a.tiles && unit0 < H, issues = warp >= WARPS - a.tiles;   // (the last warps: those without cells, mostly)
    const int mt = WARPS - 1 - warp;                         // the tile whose MMAs this warp issues
    const uint32_t acc = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(tile * a.width);
    const uint32_t peer = (uint32_t)(drains ? unit0 / U : 0);
    const uint32_t dst = map_to_rank(tc::smem_u32(recv + p * U * a.rows + (unit0 % U + lane) * 4), peer);
    const uint32_t dst_bar = map_to_rank(tc::smem_u32(got), peer);
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(a.width >> 3) << 17) | (8u << 24);
    const uint32_t a0 = (((tc::smem_u32(ops) + 2u * (uint32_t)(mt * a_group)) & 0x3FFFFu) >> 4) | (uint32_t)(a_group >> 4) << 16;
    const uint32_t bb = ((tc::smem_u32(b_ops) & 0x3FFFFu) >> 4) | (uint32_t)(B_GROUP >> 4) << 16;
    const uint32_t at0 = tmem_a + (uint32_t)(mt * 8);

    for (int s = 0; s < a.T; ++s) {
        float y[RPT];
#pragma unroll
        for (int e = 0; e < RPT; ++e) y[e] = zdh[e];
        if (cells) {
            if (s == 0) {
#pragma unroll
                for (int e = 0; e < RPT; ++e)
                    if (act[e] && a.dh_in) y[e] = a.dh_in[(size_t)(b0 + r0 + e) * H + cj];
            } else {
                // (complete before the partial sums come, save where a tile's MMAs were issued late)
                ok = ok && tc::mbar_wait(b_free, (uint32_t)((s - 1) & 1), WAIT_BUDGET);
                ok = ok && tc::mbar_wait(got, (uint32_t)((s - 1) & 1), WAIT_BUDGET);
                if (tid == 0) tc::mbar_expect_tx(got, recv_bytes);
                carry(y);
            }
        }
        if (cells) {
            float dp[RPT][3], dq[RPT][3];
#pragma unroll
            for (int e = 0; e < RPT; ++e) {
                const float z = x[e][0], r = x[e][1], g = x[e][2], q_g = x[e][3], h_old = x[e][5];
                float dh = x[e][4] + y[e];
                if (!(m[e] >> PM_H & 1)) dh *= 0.f;
                zdh[e] = z * dh;
                const float dg = (1.0f - z) * dh;
                const float dz = (h_old - g) * dh;
                const float dp_g = (1.0f - g * g) * dg;
                const float dp_r = (r * (1.0f - r)) * (dp_g * q_g);
                const float dp_z = (z * (1.0f - z)) * dz;
                dp[e][0] = dq[e][0] = dp_z;
                dp[e][1] = dq[e][1] = dp_r;
                dp[e][2] = dp_g;
                dq[e][2] = dp_g * r;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    // (a dropped gradient is multiplied by 0, so that what is not finite stays visible)
                    const float keep = (m[e] >> (PM_OUT + k) & 1) && (m[e] >> (PM_IN + k) & 1) ? 1.f : 0.f;
                    dp[e][k] *= keep;
                    dq[e][k] *= keep;
                    if (!(m[e] >> (PM_HH + k) & 1)) dq[e][k] *= 0.f;
                    if (act[e]) {
                        sum[k] += dp[e][k];
                        sum[3 + k] += dq[e][k];
                    } else {
                        dq[e][k] = zdh[e] = 0.f;
                    }
                    if (!(m[e] >> (PM_IH + k) & 1)) dp[e][k] *= 0.f;
                }
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                uint32_t w[RPT][3];
#pragma unroll
                for (int e = 0; e < RPT; ++e) split3(dq[e][k] * scale[k], w[e]);
#pragma unroll
                for (int part = 0; part < 3; ++part) {
                    unsigned char *to = b_ops + operand_at(part * a.rows + r0, k * U + cu, B_GROUP);
                    if constexpr (RPT == 4)
                        *reinterpret_cast<uint2 *>(to) = make_uint2(__byte_perm(w[0][part], w[1][part], 0x7632), __byte_perm(w[2][part], w[3][part], 0x7632));
                    else
                        *reinterpret_cast<uint32_t *>(to) = __byte_perm(w[0][part], w[1][part], 0x7632);
                }
            }
            fence_proxy_async_cta();
            tc::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(b_full);
            __syncwarp();
            cluster_arrive();            // this warp has read what came for the last step
            // (behind the arrive, whose release would wait for them)
#pragma unroll
            for (int e = 0; e < RPT; ++e)
                if (act[e])
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        dp_out[e * 3 * H + g_off[k]] = dp[e][k];
                        dq_out[e * 3 * H + g_off[k]] = dq[e][k];
                    }
            dp_out += 3 * BH;
            dq_out += 3 * BH;
        } else {
            if (lane == 0) tc::mbar_arrive(b_full);     // this warp's reads of the accumulators lie behind it
            __syncwarp();
            cluster_arrive();
        }
        if (issues) {
            if (lane == 0) {
                ok = ok && tc::mbar_wait(b_full, (uint32_t)(s & 1), WAIT_BUDGET);
                if (ok) {
                    tc::tc_fence_after_sync();
                    const uint32_t d = tmem + (uint32_t)(mt * a.width);
                    for (int k = 0; k < ks; ++k) mma_bf16(d, a0 + (uint32_t)(k * 2048 >> 4), bb + (uint32_t)(k * 2048 >> 4), idesc | 1u << 15, (uint32_t)k);
                    for (int k = 0; k < a.nt; ++k)
                        mma_bf16_ts(d, at0 + (uint32_t)(k * a.tiles * 8), bb + (uint32_t)((ks + k) * 2048 >> 4), idesc, (uint32_t)(ks + k));
                    tc::mma_commit(&acc_full[mt]);
                    tc::mma_commit(b_free);
                }
            }
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        }
        if (drains) {
            ok = ok && tc::mbar_wait(&acc_full[tile], (uint32_t)(s & 1), WAIT_BUDGET);
            ok = __all_sync(0xffffffffu, ok);
            tc::tc_fence_after_sync();
        }
        cluster_wait();                  // every CTA has read its partial sums of the last step
        if (drains && ok) {
            for (int c = 0; c < a.rows; c += 16) {
                int32_t v[3][16];
#pragma unroll
                for (int part = 0; part < 3; ++part) tc::tmem_ld16(acc + (uint32_t)(part * a.rows + c), v[part]);
                tc::tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (c + 4 * e < a.rows) {
                        uint32_t w[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            w[i] = __float_as_uint(fmaf(fmaf(__int_as_float(v[2][4 * e + i]), 0x1p-8f, __int_as_float(v[1][4 * e + i])), 0x1p-8f, __int_as_float(v[0][4 * e + i])));
                        st_async_v4(dst + (uint32_t)(c + 4 * e) * (U * 4u), w, dst_bar);
                    }
            }
            tc::tc_fence_before_sync();  // (the loads are complete: tmem_ld_wait)
        }
        __syncwarp();
        // (what the next step does not wait for: while the partial sums are on their way)
        if (cells) {
            if (s + 2 <= a.T) next();        // (the last step fetches its own once more)
            fetch();
        }
    }
    if (cells) {
        ok = ok && tc::mbar_wait(got, (uint32_t)((a.T - 1) & 1), WAIT_BUDGET);
        float y[RPT];
#pragma unroll
        for (int e = 0; e < RPT; ++e) y[e] = zdh[e];
        carry(y);
#pragma unroll
        for (int e = 0; e < RPT; ++e)
            if (act[e]) {
                const size_t at = (size_t)(b0 + r0 + e) * H + cj;
                a.dh_out[at] = a.h0_mask ? y[e] * (float)a.h0_mask[at] : y[e];
            }
#pragma unroll
        for (int k = 0; k < 6; ++k) bsum[(warp * 6 + k) * 32 + lane] = sum[k];
    }
    if (!ok && lane == 0) raise_abort(a.abort_flag, 1);
    tc::tc_fence_before_sync();
    __syncthreads();
    for (int c = tid; c < 6 * U; c += THREADS) {
        const int k = c / U, uu = c % U;
        if (p * U + uu >= H) continue;
        float s = 0.f;
        for (int w = 0; w < a.rows / RPT; ++w) s += bsum[((w * UW + uu / 32) * 6 + k) * 32 + uu % 32];
        const int g = k % 3;
        a.bias_part[((size_t)grp * 6 + (k < 3 ? 0 : 3) + (a.torch && g < 2 ? 1 - g : g)) * H + p * U + uu] = s;
    }
    if (warp == WARPS - 1) tc::tmem_dealloc(tmem, 512);
    cluster_arrive();    // nobody leaves while a peer may still store into it
    cluster_wait();
}

// What follows from H, U and Bt; false where it does not fit.
bool fill(const F32RecPlan &pl, int H, size_t smem_optin, BwdTcArgs *a) {
    const int K = 3 * pl.U;
    a->U = pl.U;
    a->P = pl.P;
    a->Bt = pl.Bt;
    a->rows = (pl.Bt + 3) & ~3;
    a->width = (3 * a->rows + 15) & ~15;
    a->tiles = (H + 127) / 128;
    a->groups = (H + 63) / 64;
    if (a->rows / 4 * (pl.U / 32) > WARPS) return false;
    for (a->nt = 0; a->nt <= K / 16; ++a->nt) {
        const int in_tmem = a->tiles * (a->width + 8 * a->nt);
        a->smem = std::max(MIN_SMEM, (size_t)a->groups * (K - 16 * a->nt) * 128 + (size_t)(3 * a->rows + 63) / 64 * K * 128 +
                                         (size_t)pl.P * pl.U * a->rows * 4 + WARPS * 6 * 32 * 4 + 1024 + 256);
        if (in_tmem > 512) return false;
        if (a->smem <= smem_optin) return true;
    }
    return false;
}

// Two rows a cell thread where sixteen warps cover them: the cells are a chain of instructions at the head of the step, and twice the
// warps have half of it each.  us a step, four rows a thread / two / one: H = 128, 32 rows 1.97 / 1.48 / 1.81; H = 256, 64 rows 2.17 / 1.82 /
// 2.21; H = 384, 256 rows 3.7 / 3.4.  With 64 units a CTA and four tiles all warps read accumulators and four issue MMAs besides:
// H = 512, 192 rows 4.4 / 4.7, 256 rows 5.3 / 5.3.
auto kernel_of(int U, int rows, int tiles) {
    const bool two = rows / 2 * (U / 32) <= WARPS && (U == 32 || tiles < 4);
    if (U == 32) return two ? k_bwd_chain_tc<32, 2> : k_bwd_chain_tc<32, 4>;
    return two ? k_bwd_chain_tc<64, 2> : k_bwd_chain_tc<64, 4>;
}

cudaLaunchConfig_t config(int P, int G, size_t smem, cudaStream_t st, cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(P * G));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)P;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

// The form for B rows, in clusters of two CTAs or more (H > 64).  32 units a CTA are the shorter step (half the MMAs) until a cluster
// has more than 20 rows: what then takes longest is the H x rows partial sums that a CTA sends (14 bytes a clock), and 64 units a
// CTA are half the CTAs a cluster, twice the clusters and half the rows.  us per step (24 steps, four rows a cell thread), 32 / 64
// units: H = 512: 128 rows 4.8 / 5.0, 256 rows 7.0 / 6.2; H = 384: 256 rows 5.5 / 4.5; H = 262: 256 rows (16 a cluster) 3.7 / 4.1.  128 units a
// CTA were slower.
bool bwd_chain_tc_plan(qgru_handle *h, int B, int sms, F32RecPlan *best) {
    const int H = h->H;
    if (best->H == H && best->B == B && best->sms == sms) return best->ok;
    *best = F32RecPlan{};
    best->H = H;
    best->B = B;
    best->sms = sms;
    if (H <= 64 || H > 512) return false;
    for (const int U : {32, 64}) {
        if (best->ok && best->Bt <= 20 && best->waves == 1) break;
        F32RecPlan pl = *best;
        pl.ok = false;
        pl.U = U;
        pl.P = (H + U - 1) / U;
        BwdTcArgs a{};
        pl.Bt = MAX_BT;
        while (pl.Bt > 0 && !fill(pl, H, (size_t)h->smem_optin, &a)) pl.Bt -= 4;
        if (pl.Bt <= 0) continue;
        const int most = pl.Bt;
        const auto kern = kernel_of(U, a.rows, a.tiles);
        cudaLaunchAttribute attr[1];
        const cudaLaunchConfig_t cfg = config(pl.P, 1, (size_t)h->smem_optin, nullptr, attr);
        int active = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)h->smem_optin) != cudaSuccess ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&active, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        active = std::min((int)((long long)active * sms / h->sm_count), sms / pl.P);
        if (active <= 0) continue;
        pl.waves = (B + active * most - 1) / (active * most);
        pl.Bt = (B + active * pl.waves - 1) / (active * pl.waves);
        pl.G = (B + pl.Bt - 1) / pl.Bt;
        if (!fill(pl, H, (size_t)h->smem_optin, &a)) continue;
        pl.smem = a.smem;
        pl.ok = true;
        if (!best->ok || pl.waves <= best->waves) *best = pl;
    }
    return best->ok;
}

int bwd_chain_tc_launch(qgru_handle *h, const F32RecPlan &pl, const BwdChainArgs &args, cudaStream_t st) {
    BwdTcArgs a{};
    static_cast<BwdChainArgs &>(a) = args;
    if (!fill(pl, h->H, (size_t)h->smem_optin, &a)) return fail(h, QGRU_ERR_UNSUPPORTED, "no plan for the chain of state gradients");
    a.abort_flag = h->d_flags + 1;
    const auto kern = kernel_of(pl.U, a.rows, a.tiles);
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)h->smem_optin));
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = config(pl.P, pl.G, a.smem, st, attr);
    CK(cudaLaunchKernelEx(&cfg, kern, a));
    h->launches++;
    return QGRU_OK;
}

}  // namespace qgru
