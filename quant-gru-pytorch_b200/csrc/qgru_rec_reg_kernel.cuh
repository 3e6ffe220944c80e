// qgru_rec_reg_kernel.cuh - the kernel of qgru_rec_reg.cu (there: what bounds it, the split).  Two translation units
// instantiate it, one for the inference cells and one for the training cells.
#pragma once
#include "qgru_rec_reg.cuh"

#include "qgru_cluster.cuh"
#include "qgru_device.cuh"
#include "qgru_handle.h"
#include "qgru_tc.cuh"

#include <type_traits>

namespace qgru {
using namespace clu;
namespace {

constexpr long long WAIT_BUDGET = 2000000000ll;   // ~1 s of SM clocks

template <bool HU>
__device__ __forceinline__ void imma(int32_t (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if constexpr (HU)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(tc::smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// until at most D - 1 of this thread's groups are in flight (D = 1 .. 3)
__device__ __forceinline__ void cp_async_wait_depth(int D) {
    if (D == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else if (D == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
}
// two neighbouring values of W*x + bw
template <typename IhT>
__device__ __forceinline__ void load_pair(const IhT *p, int &a, int &b) {
    if constexpr (sizeof(IhT) == 2) {
        const uint32_t w = *reinterpret_cast<const uint32_t *>(p);
        a = (int16_t)(w & 0xffffu);
        b = (int32_t)w >> 16;
    } else if constexpr (sizeof(IhT) == 4) {
        const int2 w = *reinterpret_cast<const int2 *>(p);
        a = w.x;
        b = w.y;
    } else {
        a = p[0];
        b = p[1];
    }
}

// Generic cell: R*h + br requantization of one channel.
struct GenLin {
    int64_t corr;
    Rescale rs;
};

__host__ __device__ constexpr size_t cell_const_bytes(int cell) {
    return cell <= CELL_INT_FAST_NOTIE ? sizeof(FastLin) : cell == CELL_INT_GENERIC || cell == CELL_INT_TRAIN ? sizeof(GenLin) : 3 * sizeof(float);
}

// State rows are 64 bytes modulo 128 apart: the four 16-byte pieces of two neighbouring rows that a quarter warp
// loads at once fall into different banks.
__host__ __device__ constexpr int state_stride(int K) { return K + (K % 128 == 0 ? 64 : 0); }
constexpr int RED_STRIDE = 33;   // words between the values of a partial-sum block: the reader's lanes spread over the banks

struct RegSmem {
    size_t tables, consts, hs, ihs, red, total;
};
__host__ __device__ inline RegSmem reg_smem(int K, int U, int KS, int NT, int D, int ih_bytes, int cell, int n_table) {
    const auto up = [](size_t v) { return (v + 127) & ~size_t(127); };
    RegSmem s;
    s.tables = 128;                                                        // barriers in front
    s.consts = s.tables + up((size_t)n_table * 4);
    s.hs = s.consts + up((size_t)3 * U * cell_const_bytes(cell));
    s.ihs = s.hs + up((size_t)2 * NT * 8 * state_stride(K));
    s.red = s.ihs + up((size_t)D * NT * 8 * 3 * U * ih_bytes);
    s.total = s.red + (KS > 1 ? up((size_t)2 * (U / 16) * KS * 12 * RED_STRIDE * 4) : 0);
    return s;
}

template <typename IhT, int KST, int Cell, bool HU, int KS, bool Few = KS == 1>
__global__ void __launch_bounds__(512, 1) k_rec_reg(const __grid_constant__ GateConsts gc, const __grid_constant__ RecRegArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr bool Tie = Cell != CELL_INT_FAST_NOTIE, Train = Cell >= CELL_INT_TRAIN;
    constexpr bool Split = KS > 1;
    constexpr int K = KS * KST * 32, HS = state_stride(K);
    const int U = a.U, P = Split ? a.P : 1, NT = a.NT, D = a.D, H = a.H;
    const RegSmem L = reg_smem(K, U, KS, NT, D, (int)sizeof(IhT), Cell, a.n_table);
    uint64_t *h_ready = reinterpret_cast<uint64_t *>(smem);      // [2], clusters only
    uint64_t *ih_full = h_ready + 2;                             // [D], one CTA only
    int32_t *tables = reinterpret_cast<int32_t *>(smem + L.tables);
    unsigned char *consts = smem + L.consts;
    unsigned char *hs = smem + L.hs;                             // [2][NT * 8][HS]
    int *red = reinterpret_cast<int *>(smem + L.red);            // [2][unit group][KS][12][RED_STRIDE]

    const int tid = threadIdx.x, NTH = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int W = NTH >> 5;
    const int p = P > 1 ? (int)cluster_rank() : 0;
    const int b0 = (blockIdx.x / P) * a.Bt, nb = min(a.Bt, a.B - b0);
    const int j0 = p * U;
    const int ug = warp / KS, ks = warp - ug * KS;               // unit group and K slice of this warp
    const int g8 = lane >> 2, q4 = lane & 3;

    // R: tile row r of a gate is unit 2 * (r & 7) + (r >> 3) of the group, so that a thread's two rows are
    // neighbouring units.  Within 64 inputs the K order is permuted (the same way for R and the state): lane
    // q4 takes 16 consecutive bytes, two words for each of two instructions.
    uint32_t R[3][KST][4];
#pragma unroll
    for (int g = 0; g < 3; ++g)
#pragma unroll
        for (int c = 0; c < KST / 2; ++c)
#pragma unroll
            for (int hi = 0; hi < 2; ++hi) {
                const int j = j0 + ug * 16 + 2 * g8 + hi, k = ks * KST * 32 + c * 64 + q4 * 16;
                uint4 w = make_uint4(0u, 0u, 0u, 0u);
                if (j < H && k < a.Hpad) w = *reinterpret_cast<const uint4 *>(a.r8 + (size_t)(g * H + j) * a.Hpad + k);
                R[g][2 * c][hi] = w.x;
                R[g][2 * c][2 + hi] = w.y;
                R[g][2 * c + 1][hi] = w.z;
                R[g][2 * c + 1][2 + hi] = w.w;
            }
    for (int i = tid; i < a.n_table; i += NTH) tables[i] = a.tables[i];
    for (int i = tid; i < 3 * U; i += NTH) {
        const int g = i / U, j = j0 + i % U;
        const bool ok = j < H;
        if constexpr (Cell <= CELL_INT_FAST_NOTIE) {
            reinterpret_cast<FastLin *>(consts)[i] = ok ? a.lc.fl[g * H + j] : FastLin{0, 0, 0, 0, 0, 0};
        } else if constexpr (Cell == CELL_INT_GENERIC || Cell == CELL_INT_TRAIN) {
            reinterpret_cast<GenLin *>(consts)[i] = ok ? GenLin{a.lc.corr[g * H + j], a.lc.rs[g * H + j]} : GenLin{0, Rescale{1, 1, 0, 0, 0, 0, 0, 0}};
        } else {
            for (int k = 0; k < 3; ++k) reinterpret_cast<float *>(consts)[k * 3 * U + i] = ok ? a.fs_chan[(size_t)k * 3 * H + g * H + j] : 0.f;
        }
    }
    // (everything up to here is the handle's own and may run beside the launches before)
    pdl_wait();
    put_stamp(a.stamp);
    // initial state: the rows of the cluster, all K inputs
    for (int i = tid; i < nb * (K >> 4); i += NTH) {
        const int b = i / (K >> 4), k = (i - b * (K >> 4)) * 16;
        uint4 w = make_uint4(0u, 0u, 0u, 0u);
        if (k < a.Hpad) w = *reinterpret_cast<const uint4 *>(a.h8 + (size_t)(b0 + b) * a.Hpad + k);
        *reinterpret_cast<uint4 *>(hs + b * HS + k) = w;
    }
    if (tid == 0) {
        tc::mbar_init(&h_ready[0], W);
        tc::mbar_init(&h_ready[1], W);
        for (int d = 0; d < D; ++d) tc::mbar_init(&ih_full[d], 1);
        tc::fence_barrier_init();
    }
    __syncthreads();
    if (P > 1) {   // no peer may send before the barriers are initialised
        cluster_arrive();
        cluster_wait();
    }
    // W*x + bw, D steps ahead.  One CTA: one bulk copy of a contiguous block per step ([rows][3][U]).  Clusters: every warp
    // fetches what its own cells read (RW rows of each tile, three gates, 16 units) in 16-byte copies and waits
    // for nobody else's; there a late issuing thread delays every CTA (H = 512, two rows: 2.35 -> 2.15 us per step with
    // the rest of the step unrolled; one CTA, two rows of H = 256: 2.6 against 2.3 with the bulk copy).
    constexpr int RW = 8 / KS, CHUNKS = RW * 3 * (int)sizeof(IhT), NC = (CHUNKS + 31) / 32;
    const size_t ih_row = (size_t)3 * U * sizeof(IhT);
    const char *ih_next = static_cast<const char *>(a.ih) + ((size_t)p * a.T * a.B + (size_t)(a.reverse ? a.T - 1 : 0) * a.B + b0 + (Split ? ks * RW : 0)) * ih_row +
                          (Split ? (size_t)ug * 16 * sizeof(IhT) : 0);
    const ptrdiff_t ih_step = (a.reverse ? -(ptrdiff_t)a.B : (ptrdiff_t)a.B) * (ptrdiff_t)ih_row;
    const unsigned char *ihs_w = smem + L.ihs + (Split ? (size_t)warp * D * NT * CHUNKS * 16 : 0);      // [D][NT][RW][3][16]
    const uint32_t ihs_u32 = tc::smem_u32(ihs_w) + (Split ? (uint32_t)lane * 16u : 0u);
    const uint32_t slot_bytes = Split ? (uint32_t)(NT * CHUNKS * 16) : (uint32_t)(NT * 8) * (uint32_t)ih_row;
    int src_off[NC], src_row[NC];
    if constexpr (Split) {
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const int c = lane + 32 * i, row = c / (3 * (int)sizeof(IhT)), r = c - row * 3 * (int)sizeof(IhT), g = r / (int)sizeof(IhT);
            src_row[i] = c < CHUNKS ? ks * RW + row : 1 << 30;
            src_off[i] = row * (int)ih_row + g * U * (int)sizeof(IhT) + (r - g * (int)sizeof(IhT)) * 16;
        }
    }
    auto fetch_ih = [&](int slot, bool more) {
        if constexpr (Split) {
            if (more) {
                const char *src = ih_next;
                uint32_t dst = ihs_u32 + (uint32_t)slot * slot_bytes;
                for (int left = nb; left > 0; left -= 8, src += 8 * ih_row, dst += CHUNKS * 16)
#pragma unroll
                    for (int i = 0; i < NC; ++i)
                        if (src_row[i] < left) cp_async16(dst + 512u * i, src + src_off[i]);
                ih_next += ih_step;
            }
            cp_async_commit();
        } else if (tid == 0 && more) {
            const uint32_t bytes = (uint32_t)nb * (uint32_t)ih_row;
            tc::mbar_expect_tx(&ih_full[slot], bytes);
            bulk_copy(ihs_u32 + (uint32_t)slot * slot_bytes, ih_next, bytes, &ih_full[slot]);
            ih_next += ih_step;
        }
    };
    for (int s = 0; s < D; ++s) fetch_ih(s, s < a.T);

    const uint32_t tab = tc::smem_u32(tables);
    const uint32_t h_bits = HU ? 9u : 8u;
    const uint32_t hs_u32 = tc::smem_u32(hs);
    bool ok = true;
    // Requantization constants of this thread's units, in registers where R leaves room for them.
    constexpr int NU = Split ? 1 : 2;                            // units per thread
    constexpr bool RegLin = Cell <= CELL_INT_FAST_NOTIE && KST <= 4;
    FastLin lin_r[RegLin ? 3 : 1][RegLin ? NU : 1];
    const int u0 = ug * 16 + (Split ? (lane & 15) : 2 * g8);     // first of them, within the CTA
    if constexpr (RegLin) {
#pragma unroll
        for (int g = 0; g < 3; ++g)
#pragma unroll
            for (int i = 0; i < NU; ++i) lin_r[g][i] = reinterpret_cast<const FastLin *>(consts)[g * U + u0 + i];
    }
    // N cells side by side: sums, W*x + bw, previous states; ui[i]: which of the thread's units.  Gate by gate over all
    // of them, so that their table lookups overlap.
    // Training: also the four values of v (zero point taken off) and the mask bits of each.
    auto cells = [&](auto n_c, const int (*acc)[2], const int (*ihv)[2], const int32_t *h_old, const int *ui, int32_t *hn, float (*vq)[4], uint32_t *keep) {
        constexpr int N = decltype(n_c)::value;
        if constexpr (Cell <= CELL_INT_FAST_NOTIE) {
            const auto lin = [&](int v, int g, int i) {
                if constexpr (RegLin) return lin_round<Tie>(v, lin_r[g][NU == 1 ? 0 : i]);
                else return lin_round<Tie>(v, reinterpret_cast<const FastLin *>(consts)[g * U + u0 + ui[i]]);
            };
            int32_t z[N], r[N];
#pragma unroll
            for (int i = 0; i < N; ++i) z[i] = fused_gate_fast(gc, tab, ACT_Z, ihv[0][i], lin(acc[0][i], 0, i));
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = fused_gate_fast(gc, tab, ACT_R, ihv[1][i], lin(acc[1][i], 1, i));
#pragma unroll
            for (int i = 0; i < N; ++i) hn[i] = fused_finish_fast<Tie>(gc, tab, ihv[2][i], lin(acc[2][i], 2, i), z[i], r[i], h_old[i]);
        } else if constexpr (Cell == CELL_INT_GENERIC) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const GenLin *f = reinterpret_cast<const GenLin *>(consts) + u0 + ui[i];
                const int32_t hz = linear_epilogue(acc[0][i], f[0].corr, f[0].rs, a.lc.zp_out, a.lc.lo, a.lc.hi);
                const int32_t hr = linear_epilogue(acc[1][i], f[U].corr, f[U].rs, a.lc.zp_out, a.lc.lo, a.lc.hi);
                const int32_t hg = linear_epilogue(acc[2][i], f[2 * U].corr, f[2 * U].rs, a.lc.zp_out, a.lc.lo, a.lc.hi);
                hn[i] = gru_cell<false>(gc, tables, ihv[0][i], ihv[1][i], ihv[2][i], hz, hr, hg, h_old[i]);
            }
        } else if constexpr (Cell == CELL_INT_TRAIN) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const GenLin *f = reinterpret_cast<const GenLin *>(consts) + u0 + ui[i];
                int32_t ih[3], hh[3], gates[3];
                uint32_t m = 0;
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    const int32_t w = (int32_t)rescale64(acc[g][i] + f[g * U].corr, f[g * U].rs) + a.lc.zp_out;
                    hh[g] = clampi(w, a.lc.lo, a.lc.hi);
                    ih[g] = clampi(ihv[g][i], gc.ih_lo, gc.ih_hi);
                    m |= (uint32_t)(hh[g] == w) << (PM_HH + g) | (uint32_t)(ih[g] == ihv[g][i]) << (PM_IH + g);
                }
                hn[i] = gru_cell_train(gc, a.n_table ? tables : nullptr, ih[0], ih[1], ih[2], hh[0], hh[1], hh[2], h_old[i], gates, m);
#pragma unroll
                for (int g = 0; g < 3; ++g) vq[i][g] = (float)(gates[g] - (int32_t)a.tc.zp[g]);
                vq[i][3] = (float)(hh[2] - (int32_t)a.tc.zp[3]);
                keep[i] = m;
            }
        } else if constexpr (Cell == CELL_FS_TRAIN) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const float *f = reinterpret_cast<const float *>(consts) + u0 + ui[i];
                float ih[3], hh[3];
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    ih[g] = (float)ihv[g][i];
                    hh[g] = fs_linear_raw(acc[g][i], f[g * U], f[(3 + g) * U], f[(6 + g) * U], a.fs.zp_hh);
                }
                keep[i] = 0;
                hn[i] = (int32_t)fs_cell_train(a.fs, a.n_table, tab, ih, hh, (float)h_old[i], vq[i], keep[i]);
#pragma unroll
                for (int k = 0; k < 4; ++k) vq[i][k] -= a.tc.zp[k];
            }
        } else {
            const auto lin = [&](int v, int g, int i) {
                const float *f = reinterpret_cast<const float *>(consts) + g * U + u0 + ui[i];
                return fs_linear(v, f[0], f[3 * U], f[6 * U], a.fs.zp_hh, a.fs.hh_lo, a.fs.hh_hi);
            };
            float ug_[N], rg_[N];
#pragma unroll
            for (int i = 0; i < N; ++i) ug_[i] = fs_sigmoid_gate_tab(a.fs, tab, 0, (float)ihv[0][i], lin(acc[0][i], 0, i));
#pragma unroll
            for (int i = 0; i < N; ++i) rg_[i] = fs_sigmoid_gate_tab(a.fs, tab, 1, (float)ihv[1][i], lin(acc[1][i], 1, i));
#pragma unroll
            for (int i = 0; i < N; ++i)
                hn[i] = (int32_t)fs_finish_tab(a.fs, tab, ug_[i], rg_[i], (float)ihv[2][i], lin(acc[2][i], 2, i), (float)h_old[i]);
        }
    };
    // outputs: running pointers of this thread's first unit and row
    const int out_j = j0 + u0;
    const ptrdiff_t out_step = a.reverse ? -(ptrdiff_t)a.out.ts : (ptrdiff_t)a.out.ts;
    float *hf = a.out.hf ? a.out.hf + (size_t)(a.reverse ? a.T - 1 : 1) * a.out.ts + (size_t)b0 * a.out.bs + out_j : nullptr;
    const int obs = (int)a.out.bs;
    // training: units j .. j + N - 1 of row n of the gate buffer, the masks and the states (two units: both exist and H is even)
    const auto keep_cells = [&](auto n_c, size_t n, size_t slot_row, int j, const float (*vq)[4], const uint32_t *keep, const float *f) {
        constexpr int N = decltype(n_c)::value;
        float *v = a.v + n * 4 * H + j;
        if constexpr (N == 2) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                *reinterpret_cast<float2 *>(v + (size_t)k * H) = make_float2(vq[0][k] * a.tc.scale[k], vq[1][k] * a.tc.scale[k]);
            *reinterpret_cast<uint32_t *>(a.pm + n * H + j) = keep[0] | keep[1] << 16;
            if (a.h_all) *reinterpret_cast<float2 *>(a.h_all + slot_row * H + j) = make_float2(f[0], f[1]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) v[(size_t)k * H] = vq[0][k] * a.tc.scale[k];
            a.pm[n * H + j] = (uint16_t)keep[0];
            if (a.h_all) a.h_all[slot_row * H + j] = f[0];
        }
    };
    // clusters: lane l of a half warp sends to CTA l
    const int ul = lane & 15;
    uint32_t peer_hs = 0, peer_bar = 0;
    if (Split && ul < P && ul != p) {
        peer_hs = map_to_rank(hs_u32, (uint32_t)ul);
        peer_bar = map_to_rank(tc::smem_u32(&h_ready[0]), (uint32_t)ul);
    }
    constexpr int RED = KS * 12 * RED_STRIDE;
    int *red_g = red + ug * RED;
    int red_buf = 0, slot = 0;
    uint32_t ih_phase = 0;
    // (a wait that has run out is not repeated: the steps go on with whatever is there, so that every barrier is met)
    for (int s = 0; s < a.T; ++s) {
        const long long out_slot = a.reverse ? (a.T - 1 - s) : (s + 1);
        const int cur = (s & 1) * NT * 8 * HS, nxt = ((s + 1) & 1) * NT * 8 * HS;
        const unsigned char *h_cur = hs + cur;
        unsigned char *h_nxt = hs + nxt;
        const bool last = s + 1 == a.T;
        if (Split && s > 0 && ok) ok = tc::mbar_wait(&h_ready[s & 1], (uint32_t)(((s - 1) >> 1) & 1), WAIT_BUDGET);
        const IhT *ih_t = reinterpret_cast<const IhT *>(ihs_w + (size_t)slot * slot_bytes) + (Split ? ul : u0);
        for (int nt = 0; nt < NT; ++nt, ih_t += Split ? RW * 48 : 24 * U) {
            const int rows = nb - nt * 8;                        // rows of this tile that exist
            if (rows <= 0) break;
            // One CTA, two to four rows: each stands in two of the eight columns, so that a thread has one row of its two units
            // to compute and not half of the threads two.  us a step, H = 256: 296 rows (2 a CTA) 2.12 -> 1.57, float storage 3.45 -> 2.21,
            // 4096 rows (28, the last tile has four) 7.3 -> 7.0.
            const bool few = Few && rows > 1 && rows <= 4;
            int32_t acc[3][4] = {};
            const unsigned char *hb = h_cur + (nt * 8 + (few ? g8 >> 1 : g8)) * HS + ks * KST * 32 + q4 * 16;
#pragma unroll
            for (int c = 0; c < KST / 2; ++c) {
                const uint4 x = *reinterpret_cast<const uint4 *>(hb + c * 64);
#pragma unroll
                for (int g = 0; g < 3; ++g) imma<HU>(acc[g], R[g][2 * c], x.x, x.y);
#pragma unroll
                for (int g = 0; g < 3; ++g) imma<HU>(acc[g], R[g][2 * c + 1], x.z, x.w);
            }
            if (nt == 0) {
                if constexpr (Split) {
                    cp_async_wait_depth(D);
                    __syncwarp();
                } else {
                    ok = ok && tc::mbar_wait(&ih_full[slot], ih_phase, WAIT_BUDGET);
                }
            }
            if constexpr (!Split) {
                // cells (units 2 g8, 2 g8 + 1) x (rows 2 q4, 2 q4 + 1), the two units of a row side by side; absent
                // rows compute with whatever is there (every lookup is clamped) and store nothing
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    if (r >= rows || (few && r)) break;          // (warp-uniform)
                    const int row = few ? q4 : 2 * q4 + r, b = nt * 8 + row;
                    const IhT *iv = ih_t + row * 3 * U;
                    const uint32_t hb2 = *reinterpret_cast<const uint16_t *>(h_cur + b * HS + out_j);
                    const int sums[3][2] = {{acc[0][r], acc[0][2 + r]}, {acc[1][r], acc[1][2 + r]}, {acc[2][r], acc[2][2 + r]}};
                    int ihv[3][2];
#pragma unroll
                    for (int g = 0; g < 3; ++g) load_pair(iv + g * U, ihv[g][0], ihv[g][1]);
                    const int32_t h_old[2] = {state_byte(hb2, h_bits), state_byte(hb2 >> 8, h_bits)};
                    const int ui[2] = {0, 1};
                    int32_t hn[2];
                    float vq[2][4];
                    uint32_t keep[2];
                    cells(std::integral_constant<int, 2>(), sums, ihv, h_old, ui, hn, vq, keep);
                    if (row < rows) {
                        *reinterpret_cast<uint16_t *>(h_nxt + b * HS + out_j) = (uint16_t)(((uint32_t)hn[0] & 0xffu) | ((uint32_t)hn[1] << 8));
                        if (a.vec2) {
                            if (out_j < H) {
                                const float2 f = make_float2((float)(hn[0] - gc.zp_h) * gc.h_scale, (float)(hn[1] - gc.zp_h) * gc.h_scale);
                                *reinterpret_cast<float2 *>(hf + b * obs) = f;
                                if (last && a.out.hn_f) *reinterpret_cast<float2 *>(a.out.hn_f + (size_t)(b0 + b) * H + out_j) = f;
                            }
                        } else {
                            if (out_j < H) put_state(a.out, out_slot, b0 + b, out_j, H, last, hn[0], gc.zp_h, gc.h_scale);
                            if (out_j + 1 < H) put_state(a.out, out_slot, b0 + b, out_j + 1, H, last, hn[1], gc.zp_h, gc.h_scale);
                        }
                        if constexpr (Train) {
                            const size_t n = (size_t)(a.reverse ? a.T - 1 - s : s) * a.B + b0 + b, at = (size_t)out_slot * a.B + b0 + b;
                            const float f[2] = {(float)(hn[0] - gc.zp_h) * gc.h_scale, (float)(hn[1] - gc.zp_h) * gc.h_scale};
                            if ((H & 1) == 0) {
                                if (out_j < H) keep_cells(std::integral_constant<int, 2>(), n, at, out_j, vq, keep, f);
                            } else {
                                if (out_j < H) keep_cells(std::integral_constant<int, 1>(), n, at, out_j, vq, keep, f);
                                if (out_j + 1 < H) keep_cells(std::integral_constant<int, 1>(), n, at, out_j + 1, vq + 1, keep + 1, f + 1);
                            }
                        }
                    }
                }
            } else {
                // partial sums of the KS slices to shared memory (two buffers: whoever writes the one after next has passed
                // the barrier between); warp ks takes rows ks * RW .. of the tile, 16 units to a half warp
                int *rb = red_g + red_buf;
                red_buf = red_buf ? 0 : (U / 16) * RED;
#pragma unroll
                for (int g = 0; g < 3; ++g)
#pragma unroll
                    for (int i = 0; i < 4; ++i) rb[(ks * 12 + g * 4 + i) * RED_STRIDE + lane] = acc[g][i];
                asm volatile("bar.sync %0, %1;" ::"r"(1 + ug), "n"(KS * 32) : "memory");
                if (ks * RW >= rows) continue;                   // (warp-uniform)
                constexpr int NR = RW / 2;                       // rows of a lane: row0 and, with two slices, row0 + 2
                const int j = out_j, row0 = ks * RW + (lane >> 4);
                const bool two = NR == 2 && ks * RW + 2 < rows;
                int32_t hn[2] = {0, 0};
                float vq[2][4];
                uint32_t keep[2];
                {
                    int sums[3][2] = {}, ihv[3][2] = {};
                    int32_t h_old[2] = {};
                    const int ui[2] = {0, 0};
                    const int *src = rb + ((ul & 1) * 2 + (row0 & 1)) * RED_STRIDE + 4 * (ul >> 1) + (row0 >> 1);
                    const IhT *iv = ih_t + (lane >> 4) * 48;
                    const unsigned char *ho = h_cur + (nt * 8 + row0) * HS + j;
#pragma unroll
                    for (int i = 0; i < NR; ++i) {
                        if (i > 0 && !two) break;
#pragma unroll
                        for (int g = 0; g < 3; ++g) {
#pragma unroll
                            for (int k = 0; k < KS; ++k) sums[g][i] += src[(k * 12 + g * 4) * RED_STRIDE + i];
                            ihv[g][i] = iv[16 * g + i * 96];
                        }
                        h_old[i] = state_byte(ho[i * 2 * HS], h_bits);
                    }
                    if (two) cells(std::integral_constant<int, NR>(), sums, ihv, h_old, ui, hn, vq, keep);
                    else cells(std::integral_constant<int, 1>(), sums, ihv, h_old, ui, hn, vq, keep);
                }
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    if (i > 0 && !two) break;
                    const int row = row0 + 2 * i;
                    // the row's 16 bytes in every lane of the half warp, then one 16-byte store per peer: with a
                    // word per store the exchange takes four times the instructions and transactions
                    uint32_t w = (uint32_t)hn[i] & 0xffu;
                    w |= __shfl_xor_sync(0xffffffffu, w, 1) << 8;
                    w |= __shfl_xor_sync(0xffffffffu, w, 2) << 16;
                    uint32_t v[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[k] = __shfl_sync(0xffffffffu, w, (lane & 16) + 4 * k);
                    if (row < rows && !last) {
                        const uint32_t at = (uint32_t)(nxt + (nt * 8 + row) * HS + (j & ~15));
                        if (ul == p) sts_v4(hs_u32 + at, v);
                        else if (ul < P) st_async_v4(peer_hs + at, v, peer_bar + (uint32_t)((s + 1) & 1) * 8u);
                    }
                }
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const int row = row0 + 2 * i;
                    if ((i == 0 || two) && row < rows && j < H) {
                        if (a.vec2) {                            // (fp32 output only)
                            const float f = (float)(hn[i] - gc.zp_h) * gc.h_scale;
                            hf[(nt * 8 + row) * obs] = f;
                            if (last && a.out.hn_f) a.out.hn_f[(size_t)(b0 + nt * 8 + row) * H + j] = f;
                        } else {
                            put_state(a.out, out_slot, b0 + nt * 8 + row, j, H, last, hn[i], gc.zp_h, gc.h_scale);
                        }
                        if constexpr (Train) {
                            const int b = b0 + nt * 8 + row;
                            const float f = (float)(hn[i] - gc.zp_h) * gc.h_scale;
                            keep_cells(std::integral_constant<int, 1>(), (size_t)(a.reverse ? a.T - 1 - s : s) * a.B + b, (size_t)out_slot * a.B + b, j,
                                       vq + i, keep + i, &f);
                        }
                    }
                }
            }
        }
        if constexpr (Split) {
            __syncwarp();
            if (lane == 0 && !last) {
                if (warp == 0) tc::mbar_expect_tx(&h_ready[(s + 1) & 1], (uint32_t)((P - 1) * nb * U));
                else tc::mbar_arrive(&h_ready[(s + 1) & 1]);
            }
        } else {
            __syncthreads();
        }
        fetch_ih(slot, s + D < a.T);
        if (++slot == D) {
            slot = 0;
            ih_phase ^= 1u;
        }
        if (hf) hf += out_step;
    }
    if (!ok && lane == 0) raise_abort(a.abort_flag, 1);
    if (Split && P > 1) {   // nobody leaves while a peer's store may be on its way
        cluster_arrive();
        cluster_wait();
    }
}

// The splits of K that occur: one warp up to 256 inputs, two up to 512, four up to 1024, at most 256 each.
template <typename IhT, int Cell, bool HU>
RegKernel pick_shape(int kst, int ks, bool few) {
    if (ks == 1) {
        switch (kst) {
            case 2: return few ? k_rec_reg<IhT, 2, Cell, HU, 1> : k_rec_reg<IhT, 2, Cell, HU, 1, false>;
            case 4: return few ? k_rec_reg<IhT, 4, Cell, HU, 1> : k_rec_reg<IhT, 4, Cell, HU, 1, false>;
            case 6: return k_rec_reg<IhT, 6, Cell, HU, 1>;
            default: return k_rec_reg<IhT, 8, Cell, HU, 1>;
        }
    }
    if (ks == 2) return kst == 6 ? k_rec_reg<IhT, 6, Cell, HU, 2> : k_rec_reg<IhT, 8, Cell, HU, 2>;
    return kst == 6 ? k_rec_reg<IhT, 6, Cell, HU, 4> : k_rec_reg<IhT, 8, Cell, HU, 4>;
}
template <typename IhT, int Cell>
RegKernel pick(int kst, int ks, bool hu, bool few) {
    return hu ? pick_shape<IhT, Cell, true>(kst, ks, few) : pick_shape<IhT, Cell, false>(kst, ks, few);
}

}  // namespace
}  // namespace qgru
