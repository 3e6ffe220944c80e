// qgru_rec_reg.cu - the recurrence with R in registers and warp-level int8 tensor instructions.
//
// A step of the recurrence is latency: a product with few batch rows, the cell, an exchange.  Here a CTA's slice
// of R (up to 196 KB) is held in registers in the order mma.sync takes its A operand (m16n8k32, eight batch
// rows per instruction), so a step reads only the state from shared memory and its sums appear in the
// registers of the threads that go on with them: no descriptors, no commit, no tensor-memory load
// between the product and the cell.  Measured on a B200: mma.sync.m16n8k32.s8 issues every 8 cycles per
// scheduler with 21 cycles latency, so the slice of 128 units of H = 512 takes 768 cycles for up to eight
// rows; the same rows on tcgen05 (whose throughput these small tiles cannot use: 16 columns at least,
// 128 x 16 x 32 per instruction, 53 cycles per issuing thread) are complete 1970 cycles after the state.
// For one row it equals dp4a (64 lanes per clock and SM).
//
// Split: clusters of P CTAs own Bt batch rows; a CTA owns U units as groups of 16 (three tiles of 16 rows of R, one
// per gate, so that one thread ends up with all three gates of a cell); K is split over KS warps per group
// where one warp's 96 registers do not hold it (H > 256), and their partial sums meet in shared memory,
// redistributed so that every warp gets an equal share of the cells.  H <= 256 is one CTA per row group:
// nothing leaves the SM and a step ends with one block barrier.  Larger layers send the new state to the
// peers with st.async, counted on their mbarrier: no fence on the sending side.  A peer can be at most
// one step ahead, so two state buffers are enough.
// W*x + bw arrives by bulk copies, D steps ahead.
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
    s.total = s.red + (KS > 1 ? up((size_t)(U / 16) * KS * 12 * RED_STRIDE * 4) : 0);
    return s;
}

template <typename IhT, int KST, int Cell, bool HU, bool Split>
__global__ void __launch_bounds__(512, 1) k_rec_reg(const __grid_constant__ GateConsts gc, const __grid_constant__ RecRegArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr bool Tie = Cell != CELL_INT_FAST_NOTIE, Train = Cell >= CELL_INT_TRAIN;
    const int U = a.U, KS = Split ? a.KS : 1, P = Split ? a.P : 1, NT = a.NT, D = a.D, H = a.H;
    const int K = KS * KST * 32, HS = state_stride(K);
    const RegSmem L = reg_smem(K, U, KS, NT, D, (int)sizeof(IhT), Cell, a.n_table);
    uint64_t *h_ready = reinterpret_cast<uint64_t *>(smem);      // [2], clusters only
    uint64_t *ih_full = h_ready + 2;                             // [D]
    int32_t *tables = reinterpret_cast<int32_t *>(smem + L.tables);
    unsigned char *consts = smem + L.consts;
    unsigned char *hs = smem + L.hs;                             // [2][NT * 8][HS]
    IhT *ihs = reinterpret_cast<IhT *>(smem + L.ihs);            // [D][rows][3][U]
    int *red = reinterpret_cast<int *>(smem + L.red);            // [unit group][KS][12][RED_STRIDE]

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
    // W*x + bw of this CTA's units and rows: one contiguous block per step
    const IhT *ih_next = reinterpret_cast<const IhT *>(a.ih) + ((size_t)p * a.T * a.B + (size_t)(a.reverse ? a.T - 1 : 0) * a.B + b0) * 3 * U;
    const ptrdiff_t ih_step = (a.reverse ? -(ptrdiff_t)a.B : (ptrdiff_t)a.B) * 3 * U;
    const uint32_t ihs_u32 = tc::smem_u32(ihs), ih_bytes = (uint32_t)(nb * 3 * U) * (uint32_t)sizeof(IhT);
    const uint32_t ih_slot_bytes = (uint32_t)(NT * 8 * 3 * U) * (uint32_t)sizeof(IhT);
    auto fetch_ih = [&](int slot) {
        tc::mbar_expect_tx(&ih_full[slot], ih_bytes);
        bulk_copy(ihs_u32 + (uint32_t)slot * ih_slot_bytes, ih_next, ih_bytes, &ih_full[slot]);
        ih_next += ih_step;
    };
    if (tid == 0)
        for (int s = 0; s < min(D, a.T); ++s) fetch_ih(s);

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
    int slot = 0;
    uint32_t ih_phase = 0;
    // (a wait that has run out is not repeated: the steps go on with whatever is there, so that every barrier is met)
    for (int s = 0; s < a.T; ++s) {
        const long long out_slot = a.reverse ? (a.T - 1 - s) : (s + 1);
        const unsigned char *h_cur = hs + (s & 1) * NT * 8 * HS;
        unsigned char *h_nxt = hs + ((s + 1) & 1) * NT * 8 * HS;
        const bool last = s + 1 == a.T;
        if (P > 1 && s > 0 && ok) ok = tc::mbar_wait(&h_ready[s & 1], (uint32_t)(((s - 1) >> 1) & 1), WAIT_BUDGET);
        const IhT *ih_s = ihs + (size_t)slot * NT * 8 * 3 * U + u0;
        bool have_ih = false;
        for (int nt = 0; nt < NT; ++nt) {
            const int rows = nb - nt * 8;                        // rows of this tile that exist
            if (rows <= 0) break;
            int32_t acc[3][4] = {};
            const unsigned char *hb = h_cur + (nt * 8 + g8) * HS + ks * KST * 32 + q4 * 16;
#pragma unroll
            for (int c = 0; c < KST / 2; ++c) {
                const uint4 x = *reinterpret_cast<const uint4 *>(hb + c * 64);
#pragma unroll
                for (int g = 0; g < 3; ++g) imma<HU>(acc[g], R[g][2 * c], x.x, x.y);
#pragma unroll
                for (int g = 0; g < 3; ++g) imma<HU>(acc[g], R[g][2 * c + 1], x.z, x.w);
            }
            if (!have_ih) {
                ok = ok && tc::mbar_wait(&ih_full[slot], ih_phase, WAIT_BUDGET);
                have_ih = true;
            }
            if constexpr (!Split) {
                // cells (units 2 g8, 2 g8 + 1) x (rows 2 q4, 2 q4 + 1), the two units of a row side by side; absent
                // rows compute with whatever is there (every lookup is clamped) and store nothing
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    if (r >= rows) continue;                     // (warp-uniform: a tile of one row)
                    const int row = 2 * q4 + r, b = nt * 8 + row;
                    const IhT *iv = ih_s + b * 3 * U;
                    const uint32_t hb2 = *reinterpret_cast<const uint16_t *>(h_cur + b * HS + out_j);
                    const int sums[3][2] = {{acc[0][r], acc[0][2 + r]}, {acc[1][r], acc[1][2 + r]}, {acc[2][r], acc[2][2 + r]}};
                    const int ihv[3][2] = {{iv[0], iv[1]}, {iv[U], iv[U + 1]}, {iv[2 * U], iv[2 * U + 1]}};
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
                // partial sums of the KS slices to shared memory; warp ks takes rows ks * (8 / KS) .. of the tile,
                // 16 units to a half warp
                int *rb = red + (size_t)ug * KS * 12 * RED_STRIDE;
#pragma unroll
                for (int g = 0; g < 3; ++g)
#pragma unroll
                    for (int i = 0; i < 4; ++i) rb[(ks * 12 + g * 4 + i) * RED_STRIDE + lane] = acc[g][i];
                asm volatile("bar.sync %0, %1;" ::"r"(1 + ug), "r"(KS * 32) : "memory");
                const int ul = lane & 15, j = out_j, per = 8 / KS;
                int32_t hn[2] = {0, 0};
                float vq[2][4];
                uint32_t keep[2];
                const int row0 = ks * per + (lane >> 4);         // this lane's rows: row0 and, with two slices, row0 + 2
                if (ks * per < rows) {                           // (warp-uniform)
                    int sums[3][2] = {}, ihv[3][2];
                    int32_t h_old[2];
                    const int ui[2] = {0, 0};
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int row = (row0 + 2 * i) & 7, b = nt * 8 + row;
                        const int *src = rb + ((ul & 1) * 2 + (row & 1)) * RED_STRIDE + 4 * (ul >> 1) + (row >> 1);
                        if (2 * i < per)
                            for (int k = 0; k < KS; ++k)
#pragma unroll
                                for (int g = 0; g < 3; ++g) sums[g][i] += src[(k * 12 + g * 4) * RED_STRIDE];
                        const IhT *iv = ih_s + b * 3 * U;
                        ihv[0][i] = iv[0];
                        ihv[1][i] = iv[U];
                        ihv[2][i] = iv[2 * U];
                        h_old[i] = state_byte(h_cur[b * HS + j], h_bits);
                    }
                    if (per == 2 || ks * per + 2 >= rows) cells(std::integral_constant<int, 1>(), sums, ihv, h_old, ui, hn, vq, keep);
                    else cells(std::integral_constant<int, 2>(), sums, ihv, h_old, ui, hn, vq, keep);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        if (2 * i >= per || ks * per + 2 * i >= rows) continue;
                        const int row = row0 + 2 * i, b = nt * 8 + row;
                        // four neighbouring units to a word in all four lanes
                        uint32_t w = (uint32_t)hn[i] & 0xffu;
                        w |= __shfl_xor_sync(0xffffffffu, w, 1) << 8;
                        const uint32_t o = __shfl_xor_sync(0xffffffffu, w, 2);
                        const uint32_t word = __shfl_sync(0xffffffffu, w | (o << 16), lane & ~3);
                        if (row < rows && !last) {
                            const uint32_t at = hs_u32 + (uint32_t)(h_nxt - hs) + (uint32_t)(b * HS + (j & ~3));
                            if ((lane & 3) == 0) sts_u32(at, word);
                            const uint32_t bar = tc::smem_u32(&h_ready[(s + 1) & 1]);
                            for (int r = lane & 3; r < P; r += 4)
                                if (r != p) st_async_u32(map_to_rank(at, (uint32_t)r), word, map_to_rank(bar, (uint32_t)r));
                        }
                    }
                }
                // the block is written again for the next tile or step
                asm volatile("bar.sync %0, %1;" ::"r"(1 + ug), "r"(KS * 32) : "memory");
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int row = row0 + 2 * i;
                    if (2 * i < per && row < rows && j < H) {
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
        if (P > 1) {
            __syncwarp();
            if (lane == 0 && !last) {
                if (warp == 0) tc::mbar_expect_tx(&h_ready[(s + 1) & 1], (uint32_t)((P - 1) * nb * U));
                else tc::mbar_arrive(&h_ready[(s + 1) & 1]);
            }
        } else {
            __syncthreads();
        }
        // (behind the barrier of a CTA of its own, or once this step's state barrier has been passed by all its
        // warps: the slot of the step before is free)
        if (tid == 0 && s + (P > 1 ? D - 1 : D) < a.T && (P == 1 || s > 0)) fetch_ih(P > 1 ? (slot == 0 ? D - 1 : slot - 1) : slot);
        if (++slot == D) {
            slot = 0;
            ih_phase ^= 1u;
        }
        if (hf) hf += out_step;
    }
    if (!ok && lane == 0) atomicOr(a.abort_flag, 1);
    if (P > 1) {   // nobody leaves while a peer's store may be on its way
        cluster_arrive();
        cluster_wait();
    }
}

typedef void (*RegKernel)(const GateConsts, const RecRegArgs);

template <typename IhT, int KST, int Cell>
RegKernel pick_split(bool hu, bool split) {
    if (split) return hu ? k_rec_reg<IhT, KST, Cell, true, true> : k_rec_reg<IhT, KST, Cell, false, true>;
    return hu ? k_rec_reg<IhT, KST, Cell, true, false> : k_rec_reg<IhT, KST, Cell, false, false>;
}
template <typename IhT, int Cell>
RegKernel pick_kst(int kst, bool hu, bool split) {
    switch (kst) {
        case 2: return pick_split<IhT, 2, Cell>(hu, split);
        case 4: return pick_split<IhT, 4, Cell>(hu, split);
        case 6: return pick_split<IhT, 6, Cell>(hu, split);
        default: return pick_split<IhT, 8, Cell>(hu, split);
    }
}
RegKernel pick(RecCell cell, int ih_bytes, int kst, bool hu, bool split) {
    switch (cell) {
        case CELL_INT_FAST: return ih_bytes == 2 ? pick_kst<int16_t, CELL_INT_FAST>(kst, hu, split) : pick_kst<int32_t, CELL_INT_FAST>(kst, hu, split);
        case CELL_INT_FAST_NOTIE:
            return ih_bytes == 2 ? pick_kst<int16_t, CELL_INT_FAST_NOTIE>(kst, hu, split) : pick_kst<int32_t, CELL_INT_FAST_NOTIE>(kst, hu, split);
        case CELL_INT_GENERIC:
            return ih_bytes == 1 ? pick_kst<int8_t, CELL_INT_GENERIC>(kst, hu, split) : pick_kst<int16_t, CELL_INT_GENERIC>(kst, hu, split);
        case CELL_INT_TRAIN: return ih_bytes == 2 ? pick_kst<int16_t, CELL_INT_TRAIN>(kst, hu, split) : pick_kst<int32_t, CELL_INT_TRAIN>(kst, hu, split);
        case CELL_FS_TRAIN: return ih_bytes == 2 ? pick_kst<int16_t, CELL_FS_TRAIN>(kst, hu, split) : pick_kst<int32_t, CELL_FS_TRAIN>(kst, hu, split);
        default: return ih_bytes == 1 ? pick_kst<int8_t, CELL_FS>(kst, hu, split) : pick_kst<int16_t, CELL_FS>(kst, hu, split);
    }
}

}  // namespace

bool rec_reg_plan(qgru_handle *h, int B, int sms, int ih_bytes, RecCell cell, int n_table, RecRegPlan *pl) {
    const int H = h->H;
    if (pl->H == H && pl->B == B && pl->sms == sms && pl->ih_bytes == ih_bytes && pl->cell == (int)cell && pl->n_table == n_table) return pl->ok;
    *pl = RecRegPlan{};
    pl->H = H;
    pl->B = B;
    pl->sms = sms;
    pl->ih_bytes = ih_bytes;
    pl->cell = (int)cell;
    pl->n_table = n_table;
    const int chunks = (H + 63) / 64;                    // of 64 inputs; at most four to a warp (96 registers)
    if (chunks > 16) return false;
    const int KS = chunks <= 4 ? 1 : chunks <= 8 ? 2 : 4;
    const int KST = 2 * ((chunks + KS - 1) / KS);
    const int groups = (H + 15) / 16, most = 16 / KS;
    const int P = (groups + most - 1) / most;
    if (P > 16) return false;
    const int U = 16 * ((groups + P - 1) / P), threads = U / 16 * KS * 32;
    const RegKernel kern = pick(cell, ih_bytes, KST, h->h_uns, KS > 1);
    const int K = KS * KST * 32;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)P);
    cfg.blockDim = dim3((unsigned)threads);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)P;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (P > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    // Rows per cluster: as few as the clusters that fit the chip at once allow.
    int D = 3, Bt = 0;
    for (int pass = 0; pass < 3; ++pass) {
        const int NT = (std::max(Bt, 1) + 7) / 8;
        for (D = 3; D > 1 && reg_smem(K, U, KS, NT, D, ih_bytes, cell, n_table).total > (size_t)h->smem_optin; --D) {}
        const size_t smem = reg_smem(K, U, KS, NT, D, ih_bytes, cell, n_table).total;
        if (smem > (size_t)h->smem_optin) {
            if (Bt <= 8) return false;
            Bt = (NT - 1) * 8;                           // more waves of clusters instead
            --pass;
            continue;
        }
        cfg.dynamicSmemBytes = smem;
        int active = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&active, kern, &cfg) != cudaSuccess || active < 1) {
            cudaGetLastError();
            return false;
        }
        active = std::max(1, std::min(active, (int)((long long)active * sms / h->sm_count)));
        pl->smem = smem;
        pl->D = D;
        const int want = (B + active - 1) / active;
        if (Bt >= want || (pass > 0 && Bt > 0)) break;
        Bt = want;
    }
    pl->KST = KST;
    pl->KS = KS;
    pl->U = U;
    pl->P = P;
    pl->Bt = Bt;
    pl->G = (B + Bt - 1) / Bt;
    pl->ok = true;
    return true;
}

int rec_reg_launch(qgru_handle *h, const RecRegPlan &pl, RecRegArgs a, RecCell cell, int ih_bytes, cudaStream_t st) {
    const RegKernel kern = pick(cell, ih_bytes, pl.KST, h->h_uns, pl.KS > 1);
    a.KS = pl.KS;
    a.U = pl.U;
    a.P = pl.P;
    a.Bt = pl.Bt;
    a.NT = (pl.Bt + 7) / 8;
    a.D = pl.D;
    // fp32 output only, through running pointers with 32-bit row offsets; where one CTA owns all units, in pairs of
    // neighbouring units (8-byte stores: every row's first unit has to be aligned)
    const bool plain = a.out.hf && !a.out.hq && !a.out.h8 && a.out.bs <= (1u << 24);
    a.vec2 = pl.KS > 1 ? plain : plain && a.H % 2 == 0 && a.out.ts % 2 == 0 && a.out.bs % 2 == 0 &&
             (reinterpret_cast<uintptr_t>(a.out.hf) & 7u) == 0 && (reinterpret_cast<uintptr_t>(a.out.hn_f) & 7u) == 0;
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
    if (pl.P > 8) CK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(pl.G * pl.P));
    cfg.blockDim = dim3((unsigned)(pl.U / 16 * pl.KS * 32));
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)pl.P;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CK(cudaLaunchKernelEx(&cfg, kern, (const GateConsts)h->gc_host, (const RecRegArgs)a));
    h->launches++;
    return QGRU_OK;
}

}  // namespace qgru
