// qgru_gemm_f32_tc.cu - the fp32 matrix product on the tensor cores: every fp32 operand times 2^24 is the exact sum of three
// bf16 values (8 + 8 + 8 significand bits), and a product of two operands is the sum of the six partial products
// hi*hi, hi*mid, mid*hi, mid*mid, hi*lo, lo*hi; the three left out are together at most 2^-23 of it, and 2^-26 in the mean.
// The factor is for small operands: the low part's last bit, 2^-149 of the operand at the least, stays a normal bf16 number
// (without it the split loses bits below 2^-110, 1e-3 of a value at 2^-124, where gradients that have vanished over many steps
// are).  The sums are multiplied by 2^-48 where they are added up.
//
// One CTA per 128 x (16 .. 256) tile of C and K part.  Eight warps fetch the fp32 operands a K slab of 32 ahead, split them in
// registers and store the three parts into swizzled shared-memory tiles (three stages of 72 KB); one thread issues the
// twelve tcgen05.mma kind::f16 of a slab, the ten small partial products first.  The tensor cores add with truncation, so a
// sum stays there for one slab only: two accumulators in tensor memory alternate, and while one is filled the
// eight warps add the other to fp32 sums in registers, rounded to nearest.  Sums are in a fixed order.
// Error against float64 (2-norm, operands uniform in +-0.5), here / fp32 multiply-adds: K = 32 5.5e-8 / 1.0e-7, K = 786 9.0e-8 / 5.2e-7,
// K = 51200 in six parts 3.1e-7 / 1.7e-6.  With a sum of two slabs in tensor memory it was 3e-7 at every K.
// Infinities, NaN and values that round to infinity in bf16 (from 2^104 up) have no such parts (inf - inf), and sums from 2^80
// up overflow in tensor memory; a CTA whose sums are not all finite multiplies its tile again with fp32 multiply-adds, so
// that the result is the one they give.
//
// us (TFLOP/s of the fp32 product) at N x K x M, fp32 pipe / here: 51200 x 1536 x 256 862 / 307 (131; its result masked 339, four
// columns at a time, one by one 425), 1536 x 51200 x 512 1860 / 513 (157; 488 without the factor of 2^24).  The MMAs alone are 1000
// cycles of a slab of 3200; bound by the eight warps' own instructions (split 1200 cycles, sums 800, stores and loads) between
// which only two warps per scheduler overlap.  What did not help: sixteen warps with half the sums each (112 registers: the
// operands in flight spill and wait); packed fp32 subtractions, sums and factors (the last: 51200 x 256 x 1536 428 us, 393 with
// single ones: spills); one K order for all operands in shared memory (transposing costs 4-byte loads).
#include <algorithm>
#include <type_traits>

#include "qgru_device.cuh"
#include "qgru_gemm_f32.cuh"
#include "qgru_handle.h"
#include "qgru_tc.cuh"

namespace qgru {
namespace {

constexpr int TM = 128;             // rows of C per tile (TMEM lanes)
constexpr int TN = 256;             // widest tile
constexpr int KS = 32;              // K slab: 64-byte rows of bf16
constexpr int ST = 3;               // stages
constexpr int WARPS = 8;            // warps that split and add; of four more one issues the MMAs
constexpr int WORK = 32 * WARPS, THREADS = WORK + 128;
constexpr int NC = TN / 32;         // groups of sixteen columns per thread
// A block of 384 threads starts with 168 registers a thread; the last four warps leave most of theirs to the others.
constexpr int REGS_WORK = 224, REGS_ISSUE = 56;
static_assert(WORK * REGS_WORK + 128 * REGS_ISSUE <= THREADS * 168, "the shares add up to what the block starts with");
constexpr int A_PART = TM * KS * 2, B_PART = TN * KS * 2;
constexpr int STAGE = 3 * (A_PART + B_PART);
constexpr size_t SMEM = (size_t)ST * STAGE + 1024 + 256;
constexpr long long WAIT_BUDGET = 2000000000ll;   // about a second of SM clocks
constexpr int C_LD = TN + 4;        // row of the staged result (floats)
static_assert(TM * C_LD * 4 <= ST * STAGE, "the result is staged where the operands were");

// An operand tile of R rows x 32 K keeps the order in which the matrix lies in memory, so that 16-byte loads go out as 8-byte
// stores.  K contiguous: rows of 64 bytes, 64-byte swizzle (16-byte chunk XOR (row / 2) mod 4), 8-row groups 512 bytes
// apart.  Rows contiguous: 64 rows x 8 K of 1024 bytes, 128 bytes a K, 128-byte swizzle (chunk XOR K mod 8); the four groups of
// K follow one another, then the next 64 rows.
template <bool RowC>
struct Layout {
    static constexpr uint32_t HI = RowC ? (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29) : (uint32_t)(512 >> 4) | (1u << 14) | (4u << 29);
    static constexpr uint32_t LO = RowC ? (uint32_t)(4096 >> 4) << 16 : 1u << 16;
    static constexpr uint32_t K16 = (RowC ? 2048 : 32) >> 4;        // the next sixteen K
    // byte offset of element (row, k), both at the start of a group of four along the contiguous side
    static __device__ __forceinline__ uint32_t at(int row, int k) {
        return RowC ? (uint32_t)((row >> 6) * 4096 + (k >> 3) * 1024 + (k & 7) * 128 + ((((row & 63) >> 3) ^ (k & 7)) << 4) + (row & 4) * 2)
                    : (uint32_t)(row * 64 + (((k >> 3) ^ ((row >> 1) & 3)) << 4) + (k & 4) * 2);
    }
};
// D fp32, A and B bf16; a bit each where rows are contiguous
__device__ __forceinline__ uint32_t idesc_bf16(int M, int N, bool a_rows, bool b_rows) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_rows ? 1u : 0u) << 15) | ((b_rows ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}
template <uint32_t AHi, uint32_t BHi>
__device__ __forceinline__ void mma_bf16(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b64 da, db;\n"
        "mov.b64 da, {%1, %5};\n"
        "mov.b64 db, {%2, %6};\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n"
        "}\n" ::"r"(d),
        "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(AHi), "n"(BHi)
        : "memory");
}

constexpr float SCALE = 0x1p24f, UNSCALE = 0x1p-48f;     // of an operand, of a product

// Four neighbours: their three bf16 parts, 8 bytes each.
__device__ __forceinline__ void split4(const float (&v)[4], uint2 (&part)[3]) {
    uint32_t w[3][2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        float x0 = v[2 * j] * SCALE, x1 = v[2 * j + 1] * SCALE;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[p][j]) : "f"(x1), "f"(x0));
            if (p == 2) break;
            x0 -= __uint_as_float(w[p][j] << 16);
            x1 -= __uint_as_float(w[p][j] & 0xffff0000u);
        }
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) part[p] = make_uint2(w[p][0], w[p][1]);
}

// A thread's share of an operand tile of R rows and 32 K: NQ groups of four values, neighbours along the contiguous side: rows
// (RowC, the operand is [K][rows]; a warp takes 128 rows of one K) or K ([rows][K]; eight threads a row).  The groups lie at
// fixed distances from the first, in memory and in the tile.
template <bool RowC, int R>
struct Share {
    static constexpr int NQ = R * KS / 4 / WORK, ACROSS = RowC ? R / 128 : 1;
    uint32_t at = 0, to = 0;            // element in the slab, byte in the tile
    int row = 0, k = 0;
    static __device__ __forceinline__ int row_of(int j) { return RowC ? j % ACROSS * 128 : j * (WORK / 8); }
    static __device__ __forceinline__ int k_of(int j) { return RowC ? j / ACROSS * WARPS : 0; }
    static __device__ __forceinline__ int to_of(int j) { return RowC ? j % ACROSS * 8192 + j / ACROSS * 1024 : j * (WORK / 8) * 64; }
    static_assert(!RowC || WARPS == 8, "eight K apart, so that the swizzle stays");
    __device__ __forceinline__ void start(int tid, long long ld) {
        row = RowC ? (tid & 31) * 4 : tid >> 3;
        k = RowC ? tid >> 5 : (tid & 7) * 4;
        at = RowC ? (uint32_t)(k * ld) + row : (uint32_t)(row * ld) + k;
        to = Layout<RowC>::at(row, k);
    }
    // Loads have no condition: what lies outside the matrix is read from its edge and dropped in keep(), so that no value
    // waits for its load before it is used, a slab later.  V values at a time (V of them are aligned, and the matrix has a multiple
    // of V along its contiguous side); rows_left and k_left say what is left of the matrix from the slab's corner on.
    template <int V, bool Whole>
    __device__ __forceinline__ void load(float (&v)[NQ][4], const float *slab, long long ld, int rows_left, int k_left) const {
#pragma unroll
        for (int j = 0; j < NQ; ++j) {
            if constexpr (Whole) {
                load_v<4>(v[j], slab + (RowC ? k_of(j) * ld + row_of(j) : row_of(j) * ld) + at);
            } else {
#pragma unroll
                for (int i = 0; i < 4; i += V) {
                    const int r = min(row + row_of(j) + (RowC ? i : 0), rows_left - (RowC ? V : 1)), kk = min(k + k_of(j) + (RowC ? 0 : i), k_left - (RowC ? 1 : V));
                    load_v<V>(v[j] + i, slab + (RowC ? kk * ld + r : r * ld + kk));
                }
            }
        }
    }
    template <int V>
    static __device__ __forceinline__ void load_v(float *v, const float *p) {
        if constexpr (V == 4) {
            const float4 q = *reinterpret_cast<const float4 *>(p);
            v[0] = q.x;
            v[1] = q.y;
            v[2] = q.z;
            v[3] = q.w;
        } else if constexpr (V == 2) {
            const float2 q = *reinterpret_cast<const float2 *>(p);
            v[0] = q.x;
            v[1] = q.y;
        } else {
            v[0] = *p;
        }
    }
    template <int V>
    __device__ __forceinline__ void keep(float (&v)[NQ][4], int rows_left, int k_left) const {
#pragma unroll
        for (int j = 0; j < NQ; ++j)
#pragma unroll
            for (int i = 0; i < 4; i += V)
                if (row + row_of(j) + (RowC ? i : 0) >= rows_left || k + k_of(j) + (RowC ? 0 : i) >= k_left)
#pragma unroll
                    for (int e = 0; e < V; ++e) v[j][i + e] = 0.f;
    }
    __device__ __forceinline__ void store(const float (&v)[NQ][4], unsigned char *tile, int width) const {
#pragma unroll
        for (int j = 0; j < NQ; ++j) {
            if (row_of(j) >= width) continue;
            uint2 q[3];
            split4(v[j], q);
#pragma unroll
            for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2 *>(tile + to + to_of(j) + i * (R * KS * 2)) = q[i];
        }
    }
    // the values themselves, [k][ld]
    __device__ __forceinline__ void store_f32(const float (&v)[NQ][4], float *s, int ld, int width) const {
#pragma unroll
        for (int j = 0; j < NQ; ++j)
            if (row_of(j) < width)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[(k + k_of(j) + (RowC ? 0 : i)) * ld + row + row_of(j) + (RowC ? i : 0)] = v[j][i];
    }
};

struct TcArgs {
    const float *A, *B;
    float *C;                  // or the K parts [z][N][M]
    long long N, K, k_part;
    int M, width;              // width of a tile: a multiple of 16, at most 256
    int accumulate, vec;       // vec: 4, 2 or 1 values of an operand at a time
    const uint8_t *mask;
    int *abort_flag;
};

template <bool ARow, bool BRow>
__global__ void __launch_bounds__(THREADS, 1) k_gemm_f32_tc(const TcArgs g) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *tiles = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(tiles + (size_t)ST * STAGE);
    uint64_t *full = bars, *empty = bars + ST, *acc_full = bars + 2 * ST, *acc_empty = acc_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    int *failed = reinterpret_cast<int *>(tmem_slot + 1), *odd = failed + 1;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long n0 = (long long)blockIdx.x * TM, j0 = (long long)blockIdx.y * g.width;
    const long long k_begin = (long long)blockIdx.z * g.k_part, k_len = min(g.K - k_begin, g.k_part);
    const int slabs = (int)((k_len + KS - 1) / KS);
    const int width = min(g.width, (int)((g.M - j0 + 15) / 16 * 16));
    if (tid == 0) {
        for (int s = 0; s < ST; ++s) {
            tc::mbar_init(&full[s], WARPS);
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&acc_full[b], 1);
            tc::mbar_init(&acc_empty[b], WARPS);
        }
        *failed = *odd = 0;
        tc::fence_barrier_init();
    }
    if (warp == WARPS) tc::tmem_alloc(tmem_slot, 512);
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    if (warp >= WARPS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_ISSUE));
        if (warp == WARPS && lane == 0) {
            const uint32_t idesc = idesc_bf16(TM, width, ARow, BRow);
            const uint32_t base = (tc::smem_u32(tiles) & 0x3FFFFu) >> 4;
            bool ok = true;
            int st = 0;
            uint32_t ph = 0;
            for (int s = 0; s < slabs && ok; ++s) {
                const int buf = s & 1;
                ok = tc::mbar_wait(&acc_empty[buf], (uint32_t)((s >> 1) & 1) ^ 1u, WAIT_BUDGET) && tc::mbar_wait(&full[st], ph, WAIT_BUDGET);
                if (!ok) break;
                tc::tc_fence_after_sync();
                const uint32_t d = tmem + (uint32_t)(buf * TN);
                using LA = Layout<ARow>;
                using LB = Layout<BRow>;
                const uint32_t at = base + (uint32_t)(st * STAGE >> 4), a = at | LA::LO, b = (at + (uint32_t)(3 * A_PART >> 4)) | LB::LO;
                constexpr uint32_t AP = A_PART >> 4, BP = B_PART >> 4;
                // (part of A, part of B): the small products first, 0 = hi, 1 = mid, 2 = lo
                constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                for (int p = 0; p < 6; ++p)
#pragma unroll
                    for (int k = 0; k < 2; ++k) mma_bf16<LA::HI, LB::HI>(d, a + PA[p] * AP + k * LA::K16, b + PB[p] * BP + k * LB::K16, idesc, (uint32_t)(p | k));
                tc::mma_commit(&empty[st]);
                tc::mma_commit(&acc_full[buf]);
                if (++st == ST) {
                    st = 0;
                    ph ^= 1u;
                }
            }
            if (!ok) atomicExch(failed, 1);
        }
        __syncwarp();
        __syncthreads();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_WORK));
        Share<ARow, TM> ca;
        Share<BRow, TN> cb;
        const long long lda = ARow ? g.N : g.K, ldb = BRow ? g.M : g.K;
        ca.start(tid, lda);
        cb.start(tid, ldb);
        const float *A0 = ARow ? g.A + k_begin * lda + n0 : g.A + n0 * lda + k_begin;
        const float *B0 = BRow ? g.B + k_begin * ldb + j0 : g.B + j0 * ldb + k_begin;
        const long long a_step = ARow ? KS * lda : KS, b_step = BRow ? KS * ldb : KS;
        const int a_left = (int)min(g.N - n0, (long long)TM), b_left = (int)min(g.M - j0, (long long)TN);
        const bool whole = g.vec == 4 && a_left == TM && b_left == TN && k_len % KS == 0;
        float va[ca.NQ][4], vb[cb.NQ][4];
        const auto left = [&](int s) { return (int)min((long long)KS, k_len - (long long)s * KS); };
        const auto load = [&](int s, auto v, auto w) {
            ca.template load<v.value, w.value>(va, A0 + s * a_step, lda, a_left, left(s));
            cb.template load<v.value, w.value>(vb, B0 + s * b_step, ldb, b_left, left(s));
        };
        const auto keep = [&](int s, auto v) {
            ca.template keep<v.value>(va, a_left, left(s));
            cb.template keep<v.value>(vb, b_left, left(s));
        };
        const int q = warp & 3, cg = warp >> 2;  // TMEM lanes 32 q .. + 31, columns 16 (cg + 2 i) .. + 15
        float sum[NC][16];
#pragma unroll
        for (int i = 0; i < NC; ++i)
#pragma unroll
            for (int e = 0; e < 16; ++e) sum[i][e] = 0.f;
        bool ok = true;
        // the sums of slab s leave tensor memory
        const auto take = [&](int s) {
            const int buf = s & 1;
            if (!tc::mbar_wait(&acc_full[buf], (uint32_t)((s >> 1) & 1), WAIT_BUDGET)) {
                ok = false;
                return;
            }
            tc::tc_fence_after_sync();
            const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * TN + cg * 16);
#pragma unroll
            for (int i = 0; i < NC; i += 2)
                if ((cg + 2 * i) * 16 < width) {
                    int32_t v[2][16];            // (the second may lie beyond the width: inside tensor memory, and not used)
                    tc::tmem_ld16(at + i * 32, v[0]);
                    tc::tmem_ld16(at + i * 32 + 32, v[1]);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int e = 0; e < 16; ++e) sum[i + h][e] = fmaf(__int_as_float(v[h][e]), UNSCALE, sum[i + h][e]);
                }
            tc::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
        };
        const auto multiply = [&](auto v, auto w) {
            load(0, v, w);
            int st = 0;
            uint32_t ph = 1;
            for (int s = 0; s < slabs; ++s) {
                if (!(ok = ok && tc::mbar_wait(&empty[st], ph, WAIT_BUDGET))) break;
                if constexpr (!w.value) keep(s, v);
                unsigned char *a = tiles + (size_t)st * STAGE, *b = a + 3 * A_PART;
                ca.store(va, a, TM);
                cb.store(vb, b, width);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&full[st]);
                if (++st == ST) {
                    st = 0;
                    ph ^= 1u;
                }
                load(min(s + 1, slabs - 1), v, w);
                if (s > 0) take(s - 1);
            }
        };
        using std::integral_constant;
        if (whole) multiply(integral_constant<int, 4>{}, std::true_type{});
        else if (g.vec == 4) multiply(integral_constant<int, 4>{}, std::false_type{});
        else if (g.vec == 2) multiply(integral_constant<int, 2>{}, std::false_type{});
        else multiply(integral_constant<int, 1>{}, std::false_type{});
        if (ok) take(slabs - 1);
        if (!ok && lane == 0) atomicExch(failed, 1);
        // (a value without parts has NaN among them, and all that it is a factor of becomes NaN)
        float big = 0.f;
#pragma unroll
        for (int i = 0; i < NC; ++i)
            if ((cg + 2 * i) * 16 < width)
#pragma unroll
                for (int e = 0; e < 16; ++e) big = fmaf(sum[i][e], 0.f, big);
        if (big != 0.f) *odd = 1;
        __syncthreads();
        const auto bar = []() { asm volatile("bar.sync 1, %0;" ::"n"(WORK) : "memory"); };
        float *cs = reinterpret_cast<float *>(tiles);
        const int r = q * 32 + lane;
        if (*odd) {
            // fp32 multiply-adds instead
            float *as = cs, *bs = as + KS * (TM + 4);
#pragma unroll
            for (int i = 0; i < NC; ++i)
#pragma unroll
                for (int e = 0; e < 16; ++e) sum[i][e] = 0.f;
            for (int s = 0; s < slabs; ++s) {
                load(s, integral_constant<int, 1>{}, std::false_type{});
                keep(s, integral_constant<int, 1>{});
                bar();
                ca.store_f32(va, as, TM + 4, TM);
                cb.store_f32(vb, bs, TN, TN);
                bar();
                for (int k = 0; k < left(s); ++k) {
                    const float x = as[k * (TM + 4) + r];
#pragma unroll
                    for (int i = 0; i < NC; ++i)
                        if ((cg + 2 * i) * 16 < width)
#pragma unroll
                            for (int e = 0; e < 16; ++e) sum[i][e] = fmaf(x, bs[k * TN + (cg + 2 * i) * 16 + e], sum[i][e]);
                }
            }
            bar();
        }
#pragma unroll
        for (int i = 0; i < NC; ++i)
            if ((cg + 2 * i) * 16 < width)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    *reinterpret_cast<float4 *>(cs + r * C_LD + (cg + 2 * i) * 16 + 4 * e) =
                        make_float4(sum[i][4 * e], sum[i][4 * e + 1], sum[i][4 * e + 2], sum[i][4 * e + 3]);
        bar();
        const int rows = (int)min((long long)TM, g.N - n0), cols = (int)min((long long)width, g.M - j0);
        const bool split = gridDim.z > 1;
        float *out = g.C + (split ? (size_t)blockIdx.z * g.N * g.M : 0) + n0 * g.M + j0;
        const uint8_t *mask = split || !g.mask ? nullptr : g.mask + n0 * g.M + j0;
        const int acc = split ? 0 : g.accumulate;
        if (g.M % 4 == 0 && ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(mask) * 4) & 15u) == 0) {
            const int c4 = cols >> 2;            // (M and the tile's width are multiples of four)
#pragma unroll 4
            for (int i = tid; i < rows * c4; i += WORK) {
                const int rr = i / c4, c = (i - rr * c4) * 4;
                const long long at = (long long)rr * g.M + c;
                float4 y = *reinterpret_cast<const float4 *>(cs + rr * C_LD + c);
                const float4 old = acc ? *reinterpret_cast<const float4 *>(out + at) : make_float4(0.f, 0.f, 0.f, 0.f);
                if (acc == 1) y = make_float4(y.x + old.x, y.y + old.y, y.z + old.z, y.w + old.w);
                if (mask) {
                    const uchar4 m = *reinterpret_cast<const uchar4 *>(mask + at);
                    y = make_float4(y.x * (float)m.x, y.y * (float)m.y, y.z * (float)m.z, y.w * (float)m.w);
                }
                if (acc == 2) y = make_float4(y.x + old.x, y.y + old.y, y.z + old.z, y.w + old.w);
                *reinterpret_cast<float4 *>(out + at) = y;
            }
        } else {
            for (int rr = warp; rr < rows; rr += WARPS)
                for (int c = lane; c < cols; c += 32) {
                    const long long at = (long long)rr * g.M + c;
                    float y = cs[rr * C_LD + c];
                    if (acc == 1) y += out[at];
                    if (mask) y *= (float)mask[at];
                    if (acc == 2) y += out[at];
                    out[at] = y;
                }
        }
    }
    if (tid == 0 && *failed) raise_abort(g.abort_flag, 2);
    tc::tc_fence_before_sync();
    __syncthreads();
    if (warp == WARPS) tc::tmem_dealloc(tmem, 512);
}

}  // namespace

bool gemm_f32_tc_fits(const GemmF32 &g) {
    // an operand's offset inside a tile: at most 256 rows of K, or 32 of N or M
    return g.K < (1 << 23) && g.N < (1ll << 26) && g.M < (1 << 23);
}

int gemm_f32_tc_tiles(const GemmF32 &g, int *width) {
    const int across = (g.M + TN - 1) / TN;
    *width = ((g.M + across - 1) / across + 15) / 16 * 16;
    return (int)((g.N + TM - 1) / TM) * ((g.M + *width - 1) / *width);
}

int gemm_f32_tc_launch(qgru_handle *h, const GemmF32 &g, int parts, long long k_part, float *out, cudaStream_t st) {
    // values that lie together and start where a vector load may: of both operands, along their contiguous sides
    const auto fits = [&](int v) {
        const long long a = g.a_trans ? g.N : g.K, b = g.b_trans ? g.K : g.M;
        return a % v == 0 && b % v == 0 && reinterpret_cast<uintptr_t>(g.A) % (4 * v) == 0 && reinterpret_cast<uintptr_t>(g.B) % (4 * v) == 0;
    };
    TcArgs a{g.A, g.B, out, g.N, g.K, k_part, g.M, 0, g.accumulate, fits(4) ? 4 : fits(2) ? 2 : 1, g.mask, h->d_flags + 1};
    gemm_f32_tc_tiles(g, &a.width);
    auto kern = g.a_trans ? (g.b_trans ? k_gemm_f32_tc<true, false> : k_gemm_f32_tc<true, true>)
                          : (g.b_trans ? k_gemm_f32_tc<false, false> : k_gemm_f32_tc<false, true>);
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM));
    const dim3 grid((unsigned)((g.N + TM - 1) / TM), (unsigned)((g.M + a.width - 1) / a.width), (unsigned)parts);
    kern<<<grid, THREADS, SMEM, st>>>(a);
    return QGRU_OK;
}

}  // namespace qgru
