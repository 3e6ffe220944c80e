// qgru_gemm_f32.cu - the fp32 matrix product: the input projection of float mode and calibration, and the three
// products of the backward pass.  Large ones run on the tensor cores (qgru_gemm_f32_tc.cu), the others here on the CUDA cores.
//
// 128 x 128 tiles of C with 8 x 8 outputs per thread, or 64 x 64 with 4 x 4, as packed pairs (fma.rn.f32x2: two IEEE
// fused multiply-adds per instruction, so that operand loads and the copies that duplicate A's value
// into both halves share the issue slots the multiply-adds leave), K in slabs of 16 through two
// shared-memory buffers, the next slab in registers while this one is multiplied.  K is split over
// gridDim.z where the tiles alone leave SMs idle (the weight gradients: a few dozen tiles, K = T * B);
// the partial tiles go to a workspace and are added in slab order, so results repeat bit for bit.
// Bound by the fp32 pipe: 45 TFLOP/s at 51200 x 1536 x 256 (dx; 24 with the unpacked 4 x 4 tiles before) and
// 46 at 512 x 51200 x 1536 (dR; 13 before, one block per tile walking all of K).
#include "qgru_gemm_f32.cuh"

#include "qgru_handle.h"

namespace qgru {
namespace {

constexpr int BK = 16;
constexpr int PART_MIN = 32;   // shortest K part

// One operand's BK x BT slab: thread-held values on their way from global to shared memory.
// Trans = false: element (row, k) at src[row * K + k]; true: at src[k * rows + row].  Stored as
// s[k][row].  Vec: every 4-element group is 16-byte aligned and whole.
template <int BT, int THREADS, bool Trans, bool Vec>
struct SlabLoader {
    static constexpr int PER = BK * BT / THREADS;   // values per thread (8 or 16)
    static_assert(PER % 4 == 0, "whole groups of four");
    float v[PER];

    __device__ __forceinline__ void load(const float *__restrict__ src, long long rows, long long K, long long r0,
                                         long long k0, long long k_end) {
#pragma unroll
        for (int i = 0; i < PER / 4; ++i) {
            const int e = (threadIdx.x + i * THREADS) * 4;
            long long r, k;
            if (Trans) {
                k = k0 + e / BT;
                r = r0 + e % BT;
            } else {
                r = r0 + e / BK;
                k = k0 + e % BK;
            }
            if (Vec) {
                const bool in = Trans ? (k < k_end && r < rows) : (r < rows && k < k_end);
                const float4 q = in ? *reinterpret_cast<const float4 *>(src + (Trans ? k * rows + r : r * K + k))
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
                v[4 * i] = q.x;
                v[4 * i + 1] = q.y;
                v[4 * i + 2] = q.z;
                v[4 * i + 3] = q.w;
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const long long rr = Trans ? r + u : r, kk = Trans ? k : k + u;
                    v[4 * i + u] = (rr < rows && kk < k_end) ? src[Trans ? kk * rows + rr : rr * K + kk] : 0.f;
                }
            }
        }
    }
    __device__ __forceinline__ void store(float (*s)[BT + 4]) const {
#pragma unroll
        for (int i = 0; i < PER / 4; ++i) {
            const int e = (threadIdx.x + i * THREADS) * 4;
            if (Trans) {
                *reinterpret_cast<float4 *>(&s[e / BT][e % BT]) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) s[e % BK + u][e / BK] = v[4 * i + u];
            }
        }
    }
};

// gridDim.z = number of K parts; part z > 1 parts write their tile to part_out[z][N * M].  A thread has TM x TM outputs,
// four neighbours each way, and with TM = 8 the four half a tile further.
template <int BT, int TM, bool ATrans, bool BTrans, bool VecA, bool VecB>
__global__ void __launch_bounds__((BT / TM) * (BT / TM), TM == 4 ? 4 : 2)
k_gemm_f32(const float *__restrict__ A, const float *__restrict__ Bm, float *__restrict__ C, long long N, long long K,
           int M, long long k_part, int accumulate, const uint8_t *__restrict__ mask, float *__restrict__ part_out) {
    static_assert(TM == 4 || TM == 8, "one or two groups of four outputs each way");
    constexpr int THREADS = (BT / TM) * (BT / TM);
    constexpr int TX = BT / TM;
    __shared__ __align__(16) float as[2][BK][BT + 4];
    __shared__ __align__(16) float bs[2][BK][BT + 4];
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const long long n0 = (long long)blockIdx.x * BT;
    const long long j0 = (long long)blockIdx.y * BT;
    const long long k_begin = (long long)blockIdx.z * k_part, k_end = min(K, k_begin + k_part);
    SlabLoader<BT, THREADS, ATrans, VecA> la;
    SlabLoader<BT, THREADS, !BTrans, VecB> lb;
    uint64_t acc[TM][TM / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TM / 2; ++j) acc[i][j] = 0ull;
    la.load(A, N, K, n0, k_begin, k_end);
    lb.load(Bm, M, K, j0, k_begin, k_end);
    la.store(as[0]);
    lb.store(bs[0]);
    __syncthreads();
    int buf = 0;
    for (long long k0 = k_begin; k0 < k_end; k0 += BK) {
        const bool more = k0 + BK < k_end;
        if (more) {
            la.load(A, N, K, n0, k0 + BK, k_end);
            lb.load(Bm, M, K, j0, k0 + BK, k_end);
        }
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            // rows ty * 4 .. + 3 (and BT / 2 + ty * 4 .. + 3), columns the same with tx: conflict-free 128-bit loads
            const float4 a0 = *reinterpret_cast<const float4 *>(&as[buf][kk][ty * 4]);
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2 *>(&bs[buf][kk][tx * 4]);
            if constexpr (TM == 8) {
                const float4 a1 = *reinterpret_cast<const float4 *>(&as[buf][kk][BT / 2 + ty * 4]);
                const ulonglong2 b1 = *reinterpret_cast<const ulonglong2 *>(&bs[buf][kk][BT / 2 + tx * 4]);
                const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint64_t aa = pack2(av[i], av[i]);
                    acc[i][0] = ffma2(aa, b0.x, acc[i][0]);
                    acc[i][1] = ffma2(aa, b0.y, acc[i][1]);
                    acc[i][2] = ffma2(aa, b1.x, acc[i][2]);
                    acc[i][3] = ffma2(aa, b1.y, acc[i][3]);
                }
            } else {
                const float av[4] = {a0.x, a0.y, a0.z, a0.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint64_t aa = pack2(av[i], av[i]);
                    acc[i][0] = ffma2(aa, b0.x, acc[i][0]);
                    acc[i][1] = ffma2(aa, b0.y, acc[i][1]);
                }
            }
        }
        if (more) {
            la.store(as[buf ^ 1]);
            lb.store(bs[buf ^ 1]);
            __syncthreads();
            buf ^= 1;
        }
    }
    const bool split = gridDim.z > 1;
    float *out = split ? part_out + (size_t)blockIdx.z * N * M : C;
    if ((split || (!accumulate && !mask)) && M % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const long long n = n0 + (i < 4 ? ty * 4 + i : BT / 2 + ty * 4 + i - 4);
            if (n >= N) continue;
#pragma unroll
            for (int g = 0; g < TM / 4; ++g) {
                const long long c = j0 + g * (BT / 2) + tx * 4;
                if (c < M) *reinterpret_cast<ulonglong2 *>(out + n * M + c) = make_ulonglong2(acc[i][2 * g], acc[i][2 * g + 1]);
            }
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const long long n = n0 + (i < 4 ? ty * 4 + i : BT / 2 + ty * 4 + i - 4);
        if (n >= N) continue;
#pragma unroll
        for (int j = 0; j < TM / 2; ++j) {
            float v[2];
            unpack2(acc[i][j], v[0], v[1]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const long long c = j0 + (j < 2 ? tx * 4 + 2 * j : BT / 2 + tx * 4 + 2 * (j - 2)) + e;
                if (c >= M) continue;
                float y = v[e];
                if (!split) {
                    if (accumulate == 1) y += out[n * M + c];
                    if (mask) y *= (float)mask[n * M + c];
                    if (accumulate == 2) y += out[n * M + c];
                }
                out[n * M + c] = y;
            }
        }
    }
}

// the K parts of a split product, added in order
__global__ void k_gemm_f32_join(const float *__restrict__ part, float *__restrict__ C, long long n, int parts, int accumulate,
                                const uint8_t *__restrict__ mask) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float y = accumulate == 1 ? C[i] : 0.f;
        for (int p = 0; p < parts; ++p) y += part[(size_t)p * n + i];
        if (mask) y *= (float)mask[i];
        if (accumulate == 2) y += C[i];
        C[i] = y;
    }
}

template <int BT, int TM, bool AT, bool BTr>
void launch(const GemmF32 &g, int parts, long long k_part, float *ws, bool va, bool vb, cudaStream_t st) {
    const dim3 grid((unsigned)((g.N + BT - 1) / BT), (unsigned)((g.M + BT - 1) / BT), (unsigned)parts);
    const int threads = (BT / TM) * (BT / TM);
    auto kern = va ? (vb ? k_gemm_f32<BT, TM, AT, BTr, true, true> : k_gemm_f32<BT, TM, AT, BTr, true, false>)
                   : (vb ? k_gemm_f32<BT, TM, AT, BTr, false, true> : k_gemm_f32<BT, TM, AT, BTr, false, false>);
    kern<<<grid, threads, 0, st>>>(g.A, g.B, g.C, g.N, g.K, g.M, k_part, g.accumulate, g.mask, ws);
}

template <int BT, int TM>
void launch_bt(const GemmF32 &g, int parts, long long k_part, float *ws, bool va, bool vb, cudaStream_t st) {
    if (g.a_trans) {
        if (g.b_trans) launch<BT, TM, true, true>(g, parts, k_part, ws, va, vb, st);
        else launch<BT, TM, true, false>(g, parts, k_part, ws, va, vb, st);
    } else {
        if (g.b_trans) launch<BT, TM, false, true>(g, parts, k_part, ws, va, vb, st);
        else launch<BT, TM, false, false>(g, parts, k_part, ws, va, vb, st);
    }
}

}  // namespace

// the parts in h->f_split into C
int gemm_f32_join(qgru_handle *h, const GemmF32 &g, int parts, cudaStream_t st) {
    const long long n = g.N * g.M;
    k_gemm_f32_join<<<grid_for(n, 256, h->sm_count), 256, 0, st>>>((const float *)h->f_split.p, g.C, n, parts, g.accumulate, g.mask);
    h->launches++;
    return QGRU_OK;
}

int gemm_f32(qgru_handle *h, const GemmF32 &g, cudaStream_t st) {
    // Tensor cores where there is work for them: a slab of 32 K takes a CTA about 1.7 us there and a tile 8 us beside its slabs.
    // us, tensor cores / fp32 pipe: 51200 x 1536 x 256 331 / 862; 12800 x 128 x 768 47 / 71; 6400 x 64 x 384 14 / 21; 384 x 3200 x 128
    // 22 / 24; below that 384 x 1600 x 128 19 / 19, 64 x 1536 x 512 20 / 17.  A narrow C fills the tile of neither (6400 x 384 x 64
    // 28 / 24, 12800 x 384 x 16 29 / 41); few K leave only the tile's own time (12800 x 16 x 768 31 / 18), and operands without two
    // neighbours in one load more of it (12801 x 77 x 600 49 / 41, 12801 x 600 x 77 66 / 76).  (Before the operands' factor of 2^24, 1 to 5 %
    // of the tensor cores' times.)
    const bool pairs = ((g.a_trans ? g.N : g.K) | (g.b_trans ? g.K : (long long)g.M)) % 2 == 0 &&
                       ((reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.B)) & 7u) == 0;
    if (g.K >= (pairs ? 64 : 256) && (double)g.N * g.K * std::max(g.M, 64) >= (g.M <= 64 ? 2.5e8 : 1.5e8) && gemm_f32_tc_fits(g)) {
        int width;
        const long long t = gemm_f32_tc_tiles(g, &width);
        long long parts = t >= h->sm_count ? 1 : std::max<long long>(1, std::min<long long>(h->sm_count / t, g.K / 64));
        const long long k_part = ((g.K + parts - 1) / parts + 31) / 32 * 32;
        parts = (g.K + k_part - 1) / k_part;
        int rc;
        if (parts > 1 && (rc = ensure(h, h->f_split, (size_t)parts * g.N * g.M * sizeof(float)))) return rc;
        if ((rc = gemm_f32_tc_launch(h, g, (int)parts, k_part, parts > 1 ? (float *)h->f_split.p : g.C, st))) return rc;
        h->launches++;
        if (parts > 1) gemm_f32_join(h, g, (int)parts, st);
        CK(cudaGetLastError());
        return QGRU_OK;
    }
    const auto al16 = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const bool va = al16(g.A) && (g.a_trans ? g.N : g.K) % 4 == 0;
    const bool vb = al16(g.B) && (g.b_trans ? g.K : (long long)g.M) % 4 == 0;
    // 128 x 128 tiles where they alone (or with few K parts) fill the SMs: half the operand traffic of 64 x 64.  Those have
    // eight warps to a tile, because a slab is latency where an SM has one tile: 4096 x 64 x 192 10 us, with two warps (8 x 8
    // outputs a thread) 15.5; 256 x 64 x 192 6.3, with two warps and two parts 18.6.  K is split while the tiles leave SMs
    // idle, in parts of two slabs or more (384 x 1600 x 64 15 us, with two warps 21; three such products of a training step
    // with two warps 97 us in parts of 128 inputs, 73 in parts of 32).
    const auto tiles = [&](int bt) { return ((g.N + bt - 1) / bt) * ((g.M + bt - 1) / bt); };
    const bool big = tiles(128) * std::max<long long>(1, g.K / 512) >= h->sm_count && g.N > 64 && g.M > 64;
    const long long t = big ? tiles(128) : tiles(64);
    const long long want = big ? 2ll * h->sm_count : 4ll * h->sm_count;
    long long parts = std::max<long long>(1, std::min({want / std::max<long long>(1, t), g.K / PART_MIN, (long long)64}));
    if (t >= h->sm_count || g.K <= 128) parts = 1;      // (adding the parts is a launch of 4 us: as long as 128 inputs)
    long long k_part = ((g.K + parts - 1) / parts + BK - 1) / BK * BK;
    parts = (g.K + k_part - 1) / k_part;
    float *ws = nullptr;
    if (parts > 1) {
        int rc;
        if ((rc = ensure(h, h->f_split, (size_t)parts * g.N * g.M * sizeof(float)))) return rc;
        ws = (float *)h->f_split.p;
    }
    if (big) launch_bt<128, 8>(g, (int)parts, k_part, ws, va, vb, st);
    else launch_bt<64, 4>(g, (int)parts, k_part, ws, va, vb, st);
    h->launches++;
    if (parts > 1) gemm_f32_join(h, g, (int)parts, st);
    CK(cudaGetLastError());
    return QGRU_OK;
}

}  // namespace qgru
