// qgru_gemm_f32.cuh - the fp32 matrix product of float mode, calibration and the backward pass.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

struct qgru_handle;

namespace qgru {

// C[n][j] (+)= sum_k A(n, k) * B(k, j), then times mask[n][j] where a mask is given (1 keep, 0 drop).
// A is stored [N][K], or [K][N] with a_trans; B is stored [K][M], or [M][K] with b_trans; C is [N][M].
// fp32 operands, fused multiply-adds in fp32, sums in a fixed order (results repeat bit for bit).
struct GemmF32 {
    const float *A;
    bool a_trans;
    const float *B;
    bool b_trans;
    float *C;
    long long N, K;
    int M;
    int accumulate = 0;              // 1: mask * (C + product), 2: C + mask * product
    const uint8_t *mask = nullptr;
};
int gemm_f32(qgru_handle *h, const GemmF32 &g, cudaStream_t st);

// The same on the tensor cores (qgru_gemm_f32_tc.cu): whether its grid and its 32-bit offsets cover the sizes; number and width of its tiles; `parts` of K into `out` (C itself with one
// part, else [parts][N][M]), added by gemm_f32_join.
bool gemm_f32_tc_fits(const GemmF32 &g);
int gemm_f32_tc_tiles(const GemmF32 &g, int *width);
int gemm_f32_join(qgru_handle *h, const GemmF32 &g, int parts, cudaStream_t st);
int gemm_f32_tc_launch(qgru_handle *h, const GemmF32 &g, int parts, long long k_part, float *out, cudaStream_t st);

// packed fp32 pairs (one register pair, element 0 in the low half)
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// two independent IEEE fused multiply-adds in one instruction
__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

}  // namespace qgru
