// Split-TF32 trailing-update GEMM on the 5th-generation tensor cores.
//   C[2M x N] (fp32, column-major, ldc) -= A[2M x K] * B[N x K]^T
// A and B are K-major fp32 operands prepared by the LU panel kernels
// (realified complex rows with the hi/lo TF32 split laid out along K).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace sieb200 {

struct GemmTC;

int gemm_tc_create(GemmTC** out);
void gemm_tc_destroy(GemmTC* g);
// The device word in which the kernels' bounded waits leave kGemmTimeout when
// they give up (the owner clears and reads it); set before the first launch.
constexpr unsigned kGemmTimeout = 3;
void gemm_tc_error_word(GemmTC* g, unsigned* word);
// Returns a SIEB200_* status.
// max_ctas > 0 caps the persistent kernel's grid, leaving the other SMs to
// concurrent work on other streams.
// layout 0: A and B are one K sweep; layout 1: [hi | lo] halves along K,
// C -= A_hi B_hi^T + A_hi B_lo^T + A_lo B_hi^T (persistent kernel).
// shift0 > 0 leaves the first shift0 columns of the first 128 rows (one row
// tile) untouched: those rows take columns [shift0, N), the others [0, N)
// (the trailing update of a block LU whose next diagonal block is factored
// concurrently).
int gemm_tc_sub(GemmTC* g, cudaStream_t stream, float* C, int64_t ldc, const float* A,
                const float* B, int64_t M2, int64_t N, int K, int max_ctas = 0, int layout = 0,
                int64_t shift0 = 0);

// Exponent of the scale of a row of L21 or a column of U12 in the FP16 split operands:
// with it the largest entry, whose exponent is max_exp, falls into [2^14, 2^15).
__host__ __device__ inline int half_exponent(int max_exp) {
    const int e = 14 - max_exp;
    return e > 126 ? 126 : (e < -126 ? -126 : e);
}
// The same update from scaled FP16 split packs (rows of ld FP16 values, hi
// columns from k0, lo columns from klo, K of each; lo kept 2^11 up; per 128 columns of
// K, one block step, a row of A is 1 / fa and a column of B 1 / fb times its value:
// fa and fb hold a float per complex row and column and step, fstride apart, the first
// step of this call first): all rows of the first w columns and the first 2 w rows of
// the others (w = N: all of C; w a multiple of 64 otherwise), the first 128 rows from
// column shift0 on. fb may be read up to 128 entries past N.
int gemm_half_sub(GemmTC* g, cudaStream_t stream, float* C, int64_t ldc, const __half* A, const __half* B, int64_t ld,
                  int64_t M2, int64_t N, int64_t w, int k0, int klo, int K, const float* fa, const float* fb,
                  int64_t fstride, int max_ctas, int64_t shift0);

// Selects the implementation: 3 = persistent tcgen05 kernel whose epilogue
// adds -acc to C by TMA reduction (default), 2 = persistent kernel that
// loads, subtracts and stores the C tile by TMA, 1 = one CTA per tile
// tcgen05 kernel, 0 = SIMT on the same packed operands (checking path).
// SIEB200_GEMM_MODE=<0..3> in the environment overrides the default;
// SIEB200_GEMM_C_SLOTS=1 moves C in one 128-column slot instead of four
// 32-column ones.
void gemm_tc_set_mode(GemmTC* g, int mode);

}  // namespace sieb200
