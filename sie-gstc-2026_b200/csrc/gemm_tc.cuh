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
// Returns a SIEB200_* status; the kernel's bounded waits report through an
// error word checked on the next synchronization (gemm_tc_check).
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
int gemm_tc_check(GemmTC* g, cudaStream_t stream);
// Whether the default kernel configuration is selected (no switch).
bool gemm_tc_default(const GemmTC* g);

// Scales of the FP16 split operands. B: the power of two that brings a largest
// magnitude (its float bits) into [2^8, 2^9), the largest entry of the matrix
// before the factorization (U12 may grow 128-fold before it leaves FP16's
// range); A = L21, whose entries are relative to the pivots, 2^6 (up to 1023). Both
// as high as the growth allows: entries below 2^-14 of a scaled value lose bits
// of lo (with scales of 1 the 20,880-unknown omega spindle took 17 refinement
// iterations instead of 15).
constexpr float kHalfScaleA = 64.f;
__host__ __device__ inline float half_scale(unsigned max_bits) {
    const unsigned e = max_bits >> 23;
    const unsigned b = (e >= 16 && e <= 253 ? 262u - e : 127u) << 23;
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    union { unsigned u; float f; } v;
    v.u = b;
    return v.f;
#endif
}
// The same update from scaled FP16 split packs (rows of ld FP16 values, hi
// columns from k0, lo columns from klo, K of each; lo kept 2^11 up, A times
// kHalfScaleA, B times half_scale(*scale_bits)): all rows of the first w columns and the first 2 w rows of the
// others (w = N: all of C; w a multiple of 64 otherwise), the first 128 rows from
// column shift0 on.
int gemm_half_sub(GemmTC* g, cudaStream_t stream, float* C, int64_t ldc, const __half* A, const __half* B, int64_t ld,
                  int64_t M2, int64_t N, int64_t w, int k0, int klo, int K, const unsigned* scale_bits, int max_ctas,
                  int64_t shift0);
// Selects the implementation: 3 = persistent tcgen05 kernel whose epilogue
// adds -acc to C by TMA reduction (default), 2 = persistent kernel that
// loads, subtracts and stores the C tile by TMA, 1 = one CTA per tile
// tcgen05 kernel, 0 = SIMT on the same packed operands (checking path).
// SIEB200_GEMM_MODE=<0..3> in the environment overrides the default;
// SIEB200_GEMM_C_SLOTS=1 moves C in one 128-column slot instead of four
// 32-column ones.
void gemm_tc_set_mode(GemmTC* g, int mode);

}  // namespace sieb200
