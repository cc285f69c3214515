// Phase factors and reciprocal square roots of the quadrature kernels.
//
// exp(j k x) for many x and one k: not a sincos of the rounded product k x but a
// table-driven reduction (P. T. P. Tang, "Table-lookup algorithms for elementary
// functions and their error analysis", 10th IEEE Symposium on Computer Arithmetic,
// 1991). x k kTurn / (2 pi) is split by FMAs into a step number and a remainder in
// [-1/2, 1/2] that keeps the product's low bits; the remainder's sine and
// cosine - 1 are short polynomials (Chebyshev interpolation over the
// remainder's range, errors 3.3e-17 and 1e-19) and the step's rotation comes
// from a table of kTurn entries in shared memory. 15 FP64 instructions, one of
// them rounding at the size of the result; absolute error below 4e-16 whatever the
// phase. The table is kept kTurnCopies times, copy c in the 16-byte bank group c, so
// that a lane reading copy lane % kTurnCopies meets no bank conflict whatever the
// steps are.
#pragma once

#include <cmath>

#include "common.cuh"

namespace sieb200 {

constexpr int kTurn = 128;      // steps per turn
constexpr int kTurnCopies = 8;
constexpr int kTurnBytes = kTurn * kTurnCopies * 2 * (int)sizeof(double);
// Step numbers have to fit 32 bits: callers keep k |x| below this.
constexpr double kPhaseMax = 1e7;

// One wavenumber: khi + klo = k kTurn / (2 pi).
struct Wave {
    double k, khi, klo;
};

inline Wave make_wave(double k) {
    // kTurn / (2 pi) = 64 / pi to twice double precision
    constexpr double hi = 0x1.45f306dc9c883p+4, lo = -1.2594353072116791651e-15;
    Wave w;
    w.k = k;
    w.khi = k * hi;
    w.klo = std::fma(k, hi, -w.khi) + k * lo;
    return w;
}

// Fills the table (all threads of the CTA; the caller synchronizes).
__device__ __forceinline__ void fill_turn_table(double2* tab) {
    for (int t = threadIdx.x; t < kTurn; t += blockDim.x) {
        double s, c;
        sincospi((double)t * (2.0 / kTurn), &s, &c);
#pragma unroll
        for (int u = 0; u < kTurnCopies; ++u) tab[t * kTurnCopies + u] = make_double2(c, s);
    }
}

// cos and sin of w.k * x; lane_tab = table + lane % kTurnCopies.
__device__ __forceinline__ void phase_cs(const double2* lane_tab, const Wave& w, double x, double& c, double& s) {
    constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: the sum's low word is the rounded addend
    const double tm = fma(x, w.khi, kMagic);
    const double2 cs = lane_tab[(__double2loint(tm) & (kTurn - 1)) * kTurnCopies];
    const double f = fma(x, w.klo, fma(x, w.khi, -(tm - kMagic)));
    const double f2 = f * f;
    const double sf = f * fma(f2, fma(f2, 2.3749742434243424e-9, -1.9713259806801761e-5), 0.04908738521234045);
    const double cf = f2 * fma(f2, fma(f2, -1.9430317098946112e-11, 2.4191809451124926e-7), -0.001204785693492353);
    c = fma(cs.x, cf, fma(-cs.y, sf, cs.x));
    s = fma(cs.y, cf, fma(cs.x, sf, cs.y));
}

// 1/sqrt(x): the hardware's approximate reciprocal square root (20 bits) refined by one
// step of Chebyshev's third-order iteration (J. F. Traub, "Iterative Methods for
// the Solution of Equations", 1964) for y^-2 = x: y (1 + e/2 + 3 e^2/8) with
// e = 1 - x y^2. Relative error below 1.7e-16.
__device__ __forceinline__ double rsqrt_refined(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// R^2 below (1e-12)^2, decided on the high words (an FP64 comparison would
// take a slot of the pipe the quadrature kernels are bound by).
__device__ __forceinline__ bool tiny_square(double R2) { return __double2hiint(R2) < 0x3AF357C3; }

}  // namespace sieb200
