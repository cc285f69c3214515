// Dense RWG-Galerkin impedance-matrix assembly (PEC T-EFIE / N-EFIE / N-MFIE,
// T-PMCHWT / N-PMCHWT / N-Muller, SIE-GSTC).
//
// Reference behaviour (paths relative to the SIE-GSTC project):
//   per face pair TL/TK      include/sie_mom/cuda/dunavant_quadrature.cuh:207-324
//   per face pair nTL/nTK    dunavant_quadrature.cuh:342-480 (surface form B),
//                            singular part 889-1040
//   RWG Gram (jump terms)    dunavant_quadrature.cuh:1261-1326
//   rotated-testing blocks   src/sie_mom/solvers/dielectric/dielectric_kernels.cu:155-500,
//                            src/sie_mom/solvers/pec_solver.cu:113-240
//   singular extraction      dunavant_quadrature.cuh:769-875,
//                            include/sie_mom/cuda/semi_analytic_integrals.cuh:35-92, 563-667
//   Green kernels            include/sie_mom/cuda/green_functions_utils.cuh:236-361
//   block placement          include/sie_mom/cuda/sie_kernels_assembly.cuh:156-272, 610-705,
//                            src/sie_mom/solvers/dielectric/dielectric_kernels.cu:23-149
//   GSTC jump-condition mass sie_kernels_assembly.cuh:460-594,
//                            include/sie_mom/cuda/gstc_tensor_utils.cuh:72-309,
//                            dunavant_quadrature.cuh:1422-1508
//
// B200 design. The reference runs one thread per face pair with 72 global
// complex atomics per pair. Here:
//   1. face_prep      one thread per face builds a geometry record and the
//                     face's quadrature points (double) once.
//   2. far_pairs      a lane (or a few) per face pair: it runs over its test
//                     points and, for each, sums over the source points only what
//                     depends on them (G, G q, g, g q), folded once per test
//                     point into the pair's complex moments in triangle-local
//                     coordinates, from which the 3x3 blocks follow:
//                       rho_m . rho_n  = (p-A_j).(q-B_i)
//                       (rho_m x rho_n) . R = (rho_m x rho_n) . (v_j - v_i).
//                     The Green kernel's phase and reciprocal square root
//                     are written for the FP64 pipe, which binds (phase.cuh).
//                     With RWG testing (m, n) and (n, m) are one evaluation.
//   3. near pairs     (centroid distance below the threshold, decided in float
//                     as the reference does): near_regular, the extracted
//                     kernel, and pair_singular, the analytic (Wilton) part,
//                     one warp per pair, lanes over the outer points.
//   4. mass_face      GSTC only: one thread per (face, tensor).
//   5. gather         one thread per (test edge, source edge) sums the <= 2x2
//                     incident face pairs and writes every block of Z exactly
//                     once per slab (with one slab Z is only stored):
//                     deterministic, no atomics.
// Face-pair blocks live in a workspace processed in slabs of test faces, so
// the largest meshes stream through a bounded buffer.

#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "phase.cuh"

namespace sieb200 {

namespace {

constexpr int kMaxQ = 80;      // Dunavant rule 20 has 79 points
constexpr int kWarps = 8;      // warps per CTA of the warp-per-pair kernels
constexpr int kMaxLine = 20;   // Gauss-Legendre points of the nTL line form
constexpr double kPi = 3.14159265358979323846;

struct FaceGeom {
    d3 v[3];
    d3 c;        // centroid ((v0 + v1) + v2) / 3, as the reference forms it
    d3 fv[3];    // free vertex of local edge j
    d3 A[3];     // fv[j] - c
    double len[3];
    double area;
    int idx[3];
    int edge[3];
};

__device__ __forceinline__ d3 ldg3(const d3* p) {
    return mk3(__ldg(&p->x), __ldg(&p->y), __ldg(&p->z));
}

// Reference-exact (no FMA contraction) centroid and distance, so that the
// float threshold test takes the same branch as the reference kernels
// (sie_kernels_assembly.cuh:195-199).
__device__ __forceinline__ float centroid_distance(const FaceGeom& a, const FaceGeom& b) {
    const double dx = __dsub_rn(a.c.x, b.c.x), dy = __dsub_rn(a.c.y, b.c.y),
                 dz = __dsub_rn(a.c.z, b.c.z);
    const double s = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    return (float)__dsqrt_rn(s);
}

// Extraction test: the dielectric kernels compare the float-rounded centroid
// distance (dielectric_kernels.cu:201-206), the PEC N-EFIE / N-MFIE kernels
// the double distance against the float threshold (pec_solver.cu:134-136).
__device__ __forceinline__ bool near_pair(const FaceGeom& a, const FaceGeom& b, float thr, int exact) {
    if (!exact) return centroid_distance(a, b) < thr;
    const double dx = __dsub_rn(a.c.x, b.c.x), dy = __dsub_rn(a.c.y, b.c.y),
                 dz = __dsub_rn(a.c.z, b.c.z);
    const double s = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    return __dsqrt_rn(s) < (double)thr;
}

__global__ void face_prep_kernel(const double* __restrict__ V, const int* __restrict__ F,
                                 const int* __restrict__ FE, int nf, const float* __restrict__ qpts,
                                 int Q, FaceGeom* __restrict__ geom, d3* __restrict__ qp) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    FaceGeom g;
    for (int a = 0; a < 3; ++a) {
        g.idx[a] = F[3 * f + a];
        g.edge[a] = FE[3 * f + a];
        g.v[a] = mk3(V[3 * g.idx[a]], V[3 * g.idx[a] + 1], V[3 * g.idx[a] + 2]);
    }
    g.c = mk3(__ddiv_rn(__dadd_rn(__dadd_rn(g.v[0].x, g.v[1].x), g.v[2].x), 3.0),
              __ddiv_rn(__dadd_rn(__dadd_rn(g.v[0].y, g.v[1].y), g.v[2].y), 3.0),
              __ddiv_rn(__dadd_rn(__dadd_rn(g.v[0].z, g.v[1].z), g.v[2].z), 3.0));
    // mesh_geometry.cuh:51-80: local edge e runs A->B, free vertex opposite,
    // sign +1 iff global index of A > global index of B.
    const int EA[3] = {0, 1, 2}, EB[3] = {1, 2, 0}, EF[3] = {2, 0, 1};
    for (int e = 0; e < 3; ++e) {
        const d3 ev = g.v[EB[e]] - g.v[EA[e]];
        const double l = sqrt(ev.x * ev.x + ev.y * ev.y + ev.z * ev.z);
        g.len[e] = (g.idx[EA[e]] > g.idx[EB[e]] ? 1.0 : -1.0) * l;
        g.fv[e] = g.v[EF[e]];
        g.A[e] = g.fv[e] - g.c;
    }
    const d3 cr = cross3(g.v[1] - g.v[0], g.v[2] - g.v[0]);
    g.area = 0.5 * sqrt(dot3(cr, cr));
    geom[f] = g;
    // mesh_geometry.cuh:211-222 with float reference coordinates.
    for (int q = 0; q < Q; ++q) {
        const double xi = (double)qpts[2 * q], eta = (double)qpts[2 * q + 1];
        const double zeta = 1.0 - xi - eta;
        qp[(size_t)f * Q + q] = mk3(g.v[0].x * zeta + g.v[1].x * xi + g.v[2].x * eta,
                                    g.v[0].y * zeta + g.v[1].y * xi + g.v[2].y * eta,
                                    g.v[0].z * zeta + g.v[1].z * xi + g.v[2].z * eta);
    }
}

// Near pairs: count (list == nullptr) or fill.
__global__ void near_pairs_kernel(const FaceGeom* __restrict__ geom, int nf, float thr, int exact,
                                  int m0, int m1, unsigned long long* counter, int2* list,
                                  unsigned long long capacity) {
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long span = (long long)(m1 - m0) * nf;
    if (id >= span) return;
    const int m = m0 + (int)(id / nf), n = (int)(id % nf);
    if (near_pair(geom[m], geom[n], thr, exact)) {
        const unsigned long long slot = atomicAdd(counter, 1ull);
        if (list && slot < capacity) list[slot] = make_int2(m, n);
    }
}

__device__ __forceinline__ void warp_sum(double& v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
}
__device__ __forceinline__ void warp_sum(cplx& v) {
    warp_sum(v.re);
    warp_sum(v.im);
}

// One point pair: kernel values for wavenumber k (standard or extracted form)
// green_functions_utils.cuh:236-288 / 295-361. Returns G (TL kernel) and g
// with TK kernel = g * (r_p - r_q).
__device__ __forceinline__ void green_std(double R, double inv_R, double i4pR, double k, cplx& G,
                                          cplx& g) {
    double s, c;
    sincos(k * R, &s, &c);
    G = cx(c * i4pR, -s * i4pR);
    const cplx wg = cx(inv_R * G.re - k * G.im, inv_R * G.im + k * G.re);
    g = wg * inv_R;
}

__device__ __forceinline__ void green_reg(double R, double k, cplx& G, cplx& g) {
    if (R < 1e-9) {
        G = cx(0.0, -k / (4.0 * kPi));
        g = cx(0.0, 0.0);
        return;
    }
    const double i4p = 1.0 / (4.0 * kPi);
    const double inv_R = 1.0 / R, inv_R2 = inv_R * inv_R, inv_R3 = inv_R2 * inv_R;
    const double i4pR = i4p * inv_R;
    double s, c;
    sincos(k * R, &s, &c);
    G = cx((c - 1.0) * i4pR, -s * i4pR);
    cplx K = cx(inv_R3, k * inv_R2) * cx(c, -s);
    K.re += -(inv_R3 + k * k * 0.5 * inv_R);
    g = K * i4p;
}

__device__ __forceinline__ d3 normalize3(d3 a) {
    const double inv = 1.0 / sqrt(dot3(a, a));
    return a * inv;
}

__device__ __forceinline__ d3 face_normal(const FaceGeom& g) {
    return normalize3(cross3(g.v[1] - g.v[0], g.v[2] - g.v[0]));
}

// The line form's unit normal: cross product divided by its length
// (dunavant_quadrature.cuh:521-525), and twice the area.
__device__ __forceinline__ d3 face_normal_div(const FaceGeom& g) {
    const d3 c = cross3(g.v[1] - g.v[0], g.v[2] - g.v[0]);
    const double l = sqrt(dot3(c, c));
    return mk3(c.x / l, c.y / l, c.z / l);
}

// ------------------------------------------------- regular quadrature ----
// Double quadrature of the Green kernel over a face pair (m test, n source).
// Inner sums per test point p, in source coordinates q about the centroid:
//   S0 = sum_q w G, Sq = sum_q w G q,  T0 = sum_q w g, Tq = sum_q w g q
// (g R is the gradient factor, R = r_p - r_q). Everything the 3 x 3 blocks
// need is linear in these, so the test point is folded in once per p, into
// one of two sets of moments:
//   RWG testing (TL, TK):
//     TL_ji = l_j l_i [ 1/4 (Spq - Sp.B_i - A_j.Sq + (A_j.B_i) S0) - S0/k^2 ]
//     TK_ji = l_j l_i / 4 [ Tpq.d - Tp.(B x d) - Tq.(d x A) + ((A x B).d) T0 ],
//     d = v_j - v_i; Tpq = sum p x Tq, the others plain products with w_p, p.
//   n x RWG testing (surface form B of nTL / nTK, dunavant_quadrature.cuh:342-480),
//   tau_j = t_p - t_j, t_p = p x n_m, t_j = A_j x n_m:
//     nTL = 1/4 (tau . rho_ni) G - 1/(2 k^2) tau . (g R),
//     nTK = 1/4 (tau x rho_ni) . (g R)   (not on the coincident face);
//     sum G tau.rho       = Stq - St.B - t_j.Sq + (t_j.B) S0
//     sum g tau.R         = TtR - t_j.TR
//     sum g (tau x rho).R = U0 - B.V1 - t_j.V2 + (t_j x B).TR
//   with, per p and P = r_p - c_n: TR = T0 P - Tq, U0 = (P x t_p).Tq,
//   V1 = TR x t_p, V2 = Tq x P.
// NT: number of T sums: 0 (TL only), NK (one per wavenumber), or 1 with
// NK = 2, where the consumer needs TK1 + TK2 only (T-PMCHWT) and the two
// wavenumbers' g are added before they are accumulated.
template <int NK, int NT>
struct PointSums {
    cplx S0[NK], Sq[NK][3];
    cplx T0[NT ? NT : 1], Tq[NT ? NT : 1][3];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int a = 0; a < NK; ++a) S0[a] = Sq[a][0] = Sq[a][1] = Sq[a][2] = cx(0, 0);
#pragma unroll
        for (int a = 0; a < (NT ? NT : 1); ++a) T0[a] = Tq[a][0] = Tq[a][1] = Tq[a][2] = cx(0, 0);
    }
    // G and g of wavenumber a already carry the source weight.
    __device__ __forceinline__ void add(const cplx (&G)[NK], const cplx (&g)[NK], double qx, double qy, double qz) {
#pragma unroll
        for (int a = 0; a < NK; ++a) {
            S0[a] += G[a];
            Sq[a][0].re = fma(G[a].re, qx, Sq[a][0].re); Sq[a][0].im = fma(G[a].im, qx, Sq[a][0].im);
            Sq[a][1].re = fma(G[a].re, qy, Sq[a][1].re); Sq[a][1].im = fma(G[a].im, qy, Sq[a][1].im);
            Sq[a][2].re = fma(G[a].re, qz, Sq[a][2].re); Sq[a][2].im = fma(G[a].im, qz, Sq[a][2].im);
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            cplx s = g[t];
            if (NT < NK) {
#pragma unroll
                for (int a = 1; a < NK; ++a) s += g[a];
            }
            T0[t] += s;
            Tq[t][0].re = fma(s.re, qx, Tq[t][0].re); Tq[t][0].im = fma(s.im, qx, Tq[t][0].im);
            Tq[t][1].re = fma(s.re, qy, Tq[t][1].re); Tq[t][1].im = fma(s.im, qy, Tq[t][1].im);
            Tq[t][2].re = fma(s.re, qz, Tq[t][2].re); Tq[t][2].im = fma(s.im, qz, Tq[t][2].im);
        }
    }
};

// Totals of one pair: S = S0, Sp (St), Sq, Spq (Stq); T = T0, Tp, Tq, Tpq
// (RWG) or TR, TtR, U0, V1, V2 (n x RWG).
template <int NK, int NT, bool ROT>
struct PairSums {
    static constexpr int NTM = ROT ? 11 : 10;
    cplx S[NK][8], T[NT ? NT : 1][NTM];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int a = 0; a < NK; ++a)
#pragma unroll
            for (int e = 0; e < 8; ++e) S[a][e] = cx(0, 0);
#pragma unroll
        for (int a = 0; a < (NT ? NT : 1); ++a)
#pragma unroll
            for (int e = 0; e < NTM; ++e) T[a][e] = cx(0, 0);
    }
    // Folds test point p in: u = p (RWG) or t_p (n x RWG), P = r_p - c_n.
    __device__ __forceinline__ void fold(const PointSums<NK, NT>& I, double w, d3 u, d3 P) {
#pragma unroll
        for (int a = 0; a < NK; ++a) {
            const cplx s0 = I.S0[a] * w, qx = I.Sq[a][0] * w, qy = I.Sq[a][1] * w, qz = I.Sq[a][2] * w;
            S[a][0] += s0;
            S[a][1] += s0 * u.x; S[a][2] += s0 * u.y; S[a][3] += s0 * u.z;
            S[a][4] += qx; S[a][5] += qy; S[a][6] += qz;
            S[a][7] += qx * u.x + qy * u.y + qz * u.z;
        }
#pragma unroll
        for (int a = 0; a < NT; ++a) {
            const cplx t0 = I.T0[a] * w, qx = I.Tq[a][0] * w, qy = I.Tq[a][1] * w, qz = I.Tq[a][2] * w;
            if (!ROT) {
                T[a][0] += t0;
                T[a][1] += t0 * u.x; T[a][2] += t0 * u.y; T[a][3] += t0 * u.z;
                T[a][4] += qx; T[a][5] += qy; T[a][6] += qz;
                T[a][7] += qz * u.y - qy * u.z;
                T[a][8] += qx * u.z - qz * u.x;
                T[a][9] += qy * u.x - qx * u.y;
            } else {
                const cplx rx = t0 * P.x - qx, ry = t0 * P.y - qy, rz = t0 * P.z - qz;
                const d3 c = cross3(P, u);
                T[a][0] += rx; T[a][1] += ry; T[a][2] += rz;
                T[a][3] += rx * u.x + ry * u.y + rz * u.z;
                T[a][4] += qx * c.x + qy * c.y + qz * c.z;
                T[a][5] += ry * u.z - rz * u.y;
                T[a][6] += rz * u.x - rx * u.z;
                T[a][7] += rx * u.y - ry * u.x;
                T[a][8] += qy * P.z - qz * P.y;
                T[a][9] += qz * P.x - qx * P.z;
                T[a][10] += qx * P.y - qy * P.x;
            }
        }
    }
    // Sums over groups of 2^lg neighbouring lanes (every lane gets the total).
    __device__ __forceinline__ void reduce(int lg) {
        for (int o = 1; o < (1 << lg); o <<= 1) {
#pragma unroll
            for (int a = 0; a < NK; ++a)
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    S[a][e].re += __shfl_xor_sync(0xffffffffu, S[a][e].re, o);
                    S[a][e].im += __shfl_xor_sync(0xffffffffu, S[a][e].im, o);
                }
#pragma unroll
            for (int a = 0; a < NT; ++a)
#pragma unroll
                for (int e = 0; e < NTM; ++e) {
                    T[a][e].re += __shfl_xor_sync(0xffffffffu, T[a][e].re, o);
                    T[a][e].im += __shfl_xor_sync(0xffffffffu, T[a][e].im, o);
                }
        }
    }
    // Values of local edges (j, i): tl per wavenumber, tk per T sum.
    __device__ __forceinline__ void expand(const FaceGeom& gm, const FaceGeom& gn, int j, int i, d3 nm, bool coinc,
                                           bool form_a, const double (&kk)[NK], cplx (&tl)[NK],
                                           cplx (&tk)[NT ? NT : 1]) const {
        const d3 B = gn.A[i];
        const d3 A = ROT ? cross3(gm.A[j], nm) : gm.A[j];  // t_j for n x RWG testing
        const double scale = gm.len[j] * gn.len[i];
        const double AB = dot3(A, B);
#pragma unroll
        for (int a = 0; a < NK; ++a) {
            cplx s = S[a][7];
            s = s - (S[a][1] * B.x + S[a][2] * B.y + S[a][3] * B.z);
            s = s - (S[a][4] * A.x + S[a][5] * A.y + S[a][6] * A.z);
            s += S[a][0] * AB;
            if (!ROT) {
                tl[a] = (s * 0.25 - S[a][0] * (1.0 / (kk[a] * kk[a]))) * scale;
            } else if (form_a) {
                tl[a] = s * (0.25 * scale);
            } else {
                // (ROT keeps one T sum per wavenumber)
                const cplx* t = T[NT == NK ? a : 0];
                const cplx g = t[3] - (t[0] * A.x + t[1] * A.y + t[2] * A.z);
                tl[a] = (s * 0.25 + g * (-0.5 / (kk[a] * kk[a]))) * scale;
            }
        }
#pragma unroll
        for (int a = 0; a < NT; ++a) {
            cplx u = cx(0, 0);
            if (!coinc && !ROT) {
                const d3 d = gm.fv[j] - gn.fv[i];
                const d3 BxD = cross3(B, d), DxA = cross3(d, A);
                u = T[a][7] * d.x + T[a][8] * d.y + T[a][9] * d.z;
                u = u - (T[a][1] * BxD.x + T[a][2] * BxD.y + T[a][3] * BxD.z);
                u = u - (T[a][4] * DxA.x + T[a][5] * DxA.y + T[a][6] * DxA.z);
                u += T[a][0] * dot3(cross3(A, B), d);
                u = u * (0.25 * scale);
            } else if (!coinc) {
                const d3 x = cross3(A, B);
                u = T[a][4];
                u = u - (T[a][5] * B.x + T[a][6] * B.y + T[a][7] * B.z);
                u = u - (T[a][8] * A.x + T[a][9] * A.y + T[a][10] * A.z);
                u += T[a][0] * x.x + T[a][1] * x.y + T[a][2] * x.z;
                u = u * (0.25 * scale);
            }
            tk[a] = u;
        }
    }
};

// Pair blocks: pairs[((m - m0) nf + n) 9 NB + (3 j + i) NB + slot], the NB
// values of one edge pair adjacent. The regular pass writes its tl to slots
// s_tl.. and its tk to slots s_tk.. (negative: not kept).
struct PairOut {
    cplx* pairs;
    int NB, s_tl, s_tk;
};
template <int NK, int NT>
__device__ __forceinline__ void put_pair(const PairOut& o, size_t row, int e, const cplx (&tl)[NK],
                                         const cplx (&tk)[NT ? NT : 1]) {
    cplx* out = o.pairs + (row * 9 + e) * o.NB;
    if (o.s_tl >= 0) {
#pragma unroll
        for (int a = 0; a < NK; ++a) out[o.s_tl + a] = tl[a];
    }
    if (NT > 0 && o.s_tk >= 0) {
#pragma unroll
        for (int a = 0; a < NT; ++a) out[o.s_tk + a] = tk[a];
    }
}

struct RuleWeights {
    double w[kMaxQ], w4[kMaxQ];  // weights, weights / (4 pi)
};
static RuleWeights make_rule_weights(const float* w, int Q) {
    RuleWeights r{};
    for (int q = 0; q < Q; ++q) {
        r.w[q] = (double)w[q];
        r.w4[q] = r.w[q] / (4.0 * kPi);
    }
    return r;
}
constexpr int kFarWarps = 4;
constexpr int kFarSmemMax = kTurnBytes + (int)sizeof(double) * 3 * kMaxQ * 32;

// Far pairs (centroid distance at or above the extraction threshold): one
// source face per lane group, 2^lg lanes sharing it (each takes every 2^lg-th
// test point); a warp works on one test face, the CTA's four warps on
// `chunk` of them against the CTA's 32 >> lg source faces, whose points sit
// in shared memory about their centroids.
// Bound: the FP64 pipe. Per Green value with its moments 52 pipe
// instructions (TL and TK, one wavenumber; 41 each with two wavenumbers and
// TK summed): 12 for R and 1/R, 15 for the phase factor, 9 for G and g, 16 to
// accumulate. What keeps it there:
//  * one lane holds a pair's moments, so no value crosses lanes unless the
//    mesh is small (lg > 0) and the 3 x 3 expansion runs on all lanes;
//  * with RWG testing (ROT = false) the blocks of (m, n) and (n, m) are each
//    other's transposes and both are written from one evaluation (m <= n);
//  * phase factors and 1/R without library calls (phase.cuh); BIG falls back
//    to sincos(k R) for meshes whose phases would not fit its step number.
// Measured: the 2000-face sphere with 61 points and two wavenumbers 54.4 ms (212 ms
// for the kernel this replaces: a warp per ordered pair, a test point per lane, sincos
// and division from the math library); the 2880-face SIE-GSTC sphere with
// equal wavenumbers 69.7 ms (435 ms). The FP64 pipe is busy 66 and 64 % of the cycles;
// what is left is the latency of dependent FP64 instructions. Three CTAs per SM cap a
// thread at 168 registers, which spills 732 bytes with two wavenumbers and 36 with
// one. The same kernel with four CTAs per SM 54.9 and 75.0 ms, with two 57.6 and
// 65.9 ms, with the source points unrolled by four 51.7 and 70.1 ms.
template <int NK, int NT, bool ROT, bool BIG>
__global__ void __launch_bounds__(kFarWarps * 32, 3)
far_pairs_kernel(const FaceGeom* __restrict__ geom, const d3* __restrict__ qp, const RuleWeights rw, int Q, int nf,
                 int m0, int m1, const Wave k0, const Wave k1, float thr, int exact, int form_a, int lg, int chunk,
                 const PairOut out) {
    extern __shared__ __align__(16) unsigned char far_smem[];
    double2* tab = reinterpret_cast<double2*>(far_smem);               // [kTurn][kTurnCopies]
    double* sq = reinterpret_cast<double*>(tab + kTurn * kTurnCopies);  // [Q][3][nt]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nt = 32 >> lg;
    const int n0 = blockIdx.y * nt;
    const int n_last = min(n0 + nt, nf) - 1;
    // Test faces of this CTA. Tiles inside the slab's own columns stop at the
    // diagonal with RWG testing.
    const bool inside = !ROT && n0 >= m0 && n_last < m1;
    const int m_end = inside ? n_last + 1 : m1;
    const int mb = m0 + blockIdx.x * chunk;
    if (mb >= m_end) return;
    const int me = min(mb + chunk, m_end);

    fill_turn_table(tab);
    for (int t = threadIdx.x; t < Q * nt; t += blockDim.x) {
        const int s = t % nt, q = t / nt, f = min(n0 + s, nf - 1);
        const d3 r = ldg3(&qp[(size_t)f * Q + q]) - ldg3(&geom[f].c);
        sq[(q * 3 + 0) * nt + s] = r.x;
        sq[(q * 3 + 1) * nt + s] = r.y;
        sq[(q * 3 + 2) * nt + s] = r.z;
    }
    __syncthreads();

    const int sub = lane & ((1 << lg) - 1), ln = lane >> lg;
    const int n = min(n0 + ln, nf - 1);
    const bool have_n = n0 + ln < nf;
    const d3 cn = ldg3(&geom[n].c);
    const double2* my_tab = tab + (lane & (kTurnCopies - 1));
    const double* my_q = sq + ln;
    const Wave kv[2] = {k0, k1};
    double kk[NK];
#pragma unroll
    for (int a = 0; a < NK; ++a) kk[a] = kv[a].k;

    for (int m = mb + warp; m < me; m += kFarWarps) {
        const FaceGeom& gm = geom[m];
        const bool mirror = !ROT && n >= m0 && n < m1;  // (n, m) lies in this slab too
        const bool mine = have_n && !(mirror && n < m) && !near_pair(gm, geom[n], thr, exact);
        if (!__any_sync(0xffffffffu, mine)) continue;
        const d3 cm = ldg3(&gm.c);
        d3 nm = mk3(0, 0, 0);
        if (ROT) nm = form_a ? face_normal_div(gm) : face_normal(gm);
        PairSums<NK, NT, ROT> tot;
        tot.clear();
#pragma unroll 1
        for (int p = sub; p < Q; p += 1 << lg) {
            const d3 rp = ldg3(&qp[(size_t)m * Q + p]);
            const d3 P = rp - cn;
            PointSums<NK, NT> in;
            in.clear();
#pragma unroll 2
            for (int q = 0; q < Q; ++q) {
                const double qx = my_q[(q * 3 + 0) * nt], qy = my_q[(q * 3 + 1) * nt], qz = my_q[(q * 3 + 2) * nt];
                const double dx = P.x - qx, dy = P.y - qy, dz = P.z - qz;
                const double R2 = fma(dz, dz, fma(dy, dy, dx * dx));
                double inv = rsqrt_refined(R2);
                if (tiny_square(R2)) inv = 0.0;  // R < 1e-12: no contribution
                const double R = R2 * inv;
                const double W = inv * rw.w4[q];
                const double i2 = inv * inv;
                cplx G[NK], g[NK];
#pragma unroll
                for (int a = 0; a < NK; ++a) {
                    double c, s;
                    if (BIG) {
                        sincos(kv[a].k * R, &s, &c);
                    } else {
                        phase_cs(my_tab, kv[a], R, c, s);
                    }
                    G[a] = cx(c * W, -s * W);
                    if (NT > 0) {
                        // g = (1/R) (1/R + j k) G
                        const double v = kv[a].k * inv;
                        g[a] = cx(fma(i2, G[a].re, -(v * G[a].im)), fma(i2, G[a].im, v * G[a].re));
                    }
                }
                in.add(G, g, qx, qy, qz);
            }
            const d3 pl = rp - cm;
            tot.fold(in, rw.w[p], ROT ? cross3(pl, nm) : pl, P);
        }
        tot.reduce(lg);
        if (!mine) continue;
        const FaceGeom& gn = geom[n];
        const bool coinc = gm.idx[0] == gn.idx[0] && gm.idx[1] == gn.idx[1] && gm.idx[2] == gn.idx[2];
        const size_t row = (size_t)(m - m0) * nf + n, rowT = (size_t)(n - m0) * nf + m;
        for (int e = sub; e < 9; e += 1 << lg) {
            const int j = e / 3, i = e - 3 * j;
            cplx tl[NK], tk[NT ? NT : 1];
            tot.expand(gm, gn, j, i, nm, coinc, form_a != 0, kk, tl, tk);
            put_pair<NK, NT>(out, row, e, tl, tk);
            if (mirror && n != m) put_pair<NK, NT>(out, rowT, i * 3 + j, tl, tk);
        }
    }
}

// Near pairs (list): the same sums with the extracted kernel, one warp per
// pair: lane groups of 32 / Q lanes share a test point (one lane each from 32
// points on). With RWG testing a pair whose mirror image lies in the slab is
// evaluated once (m <= n) and written twice.
template <int NK, int NT, bool ROT>
__global__ void __launch_bounds__(128)
near_regular_kernel(const FaceGeom* __restrict__ geom, const d3* __restrict__ qp, const RuleWeights rw, int Q, int nf,
                    int m0, int m1, const int2* __restrict__ list, int count, double k0, double k1, int form_a,
                    const PairOut out) {
    const int id = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (id >= count) return;
    const int m = list[id].x, n = list[id].y;
    const bool mirror = !ROT && n >= m0 && n < m1;
    if (mirror && n < m) return;
    const FaceGeom &gm = geom[m], &gn = geom[n];
    const d3 cm = ldg3(&gm.c), cn = ldg3(&gn.c);
    d3 nm = mk3(0, 0, 0);
    if (ROT) nm = form_a ? face_normal_div(gm) : face_normal(gm);
    const double kv[2] = {k0, k1};
    double kk[NK];
#pragma unroll
    for (int a = 0; a < NK; ++a) kk[a] = kv[a];
    const int G = Q >= 32 ? 1 : 32 / Q, PL = 32 / G;
    const int lp = lane / G, lq = lane - lp * G;
    PairSums<NK, NT, ROT> tot;
    tot.clear();
#pragma unroll 1
    for (int p = lp; p < Q && lp < PL; p += PL) {
        const d3 rp = ldg3(&qp[(size_t)m * Q + p]);
        PointSums<NK, NT> in;
        in.clear();
#pragma unroll 1
        for (int q = lq; q < Q; q += G) {
            const d3 rq = ldg3(&qp[(size_t)n * Q + q]);
            const d3 Rv = rp - rq, ql = rq - cn;
            const double R = sqrt(Rv.x * Rv.x + Rv.y * Rv.y + Rv.z * Rv.z);
            cplx Gk[NK], gk[NK];
#pragma unroll
            for (int a = 0; a < NK; ++a) {
                green_reg(R, kk[a], Gk[a], gk[a]);
                Gk[a] = Gk[a] * rw.w[q];
                gk[a] = gk[a] * rw.w[q];
            }
            in.add(Gk, gk, ql.x, ql.y, ql.z);
        }
        const d3 pl = rp - cm;
        tot.fold(in, rw.w[p], ROT ? cross3(pl, nm) : pl, rp - cn);
    }
    tot.reduce(5);
    const bool coinc = gm.idx[0] == gn.idx[0] && gm.idx[1] == gn.idx[1] && gm.idx[2] == gn.idx[2];
    if (lane < 9) {
        const int j = lane / 3, i = lane - 3 * j;
        cplx tl[NK], tk[NT ? NT : 1];
        tot.expand(gm, gn, j, i, nm, coinc, form_a != 0, kk, tl, tk);
        put_pair<NK, NT>(out, (size_t)(m - m0) * nf + n, lane, tl, tk);
        if (mirror && n != m) put_pair<NK, NT>(out, (size_t)(n - m0) * nf + m, i * 3 + j, tl, tk);
    }
}

// ------------------------------------------------------------ Wilton ----
struct Pots {
    double phi0, phi2, d;
    d3 phi1b, phi3b, r_pi;
};

// semi_analytic_integrals.cuh:35-92 and 563-667 in one pass.
__device__ Pots wilton(const d3 r, const d3 tri[3]) {
    Pots P;
    const d3 n = normalize3(cross3(tri[1] - tri[0], tri[2] - tri[0]));
    P.d = dot3(r - tri[0], n);
    P.r_pi = r - n * P.d;
    const double ad = fabs(P.d);
    const double eps9f = (double)1e-9f;
    P.phi0 = 0.0;
    P.phi2 = 0.0;
    P.phi1b = mk3(0, 0, 0);
    P.phi3b = mk3(0, 0, 0);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const d3 vs = tri[e], ve = tri[(e + 1) % 3];
        const d3 th = normalize3(ve - vs);
        const d3 u = cross3(th, n);
        const d3 rs = vs - n * dot3(n, vs);
        const d3 re = ve - n * dot3(n, ve);
        const d3 to_s = rs - P.r_pi;
        const double su = dot3(to_s, u);
        const double p0 = fabs(su);
        const double orient = su >= 0.0 ? 1.0 : -1.0;
        const double lp = dot3(re - P.r_pi, th);
        const double lm = dot3(rs - P.r_pi, th);
        const double Pp = hypot(p0, lp), Pm = hypot(p0, lm);
        const double R0 = hypot(p0, ad);
        const double Rp = hypot(Pp, ad), Rm = hypot(Pm, ad);
        const double logt = (log(Rp) + log1p(lp / Rp)) - (log(Rm) + log1p(lm / Rm));
        double at = 0.0;
        if (ad > eps9f || ad > 1e-6)
            at = atan2(p0 * lp, R0 * R0 + ad * Rp) - atan2(p0 * lm, R0 * R0 + ad * Rm);
        if (p0 > eps9f) P.phi0 += orient * (p0 * logt - (ad > eps9f ? ad * at : 0.0));
        P.phi1b = P.phi1b + u * ((R0 * R0) * logt + (lp * Rp) - (lm * Rm));
        double term = 0.0;
        if (ad > 1e-6)
            term = (1.0 / ad) * at;
        else if (p0 > 1e-9)
            term = -((lp / (p0 * Pp)) - (lm / (p0 * Pm)));
        P.phi2 += orient * term;
        P.phi3b = P.phi3b - u * logt;
    }
    P.phi1b = P.phi1b * 0.5;
    return P;
}

__device__ __forceinline__ d3 psi1(const Pots& P, d3 fv) {
    return (P.phi1b + P.r_pi * P.phi0) - fv * P.phi0;
}

// semi_analytic_integrals.cuh:481-498 (k^2/2 formed in float).
__device__ __forceinline__ d3 upsilon(const Pots& P, d3 fv, d3 r, float k) {
    const d3 phi3 = P.phi3b + (P.r_pi - fv) * P.phi2;
    const d3 ps = psi1(P, fv);
    const float k2o2 = __fmul_rn(__fmul_rn(k, k), 0.5f);
    const d3 comb = phi3 + ps * (double)k2o2;
    return cross3(r - fv, comb) * -1.0;
}

// Singular (extracted) part of the near pairs, added to the pair blocks.
// dunavant_quadrature.cuh:769-875. Lanes over outer points p.
template <int NK>
__global__ void pair_singular_kernel(const FaceGeom* __restrict__ geom, const d3* __restrict__ qp,
                                     const float* __restrict__ qw_g, int Q, int nf, int m0,
                                     const int2* __restrict__ list, int count, double k0,
                                     double k1, bool with_tk, bool sum_tk, const PairOut dst) {
    const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp_global >= count) return;
    const int2 mn = list[warp_global];
    const FaceGeom gm = geom[mn.x];
    const FaceGeom gn = geom[mn.y];
    const bool coinc = gm.idx[0] == gn.idx[0] && gm.idx[1] == gn.idx[1] && gm.idx[2] == gn.idx[2];
    const double kk[2] = {k0, k1};
    double tl[NK][9], tk[NK][9];
#pragma unroll
    for (int a = 0; a < NK; ++a)
#pragma unroll
        for (int t = 0; t < 9; ++t) { tl[a][t] = 0.0; tk[a][t] = 0.0; }

    for (int p = lane; p < Q; p += 32) {
        const d3 rp = qp[(size_t)mn.x * Q + p];
        const double wp = (double)qw_g[p];
        const Pots P = wilton(rp, gn.v);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const d3 rm = rp - gm.fv[j];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const d3 ps = psi1(P, gn.fv[i]);
                const double db = 0.25 * dot3(rm, ps);
#pragma unroll
                for (int a = 0; a < NK; ++a) {
                    tl[a][j * 3 + i] += (db - 1.0 / (kk[a] * kk[a]) * P.phi0) * wp;
                    if (with_tk && !coinc) {
                        const d3 up = upsilon(P, gn.fv[i], rp, (float)kk[a]);
                        tk[a][j * 3 + i] += 0.25 * dot3(rm, up) * wp;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int a = 0; a < NK; ++a)
#pragma unroll
        for (int t = 0; t < 9; ++t) { warp_sum(tl[a][t]); warp_sum(tk[a][t]); }
    if (lane < 9) {
        const int j = lane / 3, i = lane - 3 * j;
        const double as = 1.0 / (4.0 * kPi * gn.area);
        const double s = as * gm.len[j] * gn.len[i];
        cplx* out = dst.pairs + (((size_t)(mn.x - m0) * nf + mn.y) * 9 + lane) * dst.NB;
        double tlv[NK], tkv[NK];
#pragma unroll
        for (int a = 0; a < NK; ++a) {
            // select entry `lane` without dynamic register indexing
            tlv[a] = 0.0; tkv[a] = 0.0;
#pragma unroll
            for (int t = 0; t < 9; ++t)
                if (t == lane) { tlv[a] = tl[a][t]; tkv[a] = tk[a][t]; }
            out[dst.s_tl + a].re += tlv[a] * s;
            if (with_tk) out[dst.s_tk + (sum_tk ? 0 : a)].re += tkv[a] * s;
        }
    }
}

// ---------------------------------------------- rotated (n x RWG) testing --
// semi_analytic_integrals.cuh:108-171 (calculate_phi_0, on the testing edges
// of the line form): an edge whose end is within 1e-9 of r is skipped, and on
// an edge's line (R0 < 1e-8) the end distances are regularised by 1e-8.
__device__ double phi0_line(const d3 r, const d3 tri[3]) {
    const d3 n = normalize3(cross3(tri[1] - tri[0], tri[2] - tri[0]));
    const double d = dot3(r - tri[0], n);
    const d3 r_pi = r - n * d;
    const double ad = fabs(d);
    double phi0 = 0.0;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const d3 vs = tri[e], ve = tri[(e + 1) % 3];
        const d3 th = normalize3(ve - vs);
        const d3 u = cross3(th, n);
        const d3 rs = vs - n * dot3(n, vs);
        const d3 re = ve - n * dot3(n, ve);
        const double su = dot3(rs - r_pi, u);
        const double p0 = fabs(su);
        const double orient = su >= 0.0 ? 1.0 : -1.0;
        const double lp = dot3(re - r_pi, th);
        const double lm = dot3(rs - r_pi, th);
        const double Pp = hypot(p0, lp), Pm = hypot(p0, lm);
        const double R0 = hypot(p0, ad);
        double Rp = hypot(Pp, ad), Rm = hypot(Pm, ad);
        if (Rp < 1e-9 || Rm < 1e-9) continue;
        if (R0 < 1e-8) {
            // Rounded product, then rounded sum, as the reference's
            // sqrt(pow(R, 2) + pow(eps, 2)): where 1e-16 is below half an ulp
            // of R^2 the regularisation has no effect and, on the edge line
            // beyond its start, log1p(-1) makes the reference's value
            // infinite; the same inputs give the same values here.
            Rp = sqrt(__dadd_rn(__dmul_rn(Rp, Rp), 1e-8 * 1e-8));
            Rm = sqrt(__dadd_rn(__dmul_rn(Rm, Rm), 1e-8 * 1e-8));
        }
        const double logt = (log(Rp) + log1p(lp / Rp)) - (log(Rm) + log1p(lm / Rm));
        double at = 0.0;
        if (ad > 1e-9) at = atan2(p0 * lp, R0 * R0 + ad * Rp) - atan2(p0 * lm, R0 * R0 + ad * Rm);
        phi0 += orient * (p0 * logt - ad * at);
    }
    return phi0;
}

// Singular (extracted) part of the rotated-testing blocks of the near pairs,
// added to the pair blocks. One warp per pair, lanes over outer points.
// Surface form B (dunavant_quadrature.cuh:889-1040), per outer point with
// phi_1 = phi_1b - d phi_0 n_n and the extracted gradient phi_3b - d phi_2 n_n:
//   nTL += 1/2 tau . (phi_1 + 1/2 R_i phi_0 + gradient / k^2)
//          (the gradient left out on the coincident face),
// then e_mj e_ni / (4 pi A_n). Line form A (1040-1179): nTL += 1/4 w tau . Psi_1
// on the area, scaled alike, plus the testing-edge sum
// sum_e sum_q L_e w_q (tau . nu_e) phi_0(r_eq) scaled by e_mj e_ni / (8 pi A_m A_n k^2)
// (lanes over the 3 NG edge points). Both forms:
//   nTK += 1/4 tau . Upsilon_coul (not on the coincident face).
template <int NK, bool FORM_A>
__global__ void pair_singular_n_kernel(const FaceGeom* __restrict__ geom, const d3* __restrict__ qp,
                                       const float* __restrict__ qw_g, int Q, int nf, int m0,
                                       const int2* __restrict__ list, int count, double k0,
                                       double k1, bool with_ntk, const float* __restrict__ gl_t,
                                       const float* __restrict__ gl_w, int NG, const PairOut dst) {
    const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp_global >= count) return;
    const int2 mn = list[warp_global];
    const FaceGeom gm = geom[mn.x];
    const FaceGeom gn = geom[mn.y];
    const bool coinc = gm.idx[0] == gn.idx[0] && gm.idx[1] == gn.idx[1] && gm.idx[2] == gn.idx[2];
    const d3 nm = FORM_A ? face_normal_div(gm) : face_normal(gm);
    const d3 nn = face_normal(gn);
    const double kk[2] = {k0, k1};
    double tl[NK][9], tk[NK][9];
#pragma unroll
    for (int a = 0; a < NK; ++a)
#pragma unroll
        for (int t = 0; t < 9; ++t) { tl[a][t] = 0.0; tk[a][t] = 0.0; }

    for (int p = lane; p < Q; p += 32) {
        const d3 rp = qp[(size_t)mn.x * Q + p];
        const double wp = (double)qw_g[p];
        const Pots P = wilton(rp, gn.v);
        const d3 phi1 = P.phi1b - nn * (P.d * P.phi0);
        const d3 grad = P.phi3b - nn * (P.d * P.phi2);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const d3 tau = cross3(rp - gm.fv[j], nm);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                if (FORM_A) {
                    const double an = 0.25 * wp * dot3(tau, psi1(P, gn.fv[i]));
#pragma unroll
                    for (int a = 0; a < NK; ++a) tl[a][j * 3 + i] += an;
                } else {
                    const d3 br = phi1 + ((rp - gn.fv[i]) * 0.5) * P.phi0;
#pragma unroll
                    for (int a = 0; a < NK; ++a) {
                        const d3 V = coinc ? br : br + grad * (1.0 / (kk[a] * kk[a]));
                        tl[a][j * 3 + i] += 0.5 * dot3(tau, V) * wp;
                    }
                }
                if (with_ntk && !coinc) {
#pragma unroll
                    for (int a = 0; a < NK; ++a) {
                        const d3 up = upsilon(P, gn.fv[i], rp, (float)kk[a]);
                        tk[a][j * 3 + i] += (FORM_A ? 0.25 * wp * dot3(tau, up) : 0.25 * dot3(tau, up) * wp);
                    }
                }
            }
        }
    }
    double line[3] = {0.0, 0.0, 0.0};
    if (FORM_A) {
        for (int it = lane; it < 3 * NG; it += 32) {
            const int e = it / NG, q = it - e * NG;
            const d3 vA = gm.v[e], vB = gm.v[e == 2 ? 0 : e + 1];
            const d3 E = vB - vA;
            const double Le = sqrt(dot3(E, E));
            const d3 c = cross3(E, nm);
            const d3 nu = mk3(c.x / Le, c.y / Le, c.z / Le);
            const double t = (double)gl_t[q], wl = (double)gl_w[q];
            const d3 req = mk3(vA.x + t * (vB.x - vA.x), vA.y + t * (vB.y - vA.y), vA.z + t * (vB.z - vA.z));
            const double ph0 = phi0_line(req, gn.v);
#pragma unroll
            for (int j = 0; j < 3; ++j) line[j] += Le * wl * dot3(cross3(req - gm.fv[j], nm), nu) * ph0;
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) warp_sum(line[j]);
    }
#pragma unroll
    for (int a = 0; a < NK; ++a)
#pragma unroll
        for (int t = 0; t < 9; ++t) { warp_sum(tl[a][t]); warp_sum(tk[a][t]); }
    if (lane < 9) {
        const int j = lane / 3, i = lane - 3 * j;
        const double as = 1.0 / (4.0 * kPi * gn.area);
        const double s = as * gm.len[j] * gn.len[i];
        cplx* out = dst.pairs + (((size_t)(mn.x - m0) * nf + mn.y) * 9 + lane) * dst.NB;
        const double edges = gm.len[j] * gn.len[i];
        const double ls = FORM_A ? 1.0 / (8.0 * kPi * gm.area * gn.area) : 0.0;
        double lj = 0.0;
#pragma unroll
        for (int jj = 0; jj < 3; ++jj)
            if (jj == j) lj = line[jj];
#pragma unroll
        for (int a = 0; a < NK; ++a) {
            double tlv = 0.0, tkv = 0.0;
#pragma unroll
            for (int t = 0; t < 9; ++t)
                if (t == lane) { tlv = tl[a][t]; tkv = tk[a][t]; }
            if (FORM_A) {
                out[dst.s_tl + a].re += tlv * (edges * as) + edges * ls * lj / (kk[a] * kk[a]);
                if (with_ntk) out[dst.s_tk + a].re += tkv * (edges * as);
            } else {
                if (dst.s_tl >= 0) out[dst.s_tl + a].re += tlv * s;
                if (with_ntk) out[dst.s_tk + a].re += tkv * s;
            }
        }
    }
}

// Testing-edge line integral of the nTL form A (dunavant_quadrature.cuh:598-672),
// added to the nTL blocks of every face pair of the slab: for each test edge
// e (v_A -> v_B), Gauss-Legendre point t_q and source point p,
//   nTL_ji += l_j l_i (L_e / 2A_m) (tau_j(r_eq) . nu_e) G(r_eq, r_p) w_q w_p / k^2,
// the same for every source basis i. tau_j . nu_e is linear in t_q, so each
// warp (one face pair) accumulates sum w G and sum w t G per edge and
// wavenumber; 9 lanes expand them. Standard or extracted kernel as the pair's
// area quadrature.
template <int NK>
__global__ void __launch_bounds__(kWarps * 32)
pair_line_kernel(const FaceGeom* __restrict__ geom, const d3* __restrict__ qp,
                 const float* __restrict__ qw_g, int Q, int nf, int m0, double k0, double k1,
                 float thr, int exact, const float* __restrict__ gl_t, const float* __restrict__ gl_w,
                 int NG, const PairOut dst) {
    __shared__ double s_w[kMaxQ];
    __shared__ double s_t[20], s_wl[20];
    const int m = m0 + blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int t = threadIdx.x; t < Q; t += blockDim.x) s_w[t] = (double)qw_g[t];
    for (int t = threadIdx.x; t < NG; t += blockDim.x) { s_t[t] = (double)gl_t[t]; s_wl[t] = (double)gl_w[t]; }
    __syncthreads();
    const FaceGeom& gm = geom[m];
    const d3 nm = face_normal_div(gm);
    const d3 cr = cross3(gm.v[1] - gm.v[0], gm.v[2] - gm.v[0]);
    const double twoA = sqrt(dot3(cr, cr));
    const double kk[2] = {k0, k1};
    const int items = NG * Q;
    for (int n = warp; n < nf; n += kWarps) {
        const FaceGeom& gn = geom[n];
        const bool regular = near_pair(gm, gn, thr, exact);  // warp-uniform
        cplx M0[3][NK], M1[3][NK];
#pragma unroll
        for (int e = 0; e < 3; ++e)
#pragma unroll
            for (int a = 0; a < NK; ++a) { M0[e][a] = cx(0, 0); M1[e][a] = cx(0, 0); }
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const d3 vA = gm.v[e], vB = gm.v[e == 2 ? 0 : e + 1];
            for (int it = lane; it < items; it += 32) {
                const int q = it / Q, p = it - q * Q;
                const double t = s_t[q];
                const d3 req = mk3(vA.x + t * (vB.x - vA.x), vA.y + t * (vB.y - vA.y), vA.z + t * (vB.z - vA.z));
                const d3 rq = ldg3(&qp[(size_t)n * Q + p]);
                const d3 Rv = req - rq;
                const double R = sqrt(Rv.x * Rv.x + Rv.y * Rv.y + Rv.z * Rv.z);
                if (!regular && R < 1e-12) continue;
                const double w = s_wl[q] * s_w[p];
                const double inv_R = regular ? 0.0 : 1.0 / R;
                const double i4pR = regular ? 0.0 : 1.0 / (4.0 * kPi * R);
#pragma unroll
                for (int a = 0; a < NK; ++a) {
                    cplx G, g;
                    if (regular) green_reg(R, kk[a], G, g);
                    else green_std(R, inv_R, i4pR, kk[a], G, g);
                    const cplx Gw = G * w;
                    M0[e][a] += Gw;
                    M1[e][a] += Gw * t;
                }
            }
        }
#pragma unroll
        for (int e = 0; e < 3; ++e)
#pragma unroll
            for (int a = 0; a < NK; ++a) { warp_sum(M0[e][a]); warp_sum(M1[e][a]); }
        if (lane < 9) {
            const int j = lane / 3, i = lane - 3 * j;
            cplx acc[NK];
#pragma unroll
            for (int a = 0; a < NK; ++a) acc[a] = cx(0, 0);
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                const d3 vA = gm.v[e], vB = gm.v[e == 2 ? 0 : e + 1];
                const d3 E = vB - vA;
                const double Le = sqrt(dot3(E, E));
                const d3 c = cross3(E, nm);
                const d3 nu = mk3(c.x / Le, c.y / Le, c.z / Le);
                const double geomf = Le / twoA;
                // tau_j(r_eq) . nu_e = c0 + t c1
                const double c0 = dot3(cross3(vA - gm.fv[j], nm), nu);
                const double c1 = dot3(cross3(E, nm), nu);
#pragma unroll
                for (int a = 0; a < NK; ++a) acc[a] += (M0[e][a] * c0 + M1[e][a] * c1) * geomf;
            }
            const double scale = gm.len[j] * gn.len[i];
            cplx* out = dst.pairs + (((size_t)blockIdx.x * nf + n) * 9 + lane) * dst.NB + dst.s_tl;
#pragma unroll
            for (int a = 0; a < NK; ++a) out[a] += acc[a] * (scale / (kk[a] * kk[a]));
        }
        __syncwarp();
    }
}

// RWG Gram block <f_j, f_i> of each face (dunavant_quadrature.cuh:1261-1326)
// with the reference's float dot product, weight and scale. One thread per
// face, gram[9 f + 3 j + i].
__global__ void gram_face_kernel(const FaceGeom* __restrict__ geom, const d3* __restrict__ qp,
                                 const float* __restrict__ qw_g, int Q, int nf, double* __restrict__ gram) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const FaceGeom& g = geom[f];
    double R[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) R[e] = 0.0;
    for (int p = 0; p < Q; ++p) {
        const float wp = qw_g[p];
        const d3 rp = qp[(size_t)f * Q + p];
        d3 rho[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) rho[i] = rp - g.fv[i];
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const double d = __dadd_rn(__dadd_rn(__dmul_rn(rho[j].x, rho[i].x), __dmul_rn(rho[j].y, rho[i].y)),
                                           __dmul_rn(rho[j].z, rho[i].z));
                R[j * 3 + i] += (double)__fmul_rn(wp, (float)d);
            }
    }
    const float area = (float)g.area;
    const float sc = __fdiv_rn(1.f, __fmul_rn(4.f, area));
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float fs = __fmul_rn(__fmul_rn(sc, (float)g.len[j]), (float)g.len[i]);
            gram[(size_t)f * 9 + j * 3 + i] = R[j * 3 + i] * (double)fs;
        }
}

// ------------------------------------------------------------ GSTC mass --
// Mass block of tensor t (0..3: the Y blocks ee, em, me, mm after the perp
// transform; 4..7 the Z blocks) of face g for the 2x2 tensor block
// (t00 t01; t10 t11): out[j*3+i] for local test edge j and source edge i.
// Linear in the four tensor entries.
__device__ void mass_tensor_block(const FaceGeom& g, const d3* __restrict__ qpf, const float* __restrict__ qw_g,
                                  int Q, int basis, int t, cplx t00, cplx t01, cplx t10, cplx t11,
                                  cplx (&out)[9]) {
    // Frame: gstc_tensor_utils.cuh:72-147.
    d3 u, w;
    if (basis == 0) {
        const d3 e1 = g.v[1] - g.v[0], e2 = g.v[2] - g.v[0];
        const d3 nn = cross3(e1, e2);
        const double l1 = sqrt(dot3(e1, e1)), ln = sqrt(dot3(nn, nn));
        if (l1 < 1e-20 || ln < 1e-20) {
            u = mk3(1, 0, 0); w = mk3(0, 1, 0);
        } else {
            const d3 nh = nn * (1.0 / ln);
            u = e1 * (1.0 / l1);
            w = cross3(nh, u);
        }
    } else {
        const d3 c = mk3((g.v[0].x + g.v[1].x + g.v[2].x) / 3.0, (g.v[0].y + g.v[1].y + g.v[2].y) / 3.0,
                         (g.v[0].z + g.v[1].z + g.v[2].z) / 3.0);
        const double r = sqrt(dot3(c, c));
        if (r < 1e-12) {
            u = mk3(1, 0, 0); w = mk3(0, 1, 0);
        } else {
            double ct = c.z / r;
            ct = ct > 1.0 ? 1.0 : (ct < -1.0 ? -1.0 : ct);
            const double th = acos(ct), ph = atan2(c.y, c.x);
            const double cth = cos(th), sth = sin(th), cph = cos(ph), sph = sin(ph);
            u = mk3(cth * cph, cth * sph, -sth);
            w = mk3(-sph, cph, 0.0);
        }
    }
    // Lift the 2x2 block (gstc_tensor_utils.cuh:184-238).
    const double uc[3] = {u.x, u.y, u.z}, wc[3] = {w.x, w.y, w.z};
    cplx T[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            cplx s = cx(0, 0);
            s += t00 * (uc[i] * uc[j]);
            s += t01 * (uc[i] * wc[j]);
            s += t10 * (wc[i] * uc[j]);
            s += t11 * (wc[i] * wc[j]);
            T[i][j] = s;
        }
    if (t < 4) {
        // Y_perp = -[n]x Y [n]x with float-cast entries (gstc_tensor_utils.cuh:269-309).
        const d3 n = normalize3(cross3(g.v[1] - g.v[0], g.v[2] - g.v[0]));
        const double N[3][3] = {{0.0, (double)(float)(-n.z), (double)(float)n.y},
                                {(double)(float)n.z, 0.0, (double)(float)(-n.x)},
                                {(double)(float)(-n.y), (double)(float)n.x, 0.0}};
        cplx tmp[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                cplx s = cx(0, 0);
#pragma unroll
                for (int k = 0; k < 3; ++k) s += T[r][k] * N[k][c];
                tmp[r][c] = s;
            }
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                cplx s = cx(0, 0);
#pragma unroll
                for (int k = 0; k < 3; ++k) s += tmp[k][c] * N[r][k];
                T[r][c] = cx(-s.re, -s.im);
            }
    }
    // Mass quadrature with float geometry (dunavant_quadrature.cuh:1422-1508).
    const float area = (float)g.area;
    float el[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) el[i] = (float)g.len[i];
    cplx R[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) R[e] = cx(0, 0);
    for (int p = 0; p < Q; ++p) {
        const double wp = (double)qw_g[p];
        const d3 rp = qpf[p];
        d3 rho[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) rho[i] = rp - g.fv[i];
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const cplx tx = T[0][0] * rho[i].x + (T[0][1] * rho[i].y + T[0][2] * rho[i].z);
                const cplx ty = T[1][0] * rho[i].x + (T[1][1] * rho[i].y + T[1][2] * rho[i].z);
                const cplx tz = T[2][0] * rho[i].x + (T[2][1] * rho[i].y + T[2][2] * rho[i].z);
                const cplx ig = tx * rho[j].x + (ty * rho[j].y + tz * rho[j].z);
                R[j * 3 + i] += ig * wp;
            }
    }
    const float sc = __fdiv_rn(1.f, __fmul_rn(4.f, area));
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float fs = __fmul_rn(__fmul_rn(sc, el[j]), el[i]);
            out[j * 3 + i] = R[j * 3 + i] * (double)fs;
        }
}

// One thread per (face, tensor t in 0..7).
__global__ void mass_face_kernel(const FaceGeom* __restrict__ geom, const d3* __restrict__ qp,
                                 const float* __restrict__ qw_g, int Q, int nf,
                                 const cplx* __restrict__ tensors, int uniform, int basis,
                                 cplx* __restrict__ mass) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nf * 8) return;
    const int f = id >> 3, t = id & 7;
    const cplx* tp = tensors + (uniform ? 0 : (size_t)f * 32) + (t >= 4 ? 16 : 0);
    const int blk = t & 3, r0 = (blk >> 1) * 2, c0 = (blk & 1) * 2;
    cplx out[9];
    mass_tensor_block(geom[f], qp + (size_t)f * Q, qw_g, Q, basis, t, tp[r0 * 4 + c0], tp[r0 * 4 + c0 + 1],
                      tp[(r0 + 1) * 4 + c0], tp[(r0 + 1) * 4 + c0 + 1], out);
#pragma unroll
    for (int e = 0; e < 9; ++e) mass[((size_t)f * 8 + t) * 9 + e] = out[e];
}

// A_M'' block pattern of the 8 mass values of one (test, source) edge pair
// with the 1/2 and 1/8 factors and the eta0 scales of the M rows/columns
// (sie_kernels_assembly.cuh:565-592), added into the 4x4 region block.
__device__ __forceinline__ void add_mass_pattern(const cplx (&mv)[8], double me, double me2, cplx (&blk)[4][4]) {
    const cplx Yee = mv[0], Yem = mv[1], Yme = mv[2], Ymm = mv[3];
    const cplx Zee = mv[4], Zem = mv[5], Zme = mv[6], Zmm = mv[7];
    const double f = 0.5, fq = 0.125;
    const cplx ap = Zee * f + Ymm * fq, am = Zee * f - Ymm * fq;
    const cplx bp = Zem * f + Yme * fq, bm = Zem * f - Yme * fq;
    const cplx cp = Zme * f + Yem * fq, cm = Zme * f - Yem * fq;
    const cplx dp = Zmm * f + Yee * fq, dm = Zmm * f - Yee * fq;
    const double s1 = 1.0, se_ = me, s2 = me2;
    blk[0][0] += ap * s1; blk[0][1] += bm * se_; blk[0][2] += am * s1; blk[0][3] += bp * se_;
    blk[1][0] += cm * se_; blk[1][1] += dp * s2; blk[1][2] += cp * se_; blk[1][3] += dm * s2;
    blk[2][0] += am * s1; blk[2][1] += bp * se_; blk[2][2] += ap * s1; blk[2][3] += bm * se_;
    blk[3][0] += cp * se_; blk[3][1] += dm * s2; blk[3][2] += cm * se_; blk[3][3] += dp * s2;
}

// Adjoint contraction for the GSTC tensors: s[f*32 + k] = lambda^H
// (dZ / d record[f][k]) x, record[f] = (Lambda, Lambda^{-1}) row-major.
// Z depends on the record only through the face's own mass blocks, and
// linearly, so dZ / d entry is the mass block of a unit entry placed by the
// A_M'' pattern on the face's 3 x 3 local edge pairs. One thread per (face, t).
__global__ void tensor_grad_kernel(const FaceGeom* __restrict__ geom, const d3* __restrict__ qp,
                                   const float* __restrict__ qw_g, int Q, int nf, int ne,
                                   const int* __restrict__ FE, int basis, double me, double me2,
                                   const cplx* __restrict__ lam, const cplx* __restrict__ x,
                                   cplx* __restrict__ s_out) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nf * 8) return;
    const int f = id >> 3, t = id & 7;
    // Pattern coefficients of tensor t: the 4x4 region block of a unit value.
    cplx mv[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) mv[k] = cx(k == t ? 1.0 : 0.0, 0.0);
    cplx C[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) C[r][c] = cx(0, 0);
    add_mass_pattern(mv, me, me2, C);
    // G[j][i] = sum_{r,c} C[r][c] conj(lambda[e_j + r E]) x[e_i + c E].
    const int64_t E = ne;
    int e[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) e[k] = FE[3 * f + k];
    cplx G[9];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            cplx acc = cx(0, 0);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const cplx lv = lam[e[j] + r * E];
                const cplx lc = cx(lv.re, -lv.im);
#pragma unroll
                for (int c = 0; c < 4; ++c) acc += C[r][c] * (lc * x[e[i] + c * E]);
            }
            G[j * 3 + i] = acc;
        }
    const int blk = t & 3, r0 = (blk >> 1) * 2, c0 = (blk & 1) * 2;
    const FaceGeom g = geom[f];
#pragma unroll 1
    for (int ab = 0; ab < 4; ++ab) {
        const cplx one = cx(1, 0), zero = cx(0, 0);
        cplx out[9];
        mass_tensor_block(g, qp + (size_t)f * Q, qw_g, Q, basis, t, ab == 0 ? one : zero, ab == 1 ? one : zero,
                          ab == 2 ? one : zero, ab == 3 ? one : zero, out);
        cplx sacc = cx(0, 0);
#pragma unroll
        for (int k = 0; k < 9; ++k) sacc += G[k] * out[k];
        const int a = ab >> 1, b = ab & 1;
        s_out[(size_t)f * 32 + (t >= 4 ? 16 : 0) + (r0 + a) * 4 + (c0 + b)] = sacc;
    }
}

// ------------------------------------------------------------ gather ----
// Slots of a pair block: TL per wavenumber, then TK per wavenumber (T-EFIE
// and N-EFIE: TL only); one TL and one TK where both regions have the same
// wavenumber; TL per wavenumber and TK1 + TK2 (T-PMCHWT, which needs no more);
// the one nTK of N-MFIE.
enum { PAIR_FULL = 0, PAIR_SAME_K = 1, PAIR_SUM_TK = 2, PAIR_TK_ONLY = 3 };

struct GatherParams {
    int formulation;
    int variant;  // 0 tangential testing; 1 N-EFIE / N-PMCHWT; 2 N-MFIE / N-Muller
    int nf, ne;
    int m0, m1;
    int NB;
    int layout;  // the NB slots of an edge pair: PAIR_* below
    cplx c_jj[2], c_mm[2];
    double s_jm, s_mm;
    double me, me2;  // mass scales (float eta0, eta0^2)
    // N-Muller (dielectric_kernels.cu:433-488): z_jj = w_em[1] nTL2 - w_em[0] nTL1
    // (w_em = omega eps mu), z_jm = eps2 nTK2 - eps1 nTK1 - eps_f G,
    // z_mj = mu2 nTK2 - mu1 nTK1 - mu_f G on the same face.
    double w_em[2], eps[2], mu[2], eps_f, mu_f;
    const double* gram;  // RWG Gram blocks (N-MFIE, N-Muller), 9 per face
};

// The region block (1x1 PEC, 2x2 PMCHWT, 4x4 GSTC) of Z at test edge te and
// source edge se from the face-pair blocks of the test faces in [m0, m1);
// false when te has no incident face in the slab. FORM: the formulation, or -1
// to take it from P.
template <int FORM>
__device__ __forceinline__ bool edge_pair_block(const cplx* __restrict__ pairs, const cplx* __restrict__ mass,
                                                const int* __restrict__ inc, const GatherParams& P, int te, int se,
                                                cplx (&blk)[4][4]) {
    const int form = FORM < 0 ? P.formulation : FORM;
    const int it[2] = {inc[2 * te], inc[2 * te + 1]};
    const int is[2] = {inc[2 * se], inc[2 * se + 1]};
    bool any = false;
#pragma unroll
    for (int a = 0; a < 2; ++a)
        if (it[a] >= 0 && it[a] / 3 >= P.m0 && it[a] / 3 < P.m1) any = true;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) blk[r][c] = cx(0, 0);
    if (!any) return false;

    cplx acc[4] = {cx(0, 0), cx(0, 0), cx(0, 0), cx(0, 0)};
    cplx mass_acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) mass_acc[k] = cx(0, 0);
    bool has_mass = false;
    double gram_acc = 0.0;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        if (it[a] < 0) continue;
        const int m = it[a] / 3, j = it[a] - 3 * m;
        if (m < P.m0 || m >= P.m1) continue;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            if (is[b] < 0) continue;
            const int n = is[b] / 3, i = is[b] - 3 * n;
            const cplx* pb = pairs + (((size_t)(m - P.m0) * P.nf + n) * 9 + j * 3 + i) * P.NB;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < P.NB) acc[k] += pb[k];
            if (form == SIEB200_GSTC && m == n) {
                has_mass = true;
                const cplx* mb = mass + (size_t)m * 72 + j * 3 + i;
#pragma unroll
                for (int k = 0; k < 8; ++k) mass_acc[k] += mb[k * 9];
            }
            if (P.variant == 2 && m == n) gram_acc += P.gram[(size_t)m * 9 + j * 3 + i];
        }
    }
    if (P.layout == PAIR_SAME_K) {
        acc[3] = acc[2] = acc[1];
        acc[1] = acc[0];
    } else if (P.layout == PAIR_TK_ONLY) {
        acc[1] = acc[0];
    }
    if (form == SIEB200_PEC_EFIE && P.variant == 2) {
        // N-MFIE (pec_solver.cu:171-240): 1/2 Gram on the same face, - nTK2.
        blk[0][0] = cx(0.5 * gram_acc, 0.0) - acc[1];
    } else if (form == SIEB200_PEC_EFIE) {
        blk[0][0] = P.c_jj[1] * acc[0];
    } else if (form == SIEB200_PMCHWT && P.variant == 2) {
        // acc: nTL1, nTL2, nTK1, nTK2.
        const cplx jj = acc[1] * cx(0.0, P.w_em[1]) - acc[0] * cx(0.0, P.w_em[0]);
        const cplx jm = acc[3] * P.eps[1] - acc[2] * P.eps[0] - cx(P.eps_f * gram_acc, 0.0);
        const cplx mj = acc[3] * P.mu[1] - acc[2] * P.mu[0] - cx(P.mu_f * gram_acc, 0.0);
        blk[0][0] = jj;
        blk[0][1] = jm * P.s_jm;
        blk[1][0] = mj * P.s_jm;
        blk[1][1] = jj * (-P.s_mm);
    } else if (form == SIEB200_PMCHWT) {
        // acc: TL1, TL2, TK1, TK2 (or TL1, TL2, TK1 + TK2, 0)
        const cplx tk = acc[2] + acc[3];
        const cplx jm = tk * P.s_jm;
        blk[0][0] = P.c_jj[0] * acc[0] + P.c_jj[1] * acc[1];
        blk[0][1] = jm;
        blk[1][0] = cx(-jm.re, -jm.im);
        blk[1][1] = (P.c_mm[0] * acc[0] + P.c_mm[1] * acc[1]) * P.s_mm;
    } else {
#pragma unroll
        for (int reg = 0; reg < 2; ++reg) {
            const cplx tl = acc[reg], tk = acc[2 + reg];
            const cplx jm = tk * P.s_jm;
            const int o = 2 * reg;
            blk[o][o] = P.c_jj[reg] * tl;
            blk[o][o + 1] = jm;
            blk[o + 1][o] = cx(-jm.re, -jm.im);
            blk[o + 1][o + 1] = P.c_mm[reg] * tl;
        }
        if (has_mass) add_mass_pattern(mass_acc, P.me, P.me2, blk);
    }
    return true;
}

__device__ __forceinline__ int region_count(int formulation) {
    return formulation == SIEB200_PEC_EFIE ? 1 : (formulation == SIEB200_PMCHWT ? 2 : 4);
}

// One thread per (test edge te, source edge se); te fastest for coalesced
// column-major stores. Sums the incident face pairs with the test face in
// [m0, m1). ADD: adds into Z (zeroed before the first of several slabs); else
// the only slab, and every entry of Z is stored once without being read.
// Bound: the latency of its pair reads, so by the threads in flight; each
// formulation is its own instance, since one kernel for all keeps the 4 x 4
// blocks of SIE-GSTC in registers (36, 48 and 96 a thread now): PEC, 1920 edges
// 191 -> 103 us; T-PMCHWT, 3000 edges 780 -> 645 us; SIE-GSTC, 4320 edges
// 1720 -> 1670 us. The shape of the CTA's tile of edges makes no difference.
template <int FORM, bool ADD>
__global__ void gather_kernel(const cplx* __restrict__ pairs, const cplx* __restrict__ mass,
                              const int* __restrict__ inc, GatherParams P, cplx* __restrict__ Z,
                              int64_t ldz) {
    const int te = blockIdx.x * blockDim.x + threadIdx.x;
    const int se = blockIdx.y * blockDim.y + threadIdx.y;
    if (te >= P.ne || se >= P.ne) return;
    cplx blk[4][4];
    if (!edge_pair_block<FORM>(pairs, mass, inc, P, te, se, blk) && ADD) return;
    const int64_t E = P.ne;
    const int nr = region_count(FORM);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (c < nr && r < nr) {
                cplx* z = Z + (te + r * E) + (se + c * E) * ldz;
                *z = ADD ? *z + blk[r][c] : blk[r][c];
            }
}

// Matrix-free product: y += (the slab's rows of Z) x without storing Z. One
// warp per test edge: lanes stride over the source edges, each forming the
// same region block as gather_kernel, then a warp reduction; the warp owns
// its y entries, and slabs run in order, so the sum is deterministic.
__global__ void gather_matvec_kernel(const cplx* __restrict__ pairs, const cplx* __restrict__ mass,
                                     const int* __restrict__ inc, GatherParams P, const cplx* __restrict__ x,
                                     cplx* __restrict__ y) {
    const int te = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (te >= P.ne) return;  // warp-uniform
    const int64_t E = P.ne;
    const int nr = region_count(P.formulation);
    cplx acc[4] = {cx(0, 0), cx(0, 0), cx(0, 0), cx(0, 0)};
    bool mine = false;
    for (int se = lane; se < P.ne; se += 32) {
        cplx blk[4][4];
        if (!edge_pair_block<-1>(pairs, mass, inc, P, te, se, blk)) break;  // same answer for every se
        mine = true;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (c >= nr) break;
            const cplx xv = x[se + c * E];
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[r] += blk[r][c] * xv;  // rows >= nr of blk are zero
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        double re = acc[r].re, im = acc[r].im;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            re += __shfl_xor_sync(0xffffffffu, re, o);
            im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        acc[r] = cx(re, im);
    }
    mine = __any_sync(0xffffffffu, mine);
    if (mine && lane == 0) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (r < nr) y[te + r * E] += acc[r];
    }
}

}  // namespace

int64_t system_dimension(int formulation, int64_t ne) {
    return formulation == SIEB200_PEC_EFIE ? ne : (formulation == SIEB200_PMCHWT ? 2 * ne : 4 * ne);
}

// Mesh, rule and incidences to the device, then the per-face geometry
// records and quadrature points (shared by assembly and the adjoint
// contraction).
static int prepare_faces(sieb200_ctx* ctx, const sieb200_mesh& mesh, const float* pts, const float* wts, int Q,
                         FaceGeom** geom_out, d3** qp_out, float** dw_out, int** dFE_out) {
    const int nf = (int)mesh.num_faces, ne = (int)mesh.num_edges, nv = (int)mesh.num_vertices;
    cudaStream_t st = ctx->stream;
    // Edge -> (face*3 + local edge) incidences; at most two per edge.
    std::vector<int> inc(2 * (size_t)ne, -1);
    for (int f = 0; f < nf; ++f)
        for (int le = 0; le < 3; ++le) {
            const int e = mesh.faces_edges[3 * f + le];
            SIEB_CHECK(e >= 0 && e < ne, SIEB200_INVALID_ARG, "faces_edges entry out of range");
            if (inc[2 * e] < 0) inc[2 * e] = 3 * f + le;
            else if (inc[2 * e + 1] < 0) inc[2 * e + 1] = 3 * f + le;
            else {
                set_error("non-manifold mesh: an edge is shared by more than two faces");
                return SIEB200_INVALID_ARG;
            }
        }

    // Upload mesh, rule, incidences.
    const size_t vbytes = sizeof(double) * 3 * nv, fbytes = sizeof(int) * 3 * nf;
    SIEB_RETURN_IF(ctx->faces.reserve(vbytes + 2 * fbytes + 16 * 3));
    char* fb = ctx->faces.as<char>();
    double* dV = reinterpret_cast<double*>(fb);
    int* dF = reinterpret_cast<int*>(fb + ((vbytes + 15) / 16) * 16);
    int* dFE = dF + 3 * nf + 4;
    SIEB_TRY_CUDA(cudaMemcpyAsync(dV, mesh.vertices, vbytes, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(dF, mesh.faces, fbytes, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(dFE, mesh.faces_edges, fbytes, cudaMemcpyHostToDevice, st));
    SIEB_RETURN_IF(ctx->qw.reserve(sizeof(float) * (3 * kMaxQ + 2 * kMaxLine)));
    float* dpts = ctx->qw.as<float>();
    float* dw = dpts + 2 * kMaxQ;
    SIEB_TRY_CUDA(cudaMemcpyAsync(dpts, pts, sizeof(float) * 2 * Q, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(dw, wts, sizeof(float) * Q, cudaMemcpyHostToDevice, st));
    SIEB_RETURN_IF(ctx->inc.reserve(sizeof(int) * inc.size()));
    SIEB_TRY_CUDA(cudaMemcpyAsync(ctx->inc.ptr, inc.data(), sizeof(int) * inc.size(),
                                  cudaMemcpyHostToDevice, st));

    SIEB_RETURN_IF(ctx->geom.reserve(sizeof(FaceGeom) * nf));
    SIEB_RETURN_IF(ctx->qpts.reserve(sizeof(d3) * (size_t)nf * Q));
    FaceGeom* geom = ctx->geom.as<FaceGeom>();
    d3* qp = ctx->qpts.as<d3>();
    *geom_out = geom;
    *qp_out = qp;
    *dw_out = dw;
    *dFE_out = dFE;
    face_prep_kernel<<<(nf + 127) / 128, 128, 0, st>>>(dV, dF, dFE, nf, dpts, Q, geom, qp);
    SIEB_NOTE_LAUNCH();
    SIEB_TRY_CUDA(cudaGetLastError());

    return SIEB200_OK;
}

// The far kernel's phase step number has to fit 32 bits with room for its
// remainder: k times the mesh's extent below kPhaseMax (about 2e8 steps).
static bool far_phase_fits(const sieb200_mesh& mesh, double k) {
    double lo[3], hi[3];
    for (int c = 0; c < 3; ++c) lo[c] = hi[c] = mesh.vertices[c];
    for (int64_t v = 1; v < mesh.num_vertices; ++v)
        for (int c = 0; c < 3; ++c) {
            lo[c] = std::min(lo[c], mesh.vertices[3 * v + c]);
            hi[c] = std::max(hi[c], mesh.vertices[3 * v + c]);
        }
    const double d = (hi[0] - lo[0]) + (hi[1] - lo[1]) + (hi[2] - lo[2]);
    return k * d < kPhaseMax;
}

struct FarLaunch {
    const FaceGeom* geom;
    const d3* qp;
    const RuleWeights* rw;
    int Q, nf, m0, m1;
    double k0, k1;
    float thr;
    int exact;
    bool form_a;
    PairOut out;
    cudaStream_t st;
};

template <int NK, int NT, bool ROT>
static int launch_far(const FarLaunch& f, bool big) {
    // Lanes per pair: one where the mesh gives every SM several rounds of
    // warps (a warp takes 32 pairs then), else up to the test point count.
    const int rows = f.m1 - f.m0;
    const double pairs = (double)rows * f.nf * (ROT ? 1.0 : 0.5);
    int lg = 0;
    while ((2 << lg) <= std::min(32, std::max(1, f.Q)) && pairs * (1 << lg) / 32.0 < 8192.0) ++lg;
    const int nt = 32 >> lg;
    // Test faces per CTA: enough point pairs to pay for the table and the
    // staged points, few enough that the last wave stays short.
    const double warp_pairs = pairs * (1 << lg) / 32.0;
    int per_warp = std::max(1, std::min(16, 2048 / std::max(1, f.Q * f.Q >> lg)));
    per_warp = (int)std::max(1.0, std::min((double)per_warp, warp_pairs / 8192.0));
    const int chunk = kFarWarps * per_warp;
    const int smem = (int)(sizeof(double2) * kTurn * kTurnCopies + sizeof(double) * 3 * (size_t)f.Q * nt);
    const dim3 grid((unsigned)((rows + chunk - 1) / chunk), (unsigned)((f.nf + nt - 1) / nt));
    auto* kernel = big ? far_pairs_kernel<NK, NT, ROT, true> : far_pairs_kernel<NK, NT, ROT, false>;
    // (the largest size any rule asks for: another thread may launch the same
    // kernel with another one)
    SIEB_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFarSmemMax));
    kernel<<<grid, kFarWarps * 32, smem, f.st>>>(f.geom, f.qp, *f.rw, f.Q, f.nf, f.m0, f.m1, make_wave(f.k0),
                                                 make_wave(f.k1), f.thr, f.exact, f.form_a ? 1 : 0, lg, chunk, f.out);
    SIEB_NOTE_LAUNCH();
    SIEB_TRY_CUDA(cudaGetLastError());
    return SIEB200_OK;
}

// Assembly of Z (dx == nullptr) or, matrix-free, y = Z x with the same face
// pair blocks contracted against x slab by slab instead of written to Z.
static int assemble_or_apply(sieb200_ctx* ctx, const sieb200_mesh& mesh, const sieb200_options& opt,
                             const double* host_tensors, cplx* dZ, int64_t ldz, const cplx* dx, cplx* dy) {
    AssemblyParams ap;
    SIEB_RETURN_IF(make_assembly_params(opt, &ap));
    const int nf = (int)mesh.num_faces, ne = (int)mesh.num_edges, nv = (int)mesh.num_vertices;
    (void)nv;
    const int64_t N = system_dimension(opt.formulation, ne);
    SIEB_CHECK(dx || ldz >= N, SIEB200_INVALID_ARG, "leading dimension of Z is smaller than N");
    float pts[2 * kMaxQ], wts[kMaxQ];
    const int Q = expand_rule(opt.quadrature_rule, pts, wts);
    SIEB_CHECK(Q > 0 && Q <= kMaxQ, SIEB200_INVALID_ARG, "Dunavant quadrature rule must be in [1, 20]");
    cudaStream_t st = ctx->stream;

    FaceGeom* geom = nullptr;
    d3* qp = nullptr;
    float* dw = nullptr;
    int* dFE = nullptr;
    SIEB_RETURN_IF(prepare_faces(ctx, mesh, pts, wts, Q, &geom, &qp, &dw, &dFE));

    // GSTC mass blocks.
    cplx* dmass = nullptr;
    if (opt.formulation == SIEB200_GSTC) {
        const size_t ntens = opt.tensors_are_uniform ? 32 : (size_t)nf * 32;
        SIEB_RETURN_IF(ctx->tens.reserve(sizeof(cplx) * ntens));
        SIEB_TRY_CUDA(cudaMemcpyAsync(ctx->tens.ptr, host_tensors, sizeof(cplx) * ntens,
                                      cudaMemcpyHostToDevice, st));
        SIEB_RETURN_IF(ctx->mass.reserve(sizeof(cplx) * 72 * (size_t)nf));
        dmass = ctx->mass.as<cplx>();
        mass_face_kernel<<<(nf * 8 + 127) / 128, 128, 0, st>>>(
            geom, qp, dw, Q, nf, ctx->tens.as<cplx>(), opt.tensors_are_uniform, ap.basis, dmass);
        SIEB_NOTE_LAUNCH();
        SIEB_TRY_CUDA(cudaGetLastError());
    }

    // RWG Gram blocks for the jump terms of N-MFIE and N-Muller.
    const int variant = ap.variant;
    double* dgram = nullptr;
    if (variant == 2) {
        SIEB_RETURN_IF(ctx->mass.reserve(sizeof(double) * 9 * (size_t)nf));
        dgram = ctx->mass.as<double>();
        gram_face_kernel<<<(nf + 127) / 128, 128, 0, st>>>(geom, qp, dw, Q, nf, dgram);
        SIEB_NOTE_LAUNCH();
        SIEB_TRY_CUDA(cudaGetLastError());
    }

    // Slabs of test faces bounded by the pair-block workspace. Values per
    // edge pair (PAIR_*): TL (or nTL) per distinct wavenumber, then TK (or
    // nTK) where the formulation uses it (all but T-EFIE and N-EFIE).
    const bool pec = opt.formulation == SIEB200_PEC_EFIE;
    const bool rot = variant != 0;
    const bool tk = !(pec && variant != 2);
    const bool same_k = ap.nk == 2 && ap.k[0] == ap.k[1];
    const int NK = same_k ? 1 : ap.nk;  // distinct wavenumbers
    int layout = PAIR_FULL;
    if (pec && variant == 2) layout = PAIR_TK_ONLY;
    else if (same_k) layout = PAIR_SAME_K;
    else if (opt.formulation == SIEB200_PMCHWT && !rot) layout = PAIR_SUM_TK;
    PairOut po;
    po.NB = layout == PAIR_SUM_TK ? 3 : (layout == PAIR_TK_ONLY ? 1 : (tk ? 2 * NK : NK));
    po.s_tl = layout == PAIR_TK_ONLY ? -1 : 0;
    po.s_tk = !tk ? -1 : (layout == PAIR_TK_ONLY ? 0 : NK);
    const int exact = (pec && rot) ? 1 : 0;
    // Line form A of nTL (N-EFIE, N-PMCHWT, N-Muller): Gauss-Legendre rule on
    // [0, 1] after the Dunavant rule in the rule buffer.
    const int NG = ap.line_points;
    const bool form_a = NG > 0;
    float* dgl = ctx->qw.as<float>() + 3 * kMaxQ;
    if (form_a) {
        float glt[2 * kMaxLine];
        SIEB_CHECK(NG <= kMaxLine && gauss_legendre_rule_f(NG, glt, glt + kMaxLine) == NG, SIEB200_INVALID_ARG,
                   "Gauss-Legendre point count must be in [1, 20]");
        SIEB_TRY_CUDA(cudaMemcpyAsync(dgl, glt, sizeof(glt), cudaMemcpyHostToDevice, st));
    }
    // (The free memory, whose query takes 0.1 to 11 ms, is asked for only where
    // the workspace of earlier calls is too small; that workspace counts as free,
    // and what it holds is the least a slab takes.)
    const size_t pair_bytes = sizeof(cplx) * 9 * po.NB;
    const size_t most = (size_t)8 << 30;
    auto slab_of = [&](size_t budget) {
        return (int)std::max<size_t>(1, std::min<size_t>(nf, budget / (pair_bytes * nf)));
    };
    int slab = slab_of(most);
    if (ctx->pairs.bytes < pair_bytes * (size_t)slab * nf) {
        const size_t held = ctx->pairs.bytes;
        size_t free_b = 0;
        if (available_memory(&free_b) == SIEB200_OK)
            slab = std::max(slab_of(held), slab_of(std::min(most, (free_b + held) / 3)));
    }
    SIEB_RETURN_IF(ctx->pairs.reserve(pair_bytes * (size_t)slab * nf));
    po.pairs = ctx->pairs.as<cplx>();
    SIEB_RETURN_IF(ctx->counter.reserve(sizeof(unsigned long long)));
    unsigned long long* counter = ctx->counter.as<unsigned long long>();

    const bool one_slab = slab >= nf;
    if (dx)
        SIEB_TRY_CUDA(cudaMemsetAsync(dy, 0, sizeof(cplx) * N, st));
    else if (!one_slab)
        SIEB_TRY_CUDA(cudaMemset2DAsync(dZ, sizeof(cplx) * ldz, 0, sizeof(cplx) * N, N, st));

    GatherParams gp;
    gp.formulation = opt.formulation;
    gp.nf = nf;
    gp.ne = ne;
    gp.NB = po.NB;
    gp.layout = layout;
    gp.c_jj[0] = ap.c_jj[0]; gp.c_jj[1] = ap.c_jj[1];
    gp.c_mm[0] = ap.c_mm[0]; gp.c_mm[1] = ap.c_mm[1];
    gp.s_jm = ap.s_jm; gp.s_mm = ap.s_mm;
    gp.me = ap.mass_eta0; gp.me2 = ap.mass_eta0_sq;
    gp.variant = variant;
    for (int r = 0; r < 2; ++r) { gp.w_em[r] = ap.w_em[r]; gp.eps[r] = ap.eps[r]; gp.mu[r] = ap.mu[r]; }
    gp.eps_f = ap.eps_f; gp.mu_f = ap.mu_f;
    gp.gram = dgram;

    // The regular pass: T-PMCHWT with two wavenumbers in one launch (R and
    // the TK sums are shared); otherwise one launch per distinct wavenumber,
    // which keeps a pair's moments in registers.
    const RuleWeights rw = make_rule_weights(wts, Q);
    const int passes = layout == PAIR_SUM_TK ? 1 : NK;
    const bool big = !far_phase_fits(mesh, std::max(ap.k[0], ap.k[1]));
    // The near list of a slab, filled in one pass where the buffer kept from
    // earlier slabs and calls holds it.
    SIEB_RETURN_IF(ctx->near_list.reserve(sizeof(int2) * 32 * (size_t)slab));
    for (int m0 = 0; m0 < nf; m0 += slab) {
        const int m1 = std::min(nf, m0 + slab);
        const int rows = m1 - m0;
        const long long span = (long long)rows * nf;
        const int nb = (int)((span + 255) / 256);
        unsigned long long count = 0;
        for (int attempt = 0; attempt < 2; ++attempt) {
            const unsigned long long capacity = ctx->near_list.bytes / sizeof(int2);
            SIEB_TRY_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st));
            near_pairs_kernel<<<nb, 256, 0, st>>>(geom, nf, ap.threshold, exact, m0, m1, counter,
                                                  ctx->near_list.as<int2>(), capacity);
            SIEB_NOTE_LAUNCH();
            SIEB_TRY_CUDA(cudaGetLastError());
            SIEB_TRY_CUDA(cudaMemcpyAsync(&count, counter, sizeof(count), cudaMemcpyDeviceToHost, st));
            SIEB_TRY_CUDA(cudaStreamSynchronize(st));
            if (count <= capacity) break;
            SIEB_RETURN_IF(ctx->near_list.reserve(sizeof(int2) * count));
        }
        const int2* list = ctx->near_list.as<int2>();
        const int near_threads = 128;
        const unsigned near_blocks = (unsigned)((count * 32 + near_threads - 1) / near_threads);
        for (int a = 0; a < passes; ++a) {
            PairOut pa = po;
            if (passes == 2) {
                pa.s_tl = a;
                pa.s_tk = 2 + a;
            }
            // PEC and equal wavenumbers: the second entry
            const double ka = passes == 2 ? ap.k[a] : (layout == PAIR_SUM_TK ? ap.k[0] : ap.k[1]);
            const FarLaunch f{geom, qp, &rw, Q, nf, m0, m1, ka, ap.k[1], ap.threshold, exact, form_a, pa, st};
            if (rot) SIEB_RETURN_IF((launch_far<1, 1, true>(f, big)));
            else if (pec) SIEB_RETURN_IF((launch_far<1, 0, false>(f, big)));
            else if (layout == PAIR_SUM_TK) SIEB_RETURN_IF((launch_far<2, 1, false>(f, big)));
            else SIEB_RETURN_IF((launch_far<1, 1, false>(f, big)));
            if (count > 0) {
                if (rot)
                    near_regular_kernel<1, 1, true><<<near_blocks, near_threads, 0, st>>>(
                        geom, qp, rw, Q, nf, m0, m1, list, (int)count, ka, ap.k[1], form_a, pa);
                else if (pec)
                    near_regular_kernel<1, 0, false><<<near_blocks, near_threads, 0, st>>>(
                        geom, qp, rw, Q, nf, m0, m1, list, (int)count, ka, ap.k[1], 0, pa);
                else if (layout == PAIR_SUM_TK)
                    near_regular_kernel<2, 1, false><<<near_blocks, near_threads, 0, st>>>(
                        geom, qp, rw, Q, nf, m0, m1, list, (int)count, ka, ap.k[1], 0, pa);
                else
                    near_regular_kernel<1, 1, false><<<near_blocks, near_threads, 0, st>>>(
                        geom, qp, rw, Q, nf, m0, m1, list, (int)count, ka, ap.k[1], 0, pa);
                SIEB_NOTE_LAUNCH();
                SIEB_TRY_CUDA(cudaGetLastError());
            }
        }
        if (form_a) {
            if (NK == 1)
                pair_line_kernel<1><<<rows, kWarps * 32, 0, st>>>(geom, qp, dw, Q, nf, m0, ap.k[1], ap.k[1],
                                                                  ap.threshold, exact, dgl, dgl + kMaxLine, NG, po);
            else
                pair_line_kernel<2><<<rows, kWarps * 32, 0, st>>>(geom, qp, dw, Q, nf, m0, ap.k[0], ap.k[1],
                                                                  ap.threshold, exact, dgl, dgl + kMaxLine, NG, po);
            SIEB_NOTE_LAUNCH();
            SIEB_TRY_CUDA(cudaGetLastError());
        }
        if (count > 0) {
            const double ks = NK == 1 ? ap.k[1] : ap.k[0];
            if (rot && form_a && NK == 1)
                pair_singular_n_kernel<1, true><<<near_blocks, near_threads, 0, st>>>(
                    geom, qp, dw, Q, nf, m0, list, (int)count, ks, ap.k[1], tk, dgl, dgl + kMaxLine, NG, po);
            else if (rot && form_a)
                pair_singular_n_kernel<2, true><<<near_blocks, near_threads, 0, st>>>(
                    geom, qp, dw, Q, nf, m0, list, (int)count, ks, ap.k[1], tk, dgl, dgl + kMaxLine, NG, po);
            else if (rot && NK == 1)
                pair_singular_n_kernel<1, false><<<near_blocks, near_threads, 0, st>>>(
                    geom, qp, dw, Q, nf, m0, list, (int)count, ks, ap.k[1], tk, dgl, dgl + kMaxLine, 0, po);
            else if (rot)
                pair_singular_n_kernel<2, false><<<near_blocks, near_threads, 0, st>>>(
                    geom, qp, dw, Q, nf, m0, list, (int)count, ks, ap.k[1], tk, dgl, dgl + kMaxLine, 0, po);
            else if (NK == 1)
                pair_singular_kernel<1><<<near_blocks, near_threads, 0, st>>>(geom, qp, dw, Q, nf, m0, list, (int)count,
                                                                              ks, ap.k[1], tk, false, po);
            else
                pair_singular_kernel<2><<<near_blocks, near_threads, 0, st>>>(geom, qp, dw, Q, nf, m0, list, (int)count,
                                                                              ks, ap.k[1], tk, layout == PAIR_SUM_TK,
                                                                              po);
            SIEB_NOTE_LAUNCH();
            SIEB_TRY_CUDA(cudaGetLastError());
        }
        gp.m0 = m0;
        gp.m1 = m1;
        const dim3 gb(32, 8), gg((ne + 31) / 32, (ne + 7) / 8);
        if (dx)
            gather_matvec_kernel<<<(ne + 7) / 8, 256, 0, st>>>(po.pairs, dmass, ctx->inc.as<int>(), gp, dx, dy);
        else {
            auto* gather = gp.formulation == SIEB200_PEC_EFIE
                               ? (one_slab ? gather_kernel<SIEB200_PEC_EFIE, false> : gather_kernel<SIEB200_PEC_EFIE, true>)
                           : gp.formulation == SIEB200_PMCHWT
                               ? (one_slab ? gather_kernel<SIEB200_PMCHWT, false> : gather_kernel<SIEB200_PMCHWT, true>)
                               : (one_slab ? gather_kernel<SIEB200_GSTC, false> : gather_kernel<SIEB200_GSTC, true>);
            gather<<<gg, gb, 0, st>>>(po.pairs, dmass, ctx->inc.as<int>(), gp, dZ, ldz);
        }
        SIEB_NOTE_LAUNCH();
        SIEB_TRY_CUDA(cudaGetLastError());
    }
    return SIEB200_OK;
}

int assemble_device(sieb200_ctx* ctx, const sieb200_mesh& mesh, const sieb200_options& opt,
                    const double* host_tensors, cplx* dZ, int64_t ldz) {
    return assemble_or_apply(ctx, mesh, opt, host_tensors, dZ, ldz, nullptr, nullptr);
}

int matvec_free_device(sieb200_ctx* ctx, const sieb200_mesh& mesh, const sieb200_options& opt,
                       const double* host_tensors, const cplx* dx, cplx* dy) {
    return assemble_or_apply(ctx, mesh, opt, host_tensors, nullptr, 0, dx, dy);
}

int tensor_gradient_device(sieb200_ctx* ctx, const sieb200_mesh& mesh, const sieb200_options& opt,
                           const cplx* d_lam, const cplx* d_x, cplx* d_s) {
    SIEB_CHECK(opt.formulation == SIEB200_GSTC, SIEB200_INVALID_ARG,
               "the tensor gradient exists for the GSTC formulation only");
    AssemblyParams ap;
    SIEB_RETURN_IF(make_assembly_params(opt, &ap));
    const int nf = (int)mesh.num_faces, ne = (int)mesh.num_edges;
    float pts[2 * kMaxQ], wts[kMaxQ];
    const int Q = expand_rule(opt.quadrature_rule, pts, wts);
    SIEB_CHECK(Q > 0 && Q <= kMaxQ, SIEB200_INVALID_ARG, "Dunavant quadrature rule must be in [1, 20]");
    FaceGeom* geom = nullptr;
    d3* qp = nullptr;
    float* dw = nullptr;
    int* dFE = nullptr;
    SIEB_RETURN_IF(prepare_faces(ctx, mesh, pts, wts, Q, &geom, &qp, &dw, &dFE));
    tensor_grad_kernel<<<(nf * 8 + 127) / 128, 128, 0, ctx->stream>>>(geom, qp, dw, Q, nf, ne, dFE, ap.basis,
                                                                       ap.mass_eta0, ap.mass_eta0_sq, d_lam, d_x,
                                                                       d_s);
    SIEB_NOTE_LAUNCH();
    SIEB_TRY_CUDA(cudaGetLastError());
    return SIEB200_OK;
}

// ------------------------------------------------ surface-integral fields
// The positive surface-integral terms at observation points,
//   Q_E = j w mu L[J] + K[M],   Q_H = -K[J] + j w eps L[M]
// (surface_current_fields.hpp:12-44, kernel sie_kernels_utils.cuh:21-140).

struct FieldConsts {
    cplx cJ, cM, cJh, cMh;   // j w mu, 1, -1, j w eps
    float k;                 // the wavenumber as the quadrature helpers receive it
    float k_sq_inv;          // 1 / k^2 in float
    float threshold;         // 0.1 lambda in float
};

// Per face, for the field sums: the currents' coefficients a = sum_i l_i c_i
// and aA = sum_i l_i c_i A_i (A_i = v_i - centroid, l_i the float edge length)
// for J and M, and the quadrature points about the centroid. Structure of
// arrays over `ld` >= nf faces, so that one thread per face reads coalesced:
// rows 0-2 centroid, 3-4 a_J, 5-10 aA_J, 11-12 a_M, 13-18 aA_M, then q x 3.
constexpr int kFieldRows = 19;
__global__ void field_faces_kernel(const FaceGeom* __restrict__ geom, const d3* __restrict__ qp, int Q, int nf,
                                   const cplx* __restrict__ J, const cplx* __restrict__ M, int ld,
                                   double* __restrict__ fs) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const d3 c = geom[f].c;
    const int q = blockIdx.y;
    if (q < Q) {
        const d3 r = qp[(size_t)f * Q + q] - c;
        double* o = fs + (size_t)(kFieldRows + 3 * q) * ld + f;
        o[0] = r.x; o[ld] = r.y; o[2 * (size_t)ld] = r.z;
        return;
    }
    double v[kFieldRows];
    v[0] = c.x; v[1] = c.y; v[2] = c.z;
#pragma unroll
    for (int e = 3; e < kFieldRows; ++e) v[e] = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double el = (double)(float)geom[f].len[i];
        const d3 A = geom[f].A[i];
        const int ed = geom[f].edge[i];
        const cplx a[2] = {J[ed] * el, M ? M[ed] * el : cx(0, 0)};
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            double* o = v + 3 + 8 * t;
            o[0] += a[t].re; o[1] += a[t].im;
            o[2] += a[t].re * A.x; o[3] += a[t].im * A.x;
            o[4] += a[t].re * A.y; o[5] += a[t].im * A.y;
            o[6] += a[t].re * A.z; o[7] += a[t].im * A.z;
        }
    }
#pragma unroll
    for (int e = 0; e < kFieldRows; ++e) fs[(size_t)e * ld + f] = v[e];
}

// E and H of one face's quadrature sums S0 = sum w G, Sq = sum w G q,
// T0 = sum w g, Tq = sum w g q (grad G = g R, R = r - r_q, P = r - centroid).
// With TR = T0 P - Tq and KP = Tq x P, both linear in the edge currents:
//   L = 1/2 (a Sq - S0 aA) - a TR / k^2,  K = 1/2 (a KP - aA x TR).
__device__ __forceinline__ void add_face_fields(const PointSums<1, 1>& I, d3 P, const double (&v)[kFieldRows],
                                                const FieldConsts& fc, cplx (&e)[3], cplx (&h)[3]) {
    const cplx TR[3] = {I.T0[0] * P.x - I.Tq[0][0], I.T0[0] * P.y - I.Tq[0][1], I.T0[0] * P.z - I.Tq[0][2]};
    const cplx KP[3] = {I.Tq[0][1] * P.z - I.Tq[0][2] * P.y, I.Tq[0][2] * P.x - I.Tq[0][0] * P.z,
                        I.Tq[0][0] * P.y - I.Tq[0][1] * P.x};
    const double ik2 = (double)fc.k_sq_inv;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const double* u = v + 3 + 8 * t;
        const cplx a = cx(u[0], u[1]);
        const cplx aA[3] = {cx(u[2], u[3]), cx(u[4], u[5]), cx(u[6], u[7])};
        cplx L[3], K[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            L[c] = a * (I.Sq[0][c] * 0.5 - TR[c] * ik2) - (I.S0[0] * aA[c]) * 0.5;
            const int c1 = c == 2 ? 0 : c + 1, c2 = c == 0 ? 2 : c - 1;
            K[c] = (a * KP[c] - (aA[c1] * TR[c2] - aA[c2] * TR[c1])) * 0.5;
        }
        const cplx cE_L = fc.cJ, cH_K = fc.cJh, cE_K = fc.cM, cH_L = fc.cMh;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            e[c] += t == 0 ? cE_L * L[c] : cE_K * K[c];
            h[c] += t == 0 ? cH_K * K[c] : cH_L * L[c];
        }
    }
}

// Analytic (Wilton) part of a near face (dunavant_quadrature.cuh:1719-1770).
__device__ void add_near_fields(const FaceGeom& g, d3 r, const cplx* __restrict__ J, const cplx* __restrict__ M,
                                const FieldConsts& fc, cplx (&e)[3], cplx (&h)[3]) {
    const float A = (float)g.area;
    const float base = __fdiv_rn(1.0f, __fmul_rn(__fmul_rn(8.0f, (float)kPi), A));
    const Pots P = wilton(r, g.v);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const d3 fv = g.fv[i];
        const d3 Rf = r - fv;
        const d3 phi3 = P.phi3b + (P.r_pi - fv) * P.phi2;
        const d3 Lin = (psi1(P, fv) - (Rf * 0.5) * P.phi0) + (phi3 - Rf * P.phi2) * (double)fc.k_sq_inv;
        const d3 Kv = upsilon(P, fv, r, fc.k);
        const double ls = (double)__fmul_rn((float)g.len[i], base);
        const d3 Lv = Lin * (2.0 * ls), Kl = Kv * ls;
        const double lc[3] = {Lv.x, Lv.y, Lv.z}, kc[3] = {Kl.x, Kl.y, Kl.z};
        const int ed = g.edge[i];
        const cplx je = J[ed], me = M ? M[ed] : cx(0, 0);
        const cplx wEJ = fc.cJ * je, wEM = fc.cM * me, wHJ = fc.cJh * je, wHM = fc.cMh * me;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            e[c] += wEJ * lc[c] + wEM * kc[c];
            h[c] += wHJ * kc[c] + wHM * lc[c];
        }
    }
}

// One CTA per observation point and face chunk (blockIdx.y), one thread per
// face; the chunk's E and H go to part[point][chunk][12], or with one chunk to E and H
// themselves. Bound: the FP64
// pipe, 52 instructions per kernel value (the sums are those of the assembly,
// so the three half-RWG integrals cost nothing per value). A face whose
// centroid is within 0.1 lambda of the point takes the extracted kernel
// (green_functions_utils.cuh:142-221) and the analytic part instead.
constexpr int kFieldThreads = 128;
template <bool BIG>
__global__ void __launch_bounds__(kFieldThreads, 4)
surface_fields_kernel(const FaceGeom* __restrict__ geom, const d3* __restrict__ qp, const RuleWeights rw, int Q, int nf,
                      const double* __restrict__ fs, int ld, int faces_per_chunk, const d3* __restrict__ obs,
                      const cplx* __restrict__ J, const cplx* __restrict__ M, const FieldConsts fc, const Wave wave,
                      double* __restrict__ part, double* __restrict__ E, double* __restrict__ H) {
    __shared__ __align__(16) double2 tab[kTurn * kTurnCopies];
    __shared__ double red[kFieldThreads / 32][12];
    fill_turn_table(tab);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double2* my_tab = tab + (lane & (kTurnCopies - 1));
    const d3 r = obs[blockIdx.x];
    cplx e[3] = {cx(0, 0), cx(0, 0), cx(0, 0)}, h[3] = {cx(0, 0), cx(0, 0), cx(0, 0)};
    const int f0 = blockIdx.y * faces_per_chunk, f1 = min(nf, f0 + faces_per_chunk);
    for (int fb = f0 + 32 * warp; fb < f1; fb += kFieldThreads) {  // warp-uniform
        const int f = fb + lane;
        const bool have = f < f1;
        const double* col = fs + (have ? f : f1 - 1);
        const d3 c = mk3(col[0], col[ld], col[2 * (size_t)ld]);
        // float distance from the centroid, formed without contraction
        const double dx = __dsub_rn(r.x, c.x), dy = __dsub_rn(r.y, c.y), dz = __dsub_rn(r.z, c.z);
        const float dist = (float)__dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)),
                                                       __dmul_rn(dz, dz)));
        const bool near = have && dist < fc.threshold;
        const d3 P = mk3(dx, dy, dz);
        PointSums<1, 1> in;
        in.clear();
        if (have && !near) {
            const double* qc = col + (size_t)kFieldRows * ld;
#pragma unroll 2
            for (int q = 0; q < Q; ++q, qc += 3 * (size_t)ld) {
                const double qx = qc[0], qy = qc[ld], qz = qc[2 * (size_t)ld];
                const double ax = P.x - qx, ay = P.y - qy, az = P.z - qz;
                const double R2 = fma(az, az, fma(ay, ay, ax * ax));
                double inv = rsqrt_refined(R2);
                if (tiny_square(R2)) inv = 0.0;  // R < 1e-12: no contribution
                const double R = R2 * inv;
                const double W = inv * rw.w4[q], v = wave.k * inv, i2 = inv * inv;
                double cs, sn;
                if (BIG) sincos(wave.k * R, &sn, &cs);
                else phase_cs(my_tab, wave, R, cs, sn);
                const cplx G[1] = {cx(cs * W, -sn * W)};
                const cplx g[1] = {cx(fma(i2, G[0].re, -(v * G[0].im)), fma(i2, G[0].im, v * G[0].re))};
                in.add(G, g, qx, qy, qz);
            }
        }
        // Near faces: few against the rule's points, the warp takes them one after
        // the other, lanes over the points; many, every lane its own.
        unsigned todo = __ballot_sync(0xffffffffu, near);
        auto near_point = [&](int fn, int q, PointSums<1, 1>& s) {
            const double* qc = fs + fn + (size_t)(kFieldRows + 3 * q) * ld;
            const d3 Rv = r - qp[(size_t)fn * Q + q];
            const double R = sqrt(Rv.x * Rv.x + Rv.y * Rv.y + Rv.z * Rv.z);
            cplx G[1], g[1];
            if (R < 1e-6) {
                G[0] = cx(0.0, -wave.k / (4.0 * kPi));
                g[0] = cx(0.0, 0.0);
            } else {
                green_reg(R, wave.k, G[0], g[0]);
            }
            G[0] = G[0] * rw.w[q];
            g[0] = g[0] * rw.w[q];
            s.add(G, g, qc[0], qc[ld], qc[2 * (size_t)ld]);
        };
        if (__popc(todo) * ((Q + 31) / 32) >= Q) {
            todo = 0;
            if (near)
#pragma unroll 1
                for (int q = 0; q < Q; ++q) near_point(f, q, in);
        }
        while (todo) {
            const int b = __ffs(todo) - 1;
            todo &= todo - 1;
            PointSums<1, 1> s;
            s.clear();
#pragma unroll 1
            for (int q = lane; q < Q; q += 32) near_point(fb + b, q, s);
            warp_sum(s.S0[0]); warp_sum(s.T0[0]);
#pragma unroll
            for (int t = 0; t < 3; ++t) { warp_sum(s.Sq[0][t]); warp_sum(s.Tq[0][t]); }
            if (lane == b) in = s;
        }
        if (have) {
            double v[kFieldRows];
#pragma unroll
            for (int t = 3; t < kFieldRows; ++t) v[t] = col[(size_t)t * ld];
            add_face_fields(in, P, v, fc, e, h);
        }
        if (near) add_near_fields(geom[f], r, J, M, fc, e, h);
    }
    double v[12] = {e[0].re, e[0].im, e[1].re, e[1].im, e[2].re, e[2].im,
                    h[0].re, h[0].im, h[1].re, h[1].im, h[2].re, h[2].im};
#pragma unroll
    for (int j = 0; j < 12; ++j) warp_sum(v[j]);
    if (lane == 0)
#pragma unroll
        for (int j = 0; j < 12; ++j) red[warp][j] = v[j];
    __syncthreads();
    if (threadIdx.x < 12) {
        double t = 0.0;
        for (int w = 0; w < kFieldThreads / 32; ++w) t += red[w][threadIdx.x];
        const int j = threadIdx.x;
        if (gridDim.y == 1) (j < 6 ? E : H)[6 * (size_t)blockIdx.x + j % 6] = t;
        else part[((size_t)blockIdx.x * gridDim.y + blockIdx.y) * 12 + j] = t;
    }
}

// Sums the chunks of each point in order: E (6 values), then H.
__global__ void surface_fields_finish_kernel(const double* __restrict__ part, int64_t nobs, int chunks,
                                             cplx* __restrict__ E, cplx* __restrict__ H) {
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nobs * 12) return;
    const int64_t p = id / 12;
    const int j = (int)(id - 12 * p);
    double t = 0.0;
    for (int c = 0; c < chunks; ++c) t += part[(p * chunks + c) * 12 + j];
    reinterpret_cast<double*>(j < 6 ? E : H)[6 * p + j % 6] = t;
}

int surface_fields_device(sieb200_ctx* ctx, const sieb200_mesh& mesh, const double* j_cur, const double* m_cur,
                          int64_t nobs, const double* points, double frequency_hz, double eps_r, double mu_r,
                          double eps0, double mu0, int rule, double* E_out, double* H_out) {
    auto fin = [](double x) { return std::isfinite(x); };
    SIEB_CHECK(frequency_hz > 0 && fin(frequency_hz), SIEB200_INVALID_ARG,
               "field-evaluation frequency must be positive and finite");
    SIEB_CHECK(eps_r > 0 && mu_r > 0 && fin(eps_r) && fin(mu_r), SIEB200_INVALID_ARG,
               "field-evaluation relative permittivity and permeability must be positive and finite");
    SIEB_CHECK(eps0 > 0 && mu0 > 0 && fin(eps0) && fin(mu0), SIEB200_INVALID_ARG,
               "field-evaluation vacuum constants must be positive and finite");
    SIEB_CHECK(rule >= 1 && rule <= 20, SIEB200_INVALID_ARG, "Dunavant quadrature rule must be in [1, 20]");
    SIEB_CHECK(nobs >= 0 && nobs < (1ll << 31), SIEB200_INVALID_ARG, "observation point count out of range");
    for (int64_t p = 0; p < nobs; ++p)
        SIEB_CHECK(fin(points[3 * p]) && fin(points[3 * p + 1]) && fin(points[3 * p + 2]), SIEB200_INVALID_ARG,
                   "non-finite observation point at index " + std::to_string(p));
    if (nobs == 0) return SIEB200_OK;
    SIEB_CHECK(mesh.num_vertices > 0 && mesh.num_faces > 0 && mesh.num_edges > 0, SIEB200_INVALID_ARG,
               "field-evaluation mesh must contain vertices, faces, and edges");
    const int nf = (int)mesh.num_faces, ne = (int)mesh.num_edges;
    float pts[2 * kMaxQ], wts[kMaxQ];
    const int Q = expand_rule(rule, pts, wts);
    SIEB_CHECK(Q > 0 && Q <= kMaxQ, SIEB200_INVALID_ARG, "Dunavant quadrature rule must be in [1, 20]");
    cudaStream_t st = ctx->stream;
    FaceGeom* geom = nullptr;
    d3* qp = nullptr;
    float* dw = nullptr;
    int* dFE = nullptr;
    SIEB_RETURN_IF(prepare_faces(ctx, mesh, pts, wts, Q, &geom, &qp, &dw, &dFE));

    // surface_current_fields.cu:96-112 (medium constants) and :255-275 (coefficients).
    const double pi = std::acos(-1.0);
    const double omega = 2.0 * pi * frequency_hz;
    const double eps = eps_r * eps0, mu = mu_r * mu0;
    const double k = omega * std::sqrt(mu * eps);
    FieldConsts fc;
    fc.cJ = cx(0.0, omega * mu);
    fc.cM = cx(1.0, 0.0);
    fc.cJh = cx(-1.0, 0.0);
    fc.cMh = cx(0.0, omega * eps);
    fc.k = (float)k;
    volatile float kf = fc.k;  // float arithmetic as written, no contraction
    fc.k_sq_inv = 1.f / (kf * kf);
    volatile float lambda = (float)((double)(2.0f * (float)M_PI) / k);
    fc.threshold = 0.1f * lambda;

    // Chunks of faces per point: some 16 CTAs per SM in all, so that few
    // points still fill the GPU and the last wave is short; at least one face
    // per thread.
    const int most = (nf + kFieldThreads - 1) / kFieldThreads;
    const int64_t want = ((int64_t)ctx->sm_count * 16 + nobs - 1) / nobs;
    const int per_chunk = kFieldThreads * (int)((most + std::min<int64_t>(most, want) - 1) / std::min<int64_t>(most, want));
    const int chunks = (nf + per_chunk - 1) / per_chunk;
    const int ld = ((nf + 31) / 32) * 32;
    DeviceBuffer buf(st);
    const size_t b_obs = sizeof(d3) * (size_t)nobs, b_cur = sizeof(cplx) * (size_t)ne;
    const size_t b_out = sizeof(cplx) * 3 * (size_t)nobs;
    const size_t b_fs = sizeof(double) * (size_t)(kFieldRows + 3 * Q) * ld;
    const size_t b_part = chunks == 1 ? 0 : sizeof(double) * 12 * (size_t)nobs * chunks;
    SIEB_RETURN_IF(buf.reserve(2 * b_cur + 2 * b_out + b_fs + b_part + b_obs));
    char* b = buf.as<char>();
    cplx* dJ = reinterpret_cast<cplx*>(b);
    cplx* dM = m_cur ? dJ + ne : nullptr;
    cplx* dE = reinterpret_cast<cplx*>(b + 2 * b_cur);
    cplx* dH = dE + 3 * (size_t)nobs;
    double* fs = reinterpret_cast<double*>(b + 2 * b_cur + 2 * b_out);
    double* part = reinterpret_cast<double*>(b + 2 * b_cur + 2 * b_out + b_fs);
    d3* dobs = reinterpret_cast<d3*>(b + 2 * b_cur + 2 * b_out + b_fs + b_part);
    SIEB_TRY_CUDA(cudaMemcpyAsync(dobs, points, b_obs, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(dJ, j_cur, b_cur, cudaMemcpyHostToDevice, st));
    if (m_cur) SIEB_TRY_CUDA(cudaMemcpyAsync(dM, m_cur, b_cur, cudaMemcpyHostToDevice, st));
    field_faces_kernel<<<dim3((unsigned)most, (unsigned)(Q + 1)), kFieldThreads, 0, st>>>(geom, qp, Q, nf, dJ, dM, ld,
                                                                                         fs);
    SIEB_NOTE_LAUNCH();
    SIEB_TRY_CUDA(cudaGetLastError());
    double far = 0.0;  // no farther than this from any point to any face
    for (int64_t i = 0; i < 3 * nobs; ++i) far = std::max(far, std::fabs(points[i]));
    for (int64_t i = 0; i < 3 * mesh.num_vertices; ++i) far = std::max(far, std::fabs(mesh.vertices[i]));
    const bool big = !((double)fc.k * 4.0 * far < kPhaseMax);
    auto* kernel = big ? surface_fields_kernel<true> : surface_fields_kernel<false>;
    kernel<<<dim3((unsigned)nobs, (unsigned)chunks), kFieldThreads, 0, st>>>(
        geom, qp, make_rule_weights(wts, Q), Q, nf, fs, ld, per_chunk, dobs, dJ, dM, fc, make_wave((double)fc.k), part,
        reinterpret_cast<double*>(dE), reinterpret_cast<double*>(dH));
    SIEB_NOTE_LAUNCH();
    SIEB_TRY_CUDA(cudaGetLastError());
    if (chunks > 1) {
        surface_fields_finish_kernel<<<(unsigned)((nobs * 12 + 255) / 256), 256, 0, st>>>(part, nobs, chunks, dE, dH);
        SIEB_NOTE_LAUNCH();
        SIEB_TRY_CUDA(cudaGetLastError());
    }
    SIEB_TRY_CUDA(cudaMemcpyAsync(E_out, dE, b_out, cudaMemcpyDeviceToHost, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(H_out, dH, b_out, cudaMemcpyDeviceToHost, st));
    SIEB_TRY_CUDA(cudaStreamSynchronize(st));
    return SIEB200_OK;
}

}  // namespace sieb200
