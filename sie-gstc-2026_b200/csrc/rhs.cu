// Right-hand sides (tested incident fields) and far-field projection.
//
// RHS reference: include/sie_mom/cuda/dunavant_quadrature.cuh:1543-1611 (RWG
// testing with float edge lengths and weights), source functors
// include/sie_mom/excitation/source_functors.cuh:14-130, placements
// src/sie_mom/solvers/pec_solver.cu:242-264 (PEC),
// src/sie_mom/solvers/dielectric/dielectric_solver.cu:399-530 (T-PMCHWT,
// N-PMCHWT, N-Muller), pec_solver.cu:365-388 (T-EFIE, N-EFIE, N-MFIE) and
// include/sie_mom/cuda/sie_kernels_utils.cuh:184-232 (SIE-GSTC). The rotated
// variants test with rho x n_m (dunavant_quadrature.cuh:1569-1593).
//
// One thread per (face, source) computes the face's three tested values;
// one thread per (edge, source) gathers the <= 2 incident faces and places
// them, so every column is produced without atomics.
//
// Far field: applications/anisotropic_gstc_sphere/plot_far_field.py:88-220.
// One thread per direction sums exp(+j k0 r_hat . r_q) over the faces of a
// chunk into per-face moments, which the face's currents turn into N and L.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "phase.cuh"

namespace sieb200 {

struct DevSource {
    int kind;  // 0 plane wave, 1 dipole
    int region;
    int is_magnetic;
    double a[3], b[3];
    double k, eta;
    // placement: rows get v_E * se and v_H * sh at offsets oe, oh (in units of
    // E; a negative offset places nothing)
    double se, sh;
    int oe, oh;
    int rotated;  // n x RWG testing (dunavant_quadrature.cuh:1569-1593)
};

namespace {

__device__ void source_fields(const DevSource& s, d3 r, cplx E[3], cplx H[3]) {
    if (s.kind == 0) {
        const d3 kh = mk3(s.b[0], s.b[1], s.b[2]);
        const double kdr = dot3(kh, r) * s.k;
        double sn, cs;
        sincos(-kdr, &sn, &cs);
        const cplx ph = cx(cs, sn);
        E[0] = ph * s.a[0];
        E[1] = ph * s.a[1];
        E[2] = ph * s.a[2];
        const double ie = 1.0 / s.eta;
        H[0] = (E[2] * kh.y - E[1] * kh.z) * ie;
        H[1] = (E[0] * kh.z - E[2] * kh.x) * ie;
        H[2] = (E[1] * kh.x - E[0] * kh.y) * ie;
        return;
    }
    const d3 p = mk3(s.a[0], s.a[1], s.a[2]);
    const d3 Rv = r - mk3(s.b[0], s.b[1], s.b[2]);
    const double R = sqrt(Rv.x * Rv.x + Rv.y * Rv.y + Rv.z * Rv.z);
    if (R < 1e-6) {
        for (int c = 0; c < 3; ++c) { E[c] = cx(0, 0); H[c] = cx(0, 0); }
        return;
    }
    const d3 Rh = mk3(Rv.x / R, Rv.y / R, Rv.z / R);
    const double Rdp = Rh.x * p.x + Rh.y * p.y + Rh.z * p.z;
    const d3 Rxp = mk3(Rh.y * p.z - Rh.z * p.y, Rh.z * p.x - Rh.x * p.z, Rh.x * p.y - Rh.y * p.x);
    const d3 tri = mk3(Rxp.y * Rh.z - Rxp.z * Rh.y, Rxp.z * Rh.x - Rxp.x * Rh.z,
                       Rxp.x * Rh.y - Rxp.y * Rh.x);
    double sn, cs;
    sincos(-s.k * R, &sn, &cs);
    const cplx ph = cx(cs, sn);
    const double t1 = (s.k * s.k) / R, t2r = 1.0 / (R * R * R), t2i = s.k / (R * R);
    const double tv[3] = {3.0 * Rh.x * Rdp - p.x, 3.0 * Rh.y * Rdp - p.y, 3.0 * Rh.z * Rdp - p.z};
    const double trc[3] = {tri.x, tri.y, tri.z};
    const double rxp[3] = {Rxp.x, Rxp.y, Rxp.z};
    const cplx hc = cx(-(s.k * s.k) / (s.eta * R), s.k / (s.eta * R * R)) * ph;
    for (int c = 0; c < 3; ++c) {
        const cplx Ec = cx(t1 * trc[c] + tv[c] * t2r, tv[c] * t2i) * ph;
        const cplx Hc = cx(hc.re * -rxp[c], hc.im * -rxp[c]);
        if (s.is_magnetic) {
            E[c] = cx(Hc.re * -s.eta, Hc.im * -s.eta);
            H[c] = cx(Ec.re / s.eta, Ec.im / s.eta);
        } else {
            E[c] = Ec;
            H[c] = Hc;
        }
    }
}

__global__ void rhs_face_kernel(const double* __restrict__ V, const int* __restrict__ F, int nf,
                                const float* __restrict__ qpts, const float* __restrict__ qw,
                                int Q, const DevSource* __restrict__ src, int nsrc,
                                cplx* __restrict__ out) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = blockIdx.y;
    if (f >= nf || s >= nsrc) return;
    const DevSource S = src[s];
    int idx[3];
    d3 v[3];
    for (int a = 0; a < 3; ++a) {
        idx[a] = F[3 * f + a];
        v[a] = mk3(V[3 * idx[a]], V[3 * idx[a] + 1], V[3 * idx[a] + 2]);
    }
    const int EA[3] = {0, 1, 2}, EB[3] = {1, 2, 0}, EF[3] = {2, 0, 1};
    float el[3];
    d3 fv[3];
    d3 nm = mk3(0, 0, 0);
    if (S.rotated) {
        const d3 cr = cross3(v[1] - v[0], v[2] - v[0]);
        nm = cr * (1.0 / sqrt(dot3(cr, cr)));
    }
    for (int e = 0; e < 3; ++e) {
        const d3 ev = v[EB[e]] - v[EA[e]];
        const double l = sqrt(ev.x * ev.x + ev.y * ev.y + ev.z * ev.z);
        el[e] = (float)((idx[EA[e]] > idx[EB[e]] ? 1.0 : -1.0) * l);
        fv[e] = v[EF[e]];
    }
    cplx ve[3] = {cx(0, 0), cx(0, 0), cx(0, 0)}, vh[3] = {cx(0, 0), cx(0, 0), cx(0, 0)};
    for (int p = 0; p < Q; ++p) {
        const double wp = (double)qw[p];
        const double xi = (double)qpts[2 * p], eta = (double)qpts[2 * p + 1];
        const double zeta = 1.0 - xi - eta;
        const d3 rp = mk3(v[0].x * zeta + v[1].x * xi + v[2].x * eta,
                          v[0].y * zeta + v[1].y * xi + v[2].y * eta,
                          v[0].z * zeta + v[1].z * xi + v[2].z * eta);
        cplx E[3], H[3];
        source_fields(S, rp, E, H);
        for (int i = 0; i < 3; ++i) {
            const d3 t = S.rotated ? cross3(rp - fv[i], nm) : rp - fv[i];
            const cplx de = cx(t.x * E[0].re + t.y * E[1].re + t.z * E[2].re,
                               t.x * E[0].im + t.y * E[1].im + t.z * E[2].im);
            const cplx dh = cx(t.x * H[0].re + t.y * H[1].re + t.z * H[2].re,
                               t.x * H[0].im + t.y * H[1].im + t.z * H[2].im);
            ve[i] += de * wp;
            vh[i] += dh * wp;
        }
    }
    cplx* o = out + ((size_t)s * nf + f) * 6;
    for (int i = 0; i < 3; ++i) {
        const double sc = (double)__fmul_rn(0.5f, el[i]);
        o[i] = ve[i] * sc;
        o[3 + i] = vh[i] * sc;
    }
}

// Incident E and H of one source at observation points
// (compute_incident_field_kernel, src/sie_mom/excitation/excitation.cu:140-156):
// the same source functors as the right-hand sides, one thread per point.
__global__ void incident_fields_kernel(const double* __restrict__ pts, int64_t n, const DevSource* __restrict__ src,
                                       cplx* __restrict__ E, cplx* __restrict__ H) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const DevSource S = *src;
    cplx e[3], h[3];
    source_fields(S, mk3(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]), e, h);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        E[3 * i + c] = e[c];
        H[3 * i + c] = h[c];
    }
}

__global__ void rhs_gather_kernel(const cplx* __restrict__ face_vals, const int* __restrict__ inc,
                                  int nf, int ne, const DevSource* __restrict__ src, int nsrc,
                                  int64_t N, cplx* __restrict__ B, int64_t ldb) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = blockIdx.y;
    if (e >= ne || s >= nsrc) return;
    const DevSource S = src[s];
    cplx ve = cx(0, 0), vh = cx(0, 0);
    for (int a = 0; a < 2; ++a) {
        const int fi = inc[2 * e + a];
        if (fi < 0) continue;
        const int f = fi / 3, le = fi - 3 * f;
        const cplx* o = face_vals + ((size_t)s * nf + f) * 6;
        ve += o[le];
        vh += o[3 + le];
    }
    cplx* col = B + (int64_t)s * ldb;
    // Column zeroing happens before launch; each (row) is owned by one thread.
    if (S.oe >= 0) col[e + (int64_t)S.oe * ne] = ve * S.se;
    if (S.oh >= 0) col[e + (int64_t)S.oh * ne] = vh * S.sh;
}

// ------------------------------------------------------------ far field --
// The 7-point rule of plot_far_field.py:88-115 (double): centroid, then two
// 3-orbits.
struct FarRule {
    double xi[7], eta[7], w[7];
};
FarRule far_rule() {
    const double s15 = std::sqrt(15.0);
    const double a1 = (6.0 - s15) / 21.0, w1 = (155.0 - s15) / 1200.0;
    const double a2 = (6.0 + s15) / 21.0, w2 = (155.0 + s15) / 1200.0;
    return FarRule{{1.0 / 3.0, a1, 1.0 - 2.0 * a1, a1, a2, 1.0 - 2.0 * a2, a2},
                   {1.0 / 3.0, a1, a1, 1.0 - 2.0 * a1, a2, a2, 1.0 - 2.0 * a2},
                   {0.225, w1, w1, w1, w2, w2, w2}};
}

// Face record of the far-field sums (kFarRow doubles): centroid c; for J and
// for M a = 1/2 sum_i l_i c_i and aA = 1/2 sum_i l_i c_i A_i (A_i = v_i - c);
// the 7 points about c. With S0 = sum w e and Sq = sum w e q over the points
// (e = exp(j k0 r_hat . r_q)) the face adds a Sq - aA S0 to N (J) and L (M).
constexpr int kFarRow = 40;
__global__ void ff_faces_kernel(const double* __restrict__ V, const int* __restrict__ F, const int* __restrict__ FE,
                                int nf, const FarRule rule, const cplx* __restrict__ jc, const cplx* __restrict__ mc,
                                double* __restrict__ rec) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    int idx[3];
    d3 v[3];
    for (int a = 0; a < 3; ++a) {
        idx[a] = F[3 * f + a];
        v[a] = mk3(V[3 * idx[a]], V[3 * idx[a] + 1], V[3 * idx[a] + 2]);
    }
    const d3 c = (v[0] + v[1] + v[2]) * (1.0 / 3.0);
    double* o = rec + (size_t)f * kFarRow;
    o[0] = c.x; o[1] = c.y; o[2] = c.z;
    const int EA[3] = {0, 1, 2}, EB[3] = {1, 2, 0}, EF[3] = {2, 0, 1};
    cplx a[2] = {cx(0, 0), cx(0, 0)}, aA[2][3];
    for (int t = 0; t < 2; ++t)
        for (int k = 0; k < 3; ++k) aA[t][k] = cx(0, 0);
    for (int le = 0; le < 3; ++le) {
        const d3 ev = v[EB[le]] - v[EA[le]];
        const double len = (idx[EA[le]] > idx[EB[le]] ? 1.0 : -1.0) * sqrt(dot3(ev, ev));
        const int e = FE[3 * f + le];
        const d3 A = v[EF[le]] - c;
        const cplx co[2] = {jc[e] * (0.5 * len), mc ? mc[e] * (0.5 * len) : cx(0, 0)};
        for (int t = 0; t < 2; ++t) {
            a[t] += co[t];
            aA[t][0] += co[t] * A.x;
            aA[t][1] += co[t] * A.y;
            aA[t][2] += co[t] * A.z;
        }
    }
    for (int t = 0; t < 2; ++t) {
        double* u = o + 3 + 8 * t;
        u[0] = a[t].re; u[1] = a[t].im;
        for (int k = 0; k < 3; ++k) { u[2 + 2 * k] = aA[t][k].re; u[3 + 2 * k] = aA[t][k].im; }
    }
    for (int q = 0; q < 7; ++q) {
        const double xi = rule.xi[q], eta = rule.eta[q], zeta = 1.0 - xi - eta;
        const d3 r = v[0] * zeta + v[1] * xi + v[2] * eta - c;
        o[19 + 3 * q] = r.x; o[20 + 3 * q] = r.y; o[21 + 3 * q] = r.z;
    }
}

// Far-field operator as a matrix: rows (F_theta of direction d, then F_phi),
// columns (J of edge e, then M of edge e), row-major with 2*ne columns, so
// that [F_theta; F_phi] = A [J; M] with the same radiation vectors and
// coefficients as ff_faces_kernel / ff_directions_kernel. One thread per
// (direction, edge); the edge's incident faces and the 7-point rule are
// evaluated on the fly.
__global__ void ff_matrix_kernel(const double* __restrict__ V, const int* __restrict__ F,
                                 const int* __restrict__ inc, int ne, int64_t ndir, double k0, double eta0,
                                 const double* __restrict__ rh, const double* __restrict__ th,
                                 const double* __restrict__ ph, cplx* __restrict__ A) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t d = blockIdx.y;
    if (e >= ne) return;
    const double s15 = sqrt(15.0);
    const double a1 = (6.0 - s15) / 21.0, w1 = (155.0 - s15) / 1200.0;
    const double a2 = (6.0 + s15) / 21.0, w2 = (155.0 + s15) / 1200.0;
    const double nodes[7][2] = {{1.0 / 3.0, 1.0 / 3.0}, {a1, a1}, {1.0 - 2.0 * a1, a1},
                                {a1, 1.0 - 2.0 * a1}, {a2, a2}, {1.0 - 2.0 * a2, a2},
                                {a2, 1.0 - 2.0 * a2}};
    const double wq[7] = {0.225, w1, w1, w1, w2, w2, w2};
    const int EA[3] = {0, 1, 2}, EB[3] = {1, 2, 0}, EF[3] = {2, 0, 1};
    const d3 r = mk3(rh[3 * d], rh[3 * d + 1], rh[3 * d + 2]);
    cplx N[3] = {cx(0, 0), cx(0, 0), cx(0, 0)};
    for (int a = 0; a < 2; ++a) {
        const int fi = inc[2 * e + a];
        if (fi < 0) continue;
        const int f = fi / 3, le = fi - 3 * f;
        int idx[3];
        d3 v[3];
        for (int b = 0; b < 3; ++b) {
            idx[b] = F[3 * f + b];
            v[b] = mk3(V[3 * idx[b]], V[3 * idx[b] + 1], V[3 * idx[b] + 2]);
        }
        const d3 ev = v[EB[le]] - v[EA[le]];
        const double len = (idx[EA[le]] > idx[EB[le]] ? 1.0 : -1.0) * sqrt(dot3(ev, ev));
        for (int q = 0; q < 7; ++q) {
            const double xi = nodes[q][0], eta = nodes[q][1], zeta = 1.0 - xi - eta;
            const d3 rq = v[0] * zeta + v[1] * xi + v[2] * eta;
            const d3 rho = rq - v[EF[le]];
            double sn, cs;
            sincos(k0 * dot3(r, rq), &sn, &cs);
            const double wgt = 0.5 * len * wq[q];
            const cplx ph_ = cx(cs * wgt, sn * wgt);
            N[0] += ph_ * rho.x;
            N[1] += ph_ * rho.y;
            N[2] += ph_ * rho.z;
        }
    }
    const double* t = th + 3 * d;
    const double* p = ph + 3 * d;
    const cplx nt = N[0] * t[0] + N[1] * t[1] + N[2] * t[2];
    const cplx np = N[0] * p[0] + N[1] * p[1] + N[2] * p[2];
    const cplx coeff = cx(0.0, -k0 / (4.0 * 3.14159265358979323846));
    const int64_t cols = 2 * (int64_t)ne;
    A[d * cols + e] = coeff * (nt * eta0);
    A[(ndir + d) * cols + e] = coeff * (np * eta0);
    A[d * cols + ne + e] = coeff * np;
    A[(ndir + d) * cols + ne + e] = cx(0, 0) - coeff * nt;
}

// One thread per direction, blockIdx.y a chunk of faces whose records are
// staged in shared memory (all lanes read the same word). Bound: the FP64 pipe,
// 28 instructions per sample (3 for the path, 15 for the phase factor, 10 for
// the moments) and 51 per face. part: [chunk][N, L: 12][direction].
constexpr int kFarThreads = 128, kFarStage = 32;
template <bool BIG>
__global__ void __launch_bounds__(kFarThreads)
ff_directions_kernel(const double* __restrict__ rec, int nf, int faces_per_chunk, const FarRule rule, const Wave wave,
                     int64_t ndir, const double* __restrict__ rh, double* __restrict__ part) {
    __shared__ __align__(16) double2 tab[kTurn * kTurnCopies];
    __shared__ double sr[kFarStage * kFarRow];
    fill_turn_table(tab);
    const double2* my_tab = tab + (threadIdx.x & (kTurnCopies - 1));
    const int64_t d = (int64_t)blockIdx.x * kFarThreads + threadIdx.x;
    const int64_t dd = d < ndir ? d : ndir - 1;
    const d3 r = mk3(rh[3 * dd], rh[3 * dd + 1], rh[3 * dd + 2]);
    cplx acc[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[c] = cx(0, 0);
    const int f1 = min(nf, (int)(blockIdx.y + 1) * faces_per_chunk);
    for (int f0 = blockIdx.y * faces_per_chunk; f0 < f1; f0 += kFarStage) {
        const int n = min(kFarStage, f1 - f0);
        __syncthreads();
        for (int t = threadIdx.x; t < n * kFarRow; t += kFarThreads) sr[t] = rec[(size_t)f0 * kFarRow + t];
        __syncthreads();
        for (int f = 0; f < n; ++f) {
            const double* o = sr + f * kFarRow;
            const double x0 = r.x * o[0] + r.y * o[1] + r.z * o[2];
            cplx S0 = cx(0, 0), Sq[3] = {cx(0, 0), cx(0, 0), cx(0, 0)};
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                const double qx = o[19 + 3 * q], qy = o[20 + 3 * q], qz = o[21 + 3 * q];
                const double x = fma(r.x, qx, fma(r.y, qy, fma(r.z, qz, x0)));
                double c, s;
                if (BIG) sincos(wave.k * x, &s, &c);
                else phase_cs(my_tab, wave, x, c, s);
                const cplx e = cx(c * rule.w[q], s * rule.w[q]);
                S0 += e;
                Sq[0].re = fma(e.re, qx, Sq[0].re); Sq[0].im = fma(e.im, qx, Sq[0].im);
                Sq[1].re = fma(e.re, qy, Sq[1].re); Sq[1].im = fma(e.im, qy, Sq[1].im);
                Sq[2].re = fma(e.re, qz, Sq[2].re); Sq[2].im = fma(e.im, qz, Sq[2].im);
            }
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const double* u = o + 3 + 8 * t;
                const cplx a = cx(u[0], u[1]);
#pragma unroll
                for (int c = 0; c < 3; ++c) acc[3 * t + c] += a * Sq[c] - cx(u[2 + 2 * c], u[3 + 2 * c]) * S0;
            }
        }
    }
    if (d >= ndir) return;
    double* o = part + (size_t)blockIdx.y * 12 * ndir + d;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        o[(2 * c) * ndir] = acc[c].re;
        o[(2 * c + 1) * ndir] = acc[c].im;
    }
}

// Sums the chunks of each direction in order and projects N and L: a thread per
// direction and component, then one per direction. Latency: with all 12 components in
// a thread, 96 bytes from its neighbour's, 181 directions in 64 chunks took 36 us;
// the loads of neighbours now lie side by side, eight chunks in flight: 5.5 us.
constexpr int kFinishDirs = 32;
__global__ void __launch_bounds__(12 * kFinishDirs) ff_finish_kernel(const double* __restrict__ part, int chunks, int64_t ndir, double k0, double eta0,
                                 const double* __restrict__ th, const double* __restrict__ ph, cplx* __restrict__ ft,
                                 cplx* __restrict__ fp, double* __restrict__ U) {
    __shared__ double s[12][kFinishDirs];
    const int64_t d = (int64_t)blockIdx.x * kFinishDirs + threadIdx.x;
    if (d < ndir) {
        const double* o = part + (size_t)threadIdx.y * ndir + d;
        double sum = 0.0;
#pragma unroll 8
        for (int k = 0; k < chunks; ++k) sum += o[(size_t)k * 12 * ndir];
        s[threadIdx.y][threadIdx.x] = sum;
    }
    __syncthreads();
    if (threadIdx.y != 0 || d >= ndir) return;
    double v[12];
#pragma unroll
    for (int c = 0; c < 12; ++c) v[c] = s[c][threadIdx.x];
    const cplx Nv[3] = {cx(v[0], v[1]), cx(v[2], v[3]), cx(v[4], v[5])};
    const cplx Lv[3] = {cx(v[6], v[7]), cx(v[8], v[9]), cx(v[10], v[11])};
    const double* t = th + 3 * d;
    const double* p = ph + 3 * d;
    const cplx nt = Nv[0] * t[0] + Nv[1] * t[1] + Nv[2] * t[2];
    const cplx np = Nv[0] * p[0] + Nv[1] * p[1] + Nv[2] * p[2];
    const cplx lt = Lv[0] * t[0] + Lv[1] * t[1] + Lv[2] * t[2];
    const cplx lp = Lv[0] * p[0] + Lv[1] * p[1] + Lv[2] * p[2];
    const cplx coeff = cx(0.0, -k0 / (4.0 * 3.14159265358979323846));
    const cplx a = coeff * (nt * eta0 + lp);
    const cplx b = coeff * (np * eta0 - lt);
    ft[d] = a;
    fp[d] = b;
    U[d] = (a.re * a.re + a.im * a.im + b.re * b.re + b.im * b.im) / (2.0 * eta0);
}

}  // namespace

// Host: physical constants of one source, bound from its region's medium
// (src/sie_mom/excitation/excitation.cu:110-137) and the formulation's
// placement scales.
int prepare_sources(const sieb200_options& opt, const sieb200_source* sources, int nsrc,
                    std::vector<DevSource>* out) {
    const double pi = std::acos(-1.0);
    out->clear();
    for (int s = 0; s < nsrc; ++s) {
        const sieb200_source& in = sources[s];
        DevSource d{};
        SIEB_CHECK(in.kind == 0 || in.kind == 1, SIEB200_INVALID_ARG, "source kind must be 0 (plane wave) or 1 (dipole)");
        SIEB_CHECK(in.region == 1 || in.region == 2, SIEB200_INVALID_ARG, "source region must be interior or exterior");
        const double eps_r = in.region == 1 ? opt.eps_r_interior : opt.eps_r_exterior;
        const double mu_r = in.region == 1 ? opt.mu_r_interior : opt.mu_r_exterior;
        SIEB_CHECK(eps_r > 0 && mu_r > 0, SIEB200_INVALID_ARG, "source relative permittivity and permeability must be positive");
        const double eps = eps_r * opt.vacuum_permittivity, mu = mu_r * opt.vacuum_permeability;
        const double omega = 2.0 * pi * opt.frequency_hz;
        d.k = omega * std::sqrt(mu * eps);
        d.eta = std::sqrt(mu / eps);
        d.kind = in.kind;
        d.region = in.region;
        d.is_magnetic = in.is_magnetic;
        for (int c = 0; c < 3; ++c) { d.a[c] = in.a[c]; d.b[c] = in.b[c]; }
        for (int c = 0; c < 3; ++c)
            SIEB_CHECK(std::isfinite(in.a[c]) && std::isfinite(in.b[c]), SIEB200_INVALID_ARG,
                       "source vectors must be finite");
        if (in.kind == 0) {
            // excitation.cu:45-60: unit direction, transverse amplitude.
            const double dn = std::hypot(in.b[0], in.b[1], in.b[2]);
            const double an = std::hypot(in.a[0], in.a[1], in.a[2]);
            SIEB_CHECK(dn > 0 && std::isfinite(dn), SIEB200_INVALID_ARG, "plane-wave direction magnitude must be positive and finite");
            SIEB_CHECK(an > 0 && std::isfinite(an), SIEB200_INVALID_ARG, "plane-wave amplitude magnitude must be positive and finite");
            for (int c = 0; c < 3; ++c) d.b[c] = in.b[c] / dn;
            const double lf = d.b[0] * in.a[0] / an + d.b[1] * in.a[1] / an + d.b[2] * in.a[2] / an;
            SIEB_CHECK(std::abs(lf) <= 64.0 * 2.220446049250313e-16, SIEB200_INVALID_ARG,
                       "plane-wave electric amplitude must be transverse to propagation");
        } else {
            const double mn = std::hypot(in.a[0], in.a[1], in.a[2]);
            SIEB_CHECK(mn > 0 && std::isfinite(mn), SIEB200_INVALID_ARG, "dipole moment magnitude must be positive and finite");
        }
        d.rotated = opt.variant != SIEB200_VARIANT_T;
        if (opt.formulation == SIEB200_PEC_EFIE) {
            SIEB_CHECK(in.region == 2, SIEB200_INVALID_ARG, "PEC solver requires an exterior (region 2) source");
            if (opt.variant == SIEB200_VARIANT_N_JUMP) {
                // N-MFIE: +<f x n, H_inc> (pec_solver.cu:372-377).
                d.se = 0.0; d.sh = 1.0; d.oe = -1; d.oh = 0;
            } else {
                d.se = 1.0; d.sh = 0.0; d.oe = 0; d.oh = -1;
            }
        } else if (opt.formulation == SIEB200_PMCHWT && opt.variant == SIEB200_VARIANT_N_JUMP) {
            // N-Muller: eps V_E and -mu eta0 V_H of the source region
            // (dielectric_solver.cu:461-489).
            const double eta0 = std::sqrt(opt.vacuum_permeability / opt.vacuum_permittivity);
            d.se = eps_r * opt.vacuum_permittivity;
            d.sh = -(mu_r * opt.vacuum_permeability) * eta0;
            d.oe = 0; d.oh = 1;
        } else if (opt.formulation == SIEB200_PMCHWT) {
            const double eta0 = std::sqrt(opt.vacuum_permeability / opt.vacuum_permittivity);
            const double sign = in.region == 2 ? 1.0 : -1.0;
            d.se = sign; d.sh = sign * eta0; d.oe = 0; d.oh = 1;
        } else {
            const float mu0f = (float)opt.vacuum_permeability, eps0f = (float)opt.vacuum_permittivity;
            const double eta0 = std::sqrt((double)mu0f / (double)eps0f);
            d.se = 1.0; d.sh = eta0;
            d.oe = in.region == 1 ? 0 : 2;
            d.oh = d.oe + 1;
        }
        out->push_back(d);
    }
    return SIEB200_OK;
}

int assemble_rhs_device(sieb200_ctx* ctx, const sieb200_mesh& mesh, const sieb200_options& opt,
                        const sieb200_source* sources, int nsrc, cplx* dB, int64_t ldb) {
    std::vector<DevSource> ds;
    SIEB_RETURN_IF(prepare_sources(opt, sources, nsrc, &ds));
    const int nf = (int)mesh.num_faces, ne = (int)mesh.num_edges, nv = (int)mesh.num_vertices;
    const int64_t N = system_dimension(opt.formulation, ne);
    float pts[160], wts[80];
    const int Q = expand_rule(opt.quadrature_rule, pts, wts);
    SIEB_CHECK(Q > 0, SIEB200_INVALID_ARG, "Dunavant quadrature rule must be in [1, 20]");
    cudaStream_t st = ctx->stream;
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
    const size_t vbytes = sizeof(double) * 3 * nv, fbytes = sizeof(int) * 3 * nf;
    const size_t ibytes = sizeof(int) * inc.size();
    const size_t sbytes = sizeof(DevSource) * nsrc;
    const size_t off_f = ((vbytes + 255) / 256) * 256;
    const size_t off_i = off_f + ((fbytes + 255) / 256) * 256;
    const size_t off_s = off_i + ((ibytes + 255) / 256) * 256;
    const size_t off_q = off_s + ((sbytes + 255) / 256) * 256;
    SIEB_RETURN_IF(ctx->srcbuf.reserve(off_q + sizeof(float) * 240));
    char* base = ctx->srcbuf.as<char>();
    double* dV = reinterpret_cast<double*>(base);
    int* dF = reinterpret_cast<int*>(base + off_f);
    int* dinc = reinterpret_cast<int*>(base + off_i);
    DevSource* dsrc = reinterpret_cast<DevSource*>(base + off_s);
    float* dq = reinterpret_cast<float*>(base + off_q);
    SIEB_TRY_CUDA(cudaMemcpyAsync(dV, mesh.vertices, vbytes, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(dF, mesh.faces, fbytes, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(dinc, inc.data(), ibytes, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(dsrc, ds.data(), sbytes, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(dq, pts, sizeof(float) * 2 * Q, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(dq + 160, wts, sizeof(float) * Q, cudaMemcpyHostToDevice, st));
    SIEB_RETURN_IF(ctx->rhsbuf.reserve(sizeof(cplx) * 6 * (size_t)nf * nsrc));
    SIEB_TRY_CUDA(cudaMemset2DAsync(dB, sizeof(cplx) * ldb, 0, sizeof(cplx) * N, nsrc, st));
    rhs_face_kernel<<<dim3((nf + 127) / 128, nsrc), 128, 0, st>>>(dV, dF, nf, dq, dq + 160, Q, dsrc,
                                                                  nsrc, ctx->rhsbuf.as<cplx>());
    SIEB_NOTE_LAUNCH();
    SIEB_TRY_CUDA(cudaGetLastError());
    rhs_gather_kernel<<<dim3((ne + 127) / 128, nsrc), 128, 0, st>>>(
        ctx->rhsbuf.as<cplx>(), dinc, nf, ne, dsrc, nsrc, N, dB, ldb);
    SIEB_NOTE_LAUNCH();
    SIEB_TRY_CUDA(cudaGetLastError());
    return SIEB200_OK;
}

// evaluate_incident_fields (src/sie_mom/excitation/excitation.cu:158-210):
// host points in, host E and H (3 complex per point) out; the source's k and
// eta are bound from its region's medium as for the right-hand sides.
int incident_fields_device(sieb200_ctx* ctx, const sieb200_options& opt, const sieb200_source& source, int64_t n,
                           const double* points, double* E_out, double* H_out) {
    std::vector<DevSource> ds;
    SIEB_RETURN_IF(prepare_sources(opt, &source, 1, &ds));
    for (int64_t i = 0; i < 3 * n; ++i)
        SIEB_CHECK(std::isfinite(points[i]), SIEB200_INVALID_ARG, "incident-field observation point must be finite");
    if (n == 0) return SIEB200_OK;
    cudaStream_t st = ctx->stream;
    const size_t pbytes = sizeof(double) * 3 * (size_t)n, fbytes = sizeof(cplx) * 3 * (size_t)n;
    const size_t off_s = ((pbytes + 255) / 256) * 256;
    const size_t off_e = off_s + 256, off_h = off_e + ((fbytes + 255) / 256) * 256;
    DeviceBuffer buf(st);
    SIEB_RETURN_IF(buf.reserve(off_h + fbytes));
    char* b = buf.as<char>();
    SIEB_TRY_CUDA(cudaMemcpyAsync(b, points, pbytes, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(b + off_s, ds.data(), sizeof(DevSource), cudaMemcpyHostToDevice, st));
    incident_fields_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        reinterpret_cast<const double*>(b), n, reinterpret_cast<const DevSource*>(b + off_s),
        reinterpret_cast<cplx*>(b + off_e), reinterpret_cast<cplx*>(b + off_h));
    SIEB_NOTE_LAUNCH();
    SIEB_TRY_CUDA(cudaGetLastError());
    SIEB_TRY_CUDA(cudaMemcpyAsync(E_out, b + off_e, fbytes, cudaMemcpyDeviceToHost, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(H_out, b + off_h, fbytes, cudaMemcpyDeviceToHost, st));
    SIEB_TRY_CUDA(cudaStreamSynchronize(st));
    return SIEB200_OK;
}

int far_field_device(sieb200_ctx* ctx, const sieb200_mesh& mesh, const double* j_cur,
                     const double* m_cur, double k0, double eta0, int64_t ndir, const double* rh,
                     const double* th, const double* ph, double* f_theta, double* f_phi,
                     double* intensity) {
    const int nf = (int)mesh.num_faces, ne = (int)mesh.num_edges, nv = (int)mesh.num_vertices;
    cudaStream_t st = ctx->stream;
    // Chunks of faces: some 16 CTAs per SM in all, whole staging rounds each; small
    // meshes are cut finer, into up to 64 chunks, since a thread runs through its
    // chunk's samples one after the other (320 faces, 181 directions: 20.4 us in
    // chunks of 32, 5.4 us in chunks of 5).
    const int64_t dir_blocks = std::max<int64_t>(1, (ndir + kFarThreads - 1) / kFarThreads);
    const int64_t want = ((int64_t)ctx->sm_count * 16 + dir_blocks - 1) / dir_blocks;
    const int unit = std::min(kFarStage, std::max(4, (nf + 63) / 64));
    const int rounds = (nf + unit - 1) / unit;
    const int64_t split = std::min<int64_t>(rounds, want);
    const int per_chunk = unit * (int)((rounds + split - 1) / split);
    const int chunks = (nf + per_chunk - 1) / per_chunk;
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off += ((bytes + 255) / 256) * 256; return o; };
    const size_t oV = take(sizeof(double) * 3 * nv), oF = take(sizeof(int) * 3 * nf),
                 oFE = take(sizeof(int) * 3 * nf), oJ = take(sizeof(cplx) * ne),
                 oM = take(sizeof(cplx) * ne), oRec = take(sizeof(double) * kFarRow * nf),
                 oPart = take(sizeof(double) * 12 * (size_t)chunks * ndir),
                 oDir = take(sizeof(double) * 9 * ndir), oOut = take(sizeof(cplx) * 2 * ndir),
                 oU = take(sizeof(double) * ndir);
    DeviceBuffer buf(st);
    SIEB_RETURN_IF(buf.reserve(off));
    char* b = buf.as<char>();
    double* rec = reinterpret_cast<double*>(b + oRec);
    double* part = reinterpret_cast<double*>(b + oPart);
    SIEB_TRY_CUDA(cudaMemcpyAsync(b + oV, mesh.vertices, sizeof(double) * 3 * nv, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(b + oF, mesh.faces, sizeof(int) * 3 * nf, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(b + oFE, mesh.faces_edges, sizeof(int) * 3 * nf, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(b + oJ, j_cur, sizeof(cplx) * ne, cudaMemcpyHostToDevice, st));
    if (m_cur) SIEB_TRY_CUDA(cudaMemcpyAsync(b + oM, m_cur, sizeof(cplx) * ne, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(b + oDir, rh, sizeof(double) * 3 * ndir, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(b + oDir + sizeof(double) * 3 * ndir, th, sizeof(double) * 3 * ndir, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(b + oDir + sizeof(double) * 6 * ndir, ph, sizeof(double) * 3 * ndir, cudaMemcpyHostToDevice, st));
    const FarRule rule = far_rule();
    ff_faces_kernel<<<(nf + 127) / 128, 128, 0, st>>>(
        reinterpret_cast<double*>(b + oV), reinterpret_cast<int*>(b + oF), reinterpret_cast<int*>(b + oFE), nf, rule,
        reinterpret_cast<cplx*>(b + oJ), m_cur ? reinterpret_cast<cplx*>(b + oM) : nullptr, rec);
    SIEB_NOTE_LAUNCH();
    SIEB_TRY_CUDA(cudaGetLastError());
    if (ndir > 0) {
        double* dd = reinterpret_cast<double*>(b + oDir);
        // |r_hat . r_q| is at most |r_hat| times the sum of the largest coordinates
        double ext = 0.0, rmax = 0.0;
        for (int64_t i = 0; i < 3 * (int64_t)nv; ++i) ext = std::max(ext, std::fabs(mesh.vertices[i]));
        for (int64_t i = 0; i < 3 * ndir; ++i) rmax = std::max(rmax, std::fabs(rh[i]));
        const bool big = !(k0 * 3.0 * ext * rmax < kPhaseMax);
        auto* kernel = big ? ff_directions_kernel<true> : ff_directions_kernel<false>;
        kernel<<<dim3((unsigned)dir_blocks, (unsigned)chunks), kFarThreads, 0, st>>>(rec, nf, per_chunk, rule,
                                                                                     make_wave(k0), ndir, dd, part);
        SIEB_NOTE_LAUNCH();
        SIEB_TRY_CUDA(cudaGetLastError());
        ff_finish_kernel<<<(unsigned)((ndir + kFinishDirs - 1) / kFinishDirs), dim3(kFinishDirs, 12), 0, st>>>(
            part, chunks, ndir, k0, eta0, dd + 3 * ndir, dd + 6 * ndir, reinterpret_cast<cplx*>(b + oOut),
            reinterpret_cast<cplx*>(b + oOut) + ndir, reinterpret_cast<double*>(b + oU));
        SIEB_NOTE_LAUNCH();
        SIEB_TRY_CUDA(cudaGetLastError());
        SIEB_TRY_CUDA(cudaMemcpyAsync(f_theta, b + oOut, sizeof(cplx) * ndir, cudaMemcpyDeviceToHost, st));
        SIEB_TRY_CUDA(cudaMemcpyAsync(f_phi, b + oOut + sizeof(cplx) * ndir, sizeof(cplx) * ndir, cudaMemcpyDeviceToHost, st));
        SIEB_TRY_CUDA(cudaMemcpyAsync(intensity, b + oU, sizeof(double) * ndir, cudaMemcpyDeviceToHost, st));
    }
    SIEB_TRY_CUDA(cudaStreamSynchronize(st));
    return SIEB200_OK;
}

int far_field_matrix_device(sieb200_ctx* ctx, const sieb200_mesh& mesh, double k0, double eta0, int64_t ndir,
                            const double* rh, const double* th, const double* ph, cplx* dA) {
    const int nf = (int)mesh.num_faces, ne = (int)mesh.num_edges, nv = (int)mesh.num_vertices;
    cudaStream_t st = ctx->stream;
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
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off += ((bytes + 255) / 256) * 256; return o; };
    const size_t oV = take(sizeof(double) * 3 * nv), oF = take(sizeof(int) * 3 * nf),
                 oI = take(sizeof(int) * 2 * ne), oDir = take(sizeof(double) * 9 * ndir);
    DeviceBuffer buf(st);
    SIEB_RETURN_IF(buf.reserve(off));
    char* b = buf.as<char>();
    SIEB_TRY_CUDA(cudaMemcpyAsync(b + oV, mesh.vertices, sizeof(double) * 3 * nv, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(b + oF, mesh.faces, sizeof(int) * 3 * nf, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(b + oI, inc.data(), sizeof(int) * 2 * ne, cudaMemcpyHostToDevice, st));
    double* dd = reinterpret_cast<double*>(b + oDir);
    SIEB_TRY_CUDA(cudaMemcpyAsync(dd, rh, sizeof(double) * 3 * ndir, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(dd + 3 * ndir, th, sizeof(double) * 3 * ndir, cudaMemcpyHostToDevice, st));
    SIEB_TRY_CUDA(cudaMemcpyAsync(dd + 6 * ndir, ph, sizeof(double) * 3 * ndir, cudaMemcpyHostToDevice, st));
    ff_matrix_kernel<<<dim3((unsigned)((ne + 127) / 128), (unsigned)ndir), 128, 0, st>>>(
        reinterpret_cast<double*>(b + oV), reinterpret_cast<int*>(b + oF), reinterpret_cast<int*>(b + oI), ne,
        ndir, k0, eta0, dd, dd + 3 * ndir, dd + 6 * ndir, dA);
    SIEB_NOTE_LAUNCH();
    SIEB_TRY_CUDA(cudaGetLastError());
    SIEB_TRY_CUDA(cudaStreamSynchronize(st));
    return SIEB200_OK;
}

}  // namespace sieb200
