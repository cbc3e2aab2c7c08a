// Adjoint of the clustering energy for a fixed clustering (FP64 throughout).
//
// Forward, as a function of the vertex positions x and the per-vertex densities
// rho (the curvature-indicator slot of the metric, weight = area * rho^g):
//   face f:    cr = (p1 - p0) x (p2 - p0), area = |cr| / 2, unit normal n = cr / |cr|
//              (Common/vtkSurface.cxx:1283 area, Common/vtkQuadricTools.cxx:56-79 plane quadric)
//   vertex i:  a_i = sum_f area_f / 3, w_i = a_i rho_i^g (clamped weights are constants),
//              A_i = sum_f n n^T, b_i = A_i x_i (x_i lies on every adjacent plane)
//   cluster k: S = sum w x, W = sum w, A = sum A_i, b = sum b_i, m = S / W,
//              c = m + P (b - A m) with P the thresholded pseudo-inverse of A whose kept
//              eigenvalues are those of the forward pass (rank held fixed;
//              vtkQuadricTools.cxx:83-163), E_k = W |c|^2 - 2 c.S (vtkQEMetricForClustering.h:194-208)
// Backward: the vector-Jacobian product of L = gE * sum_k E_k + sum_k gC_k . c_k
// with respect to x and rho.  Cluster sums are recomputed, not stored.
//
// What bounds it: the FP64 pipe (2 lanes per SM and cycle, 1/64 of the float32 rate), then
// the loads of the gathers.  So values shared by several faces or corners are formed once
// (a vertex's density power and area cotangent, a face's reciprocal length), quotients by
// one divisor take one division, and the records that a gather reads are 16-byte aligned.
// At 512 x 512, K = 10,000, density exponent 1: the two face passes 441 -> 114 us (backward)
// and 52 -> 39 us, the vertex passes 91 -> 28, the cluster sums 68 -> 35 and the clusters'
// decompositions 62 -> 30-43 us; forward and backward together 1.25 -> 0.62 ms.
#include <cmath>

#include "common.cuh"
#include "primitives.cuh"
#include "state.cuh"

namespace acvd {

ACVD_DEV void put2(double* p, double a, double b) { *reinterpret_cast<double2*>(p) = make_double2(a, b); }
ACVD_DEV void get2(const double* p, double& a, double& b) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    a = v.x;
    b = v.y;
}

// r^g; the exponents of a plain density and of none need no power
ACVD_DEV double density_power(double r, double g) { return g == 1.0 ? r : (g == 0.0 ? 1.0 : pow(r, g)); }

__global__ void adj_face_fwd(AdjState a) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= a.nf) return;
    const int i0 = a.tri[3 * f], i1 = a.tri[3 * f + 1], i2 = a.tri[3 * f + 2];
    double e1[3], e2[3];
    for (int d = 0; d < 3; d++) {
        const double x0 = a.x[3 * (int64_t)i0 + d];
        e1[d] = a.x[3 * (int64_t)i1 + d] - x0;
        e2[d] = a.x[3 * (int64_t)i2 + d] - x0;
    }
    const double cr[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
    const double L = sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]);
    double n[3] = {0.0, 0.0, 0.0};
    QuotientRange range;
    range.add(L);
    for (int d = 0; d < 3; d++) range.add(cr[d]);
    if (L > 0.0 && range.holds()) {
        const double inv = 1.0 / L;
        for (int d = 0; d < 3; d++) n[d] = quotient_in_range(cr[d], L, inv);
    } else if (L > 0.0) {
        for (int d = 0; d < 3; d++) n[d] = cr[d] / L;
    }
    put2(a.face + 4 * f, n[0], n[1]);
    put2(a.face + 4 * f + 2, n[2], L);
}

__global__ void adj_vertex_fwd(AdjState a) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= a.nv) return;
    double len = 0.0, A[6] = {0, 0, 0, 0, 0, 0};
    const uint32_t j1 = a.vf_row[v + 1];
    for (uint32_t j = a.vf_row[v]; j < j1; j++) {
        const double* r = a.face + 4 * (int64_t)a.vf_face[j];
        double n0, n1, n2, L;
        get2(r, n0, n1);
        get2(r + 2, n2, L);
        len += L;
        A[0] += n0 * n0; A[1] += n0 * n1; A[2] += n0 * n2; A[3] += n1 * n1; A[4] += n1 * n2; A[5] += n2 * n2;
    }
    const double area = len / 6.0;   // a third of each face's area |cr| / 2
    a.va[v] = area;
    for (int j = 0; j < 6; j += 2) put2(a.vA + 6 * v + j, A[j], A[j + 1]);
    double w = area;
    if (a.rho) {
        const double rg = density_power(a.rho[v], a.grad);
        a.vrg[v] = rg;
        w = area * rg;
    }
    a.vw[v] = w;
}

__global__ void adj_limits(AdjState a, const double* wsum, double ratio) {
    const double mean = *wsum / (double)a.nv;
    a.lim[0] = mean / ratio;
    a.lim[1] = mean * ratio;
}

// the weight of vertex v, clamped; true if it was
ACVD_DEV bool vertex_weight(const AdjState& a, int64_t v, double& w) {
    w = a.vw[v];
    bool c = false;
    if (w > a.lim[1]) { w = a.lim[1]; c = true; }
    if (w < a.lim[0]) { w = a.lim[0]; c = true; }
    return c;
}

// Sum over a warp of C values per lane, half of them handed to the partner at each step
// (the butterfly's order of additions; 15 per lane for 13 values instead of 65).  Value
// `at` of the total ends in s[0] of the one lane with have > 0.
template <int C, int O>
ACVD_DEV void warp_sum_spread(double* s, int lane, int& at, int& have) {
    constexpr int H = (C + 1) / 2;
    const bool up = (lane & O) != 0;
#pragma unroll
    for (int j = 0; j < H; j++) {
        const double lower = s[j], upper = H + j < C ? s[H + j] : 0.0;
        const double t = __shfl_xor_sync(kFull, up ? lower : upper, O);
        s[j] = t + (up ? upper : lower);
    }
    at += up ? H : 0;
    have = up ? have - H : min(have, H);
    if constexpr (O > 1) warp_sum_spread<H, O / 2>(s, lane, at, have);
}

// one warp per cluster over its items (sorted by cluster): FP64 sums, fixed order
__global__ void adj_cluster_sums(AdjState a, const uint32_t* __restrict__ sorted, const uint32_t* __restrict__ off) {
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= a.k) return;
    double s[13];
    for (int q = 0; q < 13; q++) s[q] = 0.0;
    const uint32_t s0 = off[w], s1 = off[w + 1];
    for (uint32_t j = s0 + lane; j < s1; j += 32) {
        const int64_t i = sorted[j];
        double wi;
        vertex_weight(a, i, wi);
        const double xi[3] = {a.x[3 * i], a.x[3 * i + 1], a.x[3 * i + 2]};
        double Ai[6];
        for (int q = 0; q < 6; q += 2) get2(a.vA + 6 * i + q, Ai[q], Ai[q + 1]);
        s[0] += wi * xi[0]; s[1] += wi * xi[1]; s[2] += wi * xi[2]; s[3] += wi;
        for (int q = 0; q < 6; q++) s[4 + q] += Ai[q];
        s[10] += Ai[0] * xi[0] + Ai[1] * xi[1] + Ai[2] * xi[2];
        s[11] += Ai[1] * xi[0] + Ai[3] * xi[1] + Ai[4] * xi[2];
        s[12] += Ai[2] * xi[0] + Ai[4] * xi[1] + Ai[5] * xi[2];
    }
    int at = 0, have = 13;
    warp_sum_spread<13, 16>(s, lane, at, have);
    if (have > 0) a.cl[w * kAdjSums + at] = s[0];
}

ACVD_DEV void smul(const double a[6], const double v[3], double o[3]) {
    o[0] = a[0] * v[0] + a[1] * v[1] + a[2] * v[2];
    o[1] = a[1] * v[0] + a[3] * v[1] + a[4] * v[2];
    o[2] = a[2] * v[0] + a[4] * v[1] + a[5] * v[2];
}

// Eigenvalues and eigenvectors (columns of V) of the symmetric a = {a00, a01, a02, a11, a12,
// a22} by cyclic Jacobi rotations (Golub & Van Loan, Matrix Computations, sec. 8.5), the upper
// triangle only: w = the diagonal, o = (a01, a02, a12).  The rotation of rows p < q, the third
// row r (o[P] = a_pq, o[R] = a_pr, o[Q] = a_qr), from two reciprocal roots: with
// x = a_qq - a_pp, y = 2 a_pq and h = 1 / |(x, y)|, cos^2 = (1 + |x| h) / 2, sin = |y| h / 2 / cos.
// A cluster's decomposition is one chain of dependent FP64 operations, and there are about 2
// warps of clusters to an SM, so what counts is the chain: about 30 operations a rotation;
// with tangent and cosine by three quotients and two roots it was about 55.
// A decomposition's residual and the columns' deviation from orthonormal are half of what they
// were (on random sums of 60 normals: 1e-16 and 1.4e-16 root mean square).  At K = 10,000:
// adj_cluster 42 -> 30 us forward, 55 -> 43 with the backward.  a is a sum of n n^T of unit
// normals: no entry's square overflows.
template <int p, int q, int P, int R, int Q>
ACVD_DEV void adj_rotate(double w[3], double o[3], double V[3][3]) {
    const double x = w[q] - w[p], y = 2.0 * o[P];
    const double r2 = x * x + y * y;
    if (o[P] == 0.0 || !(r2 > 1e-290)) return;
    const double h = rsqrt(r2);
    const double c2 = 0.5 + 0.5 * (fabs(x) * h);
    const double ic = rsqrt(c2);
    const double sy = 0.5 * (x >= 0.0 ? y : -y) * h;
    double c = c2 * ic, s = sy * ic;
    const double e = 0.5 * fma(-c, c, fma(-s, s, 1.0));   // cos^2 + sin^2 = 1 to the last place
    c += c * e;
    s += s * e;
    const double t = s * ic;
    w[p] -= t * o[P];
    w[q] += t * o[P];
    o[P] = 0.0;
    const double rp = o[R], rq = o[Q];
    o[R] = c * rp - s * rq;
    o[Q] = s * rp + c * rq;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double vkp = V[k][p], vkq = V[k][q];
        V[k][p] = c * vkp - s * vkq;
        V[k][q] = s * vkp + c * vkq;
    }
}

ACVD_DEV void adj_eig3(const double a[6], double w[3], double V[3][3]) {
    double o[3] = {a[1], a[2], a[4]};
    w[0] = a[0]; w[1] = a[3]; w[2] = a[5];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) V[i][j] = i == j ? 1.0 : 0.0;
    for (int it = 0; it < 64; it++) {
        const double off = o[0] * o[0] + o[1] * o[1] + o[2] * o[2];
        const double dg = w[0] * w[0] + w[1] * w[1] + w[2] * w[2];
        if (!(off > 1e-30 * dg)) break;
        adj_rotate<0, 1, 0, 1, 2>(w, o, V);
        adj_rotate<0, 2, 1, 0, 2>(w, o, V);
        adj_rotate<1, 2, 2, 0, 1>(w, o, V);
    }
}

// per cluster: placement, energy, and (bwd) the cotangents of S, W, A, b
// gE: the cotangent of the total energy, read from dgE (device) when that is given
__global__ void adj_cluster(AdjState a, int metric, int level, double thr, bool bwd, double gE_host,
                            const double* dgE, const double* __restrict__ gC, double* __restrict__ cent) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.k) return;
    const double* r0 = a.cl + k * kAdjSums;
    double* ct = a.ct + k * kAdjCot;
    const double S[3] = {r0[0], r0[1], r0[2]};
    const double W = r0[3];
    a.ek[k] = 0.0;
    if (!(W > 0.0)) {
        for (int q = 0; bwd && q < kAdjCot; q++) ct[q] = 0.0;
        return;
    }
    const double A[6] = {r0[4], r0[5], r0[6], r0[7], r0[8], r0[9]};
    const double b[3] = {r0[10], r0[11], r0[12]};
    const double m[3] = {S[0] / W, S[1] / W, S[2] / W};
    double Am[3];
    smul(A, m, Am);
    const double r[3] = {b[0] - Am[0], b[1] - Am[1], b[2] - Am[2]};
    // eigen-decomposition and the kept set (the forward's rank decision)
    double lam[3], V[3][3];
    bool keep[3] = {false, false, false};
    double P[6] = {0, 0, 0, 0, 0, 0};
    if (metric != kIso) {
        adj_eig3(A, lam, V);
        double aw[3] = {fabs(lam[0]), fabs(lam[1]), fabs(lam[2])};
        const double mx = fmax(aw[0], fmax(aw[1], aw[2]));
        int used = 0;
        for (int it = 0; it < 3; it++) {
            int im = 0;
            if (aw[1] > aw[im]) im = 1;
            if (aw[2] > aw[im]) im = 2;
            const bool take = mx > 0.0 && aw[im] > thr * mx && used < level;
#pragma unroll
            for (int j = 0; j < 3; j++)
                if (j == im) {
                    keep[j] |= take;
                    aw[j] = -1.0;
                }
            used += take;
        }
        // P = sum_kept v v^T / lambda
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if (!keep[j]) continue;
            const double il = 1.0 / lam[j];
            P[0] += V[0][j] * V[0][j] * il; P[1] += V[0][j] * V[1][j] * il; P[2] += V[0][j] * V[2][j] * il;
            P[3] += V[1][j] * V[1][j] * il; P[4] += V[1][j] * V[2][j] * il; P[5] += V[2][j] * V[2][j] * il;
        }
    }
    double Pr[3];
    smul(P, r, Pr);
    const double c[3] = {m[0] + Pr[0], m[1] + Pr[1], m[2] + Pr[2]};
    const double cc = c[0] * c[0] + c[1] * c[1] + c[2] * c[2];
    a.ek[k] = cc * W - 2.0 * (c[0] * S[0] + c[1] * S[1] + c[2] * S[2]);
    if (cent) { cent[3 * k] = c[0]; cent[3 * k + 1] = c[1]; cent[3 * k + 2] = c[2]; }
    if (!bwd) return;
    const double gE = dgE ? *dgE : gE_host;
    // cotangent of c
    double u[3];
    for (int d = 0; d < 3; d++) u[d] = gE * 2.0 * W * (c[d] - m[d]) + (gC ? gC[3 * k + d] : 0.0);
    // M^T u = u - A P u   (M = I - P A, both symmetric)
    double Pu[3], APu[3];
    smul(P, u, Pu);
    smul(A, Pu, APu);
    const double Mu[3] = {u[0] - APu[0], u[1] - APu[1], u[2] - APu[2]};
    double GS[3];
    for (int d = 0; d < 3; d++) GS[d] = -2.0 * gE * c[d] + Mu[d] / W;
    const double GW = gE * cc - (Mu[0] * m[0] + Mu[1] * m[1] + Mu[2] * m[2]) / W;
    // b enters through P b: G_b = P u ; A enters through -P A m and through P itself
    double GA[3][3];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) GA[i][j] = -0.5 * (Pu[i] * m[j] + Pu[j] * m[i]);
    if (metric != kIso) {
        // d(u^T P r) with P = sum_kept v_j v_j^T / lam_j (first-order eigen perturbation)
        double uv[3], rv[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            uv[j] = u[0] * V[0][j] + u[1] * V[1][j] + u[2] * V[2][j];
            rv[j] = r[0] * V[0][j] + r[1] * V[1][j] + r[2] * V[2][j];
        }
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if (!keep[j]) continue;
            // eigenvalue term: -(u.v)(v.r)/lam^2 * v v^T
            const double t = -uv[j] * rv[j] / (lam[j] * lam[j]);
            for (int p = 0; p < 3; p++)
                for (int q = 0; q < 3; q++) GA[p][q] += t * V[p][j] * V[q][j];
#pragma unroll
            for (int l = 0; l < 3; l++) {
                if (l == j) continue;
                double coef;
                if (keep[l]) {
                    if (l < j) continue;   // kept pair handled once: 1/(lj(lj-ll)) + 1/(ll(ll-lj)) = -1/(lj ll)
                    coef = -1.0 / (lam[j] * lam[l]);
                } else {
                    coef = 1.0 / (lam[j] * (lam[j] - lam[l]));
                }
                const double s = coef * (uv[l] * rv[j] + uv[j] * rv[l]);
                for (int p = 0; p < 3; p++)
                    for (int q = 0; q < 3; q++) GA[p][q] += 0.5 * s * (V[p][l] * V[q][j] + V[p][j] * V[q][l]);
            }
        }
    }
    put2(ct, GS[0], GS[1]);
    put2(ct + 2, GS[2], GW);
    // compact symmetric: off-diagonal entries appear twice in A = sum n n^T
    put2(ct + 4, GA[0][0], GA[0][1] + GA[1][0]);
    put2(ct + 6, GA[0][2] + GA[2][0], GA[1][1]);
    put2(ct + 8, GA[1][2] + GA[2][1], GA[2][2]);
    put2(ct + 10, Pu[0], Pu[1]);
    put2(ct + 12, Pu[2], 0.0);
}

// Per vertex: what its item's weight, position and quadric contribute, and the cotangent of
// its dual area, which the faces around it read (a power and a division per vertex instead
// of one per face corner: the corners' three powers made adj_face_bwd 441 us at 512 x 512).
__global__ void adj_vertex_mid(AdjState a, double* __restrict__ gx, double* __restrict__ grho) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= a.nv) return;
    double g[3] = {0, 0, 0}, gr = 0.0, ga = 0.0;
    const int k = a.label[v];
    if (k >= 0 && k < a.k) {
        const double* c = a.ct + (int64_t)k * kAdjCot;
        double GS[4], Gb[3], A[6], w, AGb[3];
        get2(c, GS[0], GS[1]);
        get2(c + 2, GS[2], GS[3]);
        get2(c + 10, Gb[0], Gb[1]);
        Gb[2] = c[12];
        for (int j = 0; j < 6; j += 2) get2(a.vA + 6 * v + j, A[j], A[j + 1]);
        const bool clamped = vertex_weight(a, v, w);
        smul(A, Gb, AGb);
        for (int d = 0; d < 3; d++) g[d] = w * GS[d] + AGb[d];
        // weight cotangent: dL/dw = G_S . x + G_W
        const double gw = GS[0] * a.x[3 * v] + GS[1] * a.x[3 * v + 1] + GS[2] * a.x[3 * v + 2] + GS[3];
        if (!clamped) {
            ga = gw * (a.rho ? a.vrg[v] : 1.0) / 3.0;
            if (grho && a.rho && a.grad != 0.0)
                gr = gw * a.va[v] * a.grad * density_power(a.rho[v], a.grad - 1.0);
        }
    }
    for (int d = 0; d < 3; d++) gx[3 * v + d] = g[d];
    a.vga[v] = ga;
    if (grho) grho[v] = gr;
}

// per face: cotangents of its area and unit normal from its three corners'
// items, then of its two edge vectors
__global__ void adj_face_bwd(AdjState a) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= a.nf) return;
    double n[3], L;
    get2(a.face + 4 * f, n[0], n[1]);
    get2(a.face + 4 * f + 2, n[2], L);
    int iv[3];
    double x[3][3];
    for (int j = 0; j < 3; j++) {
        iv[j] = a.tri[3 * f + j];
        for (int d = 0; d < 3; d++) x[j][d] = a.x[3 * (int64_t)iv[j] + d];
    }
    // A_v gets n n^T, b_v gets n n^T x_v: the corners' cotangents of A add up before the
    // product with n; n . x_v is the face plane's offset for each of them
    double g_area = 0.0, g_n[3] = {0, 0, 0}, GA[6] = {0, 0, 0, 0, 0, 0}, Gb_sum[3] = {0, 0, 0};
    for (int j = 0; j < 3; j++) {
        const int k = a.label[iv[j]];
        if (k < 0 || k >= a.k) continue;
        const double* g = a.ct + (int64_t)k * kAdjCot;
        g_area += a.vga[iv[j]];
        double q[6], Gb[3];
        for (int d = 0; d < 6; d += 2) get2(g + 4 + d, q[d], q[d + 1]);
        for (int d = 0; d < 6; d++) GA[d] += q[d];
        get2(g + 10, Gb[0], Gb[1]);
        Gb[2] = g[12];
        const double gbn = Gb[0] * n[0] + Gb[1] * n[1] + Gb[2] * n[2];
        for (int d = 0; d < 3; d++) {
            Gb_sum[d] += Gb[d];
            g_n[d] += gbn * x[j][d];
        }
    }
    const double off = n[0] * x[0][0] + n[1] * x[0][1] + n[2] * x[0][2];
    // d(sum_pq GA_pq n_p n_q) / dn with the compact weights (off-diagonals counted once)
    g_n[0] += 2.0 * GA[0] * n[0] + GA[1] * n[1] + GA[2] * n[2] + off * Gb_sum[0];
    g_n[1] += GA[1] * n[0] + 2.0 * GA[3] * n[1] + GA[4] * n[2] + off * Gb_sum[1];
    g_n[2] += GA[2] * n[0] + GA[4] * n[1] + 2.0 * GA[5] * n[2] + off * Gb_sum[2];
    double g_cr[3] = {0, 0, 0};
    if (L > 0.0) {
        const double ngn = n[0] * g_n[0] + n[1] * g_n[1] + n[2] * g_n[2];
        double h[3] = {g_n[0] - n[0] * ngn, g_n[1] - n[1] * ngn, g_n[2] - n[2] * ngn};
        QuotientRange range;
        range.add(L);
        for (int d = 0; d < 3; d++) range.add(h[d]);
        if (range.holds()) {
            const double inv = 1.0 / L;
            for (int d = 0; d < 3; d++) h[d] = quotient_in_range(h[d], L, inv);
        } else {
            for (int d = 0; d < 3; d++) h[d] /= L;
        }
        for (int d = 0; d < 3; d++) g_cr[d] = 0.5 * g_area * n[d] + h[d];
    }
    double e1[3], e2[3];
    for (int d = 0; d < 3; d++) {
        e1[d] = x[1][d] - x[0][d];
        e2[d] = x[2][d] - x[0][d];
    }
    // cr = e1 x e2: g_e1 = e2 x g_cr, g_e2 = g_cr x e1
    const double ge1[3] = {e2[1] * g_cr[2] - e2[2] * g_cr[1], e2[2] * g_cr[0] - e2[0] * g_cr[2],
                           e2[0] * g_cr[1] - e2[1] * g_cr[0]};
    const double ge2[3] = {g_cr[1] * e1[2] - g_cr[2] * e1[1], g_cr[2] * e1[0] - g_cr[0] * e1[2],
                           g_cr[0] * e1[1] - g_cr[1] * e1[0]};
    double* out = a.edge + 6 * f;
    put2(out, ge1[0], ge1[1]);
    put2(out + 2, ge1[2], ge2[0]);
    put2(out + 4, ge2[1], ge2[2]);
}

// per vertex: its faces' contributions (corner 0 moves both edge vectors the other way)
__global__ void adj_vertex_bwd(AdjState a, double* __restrict__ gx) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= a.nv) return;
    double g[3] = {gx[3 * v], gx[3 * v + 1], gx[3 * v + 2]};
    const uint32_t j1 = a.vf_row[v + 1];
    for (uint32_t j = a.vf_row[v]; j < j1; j++) {
        const int64_t f = a.vf_face[j];
        const int t1 = a.tri[3 * f + 1], t2 = a.tri[3 * f + 2];
        double e[6];
        for (int d = 0; d < 6; d += 2) get2(a.edge + 6 * f + d, e[d], e[d + 1]);
        for (int d = 0; d < 3; d++) g[d] += t1 == (int)v ? e[d] : (t2 == (int)v ? e[3 + d] : -e[d] - e[3 + d]);
    }
    for (int d = 0; d < 3; d++) gx[3 * v + d] = g[d];
}

static inline unsigned nb(int64_t n, int b = 256) { return (unsigned)((n + b - 1) / b); }

cudaError_t adjoint_run(const AdjState& a, int metric, int level, double thr, double ratio, double gE,
                        const double* dgE, const double* gC, const uint32_t* sorted, const uint32_t* off,
                        double* wsum, double* cent, double* gx, double* grho, cudaStream_t s,
                        Scratch& scratch) {
    adj_face_fwd<<<nb(a.nf), 256, 0, s>>>(a);
    adj_vertex_fwd<<<nb(a.nv), 256, 0, s>>>(a);
    cudaError_t e = sum_f64(a.vw, a.nv, wsum, scratch, s);
    if (e != cudaSuccess) return e;
    adj_limits<<<1, 1, 0, s>>>(a, wsum, ratio);
    adj_cluster_sums<<<nb((int64_t)a.k * 32), 256, 0, s>>>(a, sorted, off);
    // one warp per block: 10,000 clusters in blocks of 128 left half of the SMs idle
    adj_cluster<<<nb(a.k, 32), 32, 0, s>>>(a, metric, level, thr, gx != nullptr, gE, dgE, gC, cent);
    g_launches += 5;
    if (gx) {
        adj_vertex_mid<<<nb(a.nv), 256, 0, s>>>(a, gx, grho);
        adj_face_bwd<<<nb(a.nf), 256, 0, s>>>(a);
        adj_vertex_bwd<<<nb(a.nv), 256, 0, s>>>(a, gx);
        g_launches += 3;
    }
    return cudaGetLastError();
}

size_t adjoint_bytes(int64_t nv, int64_t nf, int k) {
    return sizeof(double) * (size_t)(10 * nf + 10 * nv + (size_t)k * (kAdjSums + kAdjCot + 1) + 2);
}

// carves the work buffers out of one allocation; the records that are read in pairs come
// first, at even offsets
AdjState adjoint_state(void* base, int64_t nv, int64_t nf, int k) {
    AdjState a{};
    double* p = (double*)base;
    a.face = p; p += 4 * nf;
    a.edge = p; p += 6 * nf;
    a.vA = p; p += 6 * nv;
    a.cl = p; p += (size_t)k * kAdjSums;
    a.ct = p; p += (size_t)k * kAdjCot;
    a.lim = p; p += 2;
    a.va = p; p += nv;
    a.vw = p; p += nv;
    a.vrg = p; p += nv;
    a.vga = p; p += nv;
    a.ek = p; p += k;
    a.nv = nv; a.nf = nf; a.k = k;
    return a;
}

}  // namespace acvd
