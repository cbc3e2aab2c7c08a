// Per-vertex curvature for vertex clustering: the curvature indicator and the
// principal directions that vtkDiscreteRemeshing's pre-processing computes with
// vtkCurvatureMeasure (DiscreteRemeshing/vtkDiscreteRemeshing.h:630-637):
// polynomial fitting (method 1) on the faces of the vertex 3-ring.
//
// FP64, one thread per vertex.  This file is compiled without FMA contraction
// (build.py) and every expression keeps the operation order of the CPU
// restatement, so that each value equals it bit for bit (the divisions and
// square roots are the correctly rounded IEEE operations on both sides).
//
// What bounds it: the FP64 pipe, 2 lanes per SM and cycle.  A vertex's fit reads its 3-ring's
// faces (54 in a regular mesh) three times, about 100 FP64 operations a face and 800 for the
// 6 x 6 inverse: 5.3 ms for 524,288 vertices at that rate.  So
//  * products that depend on the face only are formed once per face;
//  * quotients by one divisor (five per face, 51 per inverse) share its reciprocal
//    (3 operations instead of about 9; what each needs to equal the division is checked on the
//    exponents, with integer operations, 0.1 % of the time);
//  * finding the 3-ring, integer work in dependent loads, has kernels of its own at their own
//    occupancy instead of idling the FP64 pipe in between: every vertex's fan of faces
//    once, then the list of each vertex's ring, in chunks of curv_chunk() vertices.
// 6.46 ms of fits and 0.76 of lists for 524,288 vertices; one kernel for both, with 8,500 FP64
// operations per vertex, took 9.9 ms with its pipe 72 % busy.
#include "../../include/acvd_gpu.h"
#include "common.cuh"
#include "primitives.cuh"
#include "state.cuh"

namespace acvd {

constexpr int kCurvMaxF = 192;    // faces of one 3-ring
constexpr int kCurvMaxV = 384;    // vertices queued for one ring step
constexpr int kCurvMaxVis = 96;   // vertices of rings 0..2
constexpr int kFitBatch = 4;

// Faces of edge e: the first two faces, in increasing id, holding both of its
// endpoints (the reference attaches faces to an edge in face order,
// Common/vtkSurfaceBase.cxx:1166-1221).  Original vertex ids.
__global__ void edge_faces_kernel(const int* __restrict__ edge_v, int64_t ne, const int* __restrict__ tri,
                                  const uint32_t* __restrict__ vf_row, const uint32_t* __restrict__ vf_face,
                                  int2* __restrict__ poly) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    const int a = edge_v[2 * e], b = edge_v[2 * e + 1];
    int f1 = -1, f2 = -1;
    for (uint32_t t = vf_row[a]; t < vf_row[a + 1] && f2 < 0; t++) {
        const int f = (int)vf_face[t];
        if (tri[3 * f] == b || tri[3 * f + 1] == b || tri[3 * f + 2] == b) {
            if (f1 < 0) f1 = f;
            else f2 = f;
        }
    }
    poly[e] = make_int2(f1, f2);
}

// Edge id of every ring slot of the internal CSR (edges in internal ids).
__global__ void slot_edges_kernel(const int* __restrict__ edge_int, int64_t ne, const int* __restrict__ row,
                                  const int* __restrict__ col, int* __restrict__ slot_edge) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    const int a = edge_int[2 * e], b = edge_int[2 * e + 1];
    for (int p = row[a]; p < row[a + 1]; p++)
        if (col[p] == b) { slot_edge[p] = (int)e; break; }
    for (int p = row[b]; p < row[b + 1]; p++)
        if (col[p] == a) { slot_edge[p] = (int)e; break; }
}

// Per face, once: the values the fit reads for every vertex whose 3-ring holds the face.
struct FaceProps {
    double an[3];     // area x unit normal
    double ab[3];     // area x barycentre
    double area;
    double bary[3];   // area-weighted barycentre
};

struct CurvMesh {
    const FaceProps* fp;
    int64_t nv;
    const int* row;         // internal ring CSR
    const int* col;
    const int* inv;         // original vertex -> item
    const int* fan;         // per item: the faces of its ring edges, each once, at 2 row[i]
    const int* fan_count;
};

// area by the side-length form (Common/vtkSurface.cxx:1283) and the
// area-weighted vertex mean (vtkSurface::GetCellMassProperties, :1380-1419)
__device__ void curv_face_mass(const double p1[3], const double p2[3], const double p3[3], double& area,
                               double bary[3]) {
    const double d12[3] = {p1[0] - p2[0], p1[1] - p2[1], p1[2] - p2[2]};
    const double d23[3] = {p2[0] - p3[0], p2[1] - p3[1], p2[2] - p3[2]};
    const double d31[3] = {p3[0] - p1[0], p3[1] - p1[1], p3[2] - p1[2]};
    const double a = d12[0] * d12[0] + d12[1] * d12[1] + d12[2] * d12[2];
    const double b = d23[0] * d23[0] + d23[1] * d23[1] + d23[2] * d23[2];
    const double c = d31[0] * d31[0] + d31[1] * d31[1] + d31[2] * d31[2];
    const double a2 = 0.25 * sqrt(fabs(4.0 * a * c - (a - b + c) * (a - b + c)));
    for (int i = 0; i < 3; i++) {
        const double t = a2 * (p1[i] + p2[i] + p3[i]);
        bary[i] = 0.0 + quotient(t, 3.0, 1.0 / 3.0);
    }
    area = 0.0 + a2;
    if (divides_well(area)) {
        const double inv = 1.0 / area;
        for (int i = 0; i < 3; i++) bary[i] = quotient(bary[i], area, inv);
    } else if (area > 0) {
        for (int i = 0; i < 3; i++) bary[i] /= area;
    }
}

// unit normal from (x3 - x2) x (x1 - x2)
__device__ void curv_normal(const double x1[3], const double x2[3], const double x3[3], double n[3]) {
    const double a[3] = {x3[0] - x2[0], x3[1] - x2[1], x3[2] - x2[2]};
    const double b[3] = {x1[0] - x2[0], x1[1] - x2[1], x1[2] - x2[2]};
    n[0] = a[1] * b[2] - a[2] * b[1];
    n[1] = a[2] * b[0] - a[0] * b[2];
    n[2] = a[0] * b[1] - a[1] * b[0];
    const double l = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    if (divides_well(l)) {
        const double inv = 1.0 / l;
        for (int k = 0; k < 3; k++) n[k] = quotient(n[k], l, inv);
    } else if (l != 0.0) {
        n[0] /= l; n[1] /= l; n[2] /= l;
    }
}

__device__ __forceinline__ void curv_normalize(double a[3]) {
    const double n = sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
    if (n != 0.0) { a[0] /= n; a[1] /= n; a[2] /= n; }
}

__device__ __forceinline__ void curv_cross(const double a[3], const double b[3], double c[3]) {
    const double x = a[1] * b[2] - a[2] * b[1], y = a[2] * b[0] - a[0] * b[2], z = a[0] * b[1] - a[1] * b[0];
    c[0] = x; c[1] = y; c[2] = z;
}

__device__ __forceinline__ double curv_dot(const double a[3], const double b[3]) {
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

__global__ void face_props_kernel(const double* __restrict__ xyz, const int* __restrict__ tri, int64_t nf,
                                  FaceProps* __restrict__ fp) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    double p1[3], p2[3], p3[3];
    for (int k = 0; k < 3; k++) {
        p1[k] = xyz[3 * (int64_t)tri[3 * f] + k];
        p2[k] = xyz[3 * (int64_t)tri[3 * f + 1] + k];
        p3[k] = xyz[3 * (int64_t)tri[3 * f + 2] + k];
    }
    FaceProps r;
    double n[3];
    curv_normal(p1, p2, p3, n);
    curv_face_mass(p1, p2, p3, r.area, r.bary);
    for (int k = 0; k < 3; k++) {
        r.an[k] = r.area * n[k];
        r.ab[k] = r.area * r.bary[k];
    }
    fp[f] = r;
}

// The faces around item i in the order its ring's edges name them (each edge's first two
// faces), each once: the order in which vtkNeighbourhoodComputation meets them.  More than
// kCurvMaxF faces are past the bound of every ring that holds the item, so that the list stops
// there: each face is looked up among those before it, and a hub of 60,000 would take this
// one thread 10^9 dependent loads.
__global__ void fan_kernel(int64_t n, const int* __restrict__ row, const int* __restrict__ slot_edge,
                           const int2* __restrict__ poly, int* fan, int* __restrict__ fan_count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int p0 = row[i], p1 = row[i + 1];
    int* out = fan + 2 * (int64_t)p0;
    int c = 0;
    auto add = [&](int f) {
        for (int j = 0; j < c; j++)
            if (out[j] == f) return;
        out[c++] = f;
    };
    for (int p = p0; p < p1 && c <= kCurvMaxF; p++) {
        const int e = slot_edge[p];
        if (e < 0) continue;
        const int2 pf = poly[e];
        if (pf.x >= 0) add(pf.x);
        if (pf.y >= 0) add(pf.y);
    }
    fan_count[i] = c;
}

// The faces of the 3-ring of vertices v0 .. v0 + n - 1 in the reference's order
// (vtkNeighbourhoodComputation::ComputeNRingCells, Common/vtkNeighbourhoodComputation.cxx:38-100:
// the vertex's own faces, then ring by ring the faces of each vertex not yet visited):
// lists[j * n + t] is the j-th face of vertex v0 + t, so that a warp's accesses to a place of
// its lists fall side by side.
// counts[t]: their number, -1 for a neighbourhood larger than the bounds above, which also
// counts in *overflow.
//
// kRingLanes lanes work on a vertex: its lists are in shared memory, a visited vertex's fan
// is looked up in them one face per lane, a ring's vertices likewise.  A thread per vertex left
// 1,281 warps with a chain of 63,000 instructions each for 40,962 vertices: 465 us, 71 so
// (524,288 vertices of a grid, where both are bound by instructions: 576 and 755 us).
constexpr int kRingThreads = 128;
constexpr int kRingLanes = 8;
constexpr int kRingGroups = kRingThreads / kRingLanes;

__global__ void __launch_bounds__(kRingThreads) ring_faces_kernel(CurvMesh m, int64_t v0, int64_t n,
                                                                  int* __restrict__ lists, int* __restrict__ counts,
                                                                  unsigned long long* __restrict__ overflow) {
    // rows of 4 (mod 32) words: the groups of a warp in different banks; -1 where nothing is listed,
    // so that a search may take four entries at a time
    __shared__ __align__(16) int s_fl[kRingGroups][kCurvMaxF + 4];
    __shared__ __align__(16) int s_vis[kRingGroups][kCurvMaxVis + 4];
    __shared__ int s_nf[kRingGroups];
    const int g = threadIdx.x / kRingLanes, l = threadIdx.x % kRingLanes;
    const int shift = (threadIdx.x & 31) & ~(kRingLanes - 1);   // the group's first lane in the warp
    const unsigned group = ((1u << kRingLanes) - 1u) << shift;
    const int64_t t0 = (int64_t)blockIdx.x * kRingGroups, t = t0 + g;
    int* fl = s_fl[g];
    int* vis = s_vis[g];
    for (int i = l; i < kCurvMaxF + 4; i += kRingLanes) fl[i] = -1;
    for (int i = l; i < kCurvMaxVis + 4; i += kRingLanes) vis[i] = -1;
    __syncwarp();
    // whether x is none of the first c entries of a list
    auto absent = [](const int* list, int c, int x) {
        bool none = true;
        for (int i = 0; i < c; i += 4) {
            const int4 q = *reinterpret_cast<const int4*>(list + i);
            none = none && q.x != x && q.y != x && q.z != x && q.w != x;
        }
        return none;
    };
    int nf = 0, nvis = 0;
    bool ok = true;
    // u joins the visited vertices; the faces of its fan that are not listed follow in order
    auto visit = [&](int u, int& queued) {
        if (nvis == kCurvMaxVis) { ok = false; return; }
        if (l == 0) vis[nvis] = u;
        nvis++;
        const int p0 = m.row[u], p1 = m.row[u + 1], c = m.fan_count[u];
        queued += p1 - p0;
        if (queued > kCurvMaxV) { ok = false; return; }
        const int* fan = m.fan + 2 * (int64_t)p0;
        for (int k0 = 0; k0 < c; k0 += kRingLanes) {
            const int f = k0 + l < c ? fan[k0 + l] : -1;
            const bool fresh = absent(fl, nf, f) && f >= 0;
            const unsigned add = (__ballot_sync(group, fresh) & group) >> shift;
            if (nf + __popc(add) > kCurvMaxF) { ok = false; return; }
            if (fresh) fl[nf + __popc(add & ((1u << l) - 1u))] = f;
            nf += __popc(add);
            __syncwarp(group);
        }
        __syncwarp(group);
    };
    if (t < n) {
        int queued = 0;
        visit(m.inv[v0 + t], queued);
        // ring r's new vertices are vis[first .. last); the next ring's candidates are their
        // neighbours in order
        int first = 0, last = nvis;
        for (int r = 1; r < 3 && ok; r++) {
            queued = 0;
            for (int k = first; k < last && ok; k++) {
                const int u = vis[k];
                const int p1 = m.row[u + 1];
                for (int p = m.row[u]; p < p1 && ok; p += kRingLanes) {
                    const int x = p + l < p1 ? m.col[p + l] : -1;
                    bool fresh = absent(vis, nvis, x) && x >= 0;
                    // a ring lists a vertex once; should it not, its first place counts
                    const unsigned same = (__match_any_sync(group, x) & group) >> shift;
                    fresh = fresh && (same & ((1u << l) - 1u)) == 0u;
                    unsigned add = (__ballot_sync(group, fresh) & group) >> shift;
                    for (; add && ok; add &= add - 1u)
                        visit(__shfl_sync(group, x, shift + __ffs((int)add) - 1), queued);
                }
            }
            first = last;
            last = nvis;
        }
        if (l == 0) {
            if (!ok) atomicAdd(overflow, 1ull);
            counts[t] = ok ? nf : -1;
        }
    }
    if (l == 0) s_nf[g] = t < n && ok ? nf : 0;
    __syncthreads();
    // the block's lists, kRingGroups vertices side by side
    int most = 0;
    for (int q = 0; q < kRingGroups; q++) most = max(most, s_nf[q]);
    const int col = threadIdx.x % kRingGroups;
    for (int j = threadIdx.x / kRingGroups; j < most; j += kRingLanes)
        if (j < s_nf[col]) lists[(int64_t)j * n + t0 + col] = s_fl[col][j];
}

// Inverse of the n x n matrix a by LU decomposition with partial pivoting
// (Doolittle), one substitution per unit vector; 0 when a pivot is exactly zero.
// SHARED: a pivot's quotients share its reciprocal; -1 if one was out of that form's range.
// (A zero may lose its sign there: it ends in sums that start from +0 or hold another term
// that is not -0, where both zeros give the same.)
template <int N, bool SHARED>
__device__ __forceinline__ int curv_lu_invert_by(const double a[N][N], double ai[N][N]) {
    double lu[N][N], rec[N];
    QuotientRange range;
    int piv[N];
    auto over_pivot = [&](double x, int k) {
        if (!SHARED) return x / lu[k][k];
        range.add(x);
        return quotient_in_range(x, lu[k][k], rec[k]);
    };
    for (int i = 0; i < N; i++)
        for (int j = 0; j < N; j++) lu[i][j] = a[i][j];
    for (int k = 0; k < N; k++) {
        int p = k;
        double best = fabs(lu[k][k]);
        for (int i = k + 1; i < N; i++) {
            const double v = fabs(lu[i][k]);
            if (v > best) { best = v; p = i; }
        }
        if (best == 0.0) return SHARED && !range.holds() ? -1 : 0;
        piv[k] = p;
        if (p != k)
            for (int j = 0; j < N; j++) { const double t = lu[k][j]; lu[k][j] = lu[p][j]; lu[p][j] = t; }
        if (SHARED) {
            range.add(lu[k][k]);
            rec[k] = 1.0 / lu[k][k];
        }
        for (int i = k + 1; i < N; i++) {
            const double f = over_pivot(lu[i][k], k);
            lu[i][k] = f;
            for (int j = k + 1; j < N; j++) lu[i][j] -= f * lu[k][j];
        }
    }
    for (int c = 0; c < N; c++) {
        double x[N];
        for (int i = 0; i < N; i++) x[i] = (i == c) ? 1.0 : 0.0;
        for (int k = 0; k < N; k++)
            if (piv[k] != k) { const double t = x[k]; x[k] = x[piv[k]]; x[piv[k]] = t; }
        for (int i = 0; i < N; i++)
            for (int j = 0; j < i; j++) x[i] -= lu[i][j] * x[j];
        for (int i = N - 1; i >= 0; i--) {
            for (int j = i + 1; j < N; j++) x[i] -= lu[i][j] * x[j];
            x[i] = over_pivot(x[i], i);
        }
        for (int i = 0; i < N; i++) ai[i][c] = x[i];
    }
    return SHARED && !range.holds() ? -1 : 1;
}

template <int N>
__device__ __noinline__ int curv_lu_invert_plain(const double a[N][N], double ai[N][N]) {
    return curv_lu_invert_by<N, false>(a, ai);
}

template <int N>
__device__ int curv_lu_invert(const double a[N][N], double ai[N][N]) {
    const int r = curv_lu_invert_by<N, true>(a, ai);
    if (r >= 0) return r;
    // copies, so that the common case's matrices need no address
    double b[N][N], bi[N][N];
    for (int i = 0; i < N; i++)
        for (int j = 0; j < N; j++) b[i][j] = a[i][j];
    const int t = curv_lu_invert_plain<N>(b, bi);
    for (int i = 0; i < N; i++)
        for (int j = 0; j < N; j++) ai[i][j] = bi[i][j];
    return t;
}

// Eigen-decomposition of the symmetric 2x2 matrix given by the upper triangle of
// a (cyclic Jacobi; Golub & Van Loan sec. 8.5): w decreasing, unit eigenvectors in
// the columns of v.
__device__ void curv_jacobi2(const double a[2][2], double w[2], double v[2][2]) {
    double m[2][2] = {{a[0][0], a[0][1]}, {a[0][1], a[1][1]}};
    v[0][0] = 1.0; v[0][1] = 0.0; v[1][0] = 0.0; v[1][1] = 1.0;
    for (int sweep = 0; sweep < 64; sweep++) {
        const double off = m[0][1] * m[0][1];
        if (off == 0.0) break;
        const double apq = m[0][1];
        if (apq == 0.0) continue;
        const double theta = (m[1][1] - m[0][0]) / (2.0 * apq);
        const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
        const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
        for (int k = 0; k < 2; k++) {
            const double mkp = m[k][0], mkq = m[k][1];
            m[k][0] = c * mkp - s * mkq;
            m[k][1] = s * mkp + c * mkq;
        }
        for (int k = 0; k < 2; k++) {
            const double mpk = m[0][k], mqk = m[1][k];
            m[0][k] = c * mpk - s * mqk;
            m[1][k] = s * mpk + c * mqk;
        }
        m[0][1] = m[1][0] = 0.0;
        for (int k = 0; k < 2; k++) {
            const double vkp = v[k][0], vkq = v[k][1];
            v[k][0] = c * vkp - s * vkq;
            v[k][1] = s * vkp + c * vkq;
        }
    }
    w[0] = m[0][0];
    w[1] = m[1][1];
    if (w[1] > w[0]) {
        const double t = w[0]; w[0] = w[1]; w[1] = t;
        for (int k = 0; k < 2; k++) { const double u = v[k][0]; v[k][0] = v[k][1]; v[k][1] = u; }
    }
}

// vtkSinglePolynomialMeasure::ComputeFitting (Common/vtkCurvatureMeasure.cxx:188-505)
// on the faces fl[0..nf): returns sqrt(k1^2 + k2^2), info = principal directions
// scaled by sqrt|k|, the larger |k| first.
// stride: between the entries of fl.
__device__ double curv_fit(const CurvMesh& m, const int* fl, int64_t stride, int nf, double* xs, double* ys, double* zs,
                           double info[6]) {
    double sarea = 0, origin[3] = {0, 0, 0}, frame[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    // kFitBatch faces at a time, their records loaded before any is used: the index and the
    // record it points to are two dependent loads, and a small mesh has few warps to hide them
    for (int j0 = 0; j0 < nf; j0 += kFitBatch) {
        int id[kFitBatch];
        double v[kFitBatch][7];
#pragma unroll
        for (int b = 0; b < kFitBatch; b++) id[b] = fl[(j0 + b < nf ? j0 + b : nf - 1) * stride];
#pragma unroll
        for (int b = 0; b < kFitBatch; b++) {
            const FaceProps& q = m.fp[id[b]];
            for (int k = 0; k < 3; k++) {
                v[b][k] = q.ab[k];
                v[b][3 + k] = q.an[k];
            }
            v[b][6] = q.area;
        }
#pragma unroll
        for (int b = 0; b < kFitBatch; b++) {
            if (j0 + b >= nf) break;
            for (int k = 0; k < 3; k++) {
                origin[k] += v[b][k];
                frame[0][k] += v[b][3 + k];
            }
            sarea += v[b][6];
        }
    }
    for (int j = 0; j < 3; j++) origin[j] = origin[j] / sarea;
    curv_normalize(frame[0]);
    for (int k = 0; k < 3; k++) frame[2][k] = frame[0][k];
    frame[1][1] = frame[2][0]; frame[1][2] = frame[2][1]; frame[1][0] = frame[2][2];
    curv_cross(frame[1], frame[2], frame[0]);
    curv_normalize(frame[0]);
    curv_cross(frame[2], frame[0], frame[1]);
    for (int i = 0; i < 6; i++) info[i] = 0;
    if (nf <= 6) return 0;
    double h = 0;
    for (int j0 = 0; j0 < nf; j0 += kFitBatch) {
        int id[kFitBatch];
        double c[kFitBatch][3];
#pragma unroll
        for (int b = 0; b < kFitBatch; b++) id[b] = fl[(j0 + b < nf ? j0 + b : nf - 1) * stride];
#pragma unroll
        for (int b = 0; b < kFitBatch; b++)
            for (int k = 0; k < 3; k++) c[b][k] = m.fp[id[b]].bary[k];
#pragma unroll
        for (int b = 0; b < kFitBatch; b++) {
            const int j = j0 + b;
            if (j >= nf) break;
            double bary[3] = {c[b][0], c[b][1], c[b][2]};
            for (int k = 0; k < 3; k++) bary[k] -= origin[k];
            const double x = curv_dot(bary, frame[0]), y = curv_dot(bary, frame[1]), z = curv_dot(bary, frame[2]);
            xs[j] = x; ys[j] = y; zs[j] = z;
            h += sqrt(x * x + y * y);
        }
    }
    h = h / ((double)nf);
    // normal equations of the conditioned Vandermonde rows (upper half, mirrored); the first
    // entry of a row is 1, and its products are the other factor
    double xxt[6][6], xxti[6][6], xyt[6], q[6];
    for (int i = 0; i < 6; i++) {
        xyt[i] = 0.0;
        for (int j = 0; j < 6; j++) xxt[i][j] = 0.0;
    }
    // The quotients by h and h^2 share reciprocals.  |x| and |y| are at most nf h: for h in
    // [2^-120, 2^120) and |x y| from 2^-250 on, both are 2^-378 or more, their squares and the
    // quotients normal numbers and the residuals exact.  Other values that are zero, or so small
    // or large, are looked at one by one.
    const double hh = h * h;
    const bool good = divides_well(hh) && divides_well(h), near_one = exponent_of(h) - 903u < 240u;
    const double rh = 1.0 / h, rhh = 1.0 / hh;
    auto squares_well = [](double v) { return exponent_of(v) - 791u < 464u || __double_as_longlong(v) << 1 == 0; };
    for (int k = 0; k < nf; k++) {
        const double x = xs[k], y = ys[k], z = zs[k];
        double r[6] = {1.0, x, y, x * x, x * y, y * y};
        if ((near_one && exponent_of(r[4]) >= 773u) || (good && squares_well(x) && squares_well(y))) {
            r[1] = quotient_in_range(x, h, rh); r[2] = quotient_in_range(y, h, rh);
            r[3] = quotient_in_range(r[3], hh, rhh); r[4] = quotient_in_range(r[4], hh, rhh);
            r[5] = quotient_in_range(r[5], hh, rhh);
        } else {
            r[1] /= h; r[2] /= h; r[3] /= hh; r[4] /= hh; r[5] /= hh;
        }
#pragma unroll
        for (int j = 1; j < 6; j++) xxt[0][j] += r[j];
        xyt[0] += z;
#pragma unroll
        for (int i = 1; i < 6; i++) {
#pragma unroll
            for (int j = i; j < 6; j++) xxt[i][j] += r[i] * r[j];
            xyt[i] += r[i] * z;
        }
    }
    xxt[0][0] = (double)nf;   // nf times 1, exactly
    for (int i = 0; i < 6; i++)
        for (int j = 0; j < i; j++) xxt[i][j] = xxt[j][i];
    if (!curv_lu_invert<6>(xxt, xxti)) return 0;
    for (int i = 0; i < 6; i++) {
        q[i] = 0.0;
        for (int k = 0; k < 6; k++) q[i] += xxti[i][k] * xyt[k];
    }
    q[1] /= h; q[2] /= h; q[3] /= h * h; q[4] /= h * h; q[5] /= h * h;
    const double E = 1.0 + q[1] * q[1], F = q[1] * q[2], G = 1.0 + q[2] * q[2];
    const double e = 2.0 * q[3] / sqrt(q[1] * q[1] + 1.0 + q[2] * q[2]);
    const double ff = 2.0 * q[4] / sqrt(q[1] * q[1] + 1.0 + q[2] * q[2]);
    const double g = 2.0 * q[5] / sqrt(q[1] * q[1] + 1.0 + q[2] * q[2]);
    double A[2][2] = {{E, F}, {F, G}}, B[2][2];
    if (!curv_lu_invert<2>(A, B)) return 0;
    A[0][0] = -(e * B[0][0] + ff * B[1][0]);
    A[1][0] = -(e * B[0][1] + ff * B[1][1]);
    A[0][1] = -(ff * B[0][0] + g * B[1][0]);
    A[1][1] = -(ff * B[0][1] + g * B[1][1]);
    double ev[2], evec[2][2];
    curv_jacobi2(A, ev, evec);
    for (int i = 0; i < 2; i++)
        for (int j = 0; j < 2; j++)
            for (int k = 0; k < 3; k++) info[k + 3 * j] += sqrt(fabs(ev[j])) * evec[i][j] * frame[i][k];
    if (fabs(ev[0]) < fabs(ev[1]))
        for (int i = 0; i < 3; i++) { const double t = info[i]; info[i] = info[i + 3]; info[i + 3] = t; }
    return sqrt(ev[0] * ev[0] + ev[1] * ev[1]);
}

// The fits of vertices v0 .. v0 + n - 1 over their face lists.  A neighbourhood that was too
// large leaves the vertex's outputs at zero.  One warp per block: the SMs differ by a warp.
// At least 12 of them to an SM: 204 registers otherwise, and 524,288 vertices took 7.81 ms
// instead of 7.73.
constexpr int kFitThreads = 32;

__global__ void __launch_bounds__(kFitThreads, 12) curvature_kernel(CurvMesh m, int64_t v0, int64_t n,
                                                                const int* __restrict__ lists,
                                                                const int* __restrict__ counts,
                                                                double* __restrict__ indicator,
                                                                float* __restrict__ dirs) {
    const int64_t t = (int64_t)blockIdx.x * kFitThreads + threadIdx.x;
    if (t >= n) return;
    const int nf = counts[t];
    double info[6] = {0, 0, 0, 0, 0, 0};
    double ind = 0.0;
    if (nf >= 0) {
        double xs[kCurvMaxF], ys[kCurvMaxF], zs[kCurvMaxF];
        ind = curv_fit(m, lists + t, n, nf, xs, ys, zs, info);
    }
    const int64_t v = v0 + t;
    indicator[v] = ind;
    for (int i = 0; i < 6; i++) dirs[6 * v + i] = (float)info[i];
}

static inline unsigned cgrid(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

// Vertices whose face lists are held at a time.  (Chunks of equal size instead of full ones
// and a rest: 1024 x 513 the same 7.87 ms, 1024 x 1000 15.1 ms instead of 14.9: what counts is
// how full the last wave of fits is, and 524,288 vertices are 8.98 waves of 12 warps to an SM.)
static int64_t curv_chunk(int64_t nv, int64_t most) { return nv < most ? nv : most; }

// Work of launch_curvature: the faces' values, the items' fans and the lists of a chunk.
size_t curvature_work_bytes(int64_t nv, int64_t nf, int64_t ne, int64_t most) {
    return (size_t)nf * sizeof(FaceProps) +
           sizeof(int) * (size_t)(4 * ne + nv + curv_chunk(nv, most) * (kCurvMaxF + 1));
}

cudaError_t launch_curvature(const double* xyz, const int* tri, int64_t nv, int64_t nf, int64_t ne,
                             const int* edge_v, const int* edge_int, const uint32_t* vf_row, const uint32_t* vf_face,
                             const int* row, const int* col, const int* inv, int2* poly, int* slot_edge, void* work,
                             int64_t most, double* indicator, float* dirs, unsigned long long* overflow, cudaStream_t s) {
    if (nv == 0) return cudaSuccess;
    cudaError_t err = cudaMemsetAsync(slot_edge, 0xff, 2 * ne * sizeof(int), s);   // -1: no edge
    if (err != cudaSuccess) return err;
    g_launches += 4;
    FaceProps* fp = (FaceProps*)work;
    const int64_t chunk = curv_chunk(nv, most);
    int* fan = (int*)(fp + nf);
    int* fan_count = fan + 4 * ne;
    int* counts = fan_count + nv;
    int* lists = counts + chunk;
    face_props_kernel<<<cgrid(nf, 256), 256, 0, s>>>(xyz, tri, nf, fp);
    edge_faces_kernel<<<cgrid(ne, 256), 256, 0, s>>>(edge_v, ne, tri, vf_row, vf_face, poly);
    slot_edges_kernel<<<cgrid(ne, 256), 256, 0, s>>>(edge_int, ne, row, col, slot_edge);
    fan_kernel<<<cgrid(nv, 256), 256, 0, s>>>(nv, row, slot_edge, poly, fan, fan_count);
    const CurvMesh m{fp, nv, row, col, inv, fan, fan_count};
    for (int64_t v0 = 0; v0 < nv; v0 += chunk) {
        const int64_t n = nv - v0 < chunk ? nv - v0 : chunk;
        g_launches += 2;
        ring_faces_kernel<<<cgrid(n, kRingGroups), kRingThreads, 0, s>>>(m, v0, n, lists, counts, overflow);
        curvature_kernel<<<cgrid(n, kFitThreads), kFitThreads, 0, s>>>(m, v0, n, lists, counts, indicator, dirs);
    }
    return cudaGetLastError();
}

}  // namespace acvd
