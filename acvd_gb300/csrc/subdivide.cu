// Midpoint subdivision of a triangle mesh, one level per launch sequence:
// vtkSurface::Subdivide (Common/vtkSurface.cxx:605-677) and the parent
// interpolation of the vertex indicator that vtkDiscreteRemeshing's
// pre-processing applies after it (DiscreteRemeshing/vtkDiscreteRemeshing.h:731-745).
//
// Output numbering is the reference's: the old vertices keep their ids, edge e
// gives vertex nV + e at its midpoint, face f gives faces 4f .. 4f+3 as
// (V1,V4,V6), (V4,V2,V5), (V5,V3,V6), (V4,V5,V6) with V4, V5, V6 the children
// of edges V1V2, V2V3, V3V1.  The reference stores the new mesh's points in a
// float vtkPoints, so every output coordinate is the float nearest to the FP64
// value (the old point, or 0.5 (P1 + P2)).
//
// What bounds it, at 524,288 vertices (187 MB in and out, 27 us at the copy rate): the FP64
// pipe, 2 lanes per SM and cycle, on which the two conversions of a rounding and the halving
// run too (79 % busy in the points kernel, 51 us), and the partial stores of 24- and 48-byte
// strides with a thread per point or face.  So a value is rounded to float on its bits, one
// FP64 addition per midpoint coordinate is left, and a warp writes its points and faces
// element by element through shared memory: 95.6 us a level before, 62.6 so.  No access
// is wider than its elements, so the caller's buffers need no alignment beyond theirs.
// (A thread per output coordinate, and four lanes per face for its three ring searches, were
// slower: 128 us.)
#include "primitives.cuh"
#include "state.cuh"

namespace acvd {

namespace {

constexpr int kSubThreads = 256;
constexpr int kSubWarps = kSubThreads / 32;

inline unsigned sgrid(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

// The rare cases of the two functions below are calls, so that they are branched around:
// inlined, the compiler ran their FP64 operations for every value and picked the result
// (FP64 pipe 44 % busy in the points kernel, 64.4 us a level against 62.6).
__device__ __noinline__ double float_rounded_rare(double v) { return (double)__double2float_rn(v); }
__device__ __noinline__ double half_rare(double v) { return 0.5 * v; }

// (double)(float)v, rounded to nearest even on the bits where the result is a normal float
__device__ __forceinline__ double float_rounded(double v) {
    const long long u = __double_as_longlong(v);
    const unsigned e = (unsigned)(u >> 52) & 0x7ffu;
    if (e - 897u < 253u) {   // 2^-126 <= |v| < 2^127: no underflow, and no overflow by rounding up
        const long long r = (u + 0x0fffffffll + ((u >> 29) & 1)) & ~0x1fffffffll;
        return __longlong_as_double(r);
    }
    if ((u << 1) == 0) return v;   // zeros
    return float_rounded_rare(v);
}

// v / 2 on the exponent
__device__ __forceinline__ double half_of(double v) {
    const long long u = __double_as_longlong(v);
    const unsigned e = (unsigned)(u >> 52) & 0x7ffu;
    if (e - 2u < 2045u) return __longlong_as_double(u - (1ll << 52));
    return (u << 1) == 0 ? v : half_rare(v);
}

// The slot of b in a's ring, -1 if it is not there.  Four slots are loaded at a time: one by
// one, each load waited for the compare before it (67.4 us a level against 64.4).
__device__ __forceinline__ int ring_slot(const int* __restrict__ row, const int* __restrict__ col, int a, int b) {
    const int p1 = row[a + 1];
    for (int p = row[a]; p < p1; p += 4) {
        int c[4];
#pragma unroll
        for (int j = 0; j < 4; j++) c[j] = p + j < p1 ? col[p + j] : -1;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (c[j] == b) return p + j;
    }
    return -1;
}

// Three independent parts of one launch, blocks of the first two alternating so that the
// ring searches' latency hides in the stream: (1) a thread per edge and end: the edge's id
// in the ring slot of its other end (a bad edge stays -1: the faces on it are reported);
// (2) a thread per edge: the midpoint, its parents and its indicator; (3) the old points'
// coordinates, float-rounded, and indicators.
__global__ void __launch_bounds__(kSubThreads) subdiv_points_kernel(
    const double* __restrict__ xyz, int64_t nv, const int* __restrict__ edge_v, int64_t ne, const int* __restrict__ row,
    const int* __restrict__ col, const double* __restrict__ ind, int* __restrict__ slot_edge,
    double* __restrict__ out_xyz, int* __restrict__ parent1, int* __restrict__ parent2, double* __restrict__ out_ind,
    unsigned edge_blocks) {
    __shared__ double s_x[kSubWarps][96];
    if (blockIdx.x >= 3u * edge_blocks) {
        const int64_t t = (int64_t)(blockIdx.x - 3u * edge_blocks) * kSubThreads + threadIdx.x;
        if (t < 3 * nv) out_xyz[t] = float_rounded(xyz[t]);
        if (out_ind && t < nv) out_ind[t] = ind[t];
        return;
    }
    const unsigned g = blockIdx.x / 3u, part = blockIdx.x - 3u * g;
    if (part < 2u) {
        const int64_t t = (int64_t)(2u * g + part) * kSubThreads + threadIdx.x;
        if (t >= 2 * ne) return;
        const int a = edge_v[t], b = edge_v[t ^ 1];
        if (a < 0 || b < 0 || a >= nv || b >= nv) return;
        const int p = ring_slot(row, col, a, b);
        if (p >= 0) slot_edge[p] = (int)(t >> 1);
        return;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t e0 = (int64_t)g * kSubThreads + 32 * w, e = e0 + lane;
    const int a = e < ne ? edge_v[2 * e] : -1, b = e < ne ? edge_v[2 * e + 1] : -1;
    const bool ok = a >= 0 && b >= 0 && a < nv && b < nv;
    if (ok) {
        for (int c = 0; c < 3; c++)
            s_x[w][3 * lane + c] = float_rounded(half_of(xyz[3 * (int64_t)a + c] + xyz[3 * (int64_t)b + c]));
        parent1[e] = a;
        parent2[e] = b;
        // CellsIndicators2[i] = (CellsIndicators2[Parent1[i]] + CellsIndicators2[Parent2[i]]) * 0.5
        if (out_ind) out_ind[nv + e] = half_of(ind[a] + ind[b]);
    }
    const unsigned have = __ballot_sync(kFull, ok);   // also orders the shared stores before the reads
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int at = lane + 32 * j;
        if ((have >> (at / 3)) & 1u) out_xyz[3 * (nv + e0) + at] = s_x[w][at];
    }
}

// A thread per face: its three edges by ring search, its 12 new corners staged (rows of 13:
// no bank conflicts) and written by the warp side by side.
__global__ void __launch_bounds__(kSubThreads) subdiv_faces_kernel(const int* __restrict__ tri, int64_t nf, int64_t nv,
                                                                   const int* __restrict__ row,
                                                                   const int* __restrict__ col,
                                                                   const int* __restrict__ slot_edge,
                                                                   int* __restrict__ out_tri,
                                                                   unsigned int* __restrict__ missing) {
    __shared__ int s_c[kSubWarps][32 * 13];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t f0 = (int64_t)blockIdx.x * kSubThreads + 32 * w, f = f0 + lane;
    bool ok = false;
    if (f < nf) {
        const int v1 = tri[3 * f], v2 = tri[3 * f + 1], v3 = tri[3 * f + 2];
        // an inactive face for vtkSurface, a vertex id out of range or an edge missing from the
        // rings: reported, not subdivided
        if (!(v1 == v2 || v1 < 0 || v2 < 0 || v3 < 0 || v1 >= nv || v2 >= nv || v3 >= nv)) {
            const int p12 = ring_slot(row, col, v1, v2), p23 = ring_slot(row, col, v2, v3),
                      p31 = ring_slot(row, col, v3, v1);
            const int e12 = p12 >= 0 ? slot_edge[p12] : -1, e23 = p23 >= 0 ? slot_edge[p23] : -1,
                      e31 = p31 >= 0 ? slot_edge[p31] : -1;
            ok = (e12 | e23 | e31) >= 0;
            const int v4 = (int)(nv + e12), v5 = (int)(nv + e23), v6 = (int)(nv + e31);
            int* o = s_c[w] + 13 * lane;
            o[0] = v1; o[1] = v4;  o[2] = v6;
            o[3] = v4; o[4] = v2;  o[5] = v5;
            o[6] = v5; o[7] = v3;  o[8] = v6;
            o[9] = v4; o[10] = v5; o[11] = v6;
        }
        if (!ok) atomicAdd(missing, 1u);
    }
    const unsigned have = __ballot_sync(kFull, ok);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 12; j++) {
        const int at = lane + 32 * j, face = at / 12;
        if ((have >> face) & 1u) out_tri[12 * f0 + at] = s_c[w][at + face];
    }
}

}  // namespace

cudaError_t launch_subdivide(const double* xyz, int64_t nv, const int* tri, int64_t nf, const int* row,
                             const int* col, const int* edge_v, int64_t ne, const double* ind, int* slot_edge,
                             double* out_xyz, int* out_tri, int* parent1, int* parent2, double* out_ind,
                             unsigned int* missing, cudaStream_t s) {
    cudaError_t err = cudaMemsetAsync(slot_edge, 0xff, 2 * (size_t)ne * sizeof(int), s);
    if (err != cudaSuccess) return err;
    if (nv + ne > 0) {
        const unsigned edges = sgrid(ne, kSubThreads);
        ++g_launches;
        subdiv_points_kernel<<<3 * edges + sgrid(3 * nv, kSubThreads), kSubThreads, 0, s>>>(
            xyz, nv, edge_v, ne, row, col, ind, slot_edge, out_xyz, parent1, parent2, out_ind, edges);
    }
    if (nf > 0) {
        ++g_launches;
        subdiv_faces_kernel<<<sgrid(nf, kSubThreads), kSubThreads, 0, s>>>(tri, nf, nv, row, col, slot_edge, out_tri,
                                                                           missing);
    }
    return cudaGetLastError();
}

}  // namespace acvd
