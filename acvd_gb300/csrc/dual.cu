// The dual (coarse) mesh of a clustering: one triangle per input face whose three labels
// are valid and distinct, in face order, the first face of every label set only
// (BuildDelaunayTriangulation, DiscreteRemeshing/vtkDiscreteRemeshing.h:1003-1152).
//
// The label sets go through a hash table that keeps the smallest face of each; a bit per
// face marks those, and the marked faces' triangles are written at the prefix sums of the
// bits.  The order of the insertions does not matter, so the result does not depend on
// thread timing.  It is bound by its launches and the label gathers of one pass over the
// faces: 4 kernels, 29 us at 1,048,576 faces and 40,000 triangles, where compacting the
// candidate faces, sorting their 63-bit keys in two 32-bit halves and compacting again took
// some 40 kernels (140 us), 14 allocations and three host round trips.
#include "state.cuh"

#include "primitives.cuh"

namespace acvd {

namespace {

constexpr unsigned long long kNoKey = ~0ull;   // no label set: labels stay below 2^21
constexpr int kDualThreads = 256;
constexpr int kDualWords = 4;                  // words of face bits per thread

inline unsigned dgrid(int64_t n, int b = kDualThreads) { return (unsigned)((n + b - 1) / b); }

__device__ __forceinline__ unsigned dual_hash(unsigned long long x) {
    x ^= x >> 31;
    x *= 0x9e3779b97f4a7c15ull;   // Fibonacci hashing (Knuth, vol. 3, 6.4)
    return (unsigned)(x >> 32);
}

// keys / first: 2^n slots (mask = slots - 1).  A set that finds no slot within `probes`
// steps sets *full.
__global__ void dual_insert_kernel(const int* __restrict__ tri, int64_t nf, const int* __restrict__ label, int k,
                                   unsigned long long* __restrict__ keys, unsigned* __restrict__ first,
                                   unsigned mask, unsigned probes, unsigned* __restrict__ full) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    int a = label[tri[3 * f]], b = label[tri[3 * f + 1]], c = label[tri[3 * f + 2]];
    if (!(a < k && b < k && c < k && a >= 0 && b >= 0 && c >= 0 && a != b && b != c && a != c)) return;
    if (a > b) { const int t = a; a = b; b = t; }
    if (b > c) { const int t = b; b = c; c = t; }
    if (a > b) { const int t = a; a = b; b = t; }
    const unsigned long long key = ((unsigned long long)a << 42) | ((unsigned long long)b << 21) | (unsigned long long)c;
    unsigned at = dual_hash(key) & mask;
    for (unsigned p = 0; p < probes; p++, at = (at + 1u) & mask) {
        unsigned long long held = *(volatile unsigned long long*)(keys + at);
        if (held == kNoKey) held = atomicCAS(keys + at, kNoKey, key);
        if (held == kNoKey || held == key) {
            atomicMin(first + at, (unsigned)f);
            return;
        }
    }
    *full = 1u;
}

__global__ void dual_mark_kernel(const unsigned* __restrict__ first, int64_t slots, unsigned* __restrict__ bits) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= slots) return;
    const unsigned f = first[s];
    if (f != ~0u) atomicOr(bits + (f >> 5), 1u << (f & 31u));
}

// marked faces of every block's words (the bits are padded to whole blocks)
__global__ void __launch_bounds__(kDualThreads) dual_count_kernel(const uint4* __restrict__ bits,
                                                                  unsigned* __restrict__ counts) {
    __shared__ unsigned s[kDualThreads / 32];
    const uint4 w = bits[(int64_t)blockIdx.x * kDualThreads + threadIdx.x];
    const unsigned n = __reduce_add_sync(kFull, __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w));
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (int q = 0; q < kDualThreads / 32; q++) t += s[q];
        counts[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(kDualThreads) dual_write_kernel(const uint4* __restrict__ bits,
                                                                  const unsigned* __restrict__ counts,
                                                                  const int* __restrict__ tri,
                                                                  const int* __restrict__ label, int* __restrict__ out,
                                                                  unsigned* __restrict__ total) {
    __shared__ unsigned s_before[kDualThreads / 32], s_warp[kDualThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // marked faces of the blocks before this one
    unsigned before = 0;
    for (unsigned b = threadIdx.x; b < blockIdx.x; b += kDualThreads) before += counts[b];
    before = __reduce_add_sync(kFull, before);
    const uint4 v = bits[(int64_t)blockIdx.x * kDualThreads + threadIdx.x];
    const unsigned w[kDualWords] = {v.x, v.y, v.z, v.w};
    unsigned mine = 0;
#pragma unroll
    for (int q = 0; q < kDualWords; q++) mine += __popc(w[q]);
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 0) s_before[wid] = before;
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    unsigned at = incl - mine;
    for (int q = 0; q < kDualThreads / 32; q++) at += s_before[q] + (q < wid ? s_warp[q] : 0u);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == kDualThreads - 1) *total = at + mine;
    const int64_t f0 = ((int64_t)blockIdx.x * kDualThreads + threadIdx.x) * (32 * kDualWords);
#pragma unroll
    for (int q = 0; q < kDualWords; q++)
        for (unsigned m = w[q]; m; m &= m - 1u) {
            const int64_t f = f0 + 32 * q + (__ffs((int)m) - 1);
            int* o = out + 3 * (int64_t)at++;
            for (int j = 0; j < 3; j++) o[j] = label[tri[3 * f + j]];
        }
}

}  // namespace

static int64_t dual_blocks(int64_t nf) {
    const int64_t per = 32 * kDualWords * kDualThreads;   // faces per block of bits
    return (nf + per - 1) / per;
}

size_t dual_work_bytes(int64_t nf, int64_t slots) {
    return (size_t)slots * 12 + (size_t)dual_blocks(nf) * (kDualWords * kDualThreads * 4 + 4) + 32;
}

cudaError_t launch_dual(const int* tri, int64_t nf, const int* label, int k, int64_t slots, unsigned probes,
                        void* work, int* out, unsigned* total_full, cudaStream_t s) {
    const int64_t nb = dual_blocks(nf);
    unsigned long long* keys = (unsigned long long*)work;
    unsigned* first = (unsigned*)(keys + slots);
    unsigned* bits = first + slots;   // slots: a multiple of 4, so 16-byte aligned
    unsigned* counts = bits + nb * kDualWords * kDualThreads;
    cudaError_t e = cudaMemsetAsync(work, 0xff, (size_t)slots * 12, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(bits, 0, (size_t)nb * kDualWords * kDualThreads * 4, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(total_full, 0, 2 * sizeof(unsigned), s);
    if (e != cudaSuccess || nf == 0) return e;
    g_launches += 4;
    dual_insert_kernel<<<dgrid(nf), kDualThreads, 0, s>>>(tri, nf, label, k, keys, first, (unsigned)(slots - 1), probes,
                                                          total_full + 1);
    dual_mark_kernel<<<dgrid(slots), kDualThreads, 0, s>>>(first, slots, bits);
    dual_count_kernel<<<(unsigned)nb, kDualThreads, 0, s>>>((const uint4*)bits, counts);
    dual_write_kernel<<<(unsigned)nb, kDualThreads, 0, s>>>((const uint4*)bits, counts, tri, label, out, total_full);
    return cudaGetLastError();
}

}  // namespace acvd
