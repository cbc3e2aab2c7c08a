// Device-wide primitives: exclusive scan, deterministic FP64 sum, stable radix sort.
#include "primitives.cuh"
#include "common.cuh"

#include <algorithm>

namespace acvd {

long long g_launches = 0;

cudaError_t Scratch::reserve(size_t need) {
    if (need <= bytes) return cudaSuccess;
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
    const size_t want = std::max(need, bytes * 2);
    cudaError_t e = cudaMalloc(&ptr, want);
    if (e == cudaSuccess) bytes = want;
    return e;
}

Scratch::~Scratch() {
    if (ptr) cudaFree(ptr);
}

// ---------------------------------------------------------------------------
// exclusive scan of uint32 (1024 threads x 2 elements per block)
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 1024;
constexpr int kScanTile = 2 * kScanThreads;

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// `in` and `out` may be the same array (in-place scans): each thread reads its
// own pair before the block's first barrier and writes it after the last, so
// neither pointer is declared __restrict__.
__global__ void __launch_bounds__(kScanThreads) scan_tile_kernel(const uint32_t* in, uint32_t* out, int64_t n,
                                                                 uint32_t* __restrict__ block_sums) {
    __shared__ uint32_t wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t base = (int64_t)blockIdx.x * kScanTile + 2 * tid;
    const uint32_t a = base < n ? in[base] : 0u;
    const uint32_t b = base + 1 < n ? in[base + 1] : 0u;
    const uint32_t pair = a + b;
    const uint32_t incl = warp_incl_scan(pair, lane);
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        const uint32_t w = wsum[lane];
        const uint32_t wi = warp_incl_scan(w, lane);
        wsum[lane] = wi - w;
        if (lane == 31 && block_sums) block_sums[blockIdx.x] = wi;
    }
    __syncthreads();
    const uint32_t excl = incl - pair + wsum[wid];
    if (base < n) out[base] = excl;
    if (base + 1 < n) out[base + 1] = excl + a;
}

__global__ void scan_add_kernel(uint32_t* __restrict__ out, int64_t n, const uint32_t* __restrict__ offs) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += offs[i / kScanTile];
}

// total = last exclusive prefix + last input (saved before an in-place scan)
__global__ void scan_total_kernel(const uint32_t* last_in, const uint32_t* out, int64_t n, uint32_t* total) {
    if (n == 0) { *total = 0; return; }
    *total = out[n - 1] + last_in[0];
}

static size_t scan_scratch_words(int64_t n) {
    size_t w = 0;
    while (n > kScanTile) {
        n = (n + kScanTile - 1) / kScanTile;
        w += (size_t)n + 1;
    }
    return w + 1;
}

static cudaError_t scan_rec(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* scratch, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int64_t nb = (n + kScanTile - 1) / kScanTile;
    if (nb == 1) {
        ++g_launches;
        scan_tile_kernel<<<1, kScanThreads, 0, s>>>(in, out, n, nullptr);
        return cudaGetLastError();
    }
    uint32_t* sums = scratch;
    ++g_launches;
    scan_tile_kernel<<<(unsigned)nb, kScanThreads, 0, s>>>(in, out, n, sums);
    cudaError_t e = scan_rec(sums, sums, nb, scratch + nb + 1, s);
    if (e != cudaSuccess) return e;
    ++g_launches;
    scan_add_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(out, n, sums);
    return cudaGetLastError();
}

cudaError_t exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* total_dev,
                               Scratch& scratch, cudaStream_t s) {
    // the total must be read before `out` overwrites `in` (in-place scan)
    const size_t words = scan_scratch_words(n) + 1;
    cudaError_t e = scratch.reserve(words * sizeof(uint32_t));
    if (e != cudaSuccess) return e;
    uint32_t* sc = (uint32_t*)scratch.ptr;
    uint32_t* last = sc + words - 1;
    if (total_dev && n > 0) {
        e = cudaMemcpyAsync(last, in + n - 1, sizeof(uint32_t), cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return e;
    }
    e = scan_rec(in, out, n, sc, s);
    if (e != cudaSuccess) return e;
    if (total_dev) {
        ++g_launches;
        scan_total_kernel<<<1, 1, 0, s>>>(last, out, n, total_dev);
        e = cudaGetLastError();
    }
    return e;
}

size_t scan_scratch_need(int64_t n) { return scan_scratch_words(n); }

cudaError_t exclusive_scan_u32_raw(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* scratch,
                                   size_t scratch_words, cudaStream_t s) {
    if (scratch_words < scan_scratch_words(n)) return cudaErrorInvalidValue;
    return scan_rec(in, out, n, scratch, s);
}

// ---------------------------------------------------------------------------
// deterministic FP64 sum: fixed-shape tree (256-thread blocks, 8 values/thread)
// ---------------------------------------------------------------------------

__global__ void sum_f64_kernel(const double* __restrict__ in, int64_t n, double* __restrict__ out) {
    sum_f64_chunk(in, n, blockIdx.x, out);
}

cudaError_t sum_f64(const double* in, int64_t n, double* out_dev, Scratch& scratch, cudaStream_t s) {
    const int64_t per = (int64_t)kSumThreads * kSumPer;
    int64_t nb = (n + per - 1) / per;
    if (nb < 1) nb = 1;
    const int64_t nb2 = (nb + per - 1) / per;
    cudaError_t e = scratch.reserve((size_t)(nb + nb2 + 2) * sizeof(double));
    if (e != cudaSuccess) return e;
    double* a = (double*)scratch.ptr;
    double* b = a + nb + 1;
    ++g_launches;
    sum_f64_kernel<<<(unsigned)nb, kSumThreads, 0, s>>>(in, n, a);
    const double* cur = a;
    int64_t m = nb;
    double* dst = b;
    double* other = a;
    while (m > 1) {
        const int64_t mb = (m + per - 1) / per;
        ++g_launches;
        sum_f64_kernel<<<(unsigned)mb, kSumThreads, 0, s>>>(cur, m, dst);
        cur = dst;
        m = mb;
        double* t = dst; dst = other; other = t;
    }
    e = cudaMemcpyAsync(out_dev, cur, sizeof(double), cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort.  Three kernels per pass: per-tile digit counts, one block
// per digit scanning its counts over the tiles, and the scatter.  A block sorts a
// tile of 256 x ITEMS elements; each of its warps walks a contiguous run of the tile
// 32 elements at a time, ranks inside a step come from __match_any_sync, so the
// order of equal digits is the input order.  The tile is put in digit order in
// shared memory before it is written, so that the stores of a digit are contiguous.
// counts are laid out digit-major: counts[digit * ntiles + tile], the digit totals
// behind them.
//
// The sorts here are short (a clustering's items by cluster: 10^4 to 2 x 10^7 pairs)
// and bound by the chain of a block's steps, not by bytes: with one warp walking 1024
// elements (32 dependent steps of a shared-memory update) a pass took 13-15 us of counts
// and 18-21 us of scatter for 10^4 pairs as for 5 x 10^5, and a scan of three to five
// launches between them; 4 or 8 elements per thread leave 4 or 8 such steps.  The coarse
// mesh of 524,288 items (18 passes) went from 3.01 to 2.41 ms, an isotropic solve of
// 10,242 items (8 passes) from 2.68 to 2.39 ms.
// ---------------------------------------------------------------------------
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;

template <int BITS, int ITEMS>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const uint32_t* __restrict__ keys, int64_t n,
                                                                  int shift, int64_t ntiles,
                                                                  uint32_t* __restrict__ counts) {
    constexpr int BINS = 1 << BITS;
    __shared__ uint32_t hist[BINS];
    for (int d = threadIdx.x; d < BINS; d += kSortThreads) hist[d] = 0u;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * (kSortThreads * ITEMS) + threadIdx.x;
    uint32_t k[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; j++) k[j] = base + j * kSortThreads < n ? keys[base + j * kSortThreads] : 0u;
#pragma unroll
    for (int j = 0; j < ITEMS; j++)
        if (base + j * kSortThreads < n) atomicAdd(&hist[(k[j] >> shift) & (BINS - 1u)], 1u);
    __syncthreads();
    for (int d = threadIdx.x; d < BINS; d += kSortThreads) counts[(int64_t)d * ntiles + blockIdx.x] = hist[d];
}

// exclusive scan of v over the block's 256 threads; total receives the sum
__device__ __forceinline__ uint32_t sort_block_scan(uint32_t v, uint32_t* wsum, uint32_t& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t incl = warp_incl_scan(v, lane);
    __syncthreads();   // an earlier scan is done with wsum
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    uint32_t before = 0u, all = 0u;
#pragma unroll
    for (int q = 0; q < kSortWarps; q++) {
        const uint32_t s = wsum[q];
        before += q < w ? s : 0u;
        all += s;
    }
    total = all;
    return before + incl - v;
}

// One block per digit: its counts over the tiles become exclusive offsets inside the
// digit, totals[digit] their sum.
__global__ void __launch_bounds__(kSortThreads) radix_rows_kernel(uint32_t* __restrict__ counts, int64_t ntiles,
                                                                  uint32_t* __restrict__ totals) {
    constexpr int PER = 4;
    __shared__ uint32_t wsum[kSortWarps];
    uint32_t* row = counts + (int64_t)blockIdx.x * ntiles;
    uint32_t carry = 0u;
    for (int64_t t0 = 0; t0 < ntiles; t0 += kSortThreads * PER) {
        const int64_t t = t0 + (int64_t)threadIdx.x * PER;
        uint32_t v[PER], sum = 0u;
#pragma unroll
        for (int j = 0; j < PER; j++) {
            v[j] = t + j < ntiles ? row[t + j] : 0u;
            sum += v[j];
        }
        uint32_t total;
        uint32_t at = carry + sort_block_scan(sum, wsum, total);
#pragma unroll
        for (int j = 0; j < PER; j++) {
            if (t + j < ntiles) row[t + j] = at;
            at += v[j];
        }
        carry += total;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

template <int BITS, int ITEMS>
__global__ void __launch_bounds__(kSortThreads) radix_scatter_kernel(
    const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals, uint32_t* __restrict__ okeys,
    uint32_t* __restrict__ ovals, int64_t n, int shift, int64_t ntiles, const uint32_t* __restrict__ offsets,
    const uint32_t* __restrict__ totals) {
    constexpr int BINS = 1 << BITS;
    constexpr int PER = BINS / kSortThreads;        // digits a thread scans
    constexpr int TILE = kSortThreads * ITEMS;
    __shared__ uint16_t run[kSortWarps][BINS];      // per warp: its elements of each digit so far
    __shared__ uint32_t sk[TILE], sv[TILE];         // the tile in digit order
    __shared__ uint32_t gpos[BINS];                 // output position of the digit's first element, less its place in the tile
    __shared__ uint16_t dpos[BINS];                 // place of the digit's first element in the tile
    __shared__ uint32_t wsum[kSortWarps];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * TILE;
    // every load first: the tile's pairs, the digits' totals and this tile's offsets
    uint32_t k[ITEMS], v[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
        const int64_t i = base + w * (32 * ITEMS) + j * 32 + lane;
        k[j] = i < n ? keys[i] : 0u;
        v[j] = i < n ? vals[i] : 0u;
    }
    uint32_t tot[PER], off[PER];
#pragma unroll
    for (int q = 0; q < PER; q++) {
        const int d = threadIdx.x * PER + q;
        tot[q] = totals[d];
        off[q] = offsets[(int64_t)d * ntiles + blockIdx.x];
    }
    for (int d = lane; d < BINS; d += 32) run[w][d] = 0;
    __syncwarp();
    // rank of every element among its warp's elements of the same digit
    uint16_t rank[ITEMS];
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
        const bool valid = base + w * (32 * ITEMS) + j * 32 + lane < n;
        const uint32_t d = valid ? (k[j] >> shift) & (BINS - 1u) : (uint32_t)BINS + lane;   // dummies: unique digits
        const unsigned peers = __match_any_sync(kFull, d);
        const uint16_t before = valid ? run[w][d] : (uint16_t)0;
        __syncwarp();
        if (valid && (peers & lt) == 0u) run[w][d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
        rank[j] = (uint16_t)(before + __popc(peers & lt));
    }
    __syncthreads();
    // digits: where each starts in the tile and in the output, and each warp's share of it
    uint32_t cnt[PER], sum = 0u, tsum = 0u;
#pragma unroll
    for (int q = 0; q < PER; q++) {
        const int d = threadIdx.x * PER + q;
        uint32_t c = 0u;
#pragma unroll
        for (int u = 0; u < kSortWarps; u++) {
            const uint32_t r = run[u][d];
            run[u][d] = (uint16_t)c;
            c += r;
        }
        cnt[q] = c;
        sum += c;
        tsum += tot[q];
    }
    uint32_t total;
    uint32_t at = sort_block_scan(sum, wsum, total);
    uint32_t gat = sort_block_scan(tsum, wsum, total);
#pragma unroll
    for (int q = 0; q < PER; q++) {
        const int d = threadIdx.x * PER + q;
        dpos[d] = (uint16_t)at;
        gpos[d] = gat + off[q] - at;
        at += cnt[q];
        gat += tot[q];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
        if (base + w * (32 * ITEMS) + j * 32 + lane >= n) continue;
        const uint32_t d = (k[j] >> shift) & (BINS - 1u);
        const uint32_t p = (uint32_t)dpos[d] + run[w][d] + rank[j];
        sk[p] = k[j];
        sv[p] = v[j];
    }
    __syncthreads();
    const int here = (int)(n - base < TILE ? n - base : TILE);
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
        const int p = j * kSortThreads + (int)threadIdx.x;
        if (p >= here) continue;
        const uint32_t key = sk[p];
        const uint32_t pos = gpos[(key >> shift) & (BINS - 1u)] + (uint32_t)p;
        okeys[pos] = key;
        ovals[pos] = sv[p];
    }
}

template <int BITS, int ITEMS>
static cudaError_t radix_pass(const uint32_t* ka, const uint32_t* va, uint32_t* kb, uint32_t* vb, int64_t n, int shift,
                              uint32_t* counts, cudaStream_t s) {
    constexpr int BINS = 1 << BITS;
    const int64_t ntiles = (n + kSortThreads * ITEMS - 1) / (kSortThreads * ITEMS);
    uint32_t* totals = counts + BINS * ntiles;
    g_launches += 3;
    radix_hist_kernel<BITS, ITEMS><<<(unsigned)ntiles, kSortThreads, 0, s>>>(ka, n, shift, ntiles, counts);
    radix_rows_kernel<<<BINS, kSortThreads, 0, s>>>(counts, ntiles, totals);
    radix_scatter_kernel<BITS, ITEMS><<<(unsigned)ntiles, kSortThreads, 0, s>>>(ka, va, kb, vb, n, shift, ntiles,
                                                                                counts, totals);
    return cudaGetLastError();
}

// 4 elements per thread up to this many pairs (512 tiles, about three blocks on each SM);
// above, 8 halve the counts' traffic
constexpr int64_t kSortShort = 512 * 4 * kSortThreads;

cudaError_t radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t* tmp_keys, uint32_t* tmp_vals, int64_t n,
                             int key_bits, Scratch& scratch, cudaStream_t s) {
    if (n <= 1) return cudaSuccess;
    // 8-bit digits, or 10-bit ones where they save a pass
    const int passes8 = (key_bits + 7) / 8, passes10 = (key_bits + 9) / 10;
    const bool wide = passes10 < passes8;
    const int passes = wide ? passes10 : passes8, bits = wide ? 10 : 8;
    const int64_t tile = kSortThreads * (n <= kSortShort && !wide ? 4 : 8);
    const int64_t bins = 1 << bits, ntiles = (n + tile - 1) / tile;
    cudaError_t e = scratch.reserve((size_t)(bins * ntiles + bins) * sizeof(uint32_t));
    if (e != cudaSuccess) return e;
    uint32_t* counts = (uint32_t*)scratch.ptr;
    uint32_t *ka = keys, *va = vals, *kb = tmp_keys, *vb = tmp_vals;
    for (int p = 0; p < passes; p++) {
        const int shift = bits * p;
        e = wide ? radix_pass<10, 8>(ka, va, kb, vb, n, shift, counts, s)
            : n <= kSortShort ? radix_pass<8, 4>(ka, va, kb, vb, n, shift, counts, s)
                              : radix_pass<8, 8>(ka, va, kb, vb, n, shift, counts, s);
        if (e != cudaSuccess) return e;
        uint32_t* t = ka; ka = kb; kb = t;
        t = va; va = vb; vb = t;
    }
    if (ka != keys) {
        e = cudaMemcpyAsync(keys, ka, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return e;
        e = cudaMemcpyAsync(vals, va, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s);
    }
    return e;
}

}  // namespace acvd
