"""The device-wide primitives against numpy (needs a GB300): compiled with a small host
entry of their own, since the C ABI does not export them."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from acvd_gb300 import build

pytestmark = pytest.mark.gpu

HARNESS = r"""
#include "@SRC@/primitives.cu"
template <class T> struct Dev {
    T* p = nullptr;
    Dev(const T* h, size_t n) {
        cudaMalloc((void**)&p, (n + 1) * sizeof(T));
        if (h) cudaMemcpy(p, h, n * sizeof(T), cudaMemcpyHostToDevice);
    }
    ~Dev() { cudaFree(p); }
};
extern "C" int test_sort(unsigned* keys, unsigned* vals, long long n, int bits) {
    Dev<unsigned> k(keys, n), v(vals, n), tk(nullptr, n), tv(nullptr, n);
    acvd::Scratch sc;
    if (acvd::radix_sort_pairs(k.p, v.p, tk.p, tv.p, n, bits, sc, 0) != cudaSuccess) return 1;
    cudaMemcpy(keys, k.p, n * 4, cudaMemcpyDeviceToHost);
    cudaMemcpy(vals, v.p, n * 4, cudaMemcpyDeviceToHost);
    return (int)cudaDeviceSynchronize();
}
// the short roots and reciprocals against the IEEE operations: counts of differing bits
__global__ void roots_kernel(unsigned long long* bad) {
    const unsigned step = gridDim.x * blockDim.x;
    for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < (1u << 24); m += step) {
        // every significand, exponents 0 and 1, then the same far up the range
        for (int e = 0; e <= 80; e += 16) {
            const float x = ldexpf(__uint_as_float(0x3f800000u + m), e);
            if (acvd::root_rn(x) != __fsqrt_rn(x)) atomicAdd(&bad[0], 1ull);
            if (acvd::recip_rn(x) != __frcp_rn(x)) atomicAdd(&bad[1], 1ull);
        }
        // t^2 + 1 lies in [1, 2]
        const float u = 1.0f + (float)m * 0x1p-24f;
        if (acvd::recip_rn(acvd::root_rn(u)) != __frcp_rn(__fsqrt_rn(u))) atomicAdd(&bad[2], 1ull);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        if (acvd::recip_rn(acvd::root_rn(2.0f)) != __frcp_rn(__fsqrt_rn(2.0f))) atomicAdd(&bad[2], 1ull);
}
// quotients by a shared reciprocal against the IEEE division: random significands, exponents
// within +-60
__global__ void quotient_kernel(unsigned long long seed, unsigned per, unsigned long long* bad) {
    unsigned long long x = seed + (unsigned long long)(blockIdx.x * blockDim.x + threadIdx.x) * 0x9e3779b97f4a7c15ull;
    auto next = [&]() {   // splitmix64 (Steele, Lea, Flood 2014)
        unsigned long long z = (x += 0x9e3779b97f4a7c15ull);
        z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
        return z ^ (z >> 31);
    };
    auto number = [&]() {
        const unsigned long long u = next();
        const unsigned long long e = 1023ull - 60ull + (next() % 121ull);
        return __longlong_as_double((long long)((u & 0x800fffffffffffffull) | (e << 52)));
    };
    unsigned long long n = 0;
    for (unsigned i = 0; i < per; i++) {
        const double b = number(), inv = 1.0 / b;
        for (int j = 0; j < 8; j++) {
            const double a = number();
            n += acvd::quotient(a, b, inv) != a / b;
        }
    }
    if (n) atomicAdd(bad, n);
}
extern "C" int test_quotients(unsigned long long seed, unsigned long long* bad) {
    Dev<unsigned long long> d(bad, 1);
    quotient_kernel<<<4096, 256>>>(seed, 512, d.p);   // 2^20 threads x 512 divisors x 8
    cudaMemcpy(bad, d.p, 8, cudaMemcpyDeviceToHost);
    return (int)cudaDeviceSynchronize();
}
extern "C" int test_roots(unsigned long long* bad) {
    Dev<unsigned long long> d(bad, 3);
    roots_kernel<<<2048, 256>>>(d.p);
    cudaMemcpy(bad, d.p, 24, cudaMemcpyDeviceToHost);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("prim")
    src, so = d / "harness.cu", d / "harness.so"
    src.write_text(HARNESS.replace("@SRC@", build.SRC))
    subprocess.run([build._nvcc(), build.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-o", str(so),
                    str(src), "-lcudart"], check=True, capture_output=True)
    return ctypes.CDLL(str(so))


# the edges of the tiles (1,024 and 2,048 pairs), of the short form (512 tiles of 1,024) and of
# the row scan (1,024 tiles), for 1 to 4 passes of 8 bits and 2 and 3 of 10
@pytest.mark.parametrize("n", [2, 31, 1023, 1024, 1025, 2049, 4097, 524287, 524289, 2100003])
@pytest.mark.parametrize("bits", [1, 8, 15, 17, 20, 24, 26, 32])
def test_radix_sort_is_stable(lib, n, bits):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    if n % 2:   # few distinct keys: long runs of equal digits
        keys = keys[rng.integers(0, min(n, 5), n)]
    vals = np.arange(n, dtype=np.uint32)
    order = np.argsort(keys, kind="stable")
    k, v = keys.copy(), vals.copy()
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert lib.test_sort(P(k), P(v), ctypes.c_longlong(n), bits) == 0
    np.testing.assert_array_equal(k, keys[order])
    np.testing.assert_array_equal(v, vals[order])


def test_short_roots_and_reciprocals_are_correctly_rounded(lib):
    bad = np.zeros(3, dtype=np.uint64)
    assert lib.test_roots(bad.ctypes.data_as(ctypes.c_void_p)) == 0
    np.testing.assert_array_equal(bad, 0)


def test_quotients_by_a_shared_reciprocal(lib):
    bad = np.zeros(1, dtype=np.uint64)
    assert lib.test_quotients(ctypes.c_ulonglong(12345), bad.ctypes.data_as(ctypes.c_void_p)) == 0
    assert bad[0] == 0
