"""Quotients by a shared reciprocal (needs a GB300), bit for bit against the IEEE division:
numerators of every exponent, the smallest and largest, zeros of both signs, infinities and
NaN, by divisors over the whole range that quotient() takes; then 2^33 random quotients, each
thread's numbers from a stretch of its own.  Compiled with and without FMA contraction, as
the files that use it are.
"""
import ctypes
import subprocess

import numpy as np
import pytest

from acvd_gb300 import build

pytestmark = pytest.mark.gpu

HARNESS = r"""
#include "@SRC@/common.cuh"
__global__ void quotients(const double* a, int na, const double* b, int nb, unsigned long long* bad) {
    for (long long i = blockIdx.x * blockDim.x + threadIdx.x; i < (long long)na * nb; i += gridDim.x * blockDim.x) {
        const double x = a[i % na], y = b[i / na];
        const double q = acvd::quotient(x, y, 1.0 / y), w = x / y;
        const bool same = __double_as_longlong(q) == __double_as_longlong(w) || (q != q && w != w);
        if (!same) atomicAdd(bad, 1ull);
    }
}
__device__ unsigned long long mix(unsigned long long z) {   // splitmix64 (Steele, Lea, Flood 2014)
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
// thread t's states are seed + gamma * [t * 18 * per, (t + 1) * 18 * per): no two threads meet
__global__ void drawn(unsigned long long seed, unsigned per, unsigned long long* bad) {
    const unsigned long long gamma = 0x9e3779b97f4a7c15ull;
    unsigned long long x = seed + gamma * (18ull * per * (blockIdx.x * blockDim.x + threadIdx.x));
    auto number = [&]() {
        const unsigned long long u = mix(x += gamma), e = 1023ull - 60ull + mix(x += gamma) % 121ull;
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
static int finish(unsigned long long* d, unsigned long long* bad) {
    cudaMemcpy(bad, d, 8, cudaMemcpyDeviceToHost);
    return (int)cudaDeviceSynchronize();
}
extern "C" int test_quotients(const double* a, int na, const double* b, int nb, unsigned long long* bad) {
    double* d;
    if (cudaMalloc(&d, (na + nb + 1) * 8) != cudaSuccess) return 1;
    unsigned long long* n = (unsigned long long*)(d + na + nb);
    cudaMemcpy(d, a, na * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(d + na, b, nb * 8, cudaMemcpyHostToDevice);
    cudaMemset(n, 0, 8);
    quotients<<<2048, 256>>>(d, na, d + na, nb, n);
    const int e = finish(n, bad);
    cudaFree(d);
    return e;
}
extern "C" int test_drawn(unsigned long long seed, unsigned long long* bad) {
    unsigned long long* n;
    if (cudaMalloc(&n, 8) != cudaSuccess) return 1;
    cudaMemset(n, 0, 8);
    drawn<<<4096, 256>>>(seed, 1024, n);   // 2^20 threads x 2^10 divisors x 8
    const int e = finish(n, bad);
    cudaFree(n);
    return e;
}
"""


@pytest.fixture(scope="module", params=["true", "false"])
def lib(tmp_path_factory, request):
    d = tmp_path_factory.mktemp("quot")
    src, so = d / "harness.cu", d / "harness.so"
    src.write_text(HARNESS.replace("@SRC@", build.SRC))
    subprocess.run([build._nvcc(), build.ARCH, "-O3", "-std=c++17", "-fmad=" + request.param, "-shared", "-Xcompiler",
                    "-fPIC", "-o", str(so), str(src), "-lcudart"], check=True, capture_output=True)
    return ctypes.CDLL(str(so))


def test_every_exponent(lib):
    rng = np.random.default_rng(3)
    frac = np.concatenate([[0, 1, (1 << 52) - 1], rng.integers(0, 1 << 52, 13)]).astype(np.uint64)
    exps = np.arange(0, 2048, dtype=np.uint64)   # denormals and zero to infinities and NaN
    mag = ((exps[:, None] << np.uint64(52)) | frac[None, :]).reshape(-1)
    a = np.concatenate([mag, mag | np.uint64(1 << 63)]).view(np.float64)
    # divisors: 2^-465 <= |b| < 2^465, its ends and powers of two among them
    e = np.concatenate([np.arange(-465, 465, 31), [-465, -464, -1, 0, 1, 463, 464]])
    b = (1.0 + rng.random((e.size, 4))) * np.exp2(e)[:, None]
    b[:, 0] = np.exp2(e)
    b[:, 1] = np.nextafter(2.0, 1.0) * np.exp2(e)
    b = np.concatenate([b.reshape(-1), -b.reshape(-1)])
    bad = np.zeros(1, dtype=np.uint64)
    P = lambda v: v.ctypes.data_as(ctypes.c_void_p)
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    assert lib.test_quotients(P(a), a.size, P(b), b.size, P(bad)) == 0
    assert bad[0] == 0


def test_drawn_quotients(lib):
    bad = np.zeros(1, dtype=np.uint64)
    assert lib.test_drawn(ctypes.c_ulonglong(987654321), bad.ctypes.data_as(ctypes.c_void_p)) == 0
    assert bad[0] == 0
