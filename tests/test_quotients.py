"""div_rcp and div_any (quotients by a divisor whose reciprocal is at hand)
against the division, bit for bit, at the edges of their ranges (|b| in
[2^-300, 2^300], |a| in [2^-500, 2^500]), just past them, at signed zeros,
infinities, NaN and subnormals, and where the quotient lies closest to the
middle of two doubles.  The functions are compiled from the kernels' header
with the FP64 kernels' flags."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = """
#include "fw_kernels.cuh"
static __global__ void k_quot(const double *a, const double *b, double *q, int n, int rcp) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const double y = __drcp_rn(b[t]);
    q[t] = rcp ? fw::div_rcp(a[t], b[t], y) : fw::div_any(a[t], b[t], y);
}
extern "C" int quot(const double *a, const double *b, double *q, int n, int rcp) {
    double *d = nullptr;
    const size_t s = (size_t)n * sizeof(double);
    if (cudaMalloc(&d, 3 * s) != cudaSuccess) return 1;
    cudaMemcpy(d, a, s, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, s, cudaMemcpyHostToDevice);
    k_quot<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * (size_t)n, n, rcp);
    const int e = (int)cudaMemcpy(q, d + 2 * (size_t)n, s, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
"""


@pytest.fixture(scope="module")
def quot(tmp_path_factory):
    d = tmp_path_factory.mktemp("quot")
    src, so = d / "quot.cu", d / "quot.so"
    src.write_text(SRC)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-fmad=false", "-shared", "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "funwave-tvd_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def run(a, b, rcp):
        a, b = (np.ascontiguousarray(x, dtype=np.float64) for x in (a, b))
        q = np.empty_like(a)
        p = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, q)]
        assert lib.quot(*p, ctypes.c_int(a.size), ctypes.c_int(rcp)) == 0
        with np.errstate(all="ignore"):
            want = a / b
        bad = np.isnan(q) != np.isnan(want)
        bad |= ~np.isnan(want) & (q.view(np.uint64) != want.view(np.uint64))
        assert not bad.any(), (a[bad][:4], b[bad][:4], q[bad][:4], want[bad][:4])
    return run


def _random(rng, n, lo, hi):
    """n doubles of both signs, exponents in [lo, hi], random mantissas with a
    share of the extreme ones."""
    m = rng.integers(0, 1 << 52, size=n, dtype=np.uint64)
    pick = rng.integers(0, 8, size=n)
    few = rng.integers(0, 16, size=n, dtype=np.uint64)
    m = np.where(pick == 0, few, np.where(pick == 1, np.uint64((1 << 52) - 1) - few, m))
    e = rng.integers(lo, hi + 1, size=n).astype(np.int64) + 1023
    s = rng.integers(0, 2, size=n, dtype=np.uint64)
    return ((s << np.uint64(63)) | (e.astype(np.uint64) << np.uint64(52)) | m).view(np.float64)


N = 1 << 20


@pytest.mark.parametrize("span", [(0, 0), (-1, 1), (-300, 299), (-300, -299), (298, 299)])
@pytest.mark.parametrize("aspan", [(0, 0), (-500, 499), (-500, -499), (498, 499)])
def test_random_quotients(quot, span, aspan):
    rng = np.random.default_rng(abs(span[0]) * 7 + abs(aspan[0]))
    a, b = _random(rng, N, *aspan), _random(rng, N, *span)
    quot(a, b, 1)
    quot(a, b, 0)


def test_quotients_near_the_middle_of_two_doubles(quot):
    # odd 54-bit integers h and 53-bit b: a = b h / 2^k rounded to 53 bits has
    # a quotient within 2^-53 of the midpoint h
    rng = np.random.default_rng(4)
    b = rng.integers(1 << 52, 1 << 53, size=N // 4)
    h = 2 * rng.integers(1 << 52, 1 << 53, size=N // 4) + 1
    a = np.array([float(int(x) * int(y)) for x, y in zip(b, h)])
    quot(a, b.astype(np.float64), 1)
    quot(np.nextafter(a, 0.0), b.astype(np.float64), 1)
    quot(np.nextafter(a, np.inf), b.astype(np.float64), 0)


def test_any_numerator_and_divisor(quot):
    rng = np.random.default_rng(5)
    edges = []
    for e in (-300.0, 300.0, -500.0, 500.0, 0.0, -1022.0, -1074.0, 1023.0):
        x = np.ldexp(1.0, int(e))
        edges += [x, np.nextafter(x, 0.0), np.nextafter(x, np.inf)]
    edges += [0.0, np.inf, np.nan, 5e-324, 1.7976931348623157e308, 3.0, 0.1]
    edges = np.array(edges + [-x for x in edges])
    a, b = (x.ravel() for x in np.meshgrid(edges, edges))
    quot(a, b, 0)
    a = _random(rng, N, -1022, 1022)
    a[::7] = rng.choice(edges, size=a[::7].size)
    b = _random(rng, N, -1022, 1022)
    b[::11] = rng.choice(edges, size=b[::11].size)
    quot(a, b, 0)
    b = _random(rng, N, -300, 299)  # div_rcp: any numerator, divisors in range
    quot(a, b, 1)
