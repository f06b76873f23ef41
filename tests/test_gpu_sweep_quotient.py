"""The sweeps' shared quotient (div_by and add_neg_quot of ofg_device.cuh) against
the division it stands for, bit by bit: every sign of zero, divisors of both signs,
subnormal numbers, infinities, NaN, the edges of the range in which no division is
made, and quotients next to a rounding boundary.  Compiled here with the flags of
both paths' units."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "ofg_device.cuh"
using namespace ofg;
// per pair: y / d, x + (-y) / d; by N = 1; by N = 5 with the pair's y in place k % 5 and others beside it
__global__ void k_quot(int n, const double *x, const double *y, const double *d, double *one, double *five, double *sub,
                       double *plain, double *plainSub) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Divisor v = make_divisor(d[i]);
    double q;
    div_by<1>(y + i, v, &q);
    one[i] = q;
    double a[5], b[5];
    const int at = i % 5;
    for (int e = 0; e < 5; ++e) a[e] = e == at ? y[i] : e + 1.0;
    div_by<5>(a, v, b);
    five[i] = b[at];
    double s = x[i];
    add_neg_quot<1>(&s, y + i, v);
    sub[i] = s;
    plain[i] = y[i] / d[i];
    plainSub[i] = x[i] + (-y[i]) / d[i];
}
extern "C" int run(int n, const double *in, double *out) {   // in: x y d, out: one five sub plain plainSub
    double *a = nullptr, *b = nullptr;
    const size_t row = size_t(n) * sizeof(double);
    if (cudaMalloc(&a, 3 * row) != cudaSuccess || cudaMalloc(&b, 5 * row) != cudaSuccess) return 1;
    int rc = cudaMemcpy(a, in, 3 * row, cudaMemcpyHostToDevice) != cudaSuccess;
    if (!rc) {
        k_quot<<<(n + 127) / 128, 128>>>(n, a, a + n, a + 2 * (size_t)n, b, b + n, b + 2 * (size_t)n, b + 3 * (size_t)n,
                                         b + 4 * (size_t)n);
        rc = cudaMemcpy(out, b, 5 * row, cudaMemcpyDeviceToHost) != cudaSuccess;
    }
    cudaFree(a);
    cudaFree(b);
    return rc;
}
"""
FLAGS = {"fp64": ["-fmad=false"], "mixed": ["-prec-div=false", "-prec-sqrt=false", "-ftz=true"]}


@pytest.fixture(scope="module", params=sorted(FLAGS))
def quotients(request, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("quot")
    (d / "quot.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    *FLAGS[request.param], "-I", os.path.join(ROOT, "oneflow_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-o", str(d / "quot.so"), str(d / "quot.cu")], check=True)
    L = C.CDLL(str(d / "quot.so"))

    def f(x, y, d):
        a = np.ascontiguousarray(np.stack([x, y, d]), np.float64)
        out = np.empty((5, len(x)))
        assert L.run(len(x), a.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p)) == 0
        return out
    return f


def same(a, b):
    return (a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))


def check(f, x, y, d):
    one, five, sub, plain, plain_sub = f(x, y, d)
    with np.errstate(all="ignore"):
        host, host_sub = y / d, x + (-y) / d
    for got, want in ((plain, host), (plain_sub, host_sub), (one, host), (five, host), (sub, host_sub)):
        ok = same(got, want)
        assert ok.all(), [(a[~ok][:4]) for a in (x, y, d, got, want)]


def test_special_numbers(quotients):
    e = [2.0 ** k for k in (-1074, -1073, -1023, -1022, -1021, -600, -301, -300, -299, -1, 0, 1, 299, 300, 301, 600, 1023)]
    v = np.array([0.0, np.inf, np.nan, 1.0 / 3.0, np.pi] + e + [np.nextafter(a, np.inf) for a in e] +
                 [np.nextafter(a, 0.0) for a in e])
    v = np.concatenate([v, -v])
    y, d = (a.ravel() for a in np.meshgrid(v, v))
    for x in (0.0, -0.0, 1.0, -np.inf):
        check(quotients, np.full(len(y), x), y, d)


@pytest.mark.parametrize("span", [3, 40, 299, 1022])
def test_random_numbers(quotients, span):
    rng = np.random.default_rng(span)
    n = 1 << 20

    def draw():
        return np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-span, span, n)) * rng.choice([-1.0, 1.0], n)
    check(quotients, draw(), draw(), draw())


def test_quotients_next_to_a_rounding_boundary(quotients):
    """y = q d rounded, and its neighbours; divisors and quotients with few or nearly all
    bits set among them"""
    rng = np.random.default_rng(5)
    n = 1 << 20

    def mantissa():
        m = rng.integers(1 << 52, 1 << 53, n)
        few = (1 << 52) + (np.int64(1) << rng.integers(0, 52, n))
        full = (1 << 53) - 1 - rng.integers(0, 4, n)
        return np.choose(rng.integers(0, 3, n), [m, few, full]).astype(np.float64)
    d, q = mantissa(), mantissa()
    y = q * d
    for k in range(-2, 3):
        t = y
        for _ in range(abs(k)):
            t = np.nextafter(t, np.inf if k > 0 else 0.0)
        check(quotients, q, t, d)
        check(quotients, q, -t, d)
