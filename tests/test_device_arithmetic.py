"""The short reciprocal, reciprocal root and quotient of csrc/wcns_dev.cuh against
their values in extended precision and against CUDA's own operators.

Bounds, from the steps themselves (u = 2^-53, one ulp of a result is between u and 2u
of it).  recip: the approximation's error e, 2^-19.9, leaves e^3 = 2^-59.7 after the third
order step, the last addition rounds once: 0.5 ulp + 2^-6.7 ulp < 0.51.  recip_sqrt: the
rounded product x*y moves e by u, half of which reaches the result (0.5 ulp at most),
5/16 e^3 and the last rounding: 0.5 + 0.5 + 2^-8 < 1.02.  div_by: Markstein's corrected
quotient of a correctly rounded reciprocal is the rounded quotient unless the first
quotient is more than one ulp off and the remainder falls near a tie; none of the
samples below may differ from CUDA's division."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from wcns_b200 import build

pytestmark = pytest.mark.gpu

PROBE = r"""
#include <cuda_runtime.h>
#include "wcns_dev.cuh"
using namespace wcns;
__global__ void k(int op, const double *a, const double *b, double *o, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double r = 0.0;
    if (op == 0) r = recip(a[i]);
    else if (op == 1) r = recip_sqrt(a[i]);
    else if (op == 2) r = div_by(a[i], b[i], 1.0 / b[i]);
    else if (op == 3) asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a[i]));
    else if (op == 4) asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a[i]));
    else if (op == 5) r = 1.0 / a[i];
    else if (op == 6) r = 1.0 / sqrt(a[i]);
    else r = a[i] / b[i];
    o[i] = r;
}
extern "C" int probe(int op, const double *a, const double *b, double *o, long long n) {
    double *d[3] = {};
    const size_t s = sizeof(double) * (size_t)n;
    cudaError_t e = cudaSuccess;
    for (int q = 0; q < 3 && e == cudaSuccess; q++) e = cudaMalloc(&d[q], s);
    if (e == cudaSuccess) e = cudaMemcpy(d[0], a, s, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d[1], b, s, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k<<<(unsigned)((n + 255) / 256), 256>>>(op, d[0], d[1], d[2], n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(o, d[2], s, cudaMemcpyDeviceToHost);
    for (double *p : d) cudaFree(p);
    return (int)e;
}
"""
RECIP, RSQRT, DIV, RCP_APPROX, RSQRT_APPROX, CUDA_RECIP, CUDA_RSQRT, CUDA_DIV = range(8)
N = 1 << 22


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("arith")
    (d / "probe.cu").write_text(PROBE)
    lib = str(d / "probe.so")
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-shared", "-I", build.CSRC, "-I", os.path.join(build.HERE, "..", "include"),
                    str(d / "probe.cu"), "-o", lib], check=True)
    fn = ctypes.CDLL(lib).probe
    fn.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 3 + [ctypes.c_longlong]

    def run(op, a, b=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = np.ascontiguousarray(np.broadcast_to(1.0 if b is None else b, a.shape), dtype=np.float64)
        out = np.empty_like(a)
        assert fn(op, a.ctypes.data, b.ctypes.data, out.ctypes.data, a.size) == 0
        return out
    return run


def _spread(rng, lo, hi, n=N):
    """Exponents evenly over the range, with mantissas next to powers of two among them."""
    x = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    near = 2.0 ** rng.integers(int(np.log2(lo)) + 1, int(np.log2(hi)), n // 8)
    x[:n // 8] = near * (1.0 + rng.integers(-64, 64, n // 8) * 2.0 ** -52)
    return x


def _ulps(got, exact):
    return float(np.max(np.abs((got.astype(np.longdouble) - exact) / np.spacing(np.abs(got)))))


def test_recip(probe):
    x = _spread(np.random.default_rng(1), 1e-28, 1e40)  # sums of weights (1.6e-23 up), densities, 1 + root
    exact = 1.0 / x.astype(np.longdouble)
    assert float(np.max(np.abs(probe(RCP_APPROX, x) / exact - 1.0))) < 2.0 ** -19.9
    assert _ulps(probe(RECIP, x), exact) <= 0.51
    assert _ulps(probe(RECIP, -x), -exact) <= 0.51
    assert float(np.max(np.abs(probe(RECIP, x) - probe(CUDA_RECIP, x)) / np.spacing(probe(CUDA_RECIP, x)))) <= 1.0


def test_recip_sqrt(probe):
    x = _spread(np.random.default_rng(2), 1e-290, 1e40)  # the floor of the roots, ratios, squared speeds and normals
    exact = 1.0 / np.sqrt(x.astype(np.longdouble))
    assert float(np.max(np.abs(probe(RSQRT_APPROX, x) / exact - 1.0))) < 2.0 ** -19.9
    got = probe(RSQRT, x)
    assert _ulps(got, exact) <= 1.02
    # CUDA's own: a rounded root, 0.5 ulp, half of which reaches the rounded reciprocal: 1 ulp at most
    assert float(np.max(np.abs(got - probe(CUDA_RSQRT, x)) / np.spacing(got))) <= 2.0


@pytest.mark.parametrize("b", [1920.0, 24.0, 12.0, 6.0, 1.4 - 1.0, None], ids=str)
def test_div_by(probe, b):
    rng = np.random.default_rng(3)
    bs = _spread(rng, 1e-12, 1e4) if b is None else np.full(N, b)  # None: volumes
    a = _spread(rng, 1e-30, 1e12) * rng.choice([-1.0, 1.0], N)
    a[:1024] = np.arange(1024.0)
    np.testing.assert_array_equal(probe(DIV, a, bs), probe(CUDA_DIV, a, bs))


def test_special_values(probe):
    """What the comments state: NaN stays NaN, a negative root is NaN, and where an
    operand is zero, infinite or subnormal recip and recip_sqrt give no finite number;
    div_by gives what a division gives."""
    inf, nan = np.inf, np.nan
    assert np.isnan(probe(RECIP, [0.0, -0.0, inf, -inf, nan])).all()
    assert np.isnan(probe(RSQRT, [0.0, -0.0, inf, nan, -1.0, -inf])).all()
    assert not np.isfinite(probe(RECIP, [1e-310, -1e-310])).any()
    assert not np.isfinite(probe(RSQRT, [1e-310])).any()
    a = np.repeat([inf, -inf, nan, 0.0, -0.0, 1.5, -1.5], 6)
    b = np.tile([1920.0, -24.0, 0.0, inf, -inf, nan], 7)
    np.testing.assert_array_equal(probe(DIV, a, b), probe(CUDA_DIV, a, b))
