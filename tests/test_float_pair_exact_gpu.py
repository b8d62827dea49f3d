"""Every routine of float_pair.cuh against its double form on the device, bit for bit, compiled here from the header:
over the lobes' ranges, around the switches to the double form and outside the ranges."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from pico_gb300 import build

pytestmark = pytest.mark.gpu

f = np.float32
SOURCE = r"""
#include "float_pair.cuh"
using namespace pico::pair;
__global__ void kernel(int what, size_t n, const float* a, const float* b, const float* c, float2* pairs, float2* doubles)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (what == 0) {
            pairs[i] = make_float2(two_pi_times(a[i]), 0.0f);
            doubles[i] = make_float2(two_pi_times_double(a[i]), 0.0f);
        } else if (what == 1) {
            pairs[i] = circle(a[i], b[i]);
            doubles[i] = circle_double(a[i], b[i]);
        } else {
            pairs[i] = make_float2(quotient_by_pi(a[i], b[i], c[i]), 0.0f);
            doubles[i] = make_float2(quotient_double(a[i], b[i], c[i]), 0.0f);
        }
    }
}
extern "C" int run(int what, size_t n, const float* a, const float* b, const float* c, float2* pairs, float2* doubles)
{
    float* in[3] = {nullptr, nullptr, nullptr};
    float2* out[2] = {nullptr, nullptr};
    const float* from[3] = {a, b, c};
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 3 && e == cudaSuccess; ++k) {
        e = cudaMalloc(&in[k], n * sizeof(float));
        if (e == cudaSuccess) e = cudaMemcpy(in[k], from[k], n * sizeof(float), cudaMemcpyHostToDevice);
    }
    for (int k = 0; k < 2 && e == cudaSuccess; ++k) e = cudaMalloc(&out[k], n * sizeof(float2));
    if (e == cudaSuccess) {
        kernel<<<1024, 256>>>(what, n, in[0], in[1], in[2], out[0], out[1]);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(pairs, out[0], n * sizeof(float2), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(doubles, out[1], n * sizeof(float2), cudaMemcpyDeviceToHost);
    for (float* p : in) cudaFree(p);
    for (float2* p : out) cudaFree(p);
    return (int)e;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs")
    (d / "pairs.cu").write_text(SOURCE)
    flags = [x for x in build._flags(d / "pairs.cu") if x not in ("-Xptxas", "-v")]
    subprocess.run([build.nvcc_path(), *flags, "-shared", "-cudart", "shared", "-o", str(d / "libpairs.so"),
                    str(d / "pairs.cu")], check=True, capture_output=True)
    lib = C.CDLL(str(d / "libpairs.so"))

    def call(what, *args):
        args = [np.ascontiguousarray(x, f) for x in np.broadcast_arrays(*(list(args) + [f(0)] * (3 - len(args))))]
        n = args[0].size
        out = [np.empty((n, 2), f) for _ in range(2)]
        assert lib.run(what, C.c_size_t(n), *[x.ctypes.data_as(C.c_void_p) for x in args + out]) == 0
        same = (out[0].view(np.uint32) == out[1].view(np.uint32)) | (np.isnan(out[0]) & np.isnan(out[1]))
        bad = np.nonzero(~same.all(axis=1))[0]
        assert len(bad) == 0, [len(bad)] + [([float(x.flat[k]).hex() for x in args], out[0][k], out[1][k]) for k in bad[:8]]

    return call


def _around(values, steps=40):
    """The floats up to `steps` ulps below and above each value."""
    v = np.array(values, f).view(np.int32)[:, None] + np.arange(-steps, steps + 1)
    return v.astype(np.int32).ravel().view(f)


ODD = np.array([0.0, -0.0, 1e-45, 1e-38, 1e-30, 3e38, np.inf, -np.inf, np.nan, -1.0, -1e-20], f)


def test_two_pi_times(run):
    rng = np.random.default_rng(1)
    run(0, rng.integers(0, 2**32, 1 << 22).astype(f) / f(2**32))
    run(0, np.concatenate([_around([0.125, 0.25, 0.5, 1.0, 1.5]), ODD, np.arange(1 << 16, dtype=f) / f(1 << 16)]))


def test_circle(run):
    rng = np.random.default_rng(2)
    u = (rng.integers(0, 2**32, (2, 1 << 22)).astype(f)) / f(2**32)
    run(1, np.sqrt(u[0]), (u[1].astype(np.float64) * np.pi * 2.0).astype(f))
    quadrants = _around([0.0, np.pi / 4, np.pi / 2, np.pi, 3 * np.pi / 2, 2 * np.pi, 6.5], 500)
    radii = np.concatenate([f(2.0) ** -np.arange(0, 60, 3, dtype=f), ODD])
    run(1, np.repeat(radii, len(quadrants)), np.tile(quadrants, len(radii)))
    run(1, np.repeat(radii, len(ODD)), np.tile(ODD, len(radii)))


def test_quotient_by_pi(run):
    rng = np.random.default_rng(3)
    n = 1 << 22
    # the Beckmann distribution: e = exp(-x), alpha of roughness 0.001 to 1, cos^4
    e = np.exp(-rng.exponential(4.0, n)).astype(f)
    alpha = np.exp(rng.uniform(np.log(1e-4), np.log(1.7), n)).astype(f)
    run(2, e, alpha, (rng.random(n) ** 4).astype(f))
    # over the exponents: results and divisors around the double form's switches, to underflow and overflow
    log = lambda lo, hi: np.exp(rng.uniform(np.log(lo), np.log(hi), n)).astype(f)   # noqa: E731
    run(2, log(1e-38, 1e38), log(1e-8, 1e8), log(1e-20, 1e20))
    edge = np.sqrt(np.array([1e-12, 1e12]) / np.pi).astype(f)   # pi a^2 c at its limits for c = 1
    for a in (edge, np.array([0.3, 1.0], f)):
        a, c, e = np.meshgrid(_around(a), _around([1.0, 0.5, 1e-12], 3),
                              np.concatenate([_around([1e-20, 1e20, 1.0], 5), ODD]), indexing="ij")
        run(2, e.ravel(), a.ravel(), c.ravel())
    a, c, e = np.meshgrid(ODD, ODD, ODD, indexing="ij")
    run(2, e.ravel(), a.ravel(), c.ravel())
