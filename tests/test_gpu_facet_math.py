"""The thermal kernel's elementary functions (csrc/facet_math.cuh) over their stated ranges, edges
of their reductions among them, against extended precision.

Tolerances, from the steps of each: the reciprocals end in one rounding (rsqrt3: and half of
that of x y), 2^-52 relative; the exponential has the table's (2^-52 at the most) and its own
last rounding, 2^-51; the logarithm below 6 the last rounding of a double there (2^-51), nine
times the rounding of ln 2 and three roundings of the series' argument, 9e-16 absolute."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cuda_runtime.h>
#include "facet_math.cuh"
__global__ void facet_math(int f, int n, const double* x, double* y) {
    __shared__ double table[kb::EXP_TABLE];
    if (threadIdx.x < kb::EXP_TABLE) table[threadIdx.x] = exp2(threadIdx.x * (1.0 / kb::EXP_TABLE));
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y[i] = f == 0 ? kb::recip3(x[i]) : f == 1 ? kb::rsqrt3(x[i])
         : f == 2 ? kb::exp_positive(x[i], table) : kb::log_kelvin(x[i]);
}
extern "C" int run(int f, int n, const double* x, double* y) {
    facet_math<<<(n + 255) / 256, 256>>>(f, n, x, y);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def facet_math(gpu, tmp_path_factory):
    from kete_b200 import build

    d = tmp_path_factory.mktemp("facet_math")
    src, lib = str(d / "probe.cu"), str(d / "probe.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build.nvcc(), *build.host_compiler(), *build.ARCH, "-O3", "-std=c++17",
                    "--shared", "-Xcompiler", "-fPIC", "-I", build.CSRC, "-o", lib, src],
                   check=True, env=dict(os.environ, TMPDIR=str(d)))
    return ctypes.CDLL(lib)


def _evaluate(lib, f, x):
    import torch

    dx = torch.from_numpy(x).cuda()
    dy = torch.empty_like(dx)
    torch.cuda.synchronize()
    run = lib.run
    run.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    assert run(f, x.size, dx.data_ptr(), dy.data_ptr()) == 0
    return dy.cpu().numpy().astype(np.longdouble)


def _around(x):
    return np.concatenate([x, np.nextafter(x, -np.inf), np.nextafter(x, np.inf)])


def test_reciprocals(facet_math):
    rng = np.random.default_rng(0)
    x = np.concatenate([10.0 ** rng.uniform(-280, 280, 200_000), 1.0 + rng.random(200_000),
                        _around(2.0 ** np.arange(-900.0, 901.0))])
    for f, want in ((0, lambda v: 1 / v), (1, lambda v: 1 / np.sqrt(v))):
        exact = want(x.astype(np.longdouble))
        assert np.abs(_evaluate(facet_math, f, x) / exact - 1).max() < 2.0**-52


def test_exponential(facet_math):
    rng = np.random.default_rng(1)
    edges = (np.arange(32_000) + 0.5) * (np.log(2.0) / 32)  # between table entries
    x = np.concatenate([rng.uniform(0, 700, 300_000), 10.0 ** rng.uniform(-300, 2.8, 100_000),
                        _around(edges[edges < 699]), [0.0]])
    exact = np.exp(x.astype(np.longdouble))
    assert np.abs(_evaluate(facet_math, 2, x) / exact - 1).max() < 2.0**-51


def test_logarithm(facet_math):
    rng = np.random.default_rng(2)
    edges = _around(np.array([2.0**e for e in (7, 8)] + [2.0 ** (e + 0.5) for e in (6, 7, 8)]))
    x = np.concatenate([rng.uniform(100, 400, 400_000), edges[(edges >= 100) & (edges <= 400)],
                        [100.0, 400.0]])
    exact = np.log(x.astype(np.longdouble))
    assert np.abs(_evaluate(facet_math, 3, x) - exact).max() < 9e-16
