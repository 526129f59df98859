"""The device functions for 1/sqrt(r2) and its powers in FP64, over squared distances from 1e-6 to
100 nm^2, values next to powers of two among them, against extended precision.

Bounds, u = 2^-53.  xrsqrt (two Newton steps): 1.5 u of roundings and, from an approximation good to
2^-19, less than 0.01 u of the method.  inv_r23: t = y^2 rounds, but e is that of the rounded t, so r^-2
has the last sum's u and e^3 < 2^-54 = 0.5 u; r^-3 has u / 2 of t, u of t y, u of the last sum and
35/16 e^3 < 1.1 u."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = """
#include "rs_device.cuh"
__global__ void k(const double *a, int n, double *y, double *p2, double *p3) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y[i] = rs::xrsqrt(a[i]);
    rs::inv_r23(a[i], p2[i], p3[i]);
}
extern "C" int run(const double *a, int n, double *out) {
    double *d;
    if (cudaMalloc(&d, 4 * sizeof(double) * n)) return 1;
    int rc = cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (!rc) {
        k<<<(n + 255) / 256, 256>>>(d, n, d + n, d + 2 * n, d + 3 * n);
        rc = cudaMemcpy(out, d + n, 3 * sizeof(double) * n, cudaMemcpyDeviceToHost);
    }
    cudaFree(d);
    return rc;
}
"""


def test_reciprocal_powers(tmp_path):
    import build
    src, lib = tmp_path / "k.cu", tmp_path / "k.so"
    src.write_text(SRC)
    subprocess.run([build.NVCC, *build.ARCH, *build.FLAGS, "-shared", "-o", str(lib), str(src), "-lcudart"],
                   check=True, cwd=os.path.dirname(build.CSRC))
    rng = np.random.default_rng(1)
    p = 2.0 ** np.arange(-20, 7)
    a = np.concatenate([10.0 ** rng.uniform(-6, 2, 1 << 20), p, np.nextafter(p, 0), np.nextafter(p, 200)])
    out = np.zeros((3, a.size))
    fp = ctypes.POINTER(ctypes.c_double)
    assert ctypes.CDLL(str(lib)).run(a.ctypes.data_as(fp), a.size, out.ctypes.data_as(fp)) == 0
    r = np.sqrt(a.astype(np.longdouble))
    u = 2.0 ** -53
    for k, (power, bound) in enumerate(((1, 1.51), (2, 1.5), (3, 3.6))):
        err = float(np.abs(out[k] * r ** power - 1).max()) / u
        print("r^-%d: %.3f u" % (power, err))
        assert err <= bound
