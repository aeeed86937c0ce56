"""The square roots and quotients that the pair passes form from the hardware's
approximations (csrc/sph_device.cuh) against CUDA's own: tile_sqrt, tile_inv and
tile_div in FP64, plain_dist and make_dist in FP32.

Bounds, in units of the last place of the result.  The last operation of each FP64
form adds a correction known to about 2^-40 of it, in one rounding: half a unit and a
little, so at most one unit from the correctly rounded result.  plain_dist's Newton
step leaves an error of the order of the approximation's square, 2^-44 relative, before
its one rounding: one unit.  make_dist keeps the root as r + e/2: 2^-24 of an
approximation good to 2^-22 is off by at most 2^-44 relative, doubled for the roundings
of e; the residual rsq - r^2 is a multiple of 2^-149, which adds 2^-150 / rsq."""
import ctypes
import subprocess

import numpy as np
import pytest

from pyticles_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "sph_device.cuh"
using namespace sph;
__global__ void k_f64(int n, const double *x, const double *d, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double ih;
    const double r = tile_sqrt(x[i], &ih);
    out[i] = r;
    out[n + i] = sqrt(x[i]);
    out[2 * n + i] = tile_inv(r, ih);
    out[3 * n + i] = 1.0 / r;
    out[4 * n + i] = tile_div(x[i], d[i]);
    out[5 * n + i] = x[i] / d[i];
}
__global__ void k_f32(int n, const float *x, float *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Dist<float> p = plain_dist<float>(x[i]), m = make_dist<float>(x[i]);
    out[i] = p.r;
    out[n + i] = __fsqrt_rn(x[i]);
    out[2 * n + i] = m.r;
    out[3 * n + i] = m.e;
}
extern "C" int run(int n, const double *x, const double *d, double *o64, const float *xf,
                   float *o32) {
    double *bx, *bd, *bo;
    float *bf, *bq;
    cudaMalloc(&bx, 8 * n); cudaMalloc(&bd, 8 * n); cudaMalloc(&bo, 48 * n);
    cudaMalloc(&bf, 4 * n); cudaMalloc(&bq, 16 * n);
    cudaMemcpy(bx, x, 8 * n, cudaMemcpyHostToDevice);
    cudaMemcpy(bd, d, 8 * n, cudaMemcpyHostToDevice);
    cudaMemcpy(bf, xf, 4 * n, cudaMemcpyHostToDevice);
    k_f64<<<(n + 255) / 256, 256>>>(n, bx, bd, bo);
    k_f32<<<(n + 255) / 256, 256>>>(n, bf, bq);
    cudaMemcpy(o64, bo, 48 * n, cudaMemcpyDeviceToHost);
    cudaMemcpy(o32, bq, 16 * n, cudaMemcpyDeviceToHost);
    cudaFree(bx); cudaFree(bd); cudaFree(bo); cudaFree(bf); cudaFree(bq);
    return (int)cudaGetLastError();
}
"""

N = 1 << 20


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("roots")
    src, lib = tmp / "roots.cu", tmp / "roots.so"
    src.write_text(SOURCE)
    cmd = [build.nvcc()] + build.ARCH + build.FLAGS + ["-I", build.CSRC, "-shared", "-cudart",
                                                       "static", str(src), "-o", str(lib)]
    subprocess.run(cmd, check=True, capture_output=True, timeout=600)
    rng = np.random.default_rng(5)
    # squared distances: near 1 (a cutoff's range), over the whole range, edges
    x = np.concatenate([rng.uniform(1e-4, 64.0, N // 2), 2.0 ** rng.uniform(-900, 900, N // 2)])
    edges = np.concatenate([2.0 ** np.arange(-60, 60), np.arange(1.0, 200.0) ** 2,
                            np.nextafter(2.0 ** np.arange(-60, 60), 0),
                            np.nextafter(2.0 ** np.arange(-60, 60), 1e300)])
    x[:len(edges)] = edges
    d = np.concatenate([rng.uniform(1e-4, 64.0, N // 2), 2.0 ** rng.uniform(-80, 80, N // 2)])
    d[:len(edges)] = edges[::-1]
    xf = np.concatenate([rng.uniform(1e-4, 64.0, N // 2), 2.0 ** rng.uniform(-120, 120, N // 2)])
    xf[:len(edges)] = edges
    xf = xf.astype(np.float32)   # all above 1e-37, below which a root reads as 0
    x[-2:], xf[-1] = (0.0, 1e-300), 0.0
    o64, o32 = np.zeros((6, N)), np.zeros((4, N), np.float32)
    p = ctypes.c_void_p
    st = ctypes.CDLL(str(lib)).run(N, p(x.ctypes.data), p(d.ctypes.data), p(o64.ctypes.data),
                                   p(xf.ctypes.data), p(o32.ctypes.data))
    assert st == 0
    return x, d, xf, o64, o32


def units(got, want):
    """|got - want| in units of want's last place, and the share that differs."""
    u = np.abs(got - want) / np.spacing(np.abs(want))
    return float(u.max()), float((u > 0).mean())


@pytest.mark.parametrize("k,what", [(0, "tile_sqrt"), (2, "tile_inv"), (4, "tile_div")])
def test_fp64(results, k, what):
    got, want = results[3][k:k + 2]
    if what != "tile_div":   # arguments below 1e-280 read as it
        assert np.allclose(got[-2:], (1e-140, None, 1e140)[k], rtol=1e-15, atol=0)
    worst, share = units(got[:-2], want[:-2])
    print(what, "units", worst, "share", share)
    assert worst <= 1.0


def test_fp32(results):
    xf, o32 = results[2][:-1], results[4][:, :-1]
    assert results[4][0, -1] == results[4][2, -1] == 0.0
    worst, share = units(o32[0], o32[1])
    print("plain_dist", "units", worst, "share", share)
    assert worst <= 1.0
    r = np.sqrt(xf.astype(np.float64))
    err = np.abs(o32[2].astype(np.float64) + 0.5 * o32[3] - r) / r
    print("make_dist", float(err.max()))
    assert np.all(err <= 2.0 ** -43 + 2.0 ** -150 / xf.astype(np.float64))

