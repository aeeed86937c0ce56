"""The splash maps where the kernel can go wrong: boxes of a few pixels, of
more than 32 columns, wider than the grid, wrapping on every side, particle
counts around a warp's, the 3D plane's edge -- against a numpy restatement of
interpolate.py:39-149.  A pixel adds at most a few hundred FP64 terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lucy(s, h, dim3):
    q = 105.0 / (np.pi * 16.0 * h ** 3) if dim3 else 5.0 / (np.pi * h ** 2)
    return np.where(s < h, q * (1 + 3 * s / h) * np.clip(1 - s / h, 0, None) ** 3, 0.0)


def image(d, L):
    d = np.where(d > L / 2, d - L, d)
    return np.where(d < -L / 2, d + L, d)


def reference(x, y, z, r, m, rho, a, h, bounds, cutoff):
    Z = np.zeros((len(x), len(y)))
    res = x[1] - x[0]
    for i in range(len(r)):
        dz = r[i, 2] - z if z is not None else 0.0
        if dz > cutoff:
            continue
        lo = [int(np.floor((r[i, k] - cutoff - bounds[2 * k]) / res)) for k in (0, 1)]
        hi = [int(np.floor((r[i, k] + cutoff - bounds[2 * k]) / res)) for k in (0, 1)]
        wrapped = []
        for k, n in ((0, len(x)), (1, len(y))):
            p = np.arange(lo[k], hi[k])
            p = np.where(p >= n, p - n, p)
            p = np.where(p < 0, p + n, p)
            wrapped.append(p[(p >= 0) & (p < n)])
        dx = image(r[i, 0] - x[wrapped[0]], bounds[1])
        dy = image(r[i, 1] - y[wrapped[1]], bounds[3])
        rsq = dx[:, None] ** 2 + dy[None, :] ** 2 + dz * dz
        w = a[i] * m[i] / rho[i] * lucy(np.sqrt(rsq), h[i], z is not None)
        np.add.at(Z, np.ix_(*wrapped), np.where(rsq < cutoff ** 2, w, 0.0))
    return Z


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n,nx,ny,cutoff", [
    (1, 20, 20, 2.0), (31, 7, 5, 2.0), (33, 40, 33, 3.0), (65, 200, 150, 1.7),
    (40, 200, 150, 4.5), (25, 9, 11, 9.0), (2000, 64, 48, 0.4),
])
def test_against_numpy(dim, n, nx, ny, cutoff):
    from pyticles_gb300 import interpolate
    rng = np.random.default_rng(100 * n + dim)
    L = 10.0
    x, y = np.arange(nx) * (L / nx), np.arange(ny) * (L / nx)
    bounds = (0.0, L, 0.0, ny * L / nx)
    r = rng.uniform(-0.2, 1.2, (n, dim)) * [L, bounds[3], L][:dim]
    m, rho, a = rng.uniform(0.5, 2, n), rng.uniform(0.5, 2, n), rng.normal(size=n)
    h = rng.uniform(0.5, 1.2, n) * cutoff
    if dim == 2:
        Z = interpolate.splash_map_2d(x, y, r, m, rho, a, h, bounds, cutoff)
        ref = reference(x, y, None, r, m, rho, a, h, bounds, cutoff)
    else:
        Z = interpolate.splash_map_3d(x, y, 4.0, r, m, rho, a, h, bounds, cutoff)
        ref = reference(x, y, 4.0, r, m, rho, a, h, bounds, cutoff)
    assert np.abs(Z - ref).max() <= 1e-12 * max(np.abs(ref).max(), 1e-300)
