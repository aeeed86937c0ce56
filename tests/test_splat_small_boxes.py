"""Splash maps of particles whose boxes have few pixels, which a lane draws by itself
(csrc/sph_splat.cu): none, one, up to the line of 36 and beyond it, in warps of one
particle and of 32, off the grid and around its edges -- against the numpy restatement.
A pixel adds at most a few hundred FP64 terms."""
import numpy as np
import pytest

from tests.test_splat_boxes import reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n,nx,ny,pixels", [
    (1, 30, 20, 0.4), (70, 30, 20, 1.0), (1300, 20, 30, 0.6), (40000, 24, 20, 0.3),
    (40000, 24, 20, 1.5), (40000, 24, 20, 3.1), (39000, 24, 20, 3.6), (20000, 24, 20, 2.2),
])
def test_against_numpy(dim, n, nx, ny, pixels):
    from pyticles_gb300 import interpolate
    rng = np.random.default_rng(10 * n + nx + dim)
    L = 10.0
    d = L / nx
    x, y = np.arange(nx) * d, np.arange(ny) * d
    bounds = (0.0, L, 0.0, ny * d)
    cutoff = pixels * d
    r = rng.uniform(-0.3, 1.3, (n, dim)) * [L, bounds[3], L][:dim]
    m, rho, a = rng.uniform(0.5, 2, n), rng.uniform(0.5, 2, n), rng.normal(size=n)
    h = rng.uniform(0.5, 1.2, n) * cutoff
    z = (4.0,) if dim == 3 else ()
    fn = interpolate.splash_map_2d if dim == 2 else interpolate.splash_map_3d
    Z = fn(x, y, *z, r, m, rho, a, h, bounds, cutoff)
    ref = reference(x, y, z[0] if z else None, r, m, rho, a, h, bounds, cutoff)
    assert np.abs(Z - ref).max() <= 1e-12 * max(np.abs(ref).max(), 1e-300)
