"""Splash maps with smoothing lengths at the ends of what the formula takes: zero,
negative, not a number, and so small that their powers vanish draw zeros (no pixel
within them), as interpolate.py's Lucy function does; ordinary ones beside them are
drawn as ever."""
import numpy as np
import pytest

from tests.test_splat_boxes import reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("h_odd", [0.0, -1.0, np.nan, 1e-120, 1e-170, 1e-320])
def test_odd_smoothing_lengths(dim, h_odd):
    from pyticles_gb300 import interpolate
    rng = np.random.default_rng(17 + dim)
    n, L, cutoff = 70, 10.0, 1.7
    x = y = np.arange(40) * (L / 40)
    bounds = (0.0, L, 0.0, L)
    r = rng.uniform(0, L, (n, dim))
    m, rho, a = rng.uniform(0.5, 2, n), rng.uniform(0.5, 2, n), rng.normal(size=n)
    h = rng.uniform(0.5, 1.2, n) * cutoff
    odd = rng.uniform(size=n) < 0.3
    z = (4.0,) if dim == 3 else ()
    fn = interpolate.splash_map_2d if dim == 2 else interpolate.splash_map_3d
    Z = fn(x, y, *z, r, m, rho, a, np.where(odd, h_odd, h), bounds, cutoff)
    keep = ~odd
    ref = reference(x, y, z[0] if z else None, r[keep], m[keep], rho[keep], a[keep], h[keep],
                    bounds, cutoff)
    assert np.abs(Z - ref).max() <= 1e-12 * np.abs(ref).max()
