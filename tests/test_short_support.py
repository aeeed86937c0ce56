"""Pairs at the edge of the short kernel's support in boxes and cells thousands of
supports wide: the cell tiles file them by an FP32 test whose rounding grows with
the distances from the cell's centre, and every pair within the support has to get
its short-kernel terms.  FP64 against the oracle, at test_tile64's tolerance."""
import numpy as np
import pytest

from pyticles_gb300 import _abi, build
from tests.test_tile64 import check, evaluate, system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


# One cell; eight cells a side, thousands of short supports wide; ordinary ones.  The
# cells get their room from the drift of a step (8 dt vmax, vmax = 2): without it a
# cell is half the cutoff.  The positions are multiples of 2^-30 and the cells' centres
# of 1/2, so that a position in its cell's frame, and every separation, is exact in FP64.
@pytest.mark.parametrize("box,cells", [(2.0 ** 18, 1), (2.0 ** 16, 8), (2.0 ** 8, 0)])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("h_short", [1.5, 0.3])
def test_dense_patch_in_a_wide_box(dim, box, cells, h_short):
    n, side = (1500, 24.0) if dim == 2 else (1500, 9.0)
    kw = dict(kernel="lucy", h_short=h_short, h_long=3.0, cutoff=3.0, tolerance=0.0, bdash=0.01,
              heat_flux=True)
    _, r, v, m, u = system(dim, n, side, 17 * dim, **kw)
    r = np.round(r * 2.0 ** 30) / 2.0 ** 30
    v *= 2.0 / np.abs(v).max()
    if cells:   # cells of half the reach, of which box / (cells + 1/2) just fits
        dt = (2.0 * box / (cells + 0.5) - 3.0) / 16.0
    else:
        dt = 1e-9
    prm = _abi.make_params(dim=dim, box=[box] * dim, viscosity=True, dt=dt, **kw)
    s = (prm, r, v, m, u)
    got, counts = evaluate(s)
    check(s, got[0], counts[0], heat=True)
