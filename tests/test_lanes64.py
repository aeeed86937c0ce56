"""FP64 simulations too sparse for cell tiles walk their windows with several lanes
per particle in a small launch (csrc/sph_pairs.cuh, walk_lanes: 32 up to 1,536
particles, eight up to 4,096): the bits of one thread per particle, which the same
simulation takes beside a larger one, and the oracle's values."""
import numpy as np
import pytest

from pyticles_gb300 import build
from tests.test_tile64 import KEYS, check, evaluate, system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


@pytest.mark.parametrize("kernel", ["lucy", "gaussian", "debrun", "cubic"])
@pytest.mark.parametrize("dim,n", [(2, 1), (2, 40), (2, 1535), (2, 1537), (2, 4096), (2, 4097),
                                   (3, 33), (3, 1536), (3, 4000)])
def test_bits_of_the_walk(dim, n, kernel):
    heat = kernel in ("cubic", "lucy")
    kw = dict(heat_flux=heat, kernel=kernel, cutoff=3.0)
    if kernel == "cubic":
        kw.update(h_short=0.75, h_long=1.5)
    if kernel == "gaussian":
        kw.update(h_short=0.7, h_long=1.0)
    # cells of half the cutoff hold 1.4 (2D) or 0.7 particles (3D)
    box = max(8.0, (n * 1.5 ** dim / (1.4 if dim == 2 else 0.7)) ** (1.0 / dim))
    s = system(dim, n, box, 100 * n + dim, **kw)
    side = 90.0 if dim == 2 else 32.0
    large = system(dim, 5000, side, 7, **kw)
    (alone,), (count,) = evaluate(s)
    (beside, big), counts = evaluate(s, large)
    assert counts[0] == count
    for k in KEYS + (("jq",) if heat else ()):
        assert np.array_equal(alone[k], beside[k]), k
    if n > 1:   # one particle has no pairs to compare
        check(s, alone, count, heat=heat)
        check(large, big, counts[1], heat=heat)
