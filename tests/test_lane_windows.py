"""Lanes per particle by the launch's windows and cells (csrc/sph_pairs.cuh,
walk_lanes): boxes of one cell, of single-cell axes, sparse ones on both sides of the
lines, alone and mixed in a batch -- the bits of one thread per particle, which the
same simulation takes beside a large one."""
import numpy as np
import pytest

from pyticles_gb300 import _abi, build
from tests.test_lanes import run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


def lattice(sides, cut, seed):
    """One particle per unit of volume in a box of `sides`, cells of half the cutoff."""
    rng = np.random.default_rng(seed)
    dim = len(sides)
    r = np.stack([g.reshape(-1) for g in np.meshgrid(*[np.arange(k) + 0.5 for k in sides],
                                                     indexing="ij")], 1)
    r += rng.uniform(-0.1, 0.1, r.shape)
    prm = _abi.make_params(dim=dim, kernel="lucy", box=[float(k) for k in sides],
                           h_short=cut / 2, h_long=cut, cutoff=cut, tolerance=0.0,
                           viscosity=True, heat_flux=True, dt=1e-4)
    n = len(r)
    return prm, r, rng.normal(0, 0.5, (n, dim)), np.ones(n), rng.uniform(-0.9, -0.7, n)


LARGE = {2: lattice((210, 210), 1.5, 1), 3: lattice((35, 35, 36), 1.5, 2)}


@pytest.mark.parametrize("sides,cut", [
    ((8, 8), 6.0), ((30, 30), 12.0), ((50, 50), 21.0),         # one cell
    ((10, 400), 6.0), ((10, 410), 6.0), ((10, 1500), 6.0),     # five cells
    ((90, 92), 1.0), ((160, 179), 1.0), ((160, 180), 1.0),     # sparse
    ((10, 10, 10), 4.4), ((10, 10, 90), 4.4), ((10, 20, 20), 4.4),
    ((10, 50, 50), 4.4), ((30, 30, 31), 1.7), ((30, 31, 31), 1.7),
])
def test_bits_of_the_walk(sides, cut):
    small = lattice(sides, cut, sum(sides))
    for a, b in zip(run([small], 2), run([small, LARGE[len(sides)]], 2)):
        assert np.array_equal(a, b), sides


@pytest.mark.parametrize("dim", [2, 3])
def test_batches_of_narrow_and_wide_boxes(dim):
    if dim == 2:
        sims = [lattice((8, 8), 6.0, k) for k in range(12)] + [lattice((40, 40), 6.0, 20),
                                                                lattice((10, 100), 6.0, 21)]
    else:
        sims = [lattice((8, 8, 8), 4.4, k) for k in range(12)] + [lattice((16, 16, 16), 4.4, 20),
                                                                   lattice((8, 8, 40), 4.4, 21)]
    for pick in (0, 12, 13):
        order = [sims[pick]] + sims[:pick] + sims[pick + 1:]
        for a, b in zip(run([sims[pick]], 2), run(order, 2)):
            assert np.array_equal(a, b), pick
