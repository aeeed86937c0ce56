"""The exported pair list of a simulation of one cell (csrc/sph_pairs.cu,
export_one_cell): sizes around a warp's, every pair or a few of them, the second of a
batch -- the oracle's pairs in its order and its squared distances, bit for bit."""
import numpy as np
import pytest

from oracle import oracle
from pyticles_gb300 import Engine, build
from tests.test_export_rows import state

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("dim,n,cutoff", [(2, 2, 6.0), (2, 32, 4.5), (2, 33, 12.0), (2, 65, 4.5),
                                          (2, 3000, 5.0), (3, 31, 12.0), (3, 97, 4.5),
                                          (3, 1500, 5.0)])
def test_rows(dim, n, cutoff, precision):
    prm, r, v, m, u = state(dim, n, 9.0, cutoff, 7 * n)
    other = state(dim, 45, 20.0, cutoff, 1)
    iap, rsq = oracle.pairs(prm, r)
    with Engine(prm, precision, max_particles=n + 45, max_sims=2) as e:
        e.add(*other)
        got = e.pairs(e.add(prm, r, v, m, u))
    assert np.array_equal(got["iap"], iap)
    assert np.array_equal(got["rsq"], rsq)
    assert np.array_equal(got["dv"], v[iap[:, 1]] - v[iap[:, 0]])
