"""FP64 simulations around the lines between cell tiles and cell windows (3072
particles; two particles per cell in 2D, one in 3D) against the oracle."""
import pytest

from pyticles_gb300 import build
from tests.test_tile64 import check, evaluate, system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


@pytest.mark.parametrize("dim,n,box", [(2, 12, 90.0), (2, 3072, 120.0), (2, 3073, 120.0),
                                       (3, 50, 30.0), (3, 3500, 17.0), (3, 3500, 21.0),
                                       (3, 3500, 30.0)])
def test_sparse_systems(dim, n, box):
    s = system(dim, n, box, n + dim)
    got, counts = evaluate(s)
    check(s, got[0], counts[0])
