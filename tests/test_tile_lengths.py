"""FP64 evaluations in units that make the lengths very large or very small: the
cell tiles test their candidates in FP32, so lengths whose squares leave its range
run on the window walk, which is FP64 throughout.  The van der Waals constants go
with the volume, so the temperatures and the balance of the terms stay what they are
at scale 1, and the tolerance is test_tile64's."""
import pytest

from pyticles_gb300 import _abi, build
from oracle import oracle
from tests.test_tile64 import check, evaluate, system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


# tiles serve cutoffs from 1e-12 on and boxes of up to 1e17
@pytest.mark.parametrize("scale", [1e-40, 1e-25, 1e-18, 1e-13, 1e-12, 1e-6, 1.0, 1e6, 1e15, 3e15,
                                   1e16, 3e17, 1e18, 1e20, 1e27])
@pytest.mark.parametrize("dim,n,box", [(2, 700, 24.0), (2, 3500, 30.0), (2, 500, 7.0),
                                       (3, 1500, 15.5)])
def test_scaled(dim, n, box, scale):
    prm, r, v, m, u = system(dim, n, box, 3 * n + dim, cutoff=3.0, tolerance=0.5)
    p = _abi.make_params(dim=dim, box=[box * scale] * dim, kernel="lucy", h_short=1.5 * scale,
                         h_long=3.0 * scale, cutoff=3.0 * scale, tolerance=0.5 * scale,
                         adash=2.0 * scale ** dim, bdash=0.01 * scale ** dim, viscosity=True,
                         dt=1e-9 * scale)
    s = (p, r * scale, v, m, u)
    got, counts = evaluate(s)
    check(s, got[0], counts[0])
    assert counts[0] == oracle.derivatives(prm, r, v, m, u)["nip"]
