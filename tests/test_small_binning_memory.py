"""The one-block binning holds its cells and slots in shared memory: sizes around
what a block has there (47 KB for cells + 2 slots, 4 bytes each, so 12,032 of
them) are binned by the one block or by the six kernels, in the same order.  A
launch of more than a block's shared memory would be refused."""
import numpy as np
import pytest

from pyticles_gb300 import Engine, _abi, build
from tests.test_zz_no_alloc import noalloc

pytestmark = pytest.mark.gpu

ROOM = 47 * 1024 // 4


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


def gas(nc, n, seed):
    """n particles in a grid of nc cells of half the cutoff (window cells of edge
    0.5, a ten-thousandth wider than they need to be)."""
    rng = np.random.default_rng(seed)
    dim = len(nc)
    box = [0.5 * k * 1.0001 for k in nc]
    prm = _abi.make_params(dim=dim, kernel="lucy", box=box, h_short=0.5, h_long=1.0, cutoff=1.0,
                           tolerance=0.0, viscosity=True, dt=1e-6)
    r = rng.uniform(0, 1, (n, dim)) * box
    return prm, r, rng.normal(0, 0.5, (n, dim)), np.ones(n), rng.uniform(0.4, 0.8, n)


def run(sims, precision, companion):
    with Engine(sims[0][0], precision, max_particles=8192, max_sims=len(sims) + 1) as e:
        ids = [e.add(*s) for s in sims]
        if companion:
            e.add(*gas((20,) * len(sims[0][0].box[:sims[0][0].dim]), 2100, 3))
        e.set_tuning(rebin=0, steps_per_graph=2)
        e.advance(3)
        e.sync()
        return e.kernels_per_step(), [(e.get_state(s), e.pair_count(s)) for s in ids]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("nc,n,sims", [
    ((90, 91), 1921, 1),        # the last sum that one block holds
    ((90, 91), 1922, 1),        # the first that it does not
    ((90, 91), 2030, 1),
    ((90, 91), 2031, 1),
    ((90, 91), 2048, 1),
    ((88, 90), 2048, 1),
    ((32, 32), 256, 8),
    ((16, 16), 64, 32),
    ((16, 16, 32), 2048, 1),
])
def test_every_size_is_binned(nc, n, sims, precision):
    systems = [gas(nc, n, 60 + k) for k in range(sims)]
    kernels, got = run(systems, precision, False)
    six, want = run(systems, precision, True)
    small = sims * (int(np.prod(nc)) + 2 * n) <= ROOM
    if precision == "mixed":   # an FP64 step has other pair passes beside the companion
        assert kernels == six - (5 if small else 0)
    for (a, ca), (b, cb) in zip(got, want):
        assert ca == cb > 0
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("nc,n", [((90, 91), 1921), ((90, 91), 2048)])
def test_without_allocation(nc, n):
    prm, r, v, m, u = gas(nc, n, 5)
    with Engine(prm, "fp64", max_particles=n) as e:
        want = e.derivatives(e.add(prm, r, v, m, u))
    got = noalloc(prm, "fp64", r, v, m, u)
    for k in ("rho", "rho_lr", "vdot", "udot"):
        assert np.array_equal(got[k], want[k]), k
