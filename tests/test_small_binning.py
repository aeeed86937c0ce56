"""Launches of at most 2048 particles are binned by one block: the canonical
order, so the bits of the same simulation in a launch that is binned by the
six kernels."""
import numpy as np
import pytest

from oracle import oracle
from pyticles_gb300 import Engine, build, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


def fluid(dim, n, seed):
    if dim == 2:
        prm, r, v, m, T0 = workloads.config_2d(48, seed, viscosity=True)
    else:
        prm, r, v, m, T0 = workloads.config_3d(13, seed)
    u = oracle.initial_energy(prm, r, v, m, T0)
    keep = np.sort(np.random.default_rng(seed).permutation(len(r))[:n])
    return prm, r[keep], v[keep], m[keep], u[keep]


@pytest.mark.parametrize("dim,n", [(2, 1), (2, 2), (2, 33), (2, 1025), (2, 2047), (2, 2048),
                                   (2, 2049), (3, 2), (3, 1024), (3, 2048)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_small_binning_keeps_the_order(dim, n, precision):
    prm, r, v, m, u = fluid(dim, n, 40 + dim)
    out = []
    for companion in (0, 600 if n > 1448 else 2100):
        with Engine(prm, precision, max_particles=8192, max_sims=3) as e:
            # a slot given back lies among the ones in use
            gone = e.add(prm, r[:1], v[:1], m[:1], u[:1]) if n < 2048 else None
            s = e.add(prm, r, v, m, u)
            if companion:
                _, r1, v1, m1, u1 = fluid(dim, companion, 50)
                e.add(prm, r1, v1, m1, u1)
            if gone is not None:
                e.remove(gone)
            e.set_tuning(rebin=0)
            e.advance(3)
            e.sync()
            out.append((e.kernels_per_step(), e.get_state(s), e.pair_count(s)))
    assert out[0][2] == out[1][2]
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)
    if n <= 2048 and precision == "mixed":
        assert out[0][0] == out[1][0] - 5
