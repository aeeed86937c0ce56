"""Small mixed-precision launches take several lanes per particle
(csrc/sph_pairs.cuh, for_pairs_lanes): a simulation's bits are those of the
thread-per-particle walk that it runs in beside a large simulation."""
import numpy as np
import pytest

from pyticles_gb300 import workloads

pytestmark = pytest.mark.gpu
KEYS = ("rho", "rho_lr", "t", "p", "pco", "vdot", "udot", "jq")


def state(maker, side, seed, **kw):
    prm, r, v, m, T0 = maker(side, seed, **kw)
    dens = len(r) / np.prod(prm.box[:prm.dim])
    return prm, r, v, m, workloads.vdw_energy(np.full(len(r), dens), T0)


def run(sims, steps):
    from pyticles_gb300 import Engine
    with Engine(sims[0][0], "mixed", max_particles=sum(len(s[1]) for s in sims),
                max_sims=len(sims)) as e:
        ids = [e.add(*s) for s in sims]
        e.advance(steps)
        e.sync()
        st, pr = e.get_state(ids[0]), e.properties(ids[0])
        return list(st) + [pr[k] for k in KEYS] + [e.last_pair_counts(1)]


# 40961 particles and more run one thread per particle
@pytest.mark.parametrize("maker,sides,big", [
    (workloads.config_2d, [3, 10, 15, 32, 64, 65, 150], 203),
    (workloads.config_3d, [4, 10, 12, 15, 16, 17, 25], 35),
])
@pytest.mark.parametrize("kernel", ["lucy", "gaussian", "debrun", "cubic"])
def test_bits_of_the_walk(maker, sides, big, kernel):
    kw = {"kernel": kernel, "heat_flux": True}
    if kernel == "gaussian":
        kw.update(h_short=0.9, h_long=1.8, cutoff=5.0)
    if kernel == "debrun" and maker is workloads.config_3d:
        # the 3D fluid's supports as this kernel's h; at half of them its rates
        # carry the companion past its cell slack (SPH_ESKIN)
        kw.update(h_short=2.735, h_long=5.148)
    large = state(maker, big, 5, **kw)
    for side in sides:
        small = state(maker, side, 7 + side, **kw)
        for a, b in zip(run([small], 2), run([small, large], 2)):
            assert np.array_equal(a, b), (side, kernel)
