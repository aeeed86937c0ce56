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


def test_masses_of_neighbouring_simulations():
    """Equal and mixed masses side by side in one warp, by lanes, by the walk and
    by pair lists: each simulation's bits are those of its size alone, and equal
    masses those of the same masses read one by one."""
    from pyticles_gb300 import Engine
    sims = []
    for k, side in enumerate((3, 4, 3, 5, 17, 4)):
        prm, r, v, m, u = state(workloads.config_2d, side, 50 + k)
        if k % 2:
            m = m * np.random.default_rng(k).uniform(0.5, 1.5, len(m))
        else:
            m = m * 1.25
        sims.append((prm, r, v, m, u))
    for pick in range(len(sims)):
        order = [sims[pick]] + sims[:pick] + sims[pick + 1:]
        for a, b in zip(run(sims[pick:pick + 1], 2), run(order, 2)):
            assert np.array_equal(a, b), pick
    # masses that differ in one far particle only: the others' pair terms are
    # summed from masses read one by one
    prm, r, v, m, u = state(workloads.config_2d, 40, 9)
    odd = m.copy()
    far = int(np.argmax(np.abs(r - 10.0).min(axis=1)))
    odd[far] = 1.5
    near = np.hypot(*((r - r[far] + 20) % 40 - 20).T) < 14.0
    with Engine(prm, "mixed", max_particles=len(r)) as e:
        s = e.add(prm, r, v, m, u)
        one = e.derivatives(s)
        e.set_state(s, r, v, odd, u)
        two = e.derivatives(s)
        for k in ("rho", "vdot", "udot"):
            assert np.array_equal(one[k][~near], two[k][~near]), k
            assert not np.array_equal(one[k], two[k])


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
