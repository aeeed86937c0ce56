"""A state set within the slack of the current binning (and lists) goes into
the current slots: the step that follows starts from the new positions and
velocities, as the oracle's does."""
import numpy as np
import pytest

from oracle import oracle
from pyticles_gb300 import Engine, build, workloads
from tests.golden_cases import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


@pytest.mark.parametrize("masses", ["kept", "changed"])
@pytest.mark.parametrize("integrator", ["ieuler", "rk4"])
@pytest.mark.parametrize("dim,precision,scheme", [(2, "mixed", 0), (2, "mixed", 2), (2, "fp64", 0),
                                                  (3, "mixed", 0), (3, "mixed", 2)])
def test_a_kept_state_is_the_start_of_the_next_step(dim, precision, scheme, integrator, masses):
    if dim == 2:
        prm, r, v, m, T0 = workloads.config_2d(32, 1006, viscosity=True, integrator=integrator)
    else:
        prm, r, v, m, T0 = workloads.config_3d(14, 1007, integrator=integrator)
    u = oracle.initial_energy(prm, r, v, m, T0)
    rng = np.random.default_rng(12)
    with Engine(prm, precision, max_particles=len(r)) as e:
        s = e.add(prm, r, v, m, u)
        e.set_tuning(pair_scheme=scheme, rebin=1, steps_per_graph=1)
        e.advance(1)
        r1, v1, u1 = e.get_state(s)
        bins = e.rebin_count()
        r2 = r1 + 1e-3 * rng.uniform(-1, 1, r.shape)
        v2 = v1 + rng.normal(0, 1, v.shape)
        # in 2D mixed precision the masses lie apart from the records
        m2 = m if masses == "kept" else m * rng.uniform(0.8, 1.2, len(m))
        e.set_state(s, r2, v2, m2, u1)
        e.advance(1)
        e.sync()
        assert e.rebin_count() == bins
        _, got, _ = e.get_state(s)
    _, ref, _, _ = oracle.advance(prm, r2, v2, m2, u1, 1)
    # the step's change of velocity is its mean rate times dt
    assert rel_l2(got - v2, ref - v2) < (1e-5 if precision == "mixed" else 1e-9)


@pytest.mark.parametrize("precision,scheme", [("mixed", 0), ("mixed", 2), ("fp64", 0)])
def test_one_simulation_of_a_batch(precision, scheme):
    """The others go on from where they were."""
    sims = []
    for k, side in enumerate((24, 32, 40)):
        prm, r, v, m, T0 = workloads.config_2d(side, 1010 + k, viscosity=True)
        sims.append((prm, r, v, m, oracle.initial_energy(prm, r, v, m, T0)))
    rng = np.random.default_rng(13)
    with Engine(sims[0][0], precision, max_particles=sum(len(s[1]) for s in sims),
                max_sims=3) as e:
        ids = [e.add(*s) for s in sims]
        e.set_tuning(pair_scheme=scheme, rebin=1, steps_per_graph=1)
        e.advance(1)
        states = [e.get_state(i) for i in ids]
        bins = e.rebin_count()
        r, v, u = states[1]
        states[1] = (r + 1e-3 * rng.uniform(-1, 1, r.shape), v + rng.normal(0, 1, v.shape), u)
        e.set_state(ids[1], states[1][0], states[1][1], sims[1][3], u)
        e.advance(1)
        e.sync()
        assert e.rebin_count() == bins
        got = [e.get_state(i)[1] for i in ids]
    for s, (r, v, u), g in zip(sims, states, got):
        _, ref, _, _ = oracle.advance(s[0], r, v, s[3], u, 1)
        assert rel_l2(g - v, ref - v) < (1e-5 if precision == "mixed" else 1e-9)
