"""FP64 cell tiles (csrc/sph_tile.cu) where they can go wrong: cells of one to
many particles (partial rounds of four, two and one), windows of more
candidates than a tile, boxes of single-cell axes, the size from which a
particle has eight lanes instead of 32, a simulation too sparse for tiles and
batches.  Against the FP64 oracle; an evaluation sums at most a few thousand
terms, whose rounding stays below 1e-12 of the largest sum."""
import numpy as np
import pytest

from oracle import oracle
from pyticles_gb300 import _abi

pytestmark = pytest.mark.gpu
TOL = 1e-12
KEYS = ("rho", "rho_lr", "t", "p", "pco", "vdot", "udot")


def system(dim, n, box, seed, **kw):
    rng = np.random.default_rng(seed)
    box = [float(box)] * dim if np.isscalar(box) else list(box)
    r = rng.uniform(0, 1, (n, dim)) * box
    v = rng.normal(0, 0.7, (n, dim))
    m = rng.uniform(0.5, 1.5, n)
    kw.setdefault("kernel", "lucy")
    kw.setdefault("h_short", 1.5)
    kw.setdefault("h_long", 3.0)
    kw.setdefault("bdash", 0.01)
    prm = _abi.make_params(dim=dim, box=box, viscosity=True, dt=1e-3, **kw)
    # temperatures of 0.4 to 0.8 (one temperature has no heat flux to compare)
    u = oracle.derivatives(prm, r, v, m, np.zeros(n))["rho"] * -prm.adash
    u += rng.uniform(0.4, 0.8, n)
    return prm, r, v, m, u


def evaluate(*systems):
    from pyticles_gb300 import Engine
    with Engine(systems[0][0], "fp64", max_particles=sum(len(s[1]) for s in systems),
                max_sims=len(systems)) as e:
        ids = [e.add(*s) for s in systems]
        out = [e.derivatives(i) for i in ids]
        e.sync()
        counts = e.last_pair_counts(len(ids))
    return out, counts


def check(sysm, got, count, heat=False):
    ref = oracle.derivatives(*sysm)
    for k in KEYS + (("jq",) if heat else ()):
        err = np.linalg.norm(got[k] - ref[k]) / max(np.linalg.norm(ref[k]), 1e-300)
        assert err < TOL, (k, err)
    assert count == ref["nip"]


@pytest.mark.parametrize("kernel", ["lucy", "gaussian", "debrun", "cubic"])
@pytest.mark.parametrize("dim,n,box", [
    (2, 700, 24.0),        # about three particles a cell: every partial round
    (2, 3072, 40.0),       # the last size with 32 lanes a particle
    (2, 3073, 40.0),       # the first with eight
    (2, 4000, 16.5),       # 33 a cell: windows of several tiles
    (2, 900, (7.0, 40.0)),   # one axis of a single cell
    (3, 1500, 15.5),       # just wide enough for windows
    (3, 600, 6.0),         # one cell
    (3, 5000, 21.0),
])
def test_against_oracle(dim, n, box, kernel):
    kw = dict(heat_flux=kernel in ("cubic", "lucy"), kernel=kernel)
    if kernel == "cubic":
        kw.update(h_short=0.75, h_long=1.5)
    if kernel == "gaussian":
        kw.update(h_short=0.7, h_long=1.0, cutoff=3.0)
    s = system(dim, n, box, 11 * n + dim, **kw)
    got, counts = evaluate(s)
    check(s, got[0], counts[0], heat=kw["heat_flux"])


def test_batch_and_sparse():
    """A batch of tiled and too sparse simulations: each one's bits alone."""
    sims = [system(2, 700, 24.0, 1), system(2, 40, 60.0, 2), system(2, 4000, 16.5, 3),
            system(2, 5, 24.0, 4), system(2, 3500, 42.0, 5)]
    got, counts = evaluate(*sims)
    for s, g, c in zip(sims, got, counts):
        check(s, g, c)
        alone, n = evaluate(s)
        assert n[0] == c
        for k in KEYS:
            assert np.array_equal(alone[0][k], g[k]), k


def test_coincident_particles():
    """Particles on top of each other: finite rates, as the oracle's."""
    prm, r, v, m, u = system(2, 800, 25.0, 6)
    r[1] = r[0]
    r[7] = r[0]
    s = (prm, r, v, m, u)
    got, counts = evaluate(s)
    check(s, got[0], counts[0])


@pytest.mark.parametrize("what", ["r", "v", "u"])
def test_non_finite_state_is_reported(what):
    from pyticles_gb300 import Engine
    prm, r, v, m, u = system(2, 800, 25.0, 7)
    with Engine(prm, "fp64", max_particles=800) as e:
        s = e.add(prm, r, v, m, u)
        bad = {"r": r.copy(), "v": v.copy(), "u": u.copy()}
        bad[what][5] = np.nan
        e.set_state(s, bad["r"], bad["v"], m, bad["u"])
        e.advance(1)
        with pytest.raises(_abi.SphError) as exc:
            e.sync()
        assert exc.value.status == _abi.SPH_ENAN
