"""The FP32 pair test's guard band (csrc/sph_engine.cu, fast_margin): pairs whose
distances lie 1e-8 to 1e-3 of the cutoff on either side of it, in every
direction, are counted as the FP64 test counts them -- by the cell windows of
every cell size, in boxes of single-cell axes, by pair lists and cluster
pairs and by the FP64 tiles."""
import numpy as np
import pytest

from oracle import oracle
from pyticles_gb300 import Engine, _abi

pytestmark = pytest.mark.gpu
CUT = 3.0


def shells(dim, box, n, seed):
    """n particles, every second one about a cutoff from its predecessor."""
    rng = np.random.default_rng(seed)
    L = np.asarray(box, dtype=float)
    a = rng.uniform(0, 1, (n // 2, dim)) * L
    e = rng.normal(size=(n // 2, dim))
    e /= np.linalg.norm(e, axis=1, keepdims=True)
    off = 10.0 ** rng.uniform(-8, -3, n // 2) * rng.choice([-1, 1], n // 2)
    b = (a + e * (CUT * (1 + off))[:, None]) % L
    r = np.concatenate([a, b])
    return r[rng.permutation(n)]


@pytest.mark.parametrize("dim,box,precision,knobs", [
    (2, (48.0, 41.0), "mixed", {"cell_ratio": 0.5}),
    (2, (48.0, 41.0), "mixed", {"cell_ratio": 0.2}),
    (2, (48.0, 41.0), "mixed", {"cell_ratio": 1.0}),
    (2, (90.0, 75.0), "mixed", {"cell_ratio": 4.0}),
    (2, (6.5, 48.0), "mixed", {"cell_ratio": 0.5}),
    (2, (35.0, 35.0), "mixed", {"cell_ratio": 4.0}),
    (2, (48.0, 41.0), "mixed", {"pair_scheme": 2}),
    (2, (48.0, 41.0), "fp64", {"cell_ratio": 0.5}),
    (2, (35.0, 35.0), "fp64", {"cell_ratio": 4.0}),
    (3, (24.0, 19.0, 21.0), "mixed", {"cell_ratio": 0.5}),
    (3, (24.0, 19.0, 21.0), "mixed", {"cell_ratio": 1.0 / 3.0}),
    (3, (7.0, 6.5, 21.0), "mixed", {"cell_ratio": 0.5}),
    (3, (24.0, 19.0, 21.0), "mixed", {"pair_scheme": 2}),
    (3, (24.0, 24.0, 24.0), "mixed", {"pair_scheme": 1}),
    (3, (24.0, 19.0, 21.0), "fp64", {"cell_ratio": 0.5}),
])
def test_pair_set_at_the_cutoff(dim, box, precision, knobs):
    n = 20000 if dim == 2 else 12000
    r = shells(dim, box, n, 1000 * dim + int(sum(box)))
    prm = _abi.make_params(dim=dim, box=list(box), h_short=1.5, h_long=CUT, bdash=1e-4, dt=1e-4)
    v, m, u = np.zeros((n, dim)), np.ones(n), np.zeros(n)
    ref, _ = oracle.pairs(prm, r)
    with Engine(prm, precision, max_particles=n) as e:
        s = e.add(prm, r, v, m, u)
        e.set_tuning(**knobs)
        assert e.pair_count(s) == len(ref)
