"""The exported pair list (csrc/sph_pairs.cu, k_pair_rows / k_pair_write) in rows
of none to thousands of partners, with particles numbered in no order, one
simulation of a batch, and each output left out -- against the oracle's list
(pairs and squared distances bit for bit)."""
import ctypes

import numpy as np
import pytest

from oracle import oracle
from pyticles_gb300 import Engine, _abi

pytestmark = pytest.mark.gpu


def state(dim, n, box, cutoff, seed):
    rng = np.random.default_rng(seed)
    r = rng.uniform(0, box, (n, dim))
    prm = _abi.make_params(dim=dim, box=[box] * dim, h_short=1.0, h_long=1.0, cutoff=cutoff,
                           tolerance=0.25, dt=1e-9)
    return prm, r, rng.normal(size=(n, dim)), np.ones(n), np.zeros(n)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("dim,n,box,cutoff", [
    (2, 1, 10.0, 1.0), (2, 50, 40.0, 1.0), (2, 900, 30.0, 2.0), (2, 1100, 9.0, 30.0),
    (2, 9000, 60.0, 1.5), (3, 700, 12.0, 2.0), (3, 2500, 9.0, 4.2),
])
def test_rows(dim, n, box, cutoff, precision):
    prm, r, v, m, u = state(dim, n, box, cutoff, n)
    other = state(dim, 60, 20.0, 1.0, 1)
    iap, rsq = oracle.pairs(prm, r)
    with Engine(prm, precision, max_particles=n + 60, max_sims=2) as e:
        e.add(*other)
        s = e.add(prm, r, v, m, u)
        for _ in range(2):
            got = e.pairs(s)
            assert np.array_equal(got["iap"], iap)
            assert np.array_equal(got["rsq"], rsq)
            assert np.array_equal(got["dv"], v[iap[:, 1]] - v[iap[:, 0]])
        d = r[iap[:, 1]] - r[iap[:, 0]]
        d = np.where(d > box / 2, d - box, np.where(d < -box / 2, d + box, d))
        assert np.array_equal(got["drij"], d)
        # the distances alone
        only = np.zeros(max(len(rsq), 1))
        k = ctypes.c_int64()
        st = _abi.lib().sph_sim_export_pairs(e._h, s, len(rsq), None, None, only.ctypes.data, None,
                                             ctypes.byref(k), _abi.SPH_HOST)
        assert st == 0 and k.value == len(rsq)
        assert np.array_equal(only[:len(rsq)], rsq)
