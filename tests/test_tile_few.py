"""FP64 cell tiles of a handful of particles (eight lanes each up to 64 particles, 32
beyond) against the oracle, alone and in a batch of many: each simulation's bits
alone."""
import numpy as np
import pytest

from pyticles_gb300 import build
from tests.test_tile64 import KEYS, check, evaluate, system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


@pytest.mark.parametrize("dim", [2, 3])
def test_batch_of_few(dim):
    sims = [system(dim, n, 6.5, 30 * n + dim, heat_flux=True)
            for n in (2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33, 40, 63, 64, 65, 66)]
    got, counts = evaluate(*sims)
    for s, g, c in zip(sims, got, counts):
        check(s, g, c, heat=True)
        (alone,), (count,) = evaluate(s)
        assert count == c
        for k in KEYS + ("jq",):
            assert np.array_equal(alone[k], g[k]), (len(s[1]), k)
