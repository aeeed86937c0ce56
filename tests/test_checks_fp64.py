"""The checking build (tests/test_checks.py) over the FP64 forms and the one-block
binning: cell tiles with their item lists, the FP64 window walk by one, eight and 32
lanes, batches of both, and 2,048 particles on both sides of the one-block line.  They
run clean and give the release build's bits."""
import os
import subprocess
import sys

import pytest

from pyticles_gb300 import build

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys, numpy as np
sys.path.insert(0, ROOT)
from pyticles_gb300 import Engine, _abi
from tests.test_tile64 import system
from tests.test_small_binning_memory import gas
assert _abi.LIB_PATH.endswith(LIBNAME), _abi.LIB_PATH
heat = dict(heat_flux=True)
groups = {
    "tiles": [system(2, 700, 24.0, 1, **heat)],
    "eight lanes": [system(2, 3500, 40.0, 2, **heat)],
    "tiles of several fills": [system(2, 4000, 16.5, 3, **heat)],
    "one cell": [system(3, 600, 6.0, 4, **heat)],
    "3D": [system(3, 1500, 15.5, 5, **heat)],
    "walk, 32 lanes": [system(2, 300, 60.0, 6, **heat)],
    "walk, 8 lanes": [system(3, 2500, 30.0, 7, **heat)],
    "walk, a thread": [system(2, 5000, 120.0, 8, **heat)],
    "batch": [system(2, 700, 24.0, 9, **heat), system(2, 40, 60.0, 10, **heat),
              system(2, 4000, 16.5, 11, **heat), system(2, 900, (7.0, 40.0), 12, **heat)],
    "one block": [gas((90, 91), 1921, 13)],
    "six kernels": [gas((90, 91), 2048, 14)],
    "one block, batch": [gas((16, 16), 64, 15 + k) for k in range(20)],
}
out = []
for name, sims in groups.items():
    for precision in ("fp64", "mixed"):
        with Engine(sims[0][0], precision, max_particles=sum(len(s[1]) for s in sims),
                    max_sims=len(sims)) as e:
            ids = [e.add(*s) for s in sims]
            e.set_tuning(steps_per_graph=2)
            for s in ids:
                d = e.derivatives(s)
                e.sync()
                out += [d[k].sum() for k in ("rho", "vdot", "udot", "jq")]
                out.append(len(e.pairs(s)["iap"]))
            e.advance(4)
            e.sync()
            out += [x.sum() for s in ids for x in e.get_state(s)]
print(repr([float(x) for x in out]))
"""


def run_child(checks):
    env = dict(os.environ, PYTICLES_CHECKS="1" if checks else "0")
    code = CHILD.replace("ROOT", repr(ROOT)).replace(
        "LIBNAME", repr("libsph_checks.so" if checks else "libsph.so"))
    res = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True,
                         text=True, timeout=600)
    assert res.returncode == 0, res.stderr[-3000:]
    return res.stdout.strip().splitlines()[-1]


def test_fp64_forms_run_clean_and_match_release():
    build.build()
    build.build(checks=True)
    assert run_child(True) == run_child(False)
