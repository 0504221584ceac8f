"""SEMISIM_MGA is the prolongation factor of every solve as it stands.  Unset, the Poisson solves
scale their coarse corrections by 1.2: set to 1.2 it changes nothing in them, bit for bit, and
set to 1.0 it takes that scaling away (the solution differs).  A child process, since the knob
is library-wide and stays set."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import os, sys
import numpy as np
import semiconductor_devices_simulator_b200 as S
from semiconductor_devices_simulator_b200 import devices as D
from semiconductor_devices_simulator_b200.abi import dptr
lib = S.load()
lib.api3b_set_persist(int(sys.argv[2]), -1)
out = []
for mga in (None, "1.2", "1.0"):
    if mga:
        os.environ["SEMISIM_MGA"] = mga
    w = (D.graph_pn_diode if sys.argv[1] == "graph" else D.pn_diode)(lib, n=(31, 17, 12))
    assert lib.b200x_prepare() == 1
    lib.b200x_init_state()
    lib.b200x_apply_bc()
    phi, F, sol = np.zeros(w.N), np.zeros(w.N), np.zeros(w.N)
    lib.b200x_get(S.ST_PHI, dptr(phi))
    i = np.arange(w.N) % 31
    phi += np.where((i > 0) & (i < 30), 5e-3 * np.random.default_rng(3).standard_normal(w.N), 0.0)
    lib.b200x_poisson(dptr(phi), dptr(F), None, None)
    lib.b200x_pcg(2000, 1e-6, dptr(sol))
    assert np.abs(sol).max() > 0.0
    out.append(sol)
assert np.array_equal(out[0], out[1]), np.abs(out[0] - out[1]).max()
assert not np.array_equal(out[0], out[2])
"""


@pytest.mark.parametrize("persist", [1, 0], ids=["persistent", "per-pass"])
@pytest.mark.parametrize("kind", ["tensor", "graph"])
def test_knob_is_the_factor(kind, persist):
    env = {k: v for k, v in os.environ.items() if k != "SEMISIM_MGA"}
    r = subprocess.run([sys.executable, "-c", CHILD, kind, str(persist)], cwd=ROOT, env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
