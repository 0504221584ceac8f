"""Newton-Poisson at fixed quasi-Fermi levels from the neutral start and over gate steps of up to
2.5 V: accumulation to inversion and back.  The Jacobian's diagonal q (n + p) / VT falls by orders of magnitude where
a step empties a node, so the line search decides rightly only when both of its norms
||F / diag|| are taken in one scaling (semiconductor_3d.c:2791-2823).  A loop that reports
convergence must leave a solved system, ||F / diag|| <= 1e-10 V: the last step is below the
Newton tolerance of 1e-12 V and the round-off floor of ~2,000 nodes lies near 1e-13 V."""
import numpy as np
import pytest

import semiconductor_devices_simulator_b200 as S
from semiconductor_devices_simulator_b200 import devices as D

pytestmark = pytest.mark.gpu
GATES = [(-1.5,), (-2.0, -0.5), (2.0, -0.5), (-1.0, 1.5), (0.5, -2.0, 1.0)]


@pytest.fixture(scope="module")
def lib():
    return S.load()


def build(lib, kind):
    if kind == "graph":
        return D.graph_nmosfet(lib, n=(14, 28, 3), diag=0.1)
    return D.nmosfet(lib, n=(14, 24, 4), h0=2e-9)


@pytest.mark.parametrize("gates", GATES, ids=lambda g: "to".join(map(str, g)))
@pytest.mark.parametrize("kind,precision", [("tensor", 0), ("tensor", 1), ("graph", 0)])
def test_newton_converges_to_the_solution(lib, kind, precision, gates):
    old = lib.api3b_set_precision(precision)
    try:
        w = build(lib, kind)
        for c in w.contacts.values():
            lib.api3_set_contact_V(c, 0.0)
        lib.api3_set_contact_V(w.contacts["gate"], gates[0])
        assert lib.b200x_prepare() == 1
        lib.b200x_init_state()
        norm = np.zeros(1)
        for v in gates:
            lib.api3_set_contact_V(w.contacts["gate"], v)
            ok = lib.b200x_poisson_newton(1e-12, 300, S.abi.dptr(norm))
            assert ok == 1 and norm[0] <= 1e-10, (v, ok, norm[0])
    finally:
        lib.api3b_set_precision(old)
