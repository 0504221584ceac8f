"""The Anderson pass at every fill of its history: depth 0 (only the state is stored), 1, 2, 5 and
the full 12 columns, with wrap-around of the slots.  The fixed point does not depend on the
depth: tightly converged currents (Gummel tolerance 1e-12 V) agree to 1e-7 or the floor, on a
tensor and on a graph mesh."""
import os

import numpy as np
import pytest

import semiconductor_devices_simulator_b200 as S
from semiconductor_devices_simulator_b200 import devices as D

pytestmark = pytest.mark.gpu
TIGHT = (2000, 1000, 500, 1e-12, 1e-9, 1.0, 1.0)


def solve(lib, depth, graph):
    os.environ["SEMISIM_AAM"] = str(depth)              # read by api3_init
    try:
        if graph:
            w = D.graph_nmosfet(lib, n=(24, 12, 3), models=4, solver=TIGHT)
        else:
            w = D.nmosfet(lib, n=(25, 13, 5), solver=TIGHT)
    finally:
        os.environ.pop("SEMISIM_AAM")
    lib.api3_set_verbose(0)
    assert lib.api3_get_aa_depth() == depth
    lib.api3_set_contact_V(w.contacts["drain"], 0.05)
    lib.api3_set_contact_V(w.contacts["gate"], 0.8)
    assert lib.api3_solve() == 1
    nc = lib.api3_get_ncon()
    return (np.array([lib.api3_get_contact_I(c) for c in range(nc)]),
            np.array([lib.api3_get_contact_Ifloor(c) for c in range(nc)]))


@pytest.mark.parametrize("graph", [False, True], ids=["tensor", "graph"])
def test_depths_share_the_fixed_point(graph):
    lib = S.load()
    try:
        i12, f12 = solve(lib, 12, graph)
        for depth in (0, 1, 2, 5):
            i, f = solve(lib, depth, graph)
            assert (np.abs(i - i12) <= np.maximum(1e-7 * np.abs(i12), np.maximum(f, f12))).all(), (depth, i, i12)
    finally:
        os.environ["SEMISIM_AAM"] = "12"
        lib.api3_init()
        os.environ.pop("SEMISIM_AAM")
