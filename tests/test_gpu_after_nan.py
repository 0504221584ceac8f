"""A solve that ran on values that are no numbers leaves nothing behind: the next solve of the
same instance, from a good state, converges as a fresh one does.  The Krylov vectors and the
hierarchies stay in device memory between solves, so whatever a sweep reads before it has written
it would carry a NaN on.  Both solvers run on a state with one NaN potential and then on the good
one: the Newton-Poisson loop (PCG) must leave ||F / diag|| <= 1e-10 V, the continuity solve (all
through api3_resolve) the currents of a fresh instance to 1e-6 relative or its floor."""
import numpy as np
import pytest

import semiconductor_devices_simulator_b200 as S
from semiconductor_devices_simulator_b200 import devices as D
from semiconductor_devices_simulator_b200.abi import dptr

pytestmark = pytest.mark.gpu
TIGHT = (2000, 1000, 500, 1e-11, 1e-8, 1.0, 1.0)


@pytest.fixture(scope="module")
def lib():
    return S.load()


def build(lib, kind):
    if kind == "graph":
        return D.graph_pn_diode(lib, n=(23, 9, 7), diag=0.3, solver=TIGHT)
    return D.pn_diode(lib, n=(23, 9, 7), solver=TIGHT)


@pytest.mark.parametrize("kind,precision", [("tensor", 0), ("tensor", 1), ("graph", 0)])
def test_newton_after_nan(lib, kind, precision):
    old = lib.api3b_set_precision(precision)
    try:
        w = build(lib, kind)
        assert lib.b200x_prepare() == 1
        lib.b200x_init_state()
        good, norm = np.zeros(w.N), np.zeros(1)
        lib.b200x_get(S.ST_PHI, dptr(good))
        bad = good.copy()
        bad[w.N // 2 + 3] = np.nan
        lib.b200x_set(S.ST_PHI, dptr(bad))
        assert lib.b200x_poisson_newton(1e-12, 300, dptr(norm)) == 0
        lib.b200x_set(S.ST_PHI, dptr(good))
        assert lib.b200x_poisson_newton(1e-12, 300, dptr(norm)) == 1
        assert norm[0] <= 1e-10, norm[0]
    finally:
        lib.api3b_set_precision(old)


@pytest.mark.parametrize("kind,precision", [("tensor", 0), ("tensor", 1), ("graph", 0)])
def test_solve_after_nan(lib, kind, precision):
    old = lib.api3b_set_precision(precision)
    try:
        I = []
        for spoil in (False, True):
            w = build(lib, kind)
            lib.api3_set_contact_V(w.contacts["cathode"], 0.0)
            if spoil:
                lib.api3_set_contact_V(w.contacts["anode"], 0.4)
                assert lib.api3_solve() == 1
                bad = np.zeros(w.N)
                lib.b200x_get(S.ST_PHI, dptr(bad))
                bad[w.N // 2 + 3] = np.nan
                lib.b200x_set(S.ST_PHI, dptr(bad))
                lib.api3_set_contact_V(w.contacts["anode"], 0.5)
                lib.api3_resolve()
            lib.api3_set_contact_V(w.contacts["anode"], 0.5)
            assert lib.api3_solve() == 1
            c = w.contacts["anode"]
            I.append((lib.api3_get_contact_I(c), lib.api3_get_contact_Ifloor(c)))
        (i0, f0), (i1, f1) = I
        assert abs(i1 - i0) <= max(1e-6 * abs(i0), f0, f1), (i0, i1)
    finally:
        lib.api3b_set_precision(old)
