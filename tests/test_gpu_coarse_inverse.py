"""Coarsest-level inverse of the persistent solves at sizes around its warp splits (16 to 64
unknowns).  Two-level hierarchies on a diode well below its Debye length, where the coarse solve
decides the convergence of the Poisson system: the persistent solve and the per-pass one (which inverts the same matrix in its own kernel) apply the same
preconditioner, so a Poisson solve takes the same number of iterations (one more or less where
the last residual falls beside the limit), and with the preconditioned residual at 1e-6 of its
start and a preconditioned condition number below 10 both solutions are within 1e-5 of the exact
one."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

import semiconductor_devices_simulator_b200 as S  # noqa: E402
from semiconductor_devices_simulator_b200 import devices as D  # noqa: E402
from semiconductor_devices_simulator_b200.abi import dptr  # noqa: E402

pytestmark = pytest.mark.gpu
SHAPES = {16: (8, 3, 3), 27: (5, 5, 5), 32: (16, 3, 3), 36: (18, 3, 4), 54: (17, 5, 3), 63: (13, 5, 5), 64: (7, 7, 7)}


@pytest.fixture(scope="module")
def lib():
    return S.load()


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "refined"])
@pytest.mark.parametrize("nc", sorted(SHAPES))
def test_coarse_inverse_sizes(lib, prec, nc):
    n = SHAPES[nc]
    assert int(np.prod([(m + 1) // 2 if m > 2 else m for m in n])) == nc
    old = lib.api3b_set_precision(prec)
    oldp = lib.api3b_set_persist(1, -1)
    try:
        w = D.pn_diode(lib, n=n, L=(1e-7, 1e-7, 1e-7), NA=1e15, ND=1e15, xj=0.5e-7)
        assert lib.b200x_prepare() == 1
        lib.b200x_init_state()
        lib.b200x_apply_bc()
        phi = np.random.default_rng(nc).uniform(-0.1, 0.1, w.N)
        F, A = np.zeros(w.N), np.zeros((7, w.N))
        lib.b200x_poisson(dptr(phi), dptr(F), dptr(A), None)
        got = {}
        for on in (1, 0):
            lib.api3b_set_persist(on, -1)
            sol = np.zeros(w.N)
            got[on] = lib.b200x_pcg(2000, 1e-6, dptr(sol)), sol
    finally:
        lib.api3b_set_persist(oldp, -1)
        lib.api3b_set_precision(old)
    (its_p, x_p), (its_g, x_g) = got[1], got[0]
    assert its_p >= 2 and abs(its_p - its_g) <= 1, (its_p, its_g)
    assert np.abs(x_p - x_g).max() <= 2e-5 * np.abs(x_g).max(), np.abs(x_p - x_g).max() / np.abs(x_g).max()
