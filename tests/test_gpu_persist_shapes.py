"""Persistent linear solves over mesh shapes where their colour-by-colour layout can go wrong:
odd and even row lengths, rows shorter than a pair of slots, dimensions that stop coarsening
before the others, a one-block hierarchy, one cluster, and a whole grid.  The systems are the
library's own (a perturbed pn diode); the solutions must meet the reference's stop rules,
recomputed in numpy with the oracle's 7-point product."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

from oracle import restate as R  # noqa: E402
import semiconductor_devices_simulator_b200 as S  # noqa: E402
from semiconductor_devices_simulator_b200 import devices as D  # noqa: E402
from semiconductor_devices_simulator_b200.abi import dptr  # noqa: E402

pytestmark = pytest.mark.gpu
SHAPES = [(5, 5, 5), (3, 40, 5), (4, 3, 66), (17, 5, 3), (65, 3, 3), (9, 9, 9), (200, 3, 4), (41, 37, 23), (130, 33, 19)]


@pytest.fixture(scope="module")
def lib():
    return S.load()


@pytest.fixture(params=[0, 1], ids=["fp64", "refined"])
def precision(lib, request):
    old = lib.api3b_set_precision(request.param)
    yield request.param
    lib.api3b_set_precision(old)


def perturbed(lib, n):
    w = D.pn_diode(lib, n=n)
    assert lib.b200x_prepare() == 1
    lib.b200x_init_state()
    lib.b200x_apply_bc()
    phi = np.zeros(w.N)
    lib.b200x_get(S.ST_PHI, dptr(phi))
    i = np.arange(w.N) % n[0]
    phi += np.where((i > 0) & (i < n[0] - 1), 5e-3 * np.random.default_rng(3).standard_normal(w.N), 0.0)
    lib.b200x_set(S.ST_PHI, dptr(phi))
    lib.b200x_rebuild_np()
    lib.b200x_upd_mob()
    return w, phi


@pytest.mark.parametrize("n", SHAPES, ids=lambda n: "x".join(map(str, n)))
def test_persistent_bicgstab_shapes(lib, precision, n):
    w, _ = perturbed(lib, n)
    dims = tuple(n)
    for hole in (0, 1):
        A, b = np.zeros((7, w.N)), np.zeros(w.N)
        lib.b200x_cont_assemble(hole, dptr(A), dptr(b), None, None)
        sol, rn, r0 = np.zeros(w.N), np.zeros(1), np.zeros(1)
        rtol, atol = 1e-8, 2e-14
        lib.b200x_bicgstab(1000, rtol, atol, -1 if hole else 1, None, dptr(sol), dptr(rn), dptr(r0))
        one = np.ones(w.N)
        start = np.linalg.norm(b - R.matvec(A, dims, one))
        tgt = max(rtol * start, atol * R.bicg_floor(A, dims, b, one))
        res = np.linalg.norm(b - R.matvec(A, dims, sol))
        assert abs(r0[0] - start) <= 1e-9 * start
        assert res <= 1.5 * tgt + 1e-300, (res, tgt)


@pytest.mark.parametrize("n", SHAPES, ids=lambda n: "x".join(map(str, n)))
def test_persistent_pcg_shapes(lib, precision, n):
    w, phi = perturbed(lib, n)
    F, A = np.zeros(w.N), np.zeros((7, w.N))
    lib.b200x_poisson(dptr(phi), dptr(F), dptr(A), None)
    sol = np.zeros(w.N)
    its = lib.b200x_pcg(2000, 1e-6, dptr(sol))
    res = np.linalg.norm(F - R.matvec(A, tuple(n), sol))
    assert res <= 1e-3 * np.linalg.norm(F), (res, its)
