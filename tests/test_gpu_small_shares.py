"""A grid share is a cap at every size: shares of 1 to 12 blocks, where the grids become clusters
of 2, 4 or 8 blocks, on tensor and graph meshes.  Every launch keeps to its share, and the
continuity system it solves meets the reference's stop rule: on tensor meshes the residual is
recomputed in numpy (half the target is left to the recurrence's drift), on graphs the solution
agrees with the per-launch path's to 1e-6 (both residuals at 1e-10 of the start's, and a condition
below 1e4)."""
import numpy as np
import pytest

import semiconductor_devices_simulator_b200 as S
from oracle import restate as R
from semiconductor_devices_simulator_b200 import devices as D
from semiconductor_devices_simulator_b200.abi import dptr, iptr

pytestmark = pytest.mark.gpu
N = (23, 9, 7)
# share: blocks of the launch, CTAs of its clusters (1,449 nodes: a few blocks' worth)
SHAPE = {0: (8, 8), 1: (1, 0), 2: (2, 2), 3: (2, 2), 4: (4, 4), 7: (4, 4), 8: (8, 8), 12: (8, 8)}


def shape(lib):
    out = np.zeros(2, np.int32)
    lib.b200x_persist_shape(iptr(out[:1]), iptr(out[1:]))
    return tuple(int(v) for v in out)


def solve(lib, n, rtol):
    sol, rn, r0 = np.zeros(n), np.zeros(1), np.zeros(1)
    x0 = 1.0 + np.random.default_rng(7).random(n)
    lib.b200x_bicgstab(1000, rtol, 0.0, 1, dptr(x0), dptr(sol), dptr(rn), dptr(r0))
    assert rn[0] <= rtol * r0[0]
    return sol, r0[0]


@pytest.mark.parametrize("kind", ["fp64", "refined", "graph"])
@pytest.mark.parametrize("share", sorted(SHAPE))
def test_launches_keep_to_their_share(kind, share):
    lib = S.load()
    h = lib.api3b_new()
    lib.api3b_use(h)
    old = lib.api3b_set_persist(1, -1)
    try:
        lib.api3b_set_precision(int(kind == "refined"))
        w = D.graph_pn_diode(lib, n=N, diag=0.2) if kind == "graph" else D.pn_diode(lib, n=N)
        assert lib.b200x_prepare() == 1
        lib.b200x_init_state()
        lib.api3b_set_share(share)
        A, b = np.zeros((7, w.N)), np.zeros(w.N)
        lib.b200x_cont_assemble(0, dptr(A), dptr(b), None, None)
        shape(lib)
        x, r0 = solve(lib, w.N, 1e-10 if kind == "graph" else 1e-8)
        assert shape(lib) == SHAPE[share]
        if kind == "graph":
            lib.api3b_set_persist(0, -1)
            y, _ = solve(lib, w.N, 1e-10)
            assert np.abs(x - y).max() <= 1e-6 * np.abs(y).max()
        else:
            assert np.linalg.norm(b - R.matvec(A, N, x)) <= 1.5e-8 * r0
    finally:
        lib.api3b_set_persist(old, -1)
        lib.api3b_use(0)
        lib.api3b_free(h)
