"""The persistent solves' workspace (about 165 bytes a node of a tensor mesh) is taken only where such
solves are on: an instance set up with them off goes without, and takes it when they are switched
on later; both solve the continuity system to the reference's stop rule (recomputed in numpy,
half the target left to the recurrence's drift)."""
import numpy as np
import pytest

import semiconductor_devices_simulator_b200 as S
from oracle import restate as R
from semiconductor_devices_simulator_b200 import devices as D
from semiconductor_devices_simulator_b200.abi import dptr, iptr

pytestmark = pytest.mark.gpu
N = (41, 37, 23)


def solve(lib, w):
    """Launch shape of the solve (0 blocks: per pass)."""
    A, b = np.zeros((7, w.N)), np.zeros(w.N)
    lib.b200x_cont_assemble(0, dptr(A), dptr(b), None, None)
    out = np.zeros(2, np.int32)
    lib.b200x_persist_shape(iptr(out[:1]), iptr(out[1:]))
    sol, rn, r0 = np.zeros(w.N), np.zeros(1), np.zeros(1)
    x0 = 1.0 + np.random.default_rng(7).random(w.N)
    lib.b200x_bicgstab(1000, 1e-8, 0.0, 1, dptr(x0), dptr(sol), dptr(rn), dptr(r0))
    lib.b200x_persist_shape(iptr(out[:1]), iptr(out[1:]))
    assert np.linalg.norm(b - R.matvec(A, N, sol)) <= 1.5e-8 * r0[0]
    return out[0]


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "refined"])
def test_workspace_follows_the_switch(precision):
    lib = S.load()
    hs = [lib.api3b_new(), lib.api3b_new()]
    old = lib.api3b_set_persist(0, -1)
    try:
        size = {}
        for h, on in zip(hs, (0, 1)):                     # set up with them off, and on
            lib.api3b_set_persist(on, -1)
            lib.api3b_use(h)
            lib.api3b_set_precision(precision)
            w = D.pn_diode(lib, n=N)
            assert lib.b200x_prepare() == 1
            lib.b200x_init_state()
            size[on] = lib.b200x_device_bytes()
            assert (solve(lib, w) > 0) == bool(on)
            assert lib.b200x_device_bytes() == size[on]
        assert 150 * w.N < size[1] - size[0] < 220 * w.N
        lib.api3b_use(hs[0])                              # on since the second instance
        assert solve(lib, w) > 0
        assert lib.b200x_device_bytes() == size[1]
        lib.api3b_set_persist(0, -1)
        assert solve(lib, w) == 0
    finally:
        lib.api3b_set_persist(old, -1)
        lib.api3b_use(0)
        for h in hs:
            lib.api3b_free(h)
