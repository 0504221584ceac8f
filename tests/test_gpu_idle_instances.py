"""The launch shape of a solve, and with it the order of its reductions, follows from its size and
its caller's settings, not from other instances of the process: a gate sweep of a 36,864-node
MOSFET is bit for bit the same with and without four idle instances of that size."""
import numpy as np
import pytest

import semiconductor_devices_simulator_b200 as S
from semiconductor_devices_simulator_b200 import devices as D
from semiconductor_devices_simulator_b200.abi import iptr

pytestmark = pytest.mark.gpu
N = (48, 32, 24)


def sweep(lib, h):
    lib.api3b_use(h)
    try:
        w = D.nmosfet(lib, n=N, vds=(0.5,), vg_max=0.2, dvg=0.1)
        assert D.start_sweep(lib, w, w.sweeps[0])
        I = D.run_sweep(lib, w, w.sweeps[0])[1]
        shape = np.zeros(2, np.int32)
        lib.b200x_persist_shape(iptr(shape[:1]), iptr(shape[1:]))
        return I, tuple(shape)
    finally:
        lib.api3b_use(0)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "refined"])
def test_idle_instances_change_nothing(precision):
    lib = S.load()
    hs = []
    try:
        out = []
        for idle in (0, 4):
            for _ in range(idle):
                hs.append(lib.api3b_new())
                lib.api3b_use(hs[-1])
                D.nmosfet(lib, n=N)
                assert lib.b200x_prepare() == 1
            hs.append(lib.api3b_new())
            lib.api3b_use(hs[-1])
            lib.api3b_set_precision(precision)
            out.append(sweep(lib, hs[-1]))
            lib.api3b_use(0)
            lib.api3b_free(hs.pop())
        assert out[0][1] == out[1][1] and out[0][1][0] > 0, (out[0][1], out[1][1])
        np.testing.assert_array_equal(out[0][0], out[1][0])
    finally:
        lib.api3b_use(0)
        for h in hs:
            lib.api3b_free(h)
