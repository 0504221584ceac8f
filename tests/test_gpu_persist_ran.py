"""The layout and cluster shapes are solved by the persistent kernels, in the launch shape that their
size calls for: a solve that was refused or abandoned falls back to the per-pass path, which passes
the residual tests too.  Blocks are a thousand nodes' worth, at least 4; one cluster of 8 up to 8
of them, clusters of 16 above while level 1 has at most three (FP32: four) nodes a thread
of one, else a plain grid.

The FP32 PCG is checked here too, at the solver's own tolerance of 1e-3: one launch, and against
the FP64 PCG at 1e-9 an error of at most 1e-2 in the energy norm (the stop rule bounds it by
1e-3 times the root of the preconditioned condition number, taken as 100 at most)."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

from oracle import restate as R  # noqa: E402
import semiconductor_devices_simulator_b200 as S  # noqa: E402
import test_gpu_persist_clusters as C  # noqa: E402
import test_gpu_persist_shapes as P  # noqa: E402
from semiconductor_devices_simulator_b200.abi import dptr, iptr  # noqa: E402

pytestmark = pytest.mark.gpu
TPB = 512


def shape(lib):
    out = np.zeros(2, np.int32)
    lib.b200x_persist_shape(iptr(out[:1]), iptr(out[1:]))
    return int(out[0]), int(out[1])


def expected_cluster(n, precision):
    worth = -(-int(np.prod(n)) // (2 * TPB))
    if worth <= 8:
        return 8
    level1 = int(np.prod([(m + 1) // 2 if m > 2 else m for m in n]))
    return 16 if level1 <= (4 if precision else 3) * 16 * TPB else 0


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "refined"])
@pytest.mark.parametrize("n", P.SHAPES + C.SHAPES, ids=lambda n: "x".join(map(str, n)))
def test_shapes_run_persistently(n, precision):
    lib = S.load()
    old, oldp = lib.api3b_set_precision(precision), lib.api3b_set_persist(1, -1)
    try:
        # (the PCG test's tolerance of 1e-6 is solved in FP64 in either precision)
        for test, prec in ((P.test_persistent_bicgstab_shapes, precision), (P.test_persistent_pcg_shapes, 0)):
            csz = expected_cluster(n, prec)
            shape(lib)
            test(lib, precision, n)
            blocks, c = shape(lib)
            assert c == csz and blocks > 0, (blocks, c, csz)
            assert blocks % c == 0 if c else blocks > 1
            if np.prod(n) <= 31 * 2 * TPB:
                assert blocks == c
    finally:
        lib.api3b_set_persist(oldp, -1)
        lib.api3b_set_precision(old)


@pytest.mark.parametrize("n", P.SHAPES + C.SHAPES, ids=lambda n: "x".join(map(str, n)))
def test_fp32_pcg(n):
    lib = S.load()
    old, oldp = lib.api3b_set_precision(0), lib.api3b_set_persist(1, -1)
    try:
        w, phi = P.perturbed(lib, n)
        F, A, x, ref = np.zeros(w.N), np.zeros((7, w.N)), np.zeros(w.N), np.zeros(w.N)
        lib.b200x_poisson(dptr(phi), dptr(F), dptr(A), None)
        lib.b200x_pcg(2000, 1e-9, dptr(ref))
        lib.api3b_set_precision(1)
        shape(lib)
        l0 = lib.b200x_launches()
        its = lib.b200x_pcg(2000, 1e-3, dptr(x))
        assert lib.b200x_launches() - l0 <= 2                # the start's fill and the solve
        assert shape(lib)[1] == expected_cluster(n, 1) and its > 0
        e = x - ref
        err = np.sqrt(e @ R.matvec(A, tuple(n), e) / (ref @ R.matvec(A, tuple(n), ref)))
        assert err <= 1e-2, (err, its)
    finally:
        lib.api3b_set_persist(oldp, -1)
        lib.api3b_set_precision(old)
