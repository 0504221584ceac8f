"""Krylov solves that run into their iteration cap or break down: the persistent kernels must
leave their loops together and stop where the per-pass solves stop.  Caps of 1 to 5 from a random
start on a continuity system with a target no few iterations reach: the iteration counts are equal;
||r|| agrees with the per-pass path to 1e-6 of the first residual in FP64 and to 1e-2 with FP32
inner solves (unit round-off 1e-16 and 6e-8 amplified by what BiCGSTAB's quotients lose in five
iterations, taken as 1e5 at most); on tensor meshes the residual of the returned solution is the
reported one to 1e-8.  A right-hand side of 1e-155 makes r.r smaller than the breakdown limit of
1e-300: one iteration, and the start is returned."""
import numpy as np
import pytest

import semiconductor_devices_simulator_b200 as S
from oracle import restate as R
from semiconductor_devices_simulator_b200 import devices as D
from semiconductor_devices_simulator_b200.abi import dptr

pytestmark = pytest.mark.gpu
# one cluster of 8 and of 16, clusters with a coarse part, a plain grid
SHAPES = [(17, 5, 3), (31, 27, 19), (41, 37, 33), (67, 65, 64)]
GRAPHS = [(23, 9, 7), (41, 22, 20)]                    # one cluster; a grid


@pytest.fixture(scope="module")
def lib():
    return S.load()


def system(lib, build, n):
    w = build(lib, n)
    assert lib.b200x_prepare() == 1
    lib.b200x_init_state()
    A, b = np.zeros((7, w.N)), np.zeros(w.N)
    lib.b200x_cont_assemble(0, dptr(A), dptr(b), None, None)
    x0 = 1.0 + np.random.default_rng(7).random(w.N)
    return w, A, b, x0


def both(lib, N, maxit, x0, rtol=1e-14):
    out = []
    old = lib.api3b_set_persist(1, -1)
    try:
        for on in (1, 0):
            lib.api3b_set_persist(on, -1)
            sol, rn, r0 = np.zeros(N), np.zeros(1), np.zeros(1)
            l0 = lib.b200x_launches()
            its = lib.b200x_bicgstab(maxit, rtol, 0.0, 1, dptr(x0), dptr(sol), dptr(rn), dptr(r0))
            out.append((its, sol, rn[0], r0[0], lib.b200x_launches() - l0))
    finally:
        lib.api3b_set_persist(old, -1)
    assert out[0][4] < out[1][4]                       # the persistent path ran
    return out


@pytest.mark.parametrize("n", SHAPES, ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "refined"])
def test_tensor_caps(lib, precision, n):
    old = lib.api3b_set_precision(precision)
    try:
        w, A, b, x0 = system(lib, lambda q, m: D.pn_diode(q, n=m), n)
        for maxit in (1, 2, 3, 5):
            p, g = both(lib, w.N, maxit, x0)
            assert p[0] == g[0] and (precision or p[0] == maxit), (maxit, p[0], g[0])
            assert abs(p[3] - g[3]) <= 1e-9 * g[3]
            assert abs(p[2] - g[2]) <= (1e-2 if precision else 1e-6) * g[3], (maxit, p[2], g[2], g[3])
            res = np.linalg.norm(b - R.matvec(A, tuple(n), p[1]))
            assert abs(res - p[2]) <= 1e-8 * p[3], (maxit, res, p[2], p[3])
    finally:
        lib.api3b_set_precision(old)


@pytest.mark.parametrize("n", GRAPHS, ids=lambda n: "x".join(map(str, n)))
def test_graph_caps(lib, n):
    w, _, _, x0 = system(lib, lambda q, m: D.graph_pn_diode(q, n=m, diag=0.2), n)
    for maxit in (1, 2, 3, 5):
        p, g = both(lib, w.N, maxit, x0)
        assert p[0] == g[0] == maxit
        assert abs(p[3] - g[3]) <= 1e-9 * g[3] and abs(p[2] - g[2]) <= 1e-6 * g[3], (maxit, p[2:4], g[2:4])
        assert np.abs(p[1] - g[1]).max() <= 1e-6 * np.abs(g[1]).max()


@pytest.mark.parametrize("kind", ["tensor", "graph"])
def test_breakdown_leaves_the_start(lib, kind):
    build = (lambda q, m: D.pn_diode(q, n=m)) if kind == "tensor" else (lambda q, m: D.graph_pn_diode(q, n=m))
    w, _, b, _ = system(lib, build, (17, 9, 5))
    lib.b200x_set(S.ST_RHS, dptr(np.ascontiguousarray(b * (1e-155 / np.linalg.norm(b)))))
    p, g = both(lib, w.N, 50, np.zeros(w.N))
    assert p[0] == g[0] == 1
    assert not p[1].any() and not g[1].any()
