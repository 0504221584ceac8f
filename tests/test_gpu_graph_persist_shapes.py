"""Persistent graph solves over hierarchies where their tables and the dense inverse can go
wrong: few nodes, more nodes than one cluster takes (grid barriers), rows of unequal degree
(diagonal edges), and a coarsest level beyond the in-register inverse.  Bias points at tight
tolerances against the per-launch solves of the same library: currents within 1e-6 relative or
the round-off floor."""
import os

import numpy as np
import pytest

import semiconductor_devices_simulator_b200 as S
from semiconductor_devices_simulator_b200 import devices as D
from semiconductor_devices_simulator_b200.abi import dptr, iptr

pytestmark = pytest.mark.gpu
TIGHT = (2000, 1000, 500, 1e-11, 1e-8, 1.0, 1.0)


@pytest.fixture(scope="module")
def lib():
    return S.load()


def both(lib, build, volts):
    out = {}
    old = lib.api3b_set_persist(1, -1)
    try:
        for on in (1, 0):
            lib.api3b_set_persist(on, -1)
            w = build(lib)
            lib.api3_set_verbose(0)
            for label, v in volts.items():
                lib.api3_set_contact_V(w.contacts[label], v)
            assert lib.api3_solve() == 1
            nc = lib.api3_get_ncon()
            psi = np.zeros(w.N)
            lib.api3_bulk_copy(0, dptr(psi))
            out[on] = (np.array([lib.api3_get_contact_I(c) for c in range(nc)]),
                       np.array([lib.api3_get_contact_Ifloor(c) for c in range(nc)]), psi)
    finally:
        lib.api3b_set_persist(old, -1)
    (i1, f1, p1), (i0, f0, p0) = out[1], out[0]
    assert (np.abs(i1 - i0) <= np.maximum(1e-6 * np.abs(i0), np.maximum(f0, f1))).all(), (i1, i0)
    assert np.abs(p1 - p0).max() <= 1e-8


@pytest.mark.parametrize("n,diag", [((9, 6, 4), 0.0), ((23, 5, 3), 0.3), ((40, 21, 21), 0.0), ((41, 22, 20), 0.2)],
                         ids=["216", "345-diagonal", "17640-grid", "18040-grid-diagonal"])
def test_graph_shapes(lib, n, diag):
    both(lib, lambda q: D.graph_pn_diode(q, n=n, diag=diag, solver=TIGHT), {"anode": 0.5, "cathode": 0.0})


def test_coarsest_level_beyond_the_register_inverse(lib):
    """Node pairs a tight gap apart with gaps between the pairs that grow along x: one round of
    matching with every node's strongest neighbour pairs them once, then stalls, so the
    coarsest level keeps half of the 600 nodes."""
    def init(q, passes, beta):                          # library-wide knobs, read by api3_init
        env = {"SEMISIM_GPASS": passes, "SEMISIM_GBETA": beta}
        os.environ.update(env)
        try:
            q.api3_init()
        finally:
            for k in env:
                os.environ.pop(k)

    def build(q):
        init(q, "1", "1.0")
        gaps = np.where(np.arange(149) % 2 == 0, 0.4e-9, 4e-9 * 1.01 ** (np.arange(149) // 2))
        xs = np.concatenate([[0.0], np.cumsum(gaps)])
        ys = zs = np.array([0.0, 1e-6])
        rp, cj, h, ar, vol, pos = D.tensor_graph(xs, ys, zs)
        N = 600
        si = q.api3_add_material(D.SI, 300.0)
        assert q.api3_set_mesh_graph(N, len(cj), iptr(rp), iptr(cj), dptr(h), dptr(ar), dptr(vol), dptr(pos))
        n_out = np.zeros(1, np.int32)
        nl = q.b200x_gmg_plan(N, iptr(rp), iptr(cj), dptr(h), dptr(ar), 1, iptr(n_out), None, None, None, None)
        assert nl == 2 and 160 < n_out[0] <= 640, (nl, n_out)
        q.api3_set_solver(*TIGHT)
        i = np.arange(N) % 150
        Nd = np.where(i >= 75, 1e23, 0.0)
        q.api3_set_node_data(iptr(np.full(N, si, np.int32)), dptr(Nd), dptr(1e23 - Nd), None)
        q.api3_clear_contacts()
        c = [q.api3_add_contact_ex(f, 0, 1, 0, 1, 0, 0, 0, 0.0, 0.0, 0.0, 0.0) for f in (0, 1)]
        for cid, plane in zip(c, (0, 149)):
            nodes = np.flatnonzero(i == plane).astype(np.int32)
            assert q.api3_set_con_nodes(cid, len(nodes), iptr(nodes), dptr(np.full(len(nodes), 0.25e-12)))
        return D.Workload("pairs", (N, 1, 1), {"anode": c[0], "cathode": c[1]}, [])
    try:
        both(lib, build, {"anode": 0.4, "cathode": 0.0})
    finally:
        init(lib, "3", "0.5")
