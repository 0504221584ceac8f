"""Labelling of floating majority blocks (float_fix) on shapes that a merging pass can get
wrong: blocks that wind through the mesh, touch only along one axis, cross warp edges inside a
row, end at row ends, and many blocks at once.  Every unanchored block must come out scaled by
one factor, every other node untouched; the blocks themselves come from scipy's labelling of
the same majority rule (semiconductor_3d.c:3159-3228)."""
import numpy as np
import pytest
from scipy import ndimage

import semiconductor_devices_simulator_b200 as S
from semiconductor_devices_simulator_b200 import devices as D
from semiconductor_devices_simulator_b200.abi import dptr, iptr

pytestmark = pytest.mark.gpu


def islands(n, fill, seed):
    """n-type nodes in a p body: random ones, a winding channel, and rows that touch the ends."""
    r = np.random.default_rng(seed)
    m = r.random((n[2], n[1], n[0])) < fill
    if n[1] >= 4:
        m[n[2] // 2, 0::2, 1:-1] = True                 # rows of a snake joined at alternate ends
        m[n[2] // 2, 1::4, -2] = True
        m[n[2] // 2, 3::4, 1] = True
    return m


@pytest.fixture(scope="module")
def lib():
    return S.load()


@pytest.mark.parametrize("graph", [False, True], ids=["tensor", "graph"])
@pytest.mark.parametrize("n,fill", [((33, 9, 7), 0.05), ((64, 5, 6), 0.3), ((7, 40, 3), 0.45), ((130, 11, 5), 0.25),
                                    ((31, 3, 2), 0.6)], ids=str)
def test_every_floating_block_is_scaled_as_one(lib, n, fill, graph):
    lib.api3_init()
    xs, ys, zs = (np.linspace(0.0, 1e-8 * (q - 1), q) for q in n)
    N = int(np.prod(n))
    si = lib.api3_add_material(D.SI, 300.0)
    if graph:
        rp, cj, h, ar, vol, pos = D.tensor_graph(xs, ys, zs)
        assert lib.api3_set_mesh_graph(N, len(cj), iptr(rp), iptr(cj), dptr(h), dptr(ar), dptr(vol), dptr(pos))
    else:
        D._grid(lib, xs, ys, zs)
    m = islands(n, fill, n[0])
    m[:, :, 0] = m[:, :, -1] = False                    # the contact planes are p
    Nd = np.ascontiguousarray(np.where(m, 1e23, 0.0).ravel())
    Na = np.ascontiguousarray(np.where(m, 0.0, 1e22).ravel())
    lib.api3_set_node_data(iptr(np.full(N, si, np.int32)), dptr(Nd), dptr(Na), None)
    lib.api3_clear_contacts()
    con = np.zeros((n[2], n[1], n[0]), bool)
    for face, plane in ((0, 0), (1, n[0] - 1)):
        c = lib.api3_add_contact_ex(face, 0, n[1] - 1, 0, n[2] - 1, 0, 0, 0, 0.0, 0.0, 0.0, 0.0)
        con[:, :, plane] = True
        if graph:
            sel = np.arange(N) % n[0] == plane
            assert lib.api3_set_con_nodes(c, int(sel.sum()), iptr(np.flatnonzero(sel).astype(np.int32)),
                                          dptr(np.full(int(sel.sum()), 1e-16)))
    assert lib.b200x_prepare() == 1
    lib.b200x_init_state(); lib.b200x_apply_bc(); lib.b200x_rebuild_np(); lib.b200x_upd_mob()
    lib.b200x_cont_assemble(0, None, None, None, None)
    get = lambda q: (lambda a: (lib.b200x_get(q, dptr(a)), a)[1])(np.zeros(N))
    nn, pp, sc = get(S.ST_N), get(S.ST_P), get(S.ST_SC)
    sol0 = 1.0 + np.random.default_rng(4).normal(0, 0.02, N)
    dn = 0.5 * np.abs(Nd - Na)
    c = sc * sol0
    maj = ((c >= pp) & (c >= dn) & (sc >= dn) & (c > 10 * 1.1e16)).reshape(m.shape) & ~con
    lab, nb = ndimage.label(maj)                        # face neighbours, as the box method's
    touch = ndimage.binary_dilation(con) & maj
    anchored = set(np.unique(lab[touch])) - {0}
    sol = sol0.copy()
    nfix = lib.b200x_float_fix(0, dptr(sol))
    ratio = (sol / sol0).reshape(m.shape)
    assert (ratio[lab == 0] == 1.0).all()
    moved = 0
    for b, sl in enumerate(ndimage.find_objects(lab), 1):
        q = ratio[sl][lab[sl] == b]
        if b in anchored:
            assert (q == 1.0).all(), b
            continue
        assert q.max() - q.min() <= 1e-14 * q.max(), (b, q.min(), q.max())
        moved += bool(abs(q[0] - 1.0) > 1e-15)
    assert nfix == moved >= 1
