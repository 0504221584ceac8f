"""Why the graph solves' coarsest inverse needs no row interchanges: its matrix has a positive
diagonal, no positive coupling, and columns whose diagonal is at least the sum of the others'
magnitudes.  Elimination keeps that, so the largest entry of a pivot column is always its diagonal,
the one that partial pivoting would take.  The operators are the library's own, Poisson and
both carriers' continuity, on a forward-biased diode (recombination on the diagonal), a MOSFET in
inversion (carrier densities over 30 decades) and one with gate tunnelling (exchange terms).
Tolerance: the column sums cancel to what recombination and contacts leave, within the rounding
of their ~1,000 terms (1e-12 of the diagonal)."""
import numpy as np
import pytest

import semiconductor_devices_simulator_b200 as S
from semiconductor_devices_simulator_b200 import devices as D
from semiconductor_devices_simulator_b200.abi import dptr, iptr

pytestmark = pytest.mark.gpu
CASES = {
    "diode": (lambda q: D.graph_pn_diode(q, n=(24, 12, 8), diag=0.3), {"anode": 0.65, "cathode": 0.0}),
    "nmos": (lambda q: D.graph_nmosfet(q, n=(24, 14, 6), diag=0.1), {"drain": 0.5, "gate": 1.0, "source": 0.0, "body": 0.0}),
    "tunnelling": (lambda q: D.graph_nmosfet(q, n=(24, 14, 6), models=7 | 32, tox=1.2e-9),
                   {"drain": 0.05, "gate": 1.0, "source": 0.0, "body": 0.0}),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_coarsest_operator_is_column_dominant(case, monkeypatch):
    lib = S.load()
    build, volts = CASES[case]
    graph, make = [], D.tensor_graph
    monkeypatch.setattr(D, "tensor_graph", lambda *a, **k: graph.append(make(*a, **k)) or graph[-1])
    w = build(lib)
    lib.api3_set_verbose(0)
    for label, v in volts.items():
        lib.api3_set_contact_V(w.contacts[label], v)
    assert lib.api3_solve() == 1
    rp, cj, h, ar, _, _ = graph[0]
    plan = lambda L, *out: lib.b200x_gmg_plan(w.N, iptr(rp), iptr(cj), dptr(h), dptr(ar), L, *out)
    n, nnz = np.zeros(1, np.int32), np.zeros(1, np.int32)
    nl = plan(0, iptr(n), iptr(nnz), None, None, None)
    assert nl >= 2
    plan(nl - 1, iptr(n), iptr(nnz), None, None, None)
    crp, ccj, agg = np.zeros(n[0] + 1, np.int32), np.zeros(nnz[0], np.int32), np.zeros(n[0], np.int32)
    plan(nl - 1, iptr(n), iptr(nnz), iptr(crp), iptr(ccj), iptr(agg))
    phi = np.zeros(w.N)
    lib.b200x_get(S.ST_PHI, dptr(phi))
    for qsign in (0, 1, -1):
        if qsign:
            lib.b200x_cont_assemble(int(qsign < 0), None, None, None, None)
        else:
            lib.b200x_poisson(dptr(phi), None, None, None)
        va, dg = np.zeros(nnz[0]), np.zeros(w.N)
        assert lib.b200x_gmg_vals(qsign, nl - 1, dptr(va), dptr(dg)) == nnz[0]
        dg = dg[:n[0]]
        off = np.zeros(n[0])
        np.add.at(off, ccj, np.abs(va))
        assert (dg > 0.0).all() and (va <= 0.0).all(), (qsign, dg.min(), va.max())
        assert (off <= dg * (1.0 + 1e-12)).all(), (qsign, (off / dg).max() - 1.0)
