"""The step with its syncs joined into fewer launches against the step that runs
every phase in the reference's order.  A copy table that breaks what the joined
order needs sends its solve the ordered way: here one more owner copy, from a
ghost that the halo copies write to a ghost that nothing reads.  Every field is
the same to the bit, ghosts included."""
import ctypes

import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

G = 4
FIELDS = ["U_H", "U_NA", "B_XI", "B_ETA", "B_ZETA", "PV_H", "PV_NA", "B_CELL", "J_CELL", "J_XI", "J_ETA", "J_ZETA",
          "E_XI", "E_ETA", "E_ZETA"]
NCOMP = {"U_H": 5, "U_NA": 5}


def _order(desc, group, keep):
    """One more owner copy in `group` (see above)."""
    from mpcns_mercury_b200 import capi
    from mpcns_mercury_b200.capi import MhdCopy

    g = desc.desc.groups[capi.GROUPS.index(group)]
    far = max(range(g.n_halo), key=lambda q: max(-g.halo[q].dst.i, -g.halo[q].dst.j, -g.halo[q].dst.k))
    near = next(q for q in range(g.n_halo) if q != far)
    rows = (MhdCopy * (g.n_owner + 1))(*[g.owner[q] for q in range(g.n_owner)])
    rows[g.n_owner].dst, rows[g.n_owner].src, rows[g.n_owner].sign = g.halo[far].dst, g.halo[near].dst, 1.0
    keep.append(rows)
    g.owner, g.n_owner = ctypes.cast(rows, ctypes.POINTER(MhdCopy)), g.n_owner + 1


def _run(batch, slot, cells, steps):
    batch.request(slot, steps)
    batch.run(steps)
    info = batch.poll()[slot]
    assert info.status == 0 and info.step == steps
    out = {}
    for f in FIELDS:
        for b, n in enumerate(cells):
            out[f, b] = batch.download(slot, f, (-G,) * 3, tuple(v + 1 + G for v in n), block=b)
    return out


def _same(a, b, what):
    for key in a:
        assert np.array_equal(a[key], b[key], equal_nan=True), (what, key, np.abs(a[key] - b[key]).max())


@pytest.mark.parametrize("n", [(3, 5, 4), (17, 8, 9)])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("resistive", [False, True])
def test_periodic_block(n, precision, resistive):
    """The periodic block's own tables, the same block from copy tables, and
    these in the reference's order."""
    if not has_gpu():
        pytest.skip("no GPU")
    from mpcns_mercury_b200 import reference_constants
    from mpcns_mercury_b200 import setup as S
    from mpcns_mercury_b200.capi import Batch, SolveDesc

    k = reference_constants(cfl=0.4)
    if resistive:
        k.resistive, k.res_max_it, k.res_rtol = 1, 50, 1e-9
    keep, got = [], []
    for kind in ("periodic", "tables", "ordered"):
        batch = Batch(1, precision)
        if kind == "periodic":
            slot = batch.add_periodic(n, G, k)
        else:
            d = SolveDesc([n], G, k, precision=precision)
            if kind == "ordered":
                _order(d, "EHALL", keep)
                _order(d, "DB", keep)
            slot = batch.add(d)
        nodes, state = S.cube_state(n, solve_id=3)
        batch.setup_geometry(slot, nodes)
        if resistive:
            eta = np.full(tuple(v + 1 for v in n) + (1,), 1e-3)
            for a, f in enumerate(("ETA_RES_XI", "ETA_RES_ETA", "ETA_RES_ZETA")):
                hi = tuple(n[q] + (q != a) for q in range(3))
                batch.upload(slot, f, np.ascontiguousarray(eta[tuple(slice(0, v) for v in hi)]), (0, 0, 0), hi)
        for name, f in (("U_H", "U_H"), ("U_Na", "U_NA"), ("B_xi", "B_XI"), ("B_eta", "B_ETA"), ("B_zeta", "B_ZETA")):
            a = state[name]
            batch.upload(slot, f, a.data, a.lo, a.hi)
        batch.sync(slot, "UCELL")
        batch.sync(slot, "BFACE")
        batch.prepare(slot)
        got.append(_run(batch, slot, [n], 3))
        batch.close()
    _same(got[1], got[2], "tables, ordered")
    _same(got[0], got[2], "periodic, ordered")


@pytest.mark.parametrize("na,nr", [(6, 5), (8, 12)])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("resistive", [False, True])
def test_shell(na, nr, precision, resistive):
    if not has_gpu():
        pytest.skip("no GPU")
    from mpcns_mercury_b200 import capi
    from mpcns_mercury_b200 import magnetosphere as M
    from mpcns_mercury_b200.capi import Batch, SolveDesc

    kw = dict(resistive=True, **M.ETA_CONFIG) if resistive else dict(resistive=False)
    case = M.ShellCase(na=na, nr=nr, **kw)
    k = M.constants(case)
    keep, got = [], []
    for ordered in (False, True):
        t = M.topology(case)
        d = SolveDesc(case.cells, G, k, precision=precision, topology=t)
        if ordered:
            _order(d, "EHALL", keep)
            if resistive:
                _order(d, "DB", keep)
        batch = Batch(1, precision)
        slot = batch.add(d)
        M.set_up(batch, case, slot=slot, k=k)
        batch.prepare(slot)
        got.append(_run(batch, slot, case.cells, 3))
        batch.close()
        capi.lib().mhd_topology_destroy(ctypes.c_void_p(t.value))
    _same(got[0], got[1], "joined, ordered")
