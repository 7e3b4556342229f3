"""Tables that break one of the rules by which the engine takes a shorter order of
a step's passes (E + Ehall summed ahead of the alias reduction, syncs joined into
fewer launches, a substep without the full Sync(dB)).  Every rule is checked
against the same tables in the order without it, which a harmless further copy
selects; all fields are the same to the bit, ghosts included."""
import ctypes

import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

G, N = 4, (6, 5, 7)
FIELDS = ["U_H", "U_NA", "B_XI", "B_ETA", "B_ZETA", "B_CELL", "J_CELL", "J_XI", "J_ETA", "J_ZETA", "E_XI", "E_ETA", "E_ZETA"]


class Tables:
    """The periodic block's copy tables, with entries added or changed."""

    def __init__(self, precision=0, resistive=False):
        from mpcns_mercury_b200 import reference_constants
        from mpcns_mercury_b200.capi import SolveDesc

        self.precision, self.resistive, self.keep = precision, resistive, []
        self.k = reference_constants(cfl=0.4)
        for q in range(19):
            self.k.bc[q] = 0.5 + 0.01 * q
        if resistive:
            self.k.resistive, self.k.res_max_it, self.k.res_rtol = 1, 50, 1e-9
        self.desc = SolveDesc([N], G, self.k, precision=precision)
        self.d = self.desc.desc

    def group(self, name):
        from mpcns_mercury_b200 import capi

        return self.d.groups[capi.GROUPS.index(name)]

    def _array(self, kind, rows):
        a = (kind * max(len(rows), 1))(*rows)
        self.keep.append(a)
        return ctypes.cast(a, ctypes.POINTER(kind))

    def set_copies(self, group, which, rows):
        from mpcns_mercury_b200.capi import MhdCopy

        g = self.group(group)
        setattr(g, which, self._array(MhdCopy, rows))
        setattr(g, "n_" + which, len(rows))

    def copies(self, group, which):
        g = self.group(group)
        t = getattr(g, which)
        return [t[q] for q in range(getattr(g, "n_" + which))]

    def add_copy(self, group, which, dst, src, sign=1.0):
        from mpcns_mercury_b200.capi import MhdCopy

        self.set_copies(group, which, self.copies(group, which) + [MhdCopy(dst, src, sign)])

    def add_set(self, group, dst, arg):
        from mpcns_mercury_b200.capi import MhdPhysOp

        g = self.group(group)
        op = MhdPhysOp()
        op.kind, op.arg, op.dst, op.src = 0, arg, dst, dst
        g.phys, g.n_phys = self._array(MhdPhysOp, [g.phys[q] for q in range(g.n_phys)] + [op]), g.n_phys + 1

    def classes(self):
        """[(owner, owner_sign, [(member, sign), ...]), ...]"""
        a = self.d.edge_aliases
        return [(a.owner[c], a.owner_sign[c], [(a.member[m], a.member_sign[m]) for m in range(a.offset[c], a.offset[c + 1])])
                for c in range(a.n_classes)]

    def set_classes(self, classes):
        from mpcns_mercury_b200.capi import MhdDof

        a = self.d.edge_aliases
        off = [0]
        for c in classes:
            off.append(off[-1] + len(c[2]))
        a.n_classes = len(classes)
        a.offset = self._array(ctypes.c_int32, off)
        a.owner = self._array(MhdDof, [c[0] for c in classes])
        a.owner_sign = self._array(ctypes.c_double, [c[1] for c in classes])
        a.member = self._array(MhdDof, [m for c in classes for m, _ in c[2]])
        a.member_sign = self._array(ctypes.c_double, [s for c in classes for _, s in c[2]])

    def hall_late(self):
        """E + Ehall summed behind the syncs: Sync(Ehall) copies an edge inside the block onto itself."""
        e = dof("EHALL_XI", 2, 2, 3)
        self.add_copy("EHALL", "owner", e, e)

    def ordered(self, group="EHALL"):
        """The syncs in their full order: an owner copy to a ghost that nothing
        reads from one that the group's halo copies write."""
        halo = self.copies(group, "halo")
        far = max(range(len(halo)), key=lambda q: max(-halo[q].dst.i, -halo[q].dst.j, -halo[q].dst.k))
        self.add_copy(group, "owner", halo[far].dst, halo[0 if far else 1].dst)

    def start(self):
        from mpcns_mercury_b200 import setup as S
        from mpcns_mercury_b200.capi import Batch

        batch = Batch(1, self.precision)
        slot = batch.add(self.desc)
        nodes, state = S.cube_state(N, solve_id=3)
        batch.setup_geometry(slot, nodes)
        if self.resistive:
            for a, f in enumerate(("ETA_RES_XI", "ETA_RES_ETA", "ETA_RES_ZETA")):
                hi = tuple(N[q] + (q != a) for q in range(3))
                batch.upload(slot, f, np.full(hi + (1,), 1e-3), (0, 0, 0), hi)
        for name, f in (("U_H", "U_H"), ("U_Na", "U_NA"), ("B_xi", "B_XI"), ("B_eta", "B_ETA"), ("B_zeta", "B_ZETA")):
            a = state[name]
            batch.upload(slot, f, a.data, a.lo, a.hi)
        batch.sync(slot, "UCELL")
        batch.sync(slot, "BFACE")
        batch.prepare(slot)
        return batch, slot

    def run(self, steps=3):
        batch, slot = self.start()
        batch.request(slot, steps)
        batch.run(steps)
        info = batch.poll()[slot]
        assert info.status == 0 and info.step == steps
        out = fields(batch, slot)
        batch.close()
        return out


def dof(field, i, j, k, comp=0):
    from mpcns_mercury_b200 import capi
    from mpcns_mercury_b200.capi import MhdDof

    return MhdDof(capi.FIELD_ID[field], 0, i, j, k, comp)


def fields(batch, slot):
    return {f: batch.download(slot, f, (-G,) * 3, tuple(v + 1 + G for v in N)) for f in FIELDS}


def same(a, b):
    for f in FIELDS:
        assert np.isfinite(b[f]).all() and np.array_equal(a[f], b[f]), (f, np.abs(a[f] - b[f]).max())


@pytest.fixture(autouse=True)
def gpu():
    if not has_gpu():
        pytest.skip("no GPU")


PRECISIONS = pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])


@PRECISIONS
def test_hall_late_changes_nothing(precision):
    """E + Ehall ahead of the syncs and behind them, on tables where both are right."""
    a, b = Tables(precision), Tables(precision)
    b.hall_late()
    same(a.run(), b.run())


@PRECISIONS
def test_alias_member_inside_the_block(precision):
    """The E alias reduction reads an edge that is not in a face of its block:
    without its Hall EMF."""
    got = []
    for late in (False, True):
        t = Tables(precision)
        c = t.classes()
        owner, sign, members = c[0]
        c[0] = (owner, sign, members + [(dof("JAC", 2, 2, 2), 1.0)])
        c[0][2][-1][0].field = owner.field
        t.set_classes(c)
        if late:
            t.hall_late()
        got.append(t.run())
    same(*got)


@PRECISIONS
def test_constant_in_an_owned_cell_of_b(precision):
    """A physical operation of Sync(B_cell) that sets an owned cell: behind the pass that computes it."""
    got = []
    for ordered in (False, True):
        t = Tables(precision)
        t.add_set("B_CELL", dof("B_CELL", 2, 0, 3, 1), 11)
        if ordered:
            t.ordered()
        got.append(t.run())
    same(*got)
    value = t.k.bc[11]
    assert got[0]["B_CELL"][2 + G, 0 + G, 3 + G, 1] == (np.float32(value) if precision else value)


def _with_member(t, member, sign=1.0):
    """`member` (an edge index) as a further member of the first class, with its owner copies."""
    c = t.classes()
    owner, osign, members = c[0]
    axis = "XI ETA ZETA".split()[owner.field]
    e = dof("JAC", *member)
    e.field = owner.field
    c[0] = (owner, osign, members + [(e, sign)])
    t.set_classes(c)
    for group, field in (("EHALL", "EHALL_"), ("EEDGE", "E_"), ("JEDGE", "J_")):
        t.add_copy(group, "owner", dof(field + axis, *member), dof(field + axis, owner.i, owner.j, owner.k), sign * osign)


@PRECISIONS
def test_ghost_alias_member(precision):
    """A class with a ghost edge: its E + Ehall comes with the owner copies of E."""
    got = []
    for ordered in (False, True):
        t = Tables(precision)
        _with_member(t, (N[0] + 2, N[1] + 2, 2))
        if ordered:
            t.ordered()
        got.append(t.run())
    same(*got)


@PRECISIONS
def test_owner_with_another_sign_as_a_member(precision):
    """The owner of a class is one of its members with a sign that is not the owner's."""
    got = []
    for ordered in (False, True):
        t = Tables(precision)
        c = t.classes()
        owner, sign, members = c[0]
        index = lambda d: (d.field, d.block, d.i, d.j, d.k)
        flipped = [(m, -s if index(m) == index(owner) else s) for m, s in members]
        assert flipped != members
        c[0] = (owner, sign, flipped)
        t.set_classes(c)
        if ordered:
            t.ordered()
        got.append(t.run())
    same(*got)


@PRECISIONS
def test_owner_copy_of_a_ghost_face_in_the_substep(precision):
    """Sync(dB) fills a ghost face by an owner copy in place of the halo copy."""
    got = []
    for owner in (False, True):
        t = Tables(precision, resistive=True)
        if owner:
            face = (-1, 2, 3)
            halo = t.copies("DB", "halo")
            row = next(h for h in halo if h.dst.field == dof("B_ETA", 0, 0, 0).field and (h.dst.i, h.dst.j, h.dst.k) == face)
            src = (row.src.i, row.src.j, row.src.k)
            t.set_copies("DB", "halo", [h for h in halo if h is not row])
            t.add_copy("DB", "owner", row.dst, row.src)
            # its four edges are those of the face it stands for
            for field, across in (("E_ZETA", 0), ("E_XI", 2)):
                for up in (0, 1):
                    e, s = [list(face), list(src)]
                    e[across] += up
                    s[across] += up
                    if all(0 <= e[a] < N[a] + 1 for a in range(3)) or field == "E_ZETA" and e[0] == 0:
                        continue
                    t.add_copy("ERES", "owner", dof(field, *e), dof(field, *s))
        got.append(t.run())
        for f in ("E_XI", "E_ETA", "E_ZETA"):  # E_res's array: its further copies go to ghosts
            got[-1][f] = got[-1][f][G:-G, G:-G, G:-G]
    same(*got)


@PRECISIONS
def test_operation_on_another_groups_field(precision):
    """Sync(Ehall) sets a density that the fluid pass reads: the step's graph runs
    the passes in the row of the step that is launched kernel by kernel."""
    from mpcns_mercury_b200 import capi

    got = []
    for eager in (False, True):
        t = Tables(precision)
        t.add_set("EHALL", dof("U_H", 3, 2, 4), 0)
        t.add_copy("EEDGE", "owner", dof("PV_H", 4, 3, 2, 3), dof("PV_NA", 4, 3, 2, 3))
        batch, slot = t.start()
        if eager:
            batch.request(slot, 3)
            ms, names, n = (ctypes.c_float * 100)(), (ctypes.c_char_p * 100)(), ctypes.c_int()
            capi.check(capi.lib().mhd_batch_step_profiled(batch.b, 3, 100, ms, names, ctypes.byref(n)), "step_profiled")
            order = [names[q].decode() for q in range(n.value)]
            assert order.index("k_fluid") > order.index("k_add_hall")
        else:
            batch.request(slot, 3)
            batch.run(3)
        info = batch.poll()[slot]
        assert info.status == 0 and info.step == 3
        got.append(fields(batch, slot))
        batch.close()
    same(*got)


def test_owner_copies_of_the_substep_that_are_not_there_already():
    """Sync(dB) with an owner copy between faces of different edges: its owner copies run, the rest is left out."""
    got = []
    for ordered in (False, True):
        t = Tables(resistive=True)
        t.add_copy("DB", "owner", dof("B_XI", 2, 2, 3), dof("B_XI", 3, 2, 3))
        t.k.res_rtol = t.d.constants.res_rtol = 1e-3
        if ordered:
            t.ordered("DB")
        got.append(t.run())
    same(*got)


def _shell_run(rule, ordered):
    """Three steps of a small shell with one entry that breaks `rule` of the joined syncs."""
    from mpcns_mercury_b200 import capi
    from mpcns_mercury_b200 import magnetosphere as M
    from mpcns_mercury_b200.capi import Batch, MhdCopy, MhdPhysOp, SolveDesc

    case = M.ShellCase(na=6, nr=5)
    k = M.constants(case)
    topo = M.topology(case)
    t = Tables.__new__(Tables)
    t.keep, t.desc = [], SolveDesc(case.cells, G, k, topology=topo)
    t.d = t.desc.desc
    hall, edge = t.group("EHALL"), t.group("EEDGE")
    if rule == "staged source set by its group":
        t.add_set("EHALL", hall.stash[0].src, 11)
    elif rule == "staged source set by the wall":
        op = MhdPhysOp()
        op.kind, op.arg, op.dst, op.src = 0, 11, edge.stash[0].src, edge.stash[0].src
        t.d.wall, t.d.n_wall = t._array(MhdPhysOp, [t.d.wall[q] for q in range(t.d.n_wall)] + [op]), t.d.n_wall + 1
    elif rule == "a slot of two groups":
        rows = [MhdCopy(c.dst, c.src, c.sign) for c in (edge.stash[q] for q in range(2 * edge.n_stash))]
        rows[0].dst.i = rows[edge.n_stash].src.i = hall.stash[0].dst.i
        edge.stash = t._array(MhdCopy, rows)
    else:  # an owned edge staged: E there takes its Hall EMF behind the staging of the joined order
        n = edge.n_stash
        rows = [edge.stash[q] for q in range(2 * n)]
        slot = MhdCopy(rows[0].dst, edge.owner[0].src, 1.0)
        slot.dst.i = t.d.n_staging
        back = MhdCopy(edge.halo[0].dst, slot.dst, 1.0)
        edge.stash, edge.n_stash = t._array(MhdCopy, rows[:n] + [slot] + rows[n:] + [back]), n + 1
        t.set_copies("EEDGE", "halo", t.copies("EEDGE", "halo")[1:])
        t.d.n_staging += 1
    if ordered:
        t.ordered("JEDGE")
    batch = Batch(1, 0)
    slot = batch.add(t.desc)
    M.set_up(batch, case, slot=slot, k=k)
    batch.prepare(slot)
    batch.request(slot, 3)
    batch.run(3)
    info = batch.poll()[slot]
    assert info.status == 0 and info.step == 3
    out = [batch.download(slot, f, (-G,) * 3, tuple(v + 1 + G for v in n), block=b) for f in FIELDS for b, n in enumerate(case.cells)]
    batch.close()
    capi.lib().mhd_topology_destroy(ctypes.c_void_p(topo.value))
    return out


@pytest.mark.parametrize("rule", ["staged source set by its group", "staged source set by the wall", "a slot of two groups",
                                  "an owned edge staged"])
def test_rules_of_the_joined_syncs(rule):
    for a, b in zip(_shell_run(rule, False), _shell_run(rule, True)):
        assert np.array_equal(a, b, equal_nan=True)
