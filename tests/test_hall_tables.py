"""k_edge_emf writes E + Ehall at once on the edges inside a block: no write of
the E alias reduction, of the singular edges or of Sync(Ehall) may land there
(the engine checks every solve's tables and falls back to the sum after the
syncs).  Here: the tables of lattices and shells, whose blocks meet in their
faces, hold no such write."""
import ctypes

import pytest

from mpcns_mercury_b200 import capi, reference_constants
from mpcns_mercury_b200 import magnetosphere as M
from mpcns_mercury_b200.capi import SolveDesc

E0 = capi.FIELD_ID["EHALL_XI"]


def _inside(axis, d, n):
    q = (d.i, d.j, d.k)
    return all(0 <= q[a] < n[a] if a == axis else 0 < q[a] < n[a] for a in range(3))


def _writes(desc):
    g = desc.groups[capi.GROUPS.index("EHALL")]
    for t, m in ((g.halo, g.n_halo), (g.owner, g.n_owner), (g.stash, 2 * g.n_stash), (g.phys, g.n_phys)):
        for q in range(m):
            d = t[q].dst
            if E0 <= d.field <= E0 + 2:
                yield d.field - E0, d
    for c in range(desc.edge_aliases.n_classes):
        yield desc.edge_aliases.owner[c].field, desc.edge_aliases.owner[c]
    for e in range(desc.singular.n_edges):
        yield desc.singular.owner[e].field, desc.singular.owner[e]


@pytest.mark.parametrize("cells,lattice", [((5, 4, 6), (1, 1, 1)), ((4, 5, 4), (2, 1, 3)), ((6, 4, 5), (2, 2, 2))])
def test_lattice_tables_write_no_edge_inside_a_block(cells, lattice):
    nb = lattice[0] * lattice[1] * lattice[2]
    d = SolveDesc([cells] * nb, 4, reference_constants(), lattice=lattice if nb > 1 else None)
    writes = list(_writes(d.desc))
    assert writes and not any(_inside(a, w, cells) for a, w in writes)
    d.close()


@pytest.mark.parametrize("na,nr,resistive", [(6, 5, False), (8, 12, True)])
def test_shell_tables_write_no_edge_inside_a_block(na, nr, resistive):
    case = M.ShellCase(na=na, nr=nr, resistive=resistive)
    t = M.topology(case)
    d = SolveDesc(case.cells, 4, M.constants(case), topology=t)
    writes = list(_writes(d.desc))
    assert writes and not any(_inside(a, w, (na, na, nr)) for a, w in writes)
    d.close()
    capi.lib().mhd_topology_destroy(ctypes.c_void_p(t.value))
