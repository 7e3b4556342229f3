"""The implicit substep on tables whose Sync(Eres) or Sync(Jedge) writes an owned
edge: both syncs then run in full, and the CG keeps its direction in an array of
its own.  Here one owner copy is repeated in the group's halo table, which
changes no value: the results are the unmodified tables' to the bit, with the CG
loop on the device and driven from the host."""
import ctypes

import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

G, N = 4, (6, 5, 7)
FIELDS = ["U_H", "U_NA", "B_XI", "B_ETA", "B_ZETA", "J_CELL"]


def _repeat_owner(desc, group, keep):
    """The first owner copy of `group` as one more halo copy."""
    from mpcns_mercury_b200 import capi
    from mpcns_mercury_b200.capi import MhdCopy

    g = desc.desc.groups[capi.GROUPS.index(group)]
    rows = (MhdCopy * (g.n_halo + 1))(*[g.halo[q] for q in range(g.n_halo)])
    rows[g.n_halo] = g.owner[0]
    keep.append(rows)
    g.halo, g.n_halo = ctypes.cast(rows, ctypes.POINTER(MhdCopy)), g.n_halo + 1


def _desc(precision, group, keep):
    from mpcns_mercury_b200 import reference_constants
    from mpcns_mercury_b200.capi import SolveDesc

    k = reference_constants(cfl=0.4)
    k.resistive, k.res_max_it, k.res_rtol = 1, 50, 1e-9
    d = SolveDesc([N], G, k, precision=precision)
    if group:
        _repeat_owner(d, group, keep)
    return d


def _add(batch, desc, solve_id):
    from mpcns_mercury_b200 import setup as S

    slot = batch.add(desc)
    nodes, state = S.cube_state(N, solve_id=solve_id)
    batch.setup_geometry(slot, nodes)
    for a, f in enumerate(("ETA_RES_XI", "ETA_RES_ETA", "ETA_RES_ZETA")):
        hi = tuple(N[q] + (q != a) for q in range(3))
        batch.upload(slot, f, np.full(hi + (1,), 1e-3), (0, 0, 0), hi)
    for name, f in (("U_H", "U_H"), ("U_Na", "U_NA"), ("B_xi", "B_XI"), ("B_eta", "B_ETA"), ("B_zeta", "B_ZETA")):
        a = state[name]
        batch.upload(slot, f, a.data, a.lo, a.hi)
    batch.sync(slot, "UCELL")
    batch.sync(slot, "BFACE")
    batch.prepare(slot)
    return slot


def _run(batch, slots, steps):
    for s in slots:
        batch.request(s, steps)
    batch.run(steps)
    infos = batch.poll()
    out = []
    for s in slots:
        assert infos[s].status == 0 and infos[s].res_iters > 0
        out.append([infos[s].res_iters] + [batch.download(s, f, (0,) * 3, N) for f in FIELDS])
    return out


def _same(a, b):
    assert a[0] == b[0]
    for f, x, y in zip(FIELDS, a[1:], b[1:]):
        assert np.array_equal(x, y), (f, np.abs(x - y).max())


@pytest.mark.parametrize("host_loop", [False, True], ids=["device", "host"])
@pytest.mark.parametrize("group", ["ERES", "JEDGE"])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_full_syncs_of_the_substep(precision, group, host_loop):
    if not has_gpu():
        pytest.skip("no GPU")
    from mpcns_mercury_b200.capi import Batch

    keep = []
    alone = {}
    for solve in (3, 5):
        batch = Batch(1, precision)
        slot = _add(batch, _desc(precision, None, keep), solve)
        alone[solve] = [_run(batch, [slot], 2)[0], _run(batch, [slot], 2)[0]]
        batch.close()

    # a batch that starts with such a solve
    batch = Batch(1, precision)
    batch.cg_host_loop(host_loop)
    slot = _add(batch, _desc(precision, group, keep), 3)
    for want in alone[3]:
        _same(_run(batch, [slot], 2)[0], want)
    batch.close()

    # one that has run without: it joins, and leaves again
    batch = Batch(2, precision)
    batch.cg_host_loop(host_loop)
    plain = _add(batch, _desc(precision, None, keep), 5)
    _same(_run(batch, [plain], 2)[0], alone[5][0])
    full = _add(batch, _desc(precision, group, keep), 3)
    got = _run(batch, [full, plain], 2)
    _same(got[0], alone[3][0])
    _same(got[1], alone[5][1])
    batch.remove(full)
    again = _add(batch, _desc(precision, None, keep), 3)
    _same(_run(batch, [again], 2)[0], alone[3][0])
    batch.close()
