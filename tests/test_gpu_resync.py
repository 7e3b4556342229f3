"""An explicit Sync(U) between steps.  On the shell's rotated seams it gives ghosts
beside owned cells other densities than the step's own sync left there; the next
step's fluxes take these, with the primitive variables as they are."""
import ctypes

import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu


def _flux(L, Q, k, gamma):
    """The Rusanov flux (Scheme_U_) of states (rho, u, v, w, p) through faces of area vector k."""
    def side(s):
        rho, u, v, w, p = s
        un = k[0] * u + k[1] * v + k[2] * w
        e = p / (gamma - 1.0) + 0.5 * rho * (u * u + v * v + w * w)
        cons = np.stack([rho, rho * u, rho * v, rho * w, e])
        f = np.stack([rho * un, rho * un * u + k[0] * p, rho * un * v + k[1] * p, rho * un * w + k[2] * p, un * (e + p)])
        return cons, f, np.abs(un) + np.sqrt(gamma * p / rho) * np.sqrt((np.array(k) ** 2).sum(0))

    (uL, fL, rL), (uQ, fQ, rQ) = side(L), side(Q)
    return 0.5 * (fL + fQ) - 0.5 * np.maximum(rL, rQ) * (uQ - uL)


# each of the two steps' results is rounded to its type (a few units in the last
# place of the largest component), and the step's increment is a difference of them
@pytest.mark.parametrize("precision,tol", [(0, 1e-13), (1, 2e-6)], ids=["fp64", "mixed"])
def test_sync_of_u_between_steps(precision, tol):
    if not has_gpu():
        pytest.skip("no GPU")
    from mpcns_mercury_b200 import capi
    from mpcns_mercury_b200 import magnetosphere as M
    from mpcns_mercury_b200.capi import Batch, SolveDesc

    case = M.ShellCase(na=6, nr=5)
    k = M.constants(case)
    before, after, dt, geo = [], [], [], []
    for sync in (False, True):
        t = M.topology(case)
        d = SolveDesc(case.cells, 4, k, precision=precision, topology=t)
        batch = Batch(1, precision)
        slot = batch.add(d)
        M.set_up(batch, case, slot=slot, k=k)
        batch.prepare(slot)
        batch.request(slot, 4)
        batch.run(3)
        if sync:
            batch.sync(slot, "UCELL")
        get = lambda f, b, hi: batch.download(slot, f, (-1,) * 3, hi, block=b)
        box = [tuple(v + 1 for v in n) for n in case.cells]
        before.append([{f: get(f, b, hi) for f in ("U_H", "U_NA", "PV_H", "PV_NA")} for b, hi in enumerate(box)])
        geo.append([{f: get(f, b, hi) for f in ("JDXI", "JDET", "JDZE", "JAC")} for b, hi in enumerate(box)])
        batch.run(1)
        info = batch.poll()[slot]
        assert info.status == 0 and info.step == 4
        dt.append(info.dt)
        after.append([{f: batch.download(slot, f, (0,) * 3, n, block=b) for f in ("U_H", "U_NA")} for b, n in enumerate(case.cells)])
        batch.close()
        capi.lib().mhd_topology_destroy(ctypes.c_void_p(t.value))
    assert dt[0] == dt[1]
    touched = 0
    for b, n in enumerate(case.cells):
        for u, pv in (("U_H", "PV_H"), ("U_NA", "PV_NA")):
            state = []
            for run in (0, 1):
                x = before[run][b]
                state.append([x[u][..., 0]] + [x[pv][..., q] for q in range(4)])
            assert all(np.array_equal(p, q) for p, q in zip(state[0][1:], state[1][1:]))
            inner = (slice(1, -1),) * 3
            assert np.array_equal(state[0][0][inner], state[1][0][inner])
            want = np.zeros((5,) + n)
            for axis, jd in enumerate(("JDXI", "JDET", "JDZE")):
                # face q of the axis lies below the cell q (arrays start at -1)
                low = [slice(1, -1)] * 3
                cell = [slice(1, -1)] * 3
                low[axis] = slice(0, -1)
                cell[axis] = slice(1, None)
                face = [geo[0][b][jd][tuple(cell)][..., q] for q in range(3)]
                f = [_flux([s[tuple(low)] for s in st], [s[tuple(cell)] for s in st], face, k.gamma) for st in state]
                diff = np.moveaxis(f[1] - f[0], axis + 1, 0)
                want -= np.moveaxis(diff[1:] - diff[:-1], 0, axis + 1) * dt[0] / geo[0][b]["JAC"][inner][..., 0]
            got = np.moveaxis(after[1][b][u] - after[0][b][u], -1, 0)
            # the wall sets the innermost layer from the one above it
            got, want = got[..., 1:], want[..., 1:]
            scale = np.abs(after[0][b][u]).max()
            touched += int((np.abs(want).max(0) > 100 * tol * scale).sum())
            assert np.abs(got - want).max() <= tol * scale, (b, u, np.abs(got - want).max() / scale, np.abs(want).max() / scale)
    assert touched > 0
