"""Explicit syncs of a periodic block with fewer cells along an axis than ghost
layers: the outer ghost layers of its face fields copy inner ghosts, and every
halo copy reads the values from before the sync (the last size has more copies
than the GPU takes at once)."""
import ctypes

import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu


def _copies(rows, n):
    """A copy table as (dst, src) index arrays (field, block, i, j, k, comp)."""
    kind = np.dtype([("dst", np.int32, 6), ("src", np.int32, 6), ("sign", float)])
    if n == 0:
        return np.zeros((0, 6), np.int32), np.zeros((0, 6), np.int32)
    t = np.frombuffer((ctypes.c_char * (n * kind.itemsize)).from_address(ctypes.addressof(rows.contents)), kind)
    return t["dst"], t["src"]


def _expected(before, group, nghost):
    """The halo copies of the block's tables on the values before, then the owner copies."""
    after = {f: a.copy() for f, a in before.items()}
    at = lambda x: tuple(x[:, 2 + a] + nghost for a in range(3))
    for rows, n, source in ((group.halo, group.n_halo, before), (group.owner, group.n_owner, after)):
        dst, src = _copies(rows, n)
        for f in after:
            m = dst[:, 0] == f
            assert np.array_equal(src[m, 0], dst[m, 0])
            after[f][at(dst[m])] = source[f][at(src[m])]
    return after


@pytest.mark.parametrize("n,nghost", [((3, 5, 4), 4), ((2, 3, 2), 4), ((2, 2, 3), 8), ((3, 300, 301), 4)])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("kind", ["periodic", "tables"])
def test_halo_copies_read_the_values_before_the_sync(n, nghost, precision, kind):
    if not has_gpu():
        pytest.skip("no GPU")
    from mpcns_mercury_b200 import capi, reference_constants
    from mpcns_mercury_b200.capi import Batch, SolveDesc

    k = reference_constants()
    d = SolveDesc([n], nghost, k, precision=precision)
    group = d.desc.groups[capi.GROUPS.index("BFACE")]
    batch = Batch(1, precision)
    slot = batch.add(d) if kind == "tables" else batch.add_periodic(n, nghost, k)
    rng = np.random.default_rng(5)
    lo = (-nghost,) * 3
    ext = {f: tuple(n[a] + (a == ax) + nghost for a in range(3)) for ax, f in enumerate(("B_XI", "B_ETA", "B_ZETA"))}
    for _ in range(20 if max(n) < 10 else 1):
        before = {f: rng.integers(-1000, 1000, tuple(h + nghost for h in hi) + (1,)).astype(float) for f, hi in ext.items()}
        for f, a in before.items():
            batch.upload(slot, f, a, lo, ext[f])
        batch.sync(slot, "BFACE")
        want = _expected({capi.FIELD_ID[f]: a for f, a in before.items()}, group, nghost)
        for f, hi in ext.items():
            assert np.array_equal(batch.download(slot, f, lo, hi), want[capi.FIELD_ID[f]]), f
    batch.close()
