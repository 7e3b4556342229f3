"""The FP64 primitive variables' quotients (momentum / density) are those of IEEE
division to the bit, over the whole range of both operands."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu


def _operands(kind, count, rng):
    """(a, b): numerators and densities."""
    sign = rng.choice([-1.0, 1.0], count)
    mant = lambda: 1.0 + rng.random(count)
    if kind == "ordinary":
        return sign * mant() * 2.0 ** rng.integers(-40, 40, count), mant() * 2.0 ** rng.integers(-30, 30, count)
    if kind == "wide":
        return sign * mant() * 2.0 ** rng.integers(-1020, 1020, count), mant() * 2.0 ** rng.integers(-39, 1020, count)
    if kind == "ends":  # around the bounds of the fast path
        a = sign * np.exp(rng.choice(np.log([1e-300, 1e-280, 1e-192, 1e-180, 1e-80, 1e280, 1e300]), count) + rng.normal(0, 4, count))
        return a, np.exp(rng.choice(np.log([1e-12, 1.0, 1e20, 1e100, 1e250]), count) + rng.normal(0, 4, count))
    # next to the rounding midpoints: b m = a 2^s + c with a midpoint m of two doubles and a small odd c
    a, b = np.empty(count), np.empty(count)
    got = 0
    while got < count:
        B = (1 << 52) | int(rng.integers(0, 1 << 52)) | 1
        if got % 3 == 0:
            B = (1 << 53) - 1 - 2 * int(rng.integers(0, 1000))
        for s in (53, 54):
            for c in (-3, -1, 1, 3):
                m = c * pow(B, -1, 1 << s) % (1 << s)
                m += 0 if m >= 1 << 53 else 1 << 53
                A, rest = divmod(B * m - c, 1 << s)
                if rest == 0 and m % 2 and 1 << 53 <= m < 1 << 54 and 1 << 52 <= A < 1 << 53 and got < count:
                    a[got], b[got] = float(A), float(B)
                    got += 1
    return a, b


@pytest.mark.parametrize("kind", ["ordinary", "wide", "ends", "midpoints", "special"])
def test_quotients_of_the_primitive_variables(kind):
    if not has_gpu():
        pytest.skip("no GPU")
    from mpcns_mercury_b200 import reference_constants
    from mpcns_mercury_b200 import setup as S
    from mpcns_mercury_b200.capi import Batch

    n, G = (32, 33, 31), 4
    cells = n[0] * n[1] * n[2]
    rng = np.random.default_rng(11)
    batch = Batch(1, 0)
    slot = batch.add_periodic(n, G, reference_constants())
    nodes, _ = S.cube_state(n)
    batch.setup_geometry(slot, nodes)
    want = {}
    for f, pv in (("U_H", "PV_H"), ("U_NA", "PV_NA")):
        if kind == "special":
            v = np.array([0.0, -0.0, 5e-324, -1e-310, 1.0, -3.0, 1e308, np.inf, -np.inf, np.nan])
            r = np.array([0.0, 1e-12, 1e-3, 1.0, 3.0, 1e30, 1e100, 1.0000001e100, 1e300, 1.7e308, np.inf, np.nan])
            a, b = rng.choice(v, (3, cells)), rng.choice(r, cells)
        elif kind == "midpoints":
            few = 3000
            q = rng.integers(0, few, cells)
            a0, b0 = _operands(kind, few, rng)
            a, b = np.stack([a0[q] * 2.0 ** e for e in (-60, 0, 40)]), b0[q]
        else:
            a0, b = _operands(kind, cells, rng)
            a = np.stack([a0, _operands(kind, cells, rng)[0], _operands(kind, cells, rng)[0]])
        u = np.stack([b, *a, np.ones(cells)], axis=-1).reshape(n + (5,))
        batch.upload(slot, f, u, (0, 0, 0), n)
        with np.errstate(all="ignore"):
            rho = np.where(b < 1e-12, 1e-12, b)
            want[pv] = np.stack([x / rho for x in a], axis=-1).reshape(n + (3,))
    batch.prepare(slot)
    for pv in want:
        got = batch.download(slot, pv, (0, 0, 0), n)[..., :3]
        same = (got.view(np.uint64) == want[pv].view(np.uint64)) | (np.isnan(got) & np.isnan(want[pv]))
        assert same.all(), (pv, int((~same).sum()), got[~same][:3], want[pv][~same][:3])
    batch.close()
