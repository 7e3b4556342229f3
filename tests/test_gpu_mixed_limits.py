"""The mixed-precision limiter at densities whose reciprocals leave the range of a
float: the ions' shares of the charge are at most 1."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rho_h,rho_na", [(1e-39, 1e-39), (1e-45, 0.0), (0.0, 2e-42), (0.0, 0.0), (1.3e-38, 1e-40)])
def test_charge_shares_at_tiny_densities(rho_h, rho_na):
    if not has_gpu():
        pytest.skip("no GPU")
    from mpcns_mercury_b200 import reference_constants
    from mpcns_mercury_b200 import setup as S
    from mpcns_mercury_b200.capi import Batch

    n, G = (4, 5, 4), 4
    batch = Batch(1, 1)
    slot = batch.add_periodic(n, G, reference_constants(cfl=0.4))
    nodes, state = S.cube_state(n, solve_id=3)
    batch.setup_geometry(slot, nodes)
    for name, f in (("U_H", "U_H"), ("U_Na", "U_NA"), ("B_xi", "B_XI"), ("B_eta", "B_ETA"), ("B_zeta", "B_ZETA")):
        a = state[name]
        data = a.data.copy()
        if f in ("U_H", "U_NA"):
            data[..., 0] = rho_h if f == "U_H" else rho_na
        batch.upload(slot, f, data, a.lo, a.hi)
    batch.sync(slot, "UCELL")
    batch.sync(slot, "BFACE")
    batch.prepare(slot)
    # velocities of densities up to 1e-20 count as 0, so the shares multiply zeros
    up = batch.download(slot, "U_PLUS", (0, 0, 0), n)
    assert np.array_equal(up, np.zeros_like(up))
    batch.close()
