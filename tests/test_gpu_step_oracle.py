"""The step's kernels against the C restatement of the reference step on
periodic cubes whose sizes reach both sides of the kernels' splits: work that
leaves the GPU idle (the fluid kernel's single-cell columns) and work that fills
it, extents below, at and off the tiles' multiples."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

# derived and work fields of the last step, beside the state
FIELDS = {"U_H": "U_H", "U_Na": "U_NA", "B_xi": "B_XI", "B_eta": "B_ETA", "B_zeta": "B_ZETA", "PV_H": "PV_H",
          "PV_Na": "PV_NA", "U_plus": "U_PLUS", "B_cell": "B_CELL", "J_cell": "J_CELL", "J_xi": "J_XI",
          "J_eta": "J_ETA", "J_zeta": "J_ZETA", "E_xi": "E_XI", "E_eta": "E_ETA", "E_zeta": "E_ZETA",
          "Ehall_xi": "EHALL_XI", "Ehall_eta": "EHALL_ETA", "Ehall_zeta": "EHALL_ZETA"}


@pytest.mark.parametrize("n", [3, 7, 16, 33, 61])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_step_matches_the_restatement(n, precision):
    if not has_gpu():
        pytest.skip("no GPU")
    import restatement
    from mpcns_mercury_b200 import Context, reference_constants
    from mpcns_mercury_b200 import setup as S
    from mpcns_mercury_b200.workloads import UPLOAD_FIELDS, capi_field

    steps = 2
    _, f = S.cube_case(n)
    ctx = Context([(n, n, n)], 4, reference_constants(cfl=0.4), precision=precision)
    for name in UPLOAD_FIELDS:
        a = f[name]
        ctx.upload(capi_field(name), a.data, a.lo, a.hi)
    ctx.sync("UCELL")
    ctx.sync("BFACE")
    ctx.prepare()
    ctx.step(steps)
    r = restatement.Restatement(n, restatement.inputs_from_fields(n, {k: (v.lo, v.hi, v.data.copy())
                                                                      for k, v in f.items()}))
    restatement.sync_state(r)
    r.update_derived()
    for _ in range(steps):
        r.step()
    # FP64: the same operations in the same order.  Mixed: state and fields in FP32 (eps 6e-8); J and E
    # are differences of neighbouring values, which loses up to the grid's 2 pi / n of a digit more
    for ref, cap in FIELDS.items():
        lo, hi, data = r.arrays[ref]
        g = [-v for v in lo]
        own = tuple(slice(g[a], hi[a]) for a in range(3))
        dev = ctx.download(cap, lo, hi)[own]
        want = data[own]
        tol = 1e-12 if precision == 0 else (2e-6 if ref[0] in "UPB" else 2e-4)
        err = np.linalg.norm((dev - want).ravel()) / np.linalg.norm(want.ravel())
        assert err <= tol, (ref, err)
    ctx.close()
