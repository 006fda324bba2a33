"""(sp sp|sp sp) integrals, whose launches give a quartet 32, 16, ... 1 lanes as the
system grows: the integrals over the functions of a cluster's first two waters do not
depend on how many more there are.  Read through the FP64 transform with unit vectors
(products with 0 and 1: exact).

Tolerance: a sum of at most 81 terms below 5, in another order: 81 * 5 * 1.1e-16 = 5e-14."""
import numpy as np
import pytest

from myqc_gb300 import MODE_TIGHT, PREC_FP64, formats, molecules

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waters", [3, 8, 10, 13, 16, 18, 20])
def test_lanes_per_quartet(ctx, basis_text, waters):
    sym, xyz = molecules.water_cluster(20, 9.0, 3)
    ctx.set_schwarz(0.0)
    out = []
    for k in (2, waters):
        sysm = formats.system_from_geometry(sym[: 3 * k], xyz[: 3 * k])
        ctx.set_system(sysm, formats.parse_mybasis_text(basis_text, sysm.atoms), None, MODE_TIGHT)
        ctx.eri_store()
        C = np.eye(ctx.n)[:, :14]
        out.append(ctx.ao2mo_iajb(C, C, C, C, PREC_FP64))
    assert np.abs(out[0]).max() > 1.0
    assert np.abs(out[1] - out[0]).max() < 5e-14
