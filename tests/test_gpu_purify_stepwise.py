"""The stepwise purification (one product and one update launch per step), which
orders above 640 take, against the eigensolver: an SCF's energy and density, at an
even order and an odd one.

Both converge the density to 1e-9 rms: energies to second order in it and the
rounding of sums of 1e5 terms of up to 1e4, 1e-8; densities within what DIIS leaves,
some hundred times the threshold, 1e-6."""
import numpy as np
import pytest

from myqc_gb300 import MODE_TIGHT, STORE_FULL, STORE_QUARTETS, formats, molecules

pytestmark = pytest.mark.gpu


@pytest.fixture
def qctx(ctx):
    ctx.set_eri_storage(STORE_QUARTETS)
    ctx.set_schwarz(1e-12)
    yield ctx
    ctx.set_eri_storage(STORE_FULL)
    ctx.set_schwarz(0.0)


@pytest.mark.parametrize("waters", [92, 93])
def test_stepwise_purification(qctx, basis_text, waters):
    sysm = molecules.water_cluster_system(waters, (27.0 * waters) ** (1 / 3), 5)
    qctx.set_system(sysm, formats.parse_mybasis_text(basis_text, sysm.atoms), None, MODE_TIGHT)
    assert qctx.n > 640
    S, H = qctx.int1e()
    qctx.eri_store()
    res = []
    for purify in (True, False):
        res.append(qctx.scf(S, H, sysm.nelcA, sysm.nelcB, conv=1e-9, conv_rms=True, diis=8, max_iter=100, purify=purify))
        assert (qctx.stat("purify_stepwise") > 0) == purify and qctx.stat("purify_persistent") == 0
    assert abs(res[0].energy - res[1].energy) < 1e-8
    assert np.abs(np.asarray(res[0].D) - np.asarray(res[1].D)).max() < 1e-6
