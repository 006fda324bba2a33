"""Matrices with infinities and NaN.

Two helium atoms with contraction coefficients of 1e100 have a finite overlap and core
Hamiltonian (1e200) and infinite two-electron integrals (1e400), so that the Fock
matrix and the eigenvalues of every iteration are not numbers."""
import numpy as np
import pytest

from myqc_gb300 import MODE_TIGHT, formats, molecules
from myqc_gb300._lib import MyQCError

pytestmark = pytest.mark.gpu


def _overflowing(basis_text):
    sysm = formats.system_from_geometry(["He", "He"], np.array([[0.0, 0, 0], [0, 0, 3.0]]))
    basis = formats.parse_mybasis_text(basis_text, sysm.atoms)
    basis.bas = basis.bas * 1e100
    return sysm, basis


@pytest.mark.parametrize("graph", [False, True])
def test_batch_neighbours_of_a_non_finite_molecule(ctx, basis_text, graph):
    """A molecule whose Fock matrix overflows (two occupied levels, ranked among
    eigenvalues that are NaN) leaves the others of its batch as they are.  Energies
    of two runs to 1e-10 rms in the density: 1e-9."""
    waters = [molecules.water_cluster_system(k, 2.0 + (27.0 * k) ** (1 / 3), k) for k in (1, 2)]
    E = []
    for extra in ([], [_overflowing(basis_text)]):
        ctx.batch_clear()
        for sysm, basis in extra:
            ctx.batch_add(sysm, basis)
        for sysm in waters:
            ctx.batch_add(sysm, formats.parse_mybasis_text(basis_text, sysm.atoms))
        out = ctx.batch_scf(conv=1e-10, conv_rms=True, diis=8, max_iter=40, graph=graph)
        assert all(out["converged"][len(extra):])
        E.append(out["energy"][len(extra):])
    ctx.batch_clear()
    assert np.abs(np.asarray(E[0]) - np.asarray(E[1])).max() < 1e-9


@pytest.mark.parametrize("conv_rms", [False, True])
@pytest.mark.parametrize("diis", [0, 6])
def test_batch_reports_a_non_finite_molecule(ctx, basis_text, diis, conv_rms):
    """Its density is not a number and it does not leave as converged."""
    ctx.batch_clear()
    for sysm, basis in [_overflowing(basis_text)] * 2:
        ctx.batch_add(sysm, basis)
    out = ctx.batch_scf(conv=1e-8, conv_rms=conv_rms, diis=diis, max_iter=12)
    ctx.batch_clear()
    assert not any(out["converged"]) and list(out["iterations"]) == [12, 12]
    assert not np.isfinite(out["energy"]).any()
    assert all(np.isnan(D).all() for D in out["D"])


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("waters,uhf", [(1, False), (2, False), (1, True), (9, False), (10, False)])
def test_scf_with_a_non_finite_density(ctx, basis_text, waters, uhf, value):
    """One density element that is no number makes the Fock matrix none, at the orders
    of the fused steps (up to 64), of the one-CTA eigensolver and with two spins."""
    sysm = molecules.water_cluster_system(waters, 1.0 + (27.0 * waters) ** (1 / 3), 5)
    ctx.set_schwarz(0.0)
    ctx.set_system(sysm, formats.parse_mybasis_text(basis_text, sysm.atoms), None, MODE_TIGHT)
    S, H = ctx.int1e()
    ctx.eri_store()
    D = np.zeros((2, ctx.n, ctx.n) if uhf else (ctx.n, ctx.n))
    D[..., 1, 1] = value
    with pytest.raises(MyQCError, match="eigensolver did not converge"):
        ctx.scf(S, H, sysm.nelcA, sysm.nelcB, uhf=uhf, conv=1e-8, max_iter=20, D_guess=D)
