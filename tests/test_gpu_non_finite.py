"""Matrices with infinities and NaN.

Two helium atoms with contraction coefficients of 1e100 have a finite overlap and core
Hamiltonian (1e200) and infinite two-electron integrals (1e400), so that the Fock
matrix and the eigenvalues of every iteration are not numbers."""
import numpy as np
import pytest

from myqc_gb300 import formats, molecules

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
