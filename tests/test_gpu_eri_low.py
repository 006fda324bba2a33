"""The early-contracted integral kernels against the oracle, every integral of
the n^4 array, in both Boys modes: molecules whose exponent sums are tabulated
(at most 512 distinct ones) and one of nine elements whose 50 exponents give
more, so that alpha and the prefactor are formed per primitive quartet; compact
and stretched geometries, so that T crosses the Boys ranges (below and above 36)
and centres coincide, lie on one axis, or lie far apart.

Tolerance: at most 81 primitive quartets of magnitude below 10, each rounded a
few times, with vectors of up to 15 bohr squared in the coefficients: 81 * 10 *
15^2 * 1e-16 / 10 (their mean size) = 2e-12; the screen leaves out terms below
1e-14 in number at most 81."""
import numpy as np
import oracle as O
import pytest

from myqc_gb300 import formats

pytestmark = pytest.mark.gpu

CASES = {
    "one centre": (["O"], [[0.3, -0.2, 0.1]]),
    "axis": (["C", "O", "H"], [[0, 0, 0], [0, 0, 1.1], [0, 0, -1.0]]),
    "water far": (["O", "H", "H", "O", "H", "H"],
                  [[0, 0, 0], [0.76, 0.59, 0], [-0.76, 0.59, 0], [0.4, 5.1, 3.3], [1.2, 5.6, 3.1], [0.0, 5.2, 4.2]]),
    "many exponents": (["H", "He", "Be", "B", "C", "N", "O", "F", "Ne"],
                       [[0, 0, 0], [1.1, 0.2, 0], [0.3, 1.4, 0.5], [2.1, 1.2, -0.4], [1.0, -1.3, 0.6],
                        [-1.2, 0.4, 1.0], [0.2, 0.3, 2.2], [-0.9, -1.1, -0.8], [1.6, 0.1, 1.7]]),
}


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("name", list(CASES))
def test_integrals_of_every_class(ctx, basis_text, ftab, name, mode):
    sym, xyz = CASES[name]
    sysm = formats.system_from_geometry(sym, np.array(xyz, dtype=float))
    basis = formats.parse_mybasis_text(basis_text, sysm.atoms)
    ctx.set_schwarz(0.0)
    ctx.set_system(sysm, basis, ftab, mode)
    XX = ctx.eri_full()
    lines = ["CARTESIAN"] + [f"{s} {x[0]!r} {x[1]!r} {x[2]!r}" for s, x in zip(sym, np.array(xyz, float).tolist())]
    mol = O.parse_zmat_text("\n".join(lines + ["END", "", "CALC= SCF", "BASIS= STO-3G", "CHARGE= 0", "MULTI= 1",
                                               "REF= RHF"]) + "\n")
    ref = O.int2e(mol, O.parse_mybasis_text(basis_text, mol.atoms), ftab, mode)
    assert np.abs(XX - ref.reshape(XX.shape, order="F")).max() < 2e-12
