"""The paths that small systems take against the ones that larger systems take.

Integrals: the class combinations launched side by side (up to 2^18 quartets: 9
waters) give what the launches in a row give for the same shells inside a system above
the line (10 waters).  A sum of at most 81 terms below 5, each rounded: 1e-13.

SCF: one launch around each Fock build (orders up to 64, no purification) and
the general steps (with purification, and above 64) reach the same energy and
density.  Converged to 1e-10 rms in the density: energies to second order in it,
densities within what DIIS leaves, some hundred times that: 1e-9 and 1e-7.

Pair tables: pairs without a surviving primitive pair (two atoms 40 A apart), in a
single system and in a batch next to other sizes: twice the energy of one, 1e-10."""
import numpy as np
import pytest

from myqc_gb300 import MODE_TIGHT, formats, molecules

pytestmark = pytest.mark.gpu


def _load(ctx, basis_text, sysm):
    ctx.set_system(sysm, formats.parse_mybasis_text(basis_text, sysm.atoms), None, MODE_TIGHT)


def test_forked_integrals(ctx, basis_text):
    sym, xyz = molecules.water_cluster(10, 7.5, 3)
    ctx.set_schwarz(0.0)
    XX = []
    for k in (10, 9):
        _load(ctx, basis_text, formats.system_from_geometry(sym[: 3 * k], xyz[: 3 * k]))
        XX.append(ctx.eri_full())
    n = ctx.n
    assert np.abs(XX[0][:n, :n, :n, :n] - XX[1]).max() < 1e-13


@pytest.mark.parametrize("waters", [1, 2, 9, 10])
def test_small_scf_equals_general(ctx, basis_text, waters):
    sysm = molecules.water_cluster_system(waters, 1.0 + (27.0 * waters) ** (1 / 3), 5)
    ctx.set_schwarz(0.0)
    _load(ctx, basis_text, sysm)
    S, H = ctx.int1e()
    ctx.eri_store()
    small, general = (ctx.scf(S, H, sysm.nelcA, sysm.nelcB, conv=1e-10, conv_rms=True, diis=8, max_iter=100, purify=p)
                      for p in (False, True))
    assert abs(small.energy - general.energy) < 1e-9
    assert np.abs(np.asarray(small.D) - np.asarray(general.D)).max() < 1e-7


def test_pairs_without_primitives(ctx, basis_text):
    ctx.set_schwarz(0.0)
    one = formats.system_from_geometry(["He"], np.zeros((1, 3)))
    two = formats.system_from_geometry(["He", "He"], np.array([[0.0, 0, 0], [0, 0, 40.0]]))
    E = []
    for sysm in (one, two):
        _load(ctx, basis_text, sysm)
        S, H = ctx.int1e()
        ctx.eri_store()
        E.append(ctx.scf(S, H, sysm.nelcA, sysm.nelcB, conv=1e-10).energy)
    assert abs(E[1] - 2 * E[0]) < 1e-10
    ctx.batch_clear()
    water = molecules.water_cluster_system(2, 5.0, 1)
    for sysm in (two, water, one):
        ctx.batch_add(sysm, formats.parse_mybasis_text(basis_text, sysm.atoms))
    out = ctx.batch_scf(conv=1e-10, diis=8, max_iter=100)
    ctx.batch_clear()
    assert abs(out["energy"][0] - 2 * out["energy"][2]) < 1e-10 and abs(out["energy"][2] - E[0]) < 1e-10
