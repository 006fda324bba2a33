"""The stored FP64 Fock build (fixed-point products of the slabs) against J and K
from the same integrals by torch in FP64, RHF and UHF: one unit per slab and
fewer rows than a fragment (n = 7), odd orders (35), more than one chunk of 128
columns (133), tiles of 1, 2 and 4 slabs, and densities with a non-finite column.

Tolerance: K's element is a sum of n slab sums, each rounded once, torch's one of
n^2 products: 133 roundings of 1.1e-16 and, for torch, sqrt(133^2) of them,
relative to sums of magnitudes a few times the largest element: 1e-12 of it."""
import numpy as np
import pytest

from myqc_gb300 import MODE_TIGHT, formats, molecules

pytestmark = pytest.mark.gpu


def _jk(torch, XX, D):
    n = D.shape[0]
    J = (XX.reshape(n * n, n * n) @ D.reshape(-1)).reshape(n, n)
    K = torch.stack([torch.einsum("jkl,jl->k", XX[i], D) for i in range(n)])
    return J, K


@pytest.mark.parametrize("waters,jc", [(1, "1"), (2, "4"), (5, "2"), (5, "4"), (19, "2")])
def test_stored_build_matches_torch(ctx, basis_text, monkeypatch, waters, jc):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("MYQC_FOCK_JC", jc)
    sysm = molecules.water_cluster_system(waters, 1.0 + (27.0 * waters) ** (1 / 3), 4)
    ctx.set_schwarz(0.0)
    ctx.set_system(sysm, formats.parse_mybasis_text(basis_text, sysm.atoms), None, MODE_TIGHT)
    XX = torch.from_numpy(ctx.eri_full()).cuda()
    n = ctx.n
    rng = np.random.default_rng(waters)
    Da, Db = (d + d.T for d in rng.standard_normal((2, n, n)))
    ta, tb = torch.from_numpy(Da).cuda(), torch.from_numpy(Db).cuda()
    (Ja, Ka), (Jb, Kb) = _jk(torch, XX, ta), _jk(torch, XX, tb)
    ref = [(Ja + Jb - Ka).cpu().numpy(), (Ja + Jb - Kb).cpu().numpy(), (Ja - 0.5 * Ka).cpu().numpy()]
    out = [*ctx.fock(Da, Db), ctx.fock(Da)]
    for g, r in zip(out, ref):
        assert np.abs(g - r).max() < 1e-12 * np.abs(r).max(), (n, jc)
    bad = Da.copy()
    bad[0, 0] = np.inf
    assert not np.isfinite(ctx.fock(bad)).all()
