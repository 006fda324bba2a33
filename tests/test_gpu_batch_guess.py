"""A guess density with an antisymmetric part: the Coulomb and exchange matrices and the
energy depend on its symmetric part alone.  One iteration's energies, sums of some 1e3
terms of at most 1e2 in two orders: 1e-10."""
import numpy as np
import pytest

from myqc_gb300 import formats, molecules

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
def test_antisymmetric_part_of_a_guess(ctx, basis_text, graph):
    systems = [molecules.water_cluster_system(k, 2.0 + (27.0 * k) ** (1 / 3), k) for k in (1, 2, 9)]
    rng = np.random.default_rng(3)

    def solve(guess, iters):
        ctx.batch_clear()
        for sysm in systems:
            ctx.batch_add(sysm, formats.parse_mybasis_text(basis_text, sysm.atoms))
        return ctx.batch_scf(conv=1e-10, diis=8, max_iter=iters, graph=graph, D_guess=guess)

    D = [np.asarray(d) for d in solve(None, 100)["D"]]
    E = []
    for size in (0.0, 0.02):
        A = [rng.uniform(-size, size, d.shape) for d in D]
        E.append(solve([d + (a - a.T) for d, a in zip(D, A)], 1)["energy"])
        assert ctx.stat("guesses_taken") == len(systems)
    ctx.batch_clear()
    assert np.abs(np.asarray(E[0]) - np.asarray(E[1])).max() < 1e-10
