"""The split transform's steps behind the quartet store (rows of non-contiguous
elements cut through shared-memory tiles) against the FP64 transform of the n^4
array: fewer rows than a tile, orders that leave remainders in both directions,
and rows of more than 256 elements; both numbers of planes.

Tolerance: each of four steps rounds its operands once to 2^-24 (2^-16) of the
row's largest element, which is up to about 30 times the row's mean size; the
signs are random: 4 * 30 * 2^-24 / 2 = 4e-6 of the largest (ia|jb), times 5 for
the largest of many; 256 times that with two planes."""
import numpy as np
import pytest

from myqc_gb300 import MODE_TIGHT, PREC_FP64, PREC_SPLIT_BF16, PREC_SPLIT_BF16X3, formats, molecules
from myqc_gb300._lib import STORE_FULL, STORE_QUARTETS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waters,dims", [(1, (5, 2, 5, 2)), (5, (7, 17, 5, 33)), (19, (2, 31, 3, 64)), (37, (3, 5, 2, 3))])
def test_store_transform_tiles(ctx, basis_text, waters, dims):
    sysm = molecules.water_cluster_system(waters, 1.0 + (27.0 * waters) ** (1 / 3), 6)
    basis = formats.parse_mybasis_text(basis_text, sysm.atoms)
    rng = np.random.default_rng(waters)
    C = [0.3 * rng.standard_normal((7 * waters, k)) for k in dims]
    ctx.set_schwarz(1e-14)
    try:
        ctx.set_system(sysm, basis, None, MODE_TIGHT)
        ctx.eri_store()
        ref = ctx.ao2mo_iajb(*C, PREC_FP64)
        ctx.set_eri_storage(STORE_QUARTETS)
        ctx.set_system(sysm, basis, None, MODE_TIGHT)
        ctx.eri_store()
        for prec, tol in ((PREC_SPLIT_BF16X3, 2e-5), (PREC_SPLIT_BF16, 5e-3)):
            got = ctx.ao2mo_iajb(*C, prec)
            assert np.abs(got - ref).max() < tol * np.abs(ref).max(), (waters, prec)
    finally:
        ctx.set_eri_storage(STORE_FULL)
        ctx.set_schwarz(0.0)
