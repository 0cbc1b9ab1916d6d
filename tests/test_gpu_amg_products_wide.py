"""The setup's block products where a row of the product has more than 256 blocks: in two runs of 256 columns
(1,184 rows and more) and in runs of 64 by four CTAs (fewer), against scipy's R A P.  Bound: that of the
setup's other tests, 1e-12 of the operator's largest entry."""

from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

from wnfea_b200.amg import AMGParams, export_system_hierarchy
from wnfea_b200.mesh import generate_c3d10_kuhn_block
from wnfea_b200.solid_solver import assemble_c3d10_sparse_3dof

pytestmark = pytest.mark.gpu


# theta 0.16: 3,265 coarse rows of up to 274 blocks; 0.1: 379 rows of up to 377 on the level after
@pytest.mark.parametrize("theta,rows", [(0.16, (1184, 10**9)), (0.1, (1, 1183))])
def test_product_rows_of_more_than_256_blocks(theta, rows):
    m, _ = generate_c3d10_kuhn_block(16 / 16, 15 / 16, 14 / 16, 16, 15, 14)
    K, _, _ = assemble_c3d10_sparse_3dof(m)
    K.system.amg_setup(AMGParams(coarse_size=60, strength_theta=theta))
    H = export_system_hierarchy(K.system)
    A = K.to_bsr().tocsr()
    covered = False
    for i, lvl in enumerate(H.levels):
        P, R = sp.csr_matrix(lvl.P), sp.csr_matrix(lvl.R)
        nxt = sp.bsr_matrix(H.levels[i + 1].A if i + 1 < len(H.levels) else H.coarse_A, blocksize=(6, 6))
        length = np.diff(nxt.indptr)
        covered |= rows[0] <= len(length) <= rows[1] and length.max() > 256
        B = sp.csr_matrix(nxt)
        Ac = (R @ (A @ P)).tocsr()
        assert abs(0.5 * (Ac + Ac.T) - B).max() <= 1e-12 * abs(B).max()
        A = B
    assert covered
