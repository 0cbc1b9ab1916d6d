"""The setup's block products at the edges of their runs (32 blocks of A's row, 64 columns of C per
CTA where rows are few): every Galerkin operator of a small and of a compact block, whose coarse rows
have up to 140 blocks, against scipy's R A P.  Bound: a coarse entry is a sum of at most a few
thousand products of the three factors, 1e-12 of the operator's largest entry (that of the setup's
other tests)."""

from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

from wnfea_b200.amg import AMGParams, export_system_hierarchy
from wnfea_b200.mesh import generate_c3d10_kuhn_block
from wnfea_b200.solid_solver import assemble_c3d10_sparse_3dof

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,longest", [((5, 4, 3), 16), ((16, 15, 14), 64)])
def test_galerkin_operators_match_scipy(cells, longest):
    m, _ = generate_c3d10_kuhn_block(1.0, 0.9, 0.8, *cells)
    K, _, _ = assemble_c3d10_sparse_3dof(m)
    K.system.amg_setup(AMGParams(coarse_size=60))
    H = export_system_hierarchy(K.system)
    A = K.to_bsr().tocsr()
    most = 0
    for i, lvl in enumerate(H.levels):
        P, R = sp.csr_matrix(lvl.P), sp.csr_matrix(lvl.R)
        nxt = H.levels[i + 1].A if i + 1 < len(H.levels) else H.coarse_A
        Ac = (R @ (A @ P)).tocsr()
        nxt = sp.bsr_matrix(nxt, blocksize=(6, 6))
        most = max(most, int(np.diff(nxt.indptr).max()))
        B = sp.csr_matrix(nxt)
        assert abs(0.5 * (Ac + Ac.T) - B).max() <= 1e-12 * abs(B).max()
        A = B
    assert most > longest
