"""Batch widths on a mesh whose rows take several passes of every row kernel's grid (32 rows per pass and CTA,
444 CTAs at most): a case has the same bits whatever batch it is solved in."""

from __future__ import annotations

import numpy as np
import pytest

from wnfea_b200.mesh import generate_c3d10_ibeam_structured, tip_load_cases
from wnfea_b200.model import solid_fixed_dofs
from wnfea_b200.solid_solver import assemble_c3d10_sparse_3dof

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_width_does_not_change_a_case_over_several_passes(precision):
    m, _ = generate_c3d10_ibeam_structured(n_slices=30, length=4.0 * 30 / 315, seed=6)
    assert len(m.mesh_nodes) > 2 * 32 * 444
    K, _, _ = assemble_c3d10_sparse_3dof(m)
    s = K.system
    s.amg_setup()
    F = tip_load_cases(m.mesh_nodes, n_cases=20, seed=9)
    F[np.asarray(solid_fixed_dofs(m), dtype=np.int64)] = 0.0
    kw = dict(rtol=1e-8, precision=precision)
    U, st = s.solve_multi(F, **kw)  # 32 wide
    assert st["status"] == 0
    for k in (12, 5):  # 16 and 8 wide
        Uk, stk = s.solve_multi(F[:, :k], **kw)
        assert np.array_equal(Uk, U[:, :k])
        assert np.array_equal(stk["case_iterations"], st["case_iterations"][:k])
