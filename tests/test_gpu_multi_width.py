"""Batches of 8, 16 and 32 load cases: a case's solution and iteration count are the same, bit for
bit, whatever batch it is solved in, and solve the system."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import solid
from wnfea_b200.mesh import generate_c3d10_ibeam_structured, generate_c3d10_kuhn_block, tip_load_cases
from wnfea_b200.model import solid_element_props, solid_fixed_dofs
from wnfea_b200.solid_solver import assemble_c3d10_sparse_3dof

pytestmark = pytest.mark.gpu


# the smallest mesh (one element row, a hierarchy that is its dense level), and one with levels
@pytest.mark.parametrize("mesh", ["bar", "ibeam"])
@pytest.mark.parametrize("precision,precond", [(0, 2), (1, 2), (0, 1)])
def test_width_does_not_change_a_case(mesh, precision, precond):
    if mesh == "bar":
        m, _ = generate_c3d10_kuhn_block(nx=2, ny=1, nz=1)
    else:
        m, _ = generate_c3d10_ibeam_structured(n_slices=9, length=4.0 * 9 / 315, seed=3)
    K, _, _ = assemble_c3d10_sparse_3dof(m)
    s = K.system
    F = tip_load_cases(m.mesh_nodes, n_cases=37, seed=5)
    fixed = np.asarray(solid_fixed_dofs(m), dtype=np.int64)
    F[fixed] = 0.0
    kw = dict(rtol=1e-8, max_iter=4000, precision=precision, precond=precond)
    if precond == 2:
        s.amg_setup()
    U, st = s.solve_multi(F, **kw)  # 32 + 8
    assert st["status"] == 0
    for k in (1, 8, 9, 16, 17):
        Uk, stk = s.solve_multi(F[:, :k], **kw)
        assert np.array_equal(Uk, U[:, :k])
        assert np.array_equal(stk["case_iterations"], st["case_iterations"][:k])
    assert np.array_equal(s.solve_multi(F[:, 32:], **kw)[0], U[:, 32:])
    Ko, _, _ = solid.assemble(m.mesh_nodes, m.solid_elements, solid_element_props(m), F[:, 0], fixed)
    # the rounded solution's own residual: rtol plus the rounding level of K u
    eps = np.finfo(float).eps
    level = 100 * eps * np.linalg.norm(abs(Ko) @ np.abs(U), axis=0)
    assert (np.linalg.norm(Ko @ U - F, axis=0) <= 1e-8 * np.linalg.norm(F, axis=0) + level).all()
