"""Small systems (one cluster kernel per solve): every preconditioner against a direct solution, around the
sizes where the paths change, and the ends of a solve that are not convergence."""

from __future__ import annotations

import numpy as np
import pytest
from scipy.sparse.linalg import splu

from oracle import solid
from wnfea_b200.mesh import generate_c3d10_kuhn_block
from wnfea_b200.model import solid_element_props, solid_fixed_dofs
from wnfea_b200.solid_solver import assemble_c3d10_sparse_3dof

pytestmark = pytest.mark.gpu


def _system(nx, ny, nz, seed):
    m, _ = generate_c3d10_kuhn_block(0.05 * nx, 0.05 * ny, 0.05 * nz, nx, ny, nz)
    K, _, _ = assemble_c3d10_sparse_3dof(m)
    rng = np.random.default_rng(seed)
    F = rng.standard_normal(K.shape[0]) * 100.0
    fixed = np.asarray(solid_fixed_dofs(m), dtype=np.int64)
    F[fixed] = 0.0
    Ko, _, _ = solid.assemble(m.mesh_nodes, m.solid_elements, solid_element_props(m), F, fixed)
    return K.system, F, Ko


# 27 nodes (fewer than the lanes of a CTA, CTAs without rows), 125, 585 (two levels), 1,025 and 1,105 (the
# matrix in shared memory, and not), 2,023 and 2,125 (the last size of the cluster, and the launched kernels)
@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (2, 2, 2), (6, 4, 2), (20, 2, 2), (8, 6, 2), (8, 8, 3), (8, 12, 2)])
@pytest.mark.parametrize("precond", [0, 1, 2, 3])
@pytest.mark.parametrize("precision", [0, 1])
def test_solution_matches_direct(nx, ny, nz, precond, precision):
    s, F, Ko = _system(nx, ny, nz, nx + precond)
    if precond == 2:
        s.amg_setup()
    rtol = 1e-10
    u, st = s.solve(F, rtol=rtol, max_iter=20000, precond=precond, precision=precision)
    assert st["status"] == 0 and st["rel_res"] <= rtol and st["iterations"] > 0
    assert st["algorithmic_bytes"] > 0
    ref = splu(Ko.tocsc()).solve(F)
    # a residual of rtol ||F|| moves u by at most rtol ||K^-1|| ||F||; for these loads ||K^-1|| ||F|| stays
    # below 1e3 ||u|| (a bending bar), and the direct solution carries its own rounding
    assert np.linalg.norm(u - ref) <= 1e-7 * np.linalg.norm(ref)
    u2, st2 = s.solve(F, rtol=rtol, max_iter=20000, precond=precond, precision=precision)
    assert np.array_equal(u, u2) and st2["iterations"] == st["iterations"]


@pytest.mark.parametrize("precond", [1, 2])
def test_ends_other_than_convergence(precond):
    s, F, Ko = _system(20, 2, 2, 3)
    s.amg_setup()
    u, st = s.solve(F, rtol=1e-12, max_iter=3, precond=precond)
    assert st["status"] == -5 and st["iterations"] == 3
    u, st = s.solve(np.zeros_like(F), precond=precond)
    assert st["status"] == 0 and st["iterations"] == 0 and not u.any()
    Fn = F.copy()
    Fn[40] = np.nan
    u, st = s.solve(Fn, precond=precond)
    assert st["status"] == -4
    # the handle still solves
    u, st = s.solve(F, rtol=1e-9, max_iter=5000, precond=precond)
    assert st["status"] == 0 and np.linalg.norm(F - Ko @ u) <= 2e-9 * np.linalg.norm(F)
