"""Small systems without AMG: the one-kernel solve adds its dot products in the order of the launched kernels
(which a profiled solve runs), so that iterates, counts and residuals are theirs bit for bit, also where
the solve stops at its iteration limit, and no solve runs twice."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from wnfea_b200.amg import AMGParams
from wnfea_b200.mesh import generate_c3d10_kuhn_block, tip_load_cases
from wnfea_b200.model import solid_fixed_dofs
from wnfea_b200.solid_solver import assemble_c3d10_sparse_3dof

pytestmark = pytest.mark.gpu


def _system(nx, ny, nz, seed):
    m, _ = generate_c3d10_kuhn_block(0.05 * nx, 0.05 * ny, 0.05 * nz, nx, ny, nz)
    K, _, _ = assemble_c3d10_sparse_3dof(m)
    F = tip_load_cases(m.mesh_nodes, 1, seed=seed)[:, 0]
    F[np.asarray(solid_fixed_dofs(m), dtype=np.int64)] = 0.0
    return K.system, np.ascontiguousarray(F)


def _same(s, F, **kw):
    u, st = s.solve(F, **kw)
    v, sv = s.solve(F, profile=True, **kw)
    assert np.array_equal(u, v)
    assert st["iterations"] == sv["iterations"] and st["status"] == sv["status"]
    assert st["rel_res"] == sv["rel_res"]
    return st


# 27 nodes (CTAs without rows), 99, 585, 603 (slender: two outer passes), 1,025 and 1,105 (the matrix in shared
# memory), 1,815 and 2,023 (in L2)
@pytest.mark.parametrize("cells", [(1, 1, 1), (5, 1, 1), (6, 4, 2), (25, 1, 1), (20, 2, 2), (8, 6, 2), (7, 5, 5),
                                   (8, 8, 3)])
@pytest.mark.parametrize("precond", [0, 1, 3])
def test_same_bits_as_the_launched_kernels(cells, precond):
    s, F = _system(*cells, seed=sum(cells))
    st = _same(s, F, rtol=1e-6, max_iter=2000, precond=precond)
    if precond:
        assert st["status"] == 0


# bars that the default 2,000 iterations do not bring to 1e-6, and a limit of a few iterations
@pytest.mark.parametrize("cells,limit", [((37, 1, 1), 2000), ((34, 2, 1), 2000), ((20, 2, 2), 3)])
@pytest.mark.parametrize("precond", [0, 1])
def test_iteration_limit_returns_the_iterate_once(cells, limit, precond):
    s, F = _system(*cells, seed=7)
    st = _same(s, F, rtol=1e-6, max_iter=limit, precond=precond)
    assert st["status"] == -5 and st["iterations"] == limit
    assert st["kernel_launches"] < 20
    st = s.solve(F, rtol=1e-6, max_iter=limit, precond=precond, precision=1)[1]
    assert st["status"] == -5 and st["iterations"] == limit and st["kernel_launches"] < 20


# a launch runs 2,048 iterations at most (128 with AMG), whatever the caller's limit, and the next goes on
# with the same bits
@pytest.mark.parametrize("cells", [(37, 1, 1), (34, 2, 1)])
@pytest.mark.parametrize("precond", [0, 1, 3])
def test_long_solves_take_several_launches(cells, precond):
    s, F = _system(*cells, seed=11)
    kw = dict(rtol=1e-30, precond=precond, max_outer=1)
    launches = [s.solve(F, max_iter=n, **kw)[1]["kernel_launches"] for n in (2048, 2049)]
    assert launches[1] == launches[0] + 1
    st = _same(s, F, max_iter=5000, **kw)
    # (a Jacobi solve's recurrence may reach 1e-30 within one launch more)
    assert st["iterations"] > 2048 and st["kernel_launches"] >= launches[1]


# (sizes whose matrix copies fit shared memory)
@pytest.mark.parametrize("cells,precision", [((20, 2, 2), 0), ((12, 2, 2), 1)])
def test_long_amg_solve_takes_several_launches(cells, precision):
    s, F = _system(*cells, seed=13)
    s.amg_setup(AMGParams(cheb_safety=1e6))  # hardly any smoothing: some hundred iterations
    u, st = s.solve(F, rtol=1e-13, precond=2, precision=precision, max_outer=1)
    v, sv = s.solve(F, rtol=1e-13, precond=2, precision=precision, max_outer=1, profile=True)
    few = s.solve(F, rtol=1e-2, precond=2, precision=precision, max_outer=1)[1]
    assert st["iterations"] > 128 >= few["iterations"]
    assert st["kernel_launches"] == few["kernel_launches"] + (st["iterations"] - 1) // 128
    # the launched kernels' sums run in another order; a lost direction would cost a start from scratch
    assert abs(st["iterations"] - sv["iterations"]) <= 0.05 * sv["iterations"]
    assert np.linalg.norm(u - v) <= 1e-9 * np.linalg.norm(v)


# tetrahedra apart from one another, clamped on a face: rows of 10 blocks, so that a row tile has 51 rows and a warp's
# share of it two passes
@pytest.mark.parametrize("precond", [0, 1, 3])
def test_tiles_of_many_short_rows(precond):
    m, _ = generate_c3d10_kuhn_block(1.0, 1.0, 1.0, 1, 1, 1)
    tet = m.mesh_nodes[m.solid_elements[0]]
    rng = np.random.default_rng(5)
    n_tets = 57
    scale = rng.uniform(0.2, 3.0, (n_tets, 1, 1))
    nodes = (scale * tet + 4.0 * np.arange(n_tets)[:, None, None]).reshape(-1, 3)
    face = [0, 1, 2, 4, 5, 6]  # vertices 0, 1, 2 and the nodes amid their edges
    supports = [dataclasses.replace(m.supports[0], node_id=10 * t + a) for t in range(n_tets) for a in face]
    m = dataclasses.replace(m, mesh_nodes=nodes, solid_elements=np.arange(10 * n_tets, dtype=np.int32).reshape(-1, 10),
                            supports=supports, loads=[])
    K, _, _ = assemble_c3d10_sparse_3dof(m)
    s = K.system
    assert np.all(np.diff(s.pattern()[0]) == 10)
    F = rng.standard_normal(K.shape[0]) * 100.0
    F[np.asarray(solid_fixed_dofs(m), dtype=np.int64)] = 0.0
    st = _same(s, F, rtol=1e-10, max_iter=2000, precond=precond)
    assert st["iterations"] > 3 and (precond == 0 or st["status"] == 0)
