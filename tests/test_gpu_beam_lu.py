"""Dense LU of the frame tangent at the edges of its panel shapes and bands, against numpy."""

from __future__ import annotations

import numpy as np
import pytest

from wnfea_b200.beam import BeamFrame
from wnfea_b200.frames import generate_frame_grid

pytestmark = pytest.mark.gpu


# the panel's columns and rows per thread follow the half bandwidth 6 ny + 5 (or any, when shuffled):
# one panel, a ragged last panel, the last 32-column band and the first 16-column one, 8 columns,
# and bands as wide as the matrix
@pytest.mark.parametrize("nx,ny,shuffle", [(2, 2, False), (3, 2, False), (11, 3, False), (7, 9, True), (2, 79, False),
                                           (2, 80, False), (2, 165, False), (2, 200, True), (2, 256, True)])
def test_dense_lu_matches_numpy(nx, ny, shuffle):
    m = generate_frame_grid(nx, ny, seed=nx + ny)
    if shuffle:
        perm = np.random.default_rng(5).permutation(nx * ny)  # old node i becomes perm[i]
        m.mesh_nodes = m.mesh_nodes[np.argsort(perm)]
        m.mesh_elements = perm[m.mesh_elements].astype(np.int32)
        for s in m.supports:
            s.node_id = int(perm[s.node_id])
    fr = BeamFrame(m)
    mask = np.zeros(fr.n, dtype=np.uint8)
    for s in m.supports[:1]:
        mask[6 * s.node_id:6 * s.node_id + 6] = 1
    fr.set_fixed(mask)
    U = np.random.default_rng(1).standard_normal(fr.n) * 1e-2 * (1 - mask)
    fr.assemble_tangent(U, apply_bcs=True)
    K = fr.tangent_bsr().toarray()
    b = np.random.default_rng(2).standard_normal(fr.n)
    x, _, rel, status = fr.solve(b, method="dense")
    assert status == 0
    # backward stability of partial pivoting: n eps times the (small) growth of the factors
    eps = np.finfo(float).eps
    scale = np.abs(K) @ np.abs(x) + np.abs(b)
    assert np.abs(K @ x - b).max() <= 16 * fr.n * eps * scale.max()
    assert np.isfinite(rel)
    # the same system again: bit for bit
    assert np.array_equal(x, fr.solve(b, method="dense")[0])


def test_dense_lu_reports_a_singular_tangent():
    m = generate_frame_grid(4, 5, E=0.0)
    fr = BeamFrame(m)
    fr.assemble_tangent(np.zeros(fr.n), apply_bcs=True)
    assert fr.solve(np.ones(fr.n), method="dense")[3] == -4
