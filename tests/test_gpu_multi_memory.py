"""Batches of several widths on one handle: the device vectors of the widest serve the others, and a new
hierarchy replaces the old one's vectors, with the same solutions."""

from __future__ import annotations

import numpy as np
import pytest

from wnfea_b200.mesh import generate_c3d10_kuhn_block, tip_load_cases
from wnfea_b200.model import solid_fixed_dofs
from wnfea_b200.solid_solver import assemble_c3d10_sparse_3dof

pytestmark = pytest.mark.gpu


def _used():
    """Bytes in use from the device's default memory pool, the library's allocations."""
    import torch
    from cuda.bindings import runtime as rt

    torch.cuda.synchronize()
    pool = rt.cudaDeviceGetDefaultMemPool(0)[1]
    return int(rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)[1])


def test_widths_share_their_vectors():
    m, _ = generate_c3d10_kuhn_block(2.0, 1.0, 1.0, 20, 9, 8)
    K, _, _ = assemble_c3d10_sparse_3dof(m)
    s = K.system
    F = tip_load_cases(m.mesh_nodes, n_cases=40, seed=2)
    F[np.asarray(solid_fixed_dofs(m), dtype=np.int64)] = 0.0
    s.amg_setup()
    n = len(F)
    for precision in (0, 1):
        kw = dict(rtol=1e-8, precision=precision)
        U, st = s.solve_multi(F, **kw)  # 32 + 8
        assert st["status"] == 0
        full = _used()
        for k in (40, 16, 5, 40, 32, 12):
            assert np.array_equal(s.solve_multi(F[:, :k], **kw)[0], U[:, :k])
        # nothing that grows with the mesh (16 cases alone hold more than 16 vectors of 16 columns)
        assert _used() - full <= 1 << 20 < 8 * 16 * n
        # narrow first: the vectors grow, and the narrow batch's captured launches follow them
        s.amg_setup()
        for k in (5, 16, 40, 5, 16):
            assert np.array_equal(s.solve_multi(F[:, :k], **kw)[0], U[:, :k])
        assert _used() - full <= 1 << 20
