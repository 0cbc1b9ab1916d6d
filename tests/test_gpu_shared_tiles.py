"""Streamed tiles of few long rows, which all consumer warps share: V-cycles of blocks whose packed coarse
levels have rows from about 20 to 140 blocks (a tile of 256 blocks: many rows, down to one) against the
oracle's V-cycle on the exported hierarchy.

Bounds: those of the other V-cycle tests (1e-10 in FP64, 1e-4 in FP32 of the largest entry)."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import amg as oamg
from wnfea_b200 import _lib
from wnfea_b200.amg import AMGParams, export_system_hierarchy
from wnfea_b200.mesh import generate_c3d10_kuhn_block
from wnfea_b200.solid_solver import assemble_c3d10_sparse_3dof

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(5, 4, 3), (8, 7, 6), (16, 15, 14), (40, 4, 4)])
def test_vcycle_with_tiles_of_few_rows(cells):
    import torch

    m, _ = generate_c3d10_kuhn_block(1.0, 0.9, 0.8, *cells)
    K, _, _ = assemble_c3d10_sparse_3dof(m)
    s = K.system
    prm = AMGParams(stream_min_mb=0.0, coarse_size=60)
    s.amg_setup(prm)
    H = export_system_hierarchy(s)
    n = K.shape[0]
    b = np.random.default_rng(11).standard_normal(n)
    b[s.fixed_mask.astype(bool)] = 0.0
    r = torch.from_numpy(b).cuda()
    r32 = r.float()
    z, z32 = torch.empty_like(r), torch.empty_like(r32)
    _lib.call("wn_amg_vcycle_device", s.handle, 0, r.data_ptr(), z.data_ptr(), 0)
    _lib.call("wn_amg_vcycle_device", s.handle, 1, r32.data_ptr(), z32.data_ptr(), 0)
    torch.cuda.synchronize()
    A = K.to_bsr().tocsr()
    kw = dict(degree=1, lower=prm.cheb_lower, safety=prm.cheb_safety)
    ref = oamg.vcycle(A, H, b, **kw)
    ref32 = oamg.vcycle(A, H, r32.double().cpu().numpy(), **kw)
    assert np.abs(z.cpu().numpy() - ref).max() <= 1e-10 * np.abs(ref).max()
    assert np.abs(z32.cpu().numpy() - ref32).max() <= 1e-4 * np.abs(ref32).max()
