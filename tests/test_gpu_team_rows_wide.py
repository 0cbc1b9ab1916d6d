"""Rows of 160 to 250 blocks: V-cycles whose levels have such rows without a pack, spread over eight warps (6x6 and
6x3 blocks; more rows than the grid holds at once), and with one, in streamed tiles of one or two rows,
against the oracle's V-cycle on the exported hierarchy.

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


def _long_rows(H, packed):
    """(block columns, packed, rows) of the hierarchy's 6-row matrices with such rows on average."""
    found = []
    for i, lv in enumerate(H.levels):
        for M, bc in ([(lv.A, 6)] if i else []) + [(lv.R, 6 if i else 3)]:
            length = np.diff(M.indptr)
            is_packed = packed and length.max() <= (256 if bc == 6 else 512)  # (a row fits a tile)
            if length.mean() >= 160:
                found.append((bc, bool(is_packed), len(length)))
    return found


# strength thresholds at which this block's hierarchy has such rows: 0.16, 3,265 rows of 165 blocks; 0.0895, 242 of
# 206 and a restriction of 225; 0.003, a first restriction of 512 rows of 199
@pytest.mark.parametrize("theta,stream_min_mb,bc,rows", [(0.16, -1.0, 6, 3000), (0.0895, -1.0, 6, 200),
                                                         (0.0895, 0.0, 6, 200), (0.003, -1.0, 3, 300),
                                                         (0.003, 0.0, 3, 300)])
def test_vcycle_with_very_long_rows(theta, stream_min_mb, bc, rows):
    import torch

    m, _ = generate_c3d10_kuhn_block(16 / 16, 15 / 16, 14 / 16, 16, 15, 14)
    K, _, _ = assemble_c3d10_sparse_3dof(m)
    s = K.system
    prm = AMGParams(stream_min_mb=stream_min_mb, strength_theta=theta, coarse_size=60)
    s.amg_setup(prm)
    H = export_system_hierarchy(s)
    packed = stream_min_mb == 0.0
    found = _long_rows(H, packed)
    assert any(c == bc and p == packed and n >= rows for c, p, n in found), found
    n = K.shape[0]
    b = np.random.default_rng(17).standard_normal(n)
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
