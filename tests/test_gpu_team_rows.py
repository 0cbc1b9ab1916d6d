"""Rows of many blocks spread over several warps: a V-cycle whose levels have such rows, against the
oracle's V-cycle on the exported hierarchy."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import amg as oamg
from wnfea_b200 import _lib
from wnfea_b200.amg import AMGParams, export_system_hierarchy
from wnfea_b200.mesh import generate_c3d10_kuhn_block
from wnfea_b200.solid_solver import assemble_c3d10_sparse_3dof

pytestmark = pytest.mark.gpu


# a compact block: its coarse rows reach every other aggregate; stream_min_mb < 0 keeps every coarse
# matrix without a pack, 0 packs them all
@pytest.mark.parametrize("stream_min_mb", [-1.0, 0.0])
@pytest.mark.parametrize("degree", [1, 2])
def test_vcycle_with_long_coarse_rows(stream_min_mb, degree):
    import torch

    m, _ = generate_c3d10_kuhn_block(1.0, 1.0, 1.0, 11, 10, 9)
    K, F, _ = assemble_c3d10_sparse_3dof(m)
    s = K.system
    prm = AMGParams(stream_min_mb=stream_min_mb, smoother_degree=degree, coarse_size=60)
    s.amg_setup(prm)
    H = export_system_hierarchy(s)
    mean = [lv.A.indices.size / lv.n_nodes for lv in H.levels[1:]]
    assert max(mean) >= 64, mean  # rows that take the path
    n = K.shape[0]
    rng = np.random.default_rng(3)
    b = rng.standard_normal(n)
    b[s.fixed_mask.astype(bool)] = 0.0
    r = torch.from_numpy(b).cuda()
    z = torch.empty_like(r)
    _lib.call("wn_amg_vcycle_device", s.handle, 0, r.data_ptr(), z.data_ptr(), 0)
    z32 = torch.empty(n, dtype=torch.float32, device="cuda")
    r32 = r.float()
    _lib.call("wn_amg_vcycle_device", s.handle, 1, r32.data_ptr(), z32.data_ptr(), 0)
    torch.cuda.synchronize()
    A = K.to_bsr().tocsr()
    kw = dict(degree=degree, lower=prm.cheb_lower, safety=prm.cheb_safety)
    ref = oamg.vcycle(A, H, b, **kw)
    ref32 = oamg.vcycle(A, H, r32.double().cpu().numpy(), **kw)
    assert np.abs(z.cpu().numpy() - ref).max() <= 1e-10 * np.abs(ref).max()
    assert np.abs(z32.cpu().numpy() - ref32).max() <= 1e-4 * np.abs(ref32).max()
