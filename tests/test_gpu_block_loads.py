"""A frame's V-cycle (6-DOF fine level) on a vector that starts off a 16-byte boundary: the streamed
kernels load a node's values in pairs and leave such a vector to the row kernels.

Bound: the two ways add a row's products in different orders; a V-cycle's sums have at most a few
hundred terms per row and level, so 1e-11 (FP64) and 1e-4 (FP32) of the largest entry."""

from __future__ import annotations

import numpy as np
import pytest

from wnfea_b200 import _lib
from wnfea_b200.amg import AMGParams
from wnfea_b200.beam import frame_linear_system
from wnfea_b200.frames import generate_space_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [1, 2])
def test_vcycle_of_an_unaligned_vector(degree):
    import torch

    frame, s, F = frame_linear_system(generate_space_frame(8, 8, 8, seed=1))
    s.amg_setup(AMGParams(coarse_size=300, smoother_degree=degree, stream_min_mb=0.0))
    n = np.asarray(F).size
    b = torch.from_numpy(np.random.default_rng(5).standard_normal(n)).cuda()
    for prec, dt, tol in ((0, torch.float64, 1e-11), (1, torch.float32, 1e-4)):
        r = b.to(dt)
        off = torch.empty(n + 1, dtype=dt, device="cuda")[1:]
        off.copy_(r)
        assert off.data_ptr() % 16 != 0
        z, zo = torch.empty_like(r), torch.empty_like(r)
        _lib.call("wn_amg_vcycle_device", s._h, prec, r.data_ptr(), z.data_ptr(), 0)
        _lib.call("wn_amg_vcycle_device", s._h, prec, off.data_ptr(), zo.data_ptr(), 0)
        torch.cuda.synchronize()
        assert (z - zo).abs().max().item() <= tol * z.abs().max().item()
