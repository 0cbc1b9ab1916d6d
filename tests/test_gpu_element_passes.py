"""Element forces, energies and stresses at the edges of the element kernels' runs (32 elements per
warp, four warps per block, two blocks per SM in one wave), on curved elements off the origin,
against the oracle.

Bounds: an element's force is a sum of 4 x 6 x 10 products per component whose terms are at most
about the element's largest force times its conditioning; 1e-12 of that force (the bound of the
element tests beside this one) and for stresses 1e-12 of the largest stress."""

from __future__ import annotations

import numpy as np
import pytest

import wnfea_b200 as wn
from oracle import c3d10 as oc3d10

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 31, 32, 33, 127, 129, 2 * 148 * 128 + 33])
def test_runs_of_elements_match_oracle(m, golden):
    g = golden("c3d10_element.npz")
    rng = np.random.default_rng(m)
    base = np.where(rng.random(m)[:, None, None] < 0.5, g["tet"], g["curved"])
    coords = base * rng.uniform(0.5, 2.0, (m, 1, 1)) + rng.standard_normal((m, 1, 3))
    u = rng.standard_normal((m, 30)) * 1e-3
    E, nu = rng.uniform(1e9, 3e11, m), rng.uniform(0.0, 0.45, m)
    props = np.stack([E, nu], axis=1)
    f = wn.element_internal_forces_c3d10(coords, u, E, nu)
    f_o = oc3d10.element_internal_forces_batch(coords, u, props)
    assert (np.abs(f - f_o).max(axis=1) <= 1e-12 * np.abs(f_o).max(axis=1)).all()
    sig, vm, _ = wn.element_stresses_c3d10(coords, u, E, nu)
    sig_o, vm_o = oc3d10.element_stresses_batch(coords, u, props)[:2]
    assert (np.abs(sig - sig_o).max(axis=(1, 2)) <= 1e-12 * np.abs(sig_o).max(axis=(1, 2))).all()
    assert (np.abs(vm - vm_o) <= 1e-12 * vm_o.max(axis=1)[:, None]).all()
