"""The coupling with staged lattice velocities (the large tiled launches' own kernel) where it can go
wrong: blocks that end one body and begin the next, blocks whose stencils do not fit the tile,
stencils beside walls and past the lattice's faces, inactive particles, block remainders.

Forces, valid weights, masks and counters against the coupling that reads the lattice directly, on
the same state: the same values in the same order, so equal. The reaction is summed by atomics in
order of arrival: all terms of a node point along the flow here, at most a few hundred of them, so
both float32 sums are within 300 u = 2e-5 of exact and typically its square root (1e-6): 1e-5."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from fsi.config import CouplingConfig
from fsi.coupling import LBMMpmCoupler
from fsi.lbm3d import LBMSolver3D
from fsi.mpm3d import MPMSolver3D
from helpers import periodic_lbm, rel_l2, small_mpm

pytestmark = pytest.mark.gpu


def _positions(case, rng):
    if case == "two_bodies":
        return np.concatenate([rng.uniform(5, 9, (300, 3)), rng.uniform(25, 31, (333, 3))])
    if case == "scattered":
        return rng.uniform(2, 36, (700, 3))
    if case == "walls":  # the mask's solid layers and balls lie among these
        return np.concatenate([rng.uniform((5, 0.5, 5), (9, 3, 9), (257, 3)), rng.uniform(17, 22, (255, 3))])
    if case == "faces":
        return np.concatenate([rng.uniform(-1.5, 2, (200, 3)), rng.uniform(37, 41, (120, 3))])
    return rng.uniform(10, 12, (1, 3))  # one


@pytest.mark.parametrize("build", [False, True])
@pytest.mark.parametrize("case", ["one", "two_bodies", "scattered", "walls", "faces"])
def test_staged_coupling_equals_direct(case, build):
    rng = np.random.default_rng(len(case))
    pos = _positions(case, rng).astype(np.float32)
    solid = np.zeros((40, 40, 40), np.int32)
    solid[:, 0] = solid[:, -1] = 1
    solid[18:20, 18:21, 19:21] = 1
    lbm = LBMSolver3D(periodic_lbm(nx=40, ny=40, nz=40, initial_velocity=(1e-2, 2e-3, 1e-3)))
    lbm.initialize(solid)
    for _ in range(3):
        lbm.step()
    mpm = MPMSolver3D(small_mpm(nx=40, ny=40, nz=40, max_particles=1000))
    mpm.initialize_particles_from_numpy(pos, np.zeros_like(pos), 1.0, 0.125)
    if len(pos) > 1:
        mpm._active[::9] = 0
    cfg = CouplingConfig(gamma=0.1, force_limit=1e-3, build_solid_volume_fraction=build)
    c = LBMMpmCoupler(cfg, lbm, mpm)
    c.compute_coupling_forces(0.25)
    want = [mpm.particle_forces_numpy(), c.particle_valid_weights_numpy(), c.particle_coupling_mask_numpy()]
    counts, reaction = c._counters[:3].clone(), c.coupling_force_numpy()
    c.clear_coupling_fields()
    mpm.clear_particle_force()
    mpm.desc.coupling_fold = 2  # the coupling in a kernel of its own
    c._coupled_substep(0.25, 0.25, build)
    got = [mpm.particle_forces_numpy(), c.particle_valid_weights_numpy(), c.particle_coupling_mask_numpy()]
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)
    assert torch.equal(c._counters[:3], counts)
    assert rel_l2(c.coupling_force_numpy(), reaction) < 1e-5
