"""The tiled P2G and the staged coupling with cells that are not of size 1, on another stream than the
default, and with a particle whose velocity is NaN.

Against the oracle one substep from C = 0: at most 8 * 27 terms meet in a node here, both float32 sums
are within 216 u = 1.3e-5 of exact relative to the sum of magnitudes and typically its square root: 1e-5
on v. Staged against direct coupling: forces, weights and masks equal, the reaction within 1e-5."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from fsi.config import CouplingConfig, MPMConfig
from fsi.coupling import LBMMpmCoupler
from fsi.lbm3d import LBMSolver3D
from fsi.mpm3d import MPMSolver3D
from helpers import periodic_lbm, rel_l2
from oracle import oracle as O

pytestmark = pytest.mark.gpu
N = 32


def _body(dx, rng):
    idx = np.stack(np.meshgrid(*[np.arange(9)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return (dx * (8.0 + 0.5 * (idx + rng.uniform(0, 1, idx.shape)))).astype(np.float32)


@pytest.mark.parametrize("dx", [0.5, 0.3, 2.0])
def test_runs_in_cells_of_another_size(dx):
    rng = np.random.default_rng(int(10 * dx))
    pos = _body(dx, rng)
    vel = rng.normal(0, 1e-2, pos.shape).astype(np.float32)
    cfg = MPMConfig(nx=N, ny=N, nz=N, max_particles=1000, dx=dx, dt=1e-3, youngs_modulus=100.0,
                    gravity=(0.0, -1e-3, 0.0), boundary_width=2)
    g, o = MPMSolver3D(cfg), O.MPMSolver3D(cfg, polar="device")
    for s in (g, o):
        s.initialize_particles_from_numpy(pos, vel, particle_volume=0.125 * dx ** 3)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        g.substep()
    stream.synchronize()
    o.substep()
    assert rel_l2(g.velocities_numpy(), o.velocities_numpy()) < 1e-5
    assert rel_l2(g.positions_numpy(), o.positions_numpy()) < 1e-6


@pytest.mark.parametrize("dx", [0.5, 2.0])
def test_staged_coupling_in_cells_of_another_size(dx):
    rng = np.random.default_rng(int(10 * dx))
    pos = _body(dx, rng)
    lbm = LBMSolver3D(periodic_lbm(nx=N, ny=N, nz=N, initial_velocity=(1e-2, 2e-3, 1e-3)))
    lbm.initialize(np.zeros((N, N, N), np.int32))
    mpm = MPMSolver3D(MPMConfig(nx=N, ny=N, nz=N, max_particles=1000, dx=dx, dt=1e-3, youngs_modulus=100.0,
                                boundary_width=2, gravity=(0.0, 0.0, 0.0)))
    mpm.initialize_particles_from_numpy(pos, np.zeros_like(pos), particle_volume=0.125 * dx ** 3)
    c = LBMMpmCoupler(CouplingConfig(gamma=0.1), lbm, mpm)
    c.compute_coupling_forces(0.25)
    want = [mpm.particle_forces_numpy(), c.particle_valid_weights_numpy(), c.particle_coupling_mask_numpy()]
    reaction = c.coupling_force_numpy()
    c.clear_coupling_fields()
    mpm.clear_particle_force()
    mpm.desc.coupling_fold = 2  # the coupling in a kernel of its own
    c._coupled_substep(1e-3, 0.25, True)
    got = [mpm.particle_forces_numpy(), c.particle_valid_weights_numpy(), c.particle_coupling_mask_numpy()]
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)
    assert rel_l2(c.coupling_force_numpy(), reaction) < 1e-5


def test_a_nan_velocity_reaches_the_same_particles():
    rng = np.random.default_rng(5)
    pos = _body(1.0, rng)
    vel = rng.normal(0, 1e-2, pos.shape).astype(np.float32)
    vel[300, 1] = np.nan
    cfg = MPMConfig(nx=N, ny=N, nz=N, max_particles=1000, dt=1e-2, youngs_modulus=100.0,
                    gravity=(0.0, 0.0, 0.0), boundary_width=2)
    g, o = MPMSolver3D(cfg), O.MPMSolver3D(cfg, polar="device")
    for s in (g, o):
        s.initialize_particles_from_numpy(pos, vel, particle_volume=0.125)
        s.substep()
    hit = np.isnan(o.velocities_numpy())
    assert hit.any() and not hit.all()
    np.testing.assert_array_equal(np.isnan(g.velocities_numpy()), hit)
    assert rel_l2(g.velocities_numpy()[~hit], o.velocities_numpy()[~hit]) < 1e-5
