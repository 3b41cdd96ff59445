"""Particles at infinity and beyond the range of cell numbers: they meet no node, so a substep leaves
them without velocity at the position limits, and the other particles as they are without them.

The others' sums differ by the order of arrival alone: at most 8 * 27 terms meet in a node, within
216 * 6e-8 = 1.3e-5 of exact on both sides, typically its square root: 1e-5 on v."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from fsi.config import CouplingConfig, MPMConfig
from fsi.coupling import LBMMpmCoupler
from fsi.lbm3d import LBMSolver3D
from fsi.mpm3d import MPMSolver3D
from helpers import periodic_lbm, rel_l2

pytestmark = pytest.mark.gpu
N = 40
FAR = np.array([[np.inf, 10, 10], [10, np.inf, 10], [10, 10, 3e9], [np.inf] * 3, [-np.inf, 10, 10], [-3e9] * 3],
               np.float32)


def _solver(mode, pos, extra):
    cfg = MPMConfig(nx=N, ny=N, nz=N, max_particles=1000, dt=1e-2, youngs_modulus=100.0,
                    gravity=(0.0, 0.0, 0.0), boundary_width=2, p2g_mode=mode)
    m = MPMSolver3D(cfg)
    p = np.concatenate([pos, np.full((extra, 3), 10.0, np.float32)])
    vel = np.random.default_rng(1).normal(0, 1e-2, pos.shape).astype(np.float32)
    m.initialize_particles_from_numpy(p, np.concatenate([vel, np.zeros((extra, 3), np.float32)]),
                                      particle_volume=0.125)
    if extra:
        m._x[:, len(pos):len(p)] = torch.from_numpy(FAR.T.copy()).cuda()
    return m


@pytest.mark.parametrize("mode,coupled,storage", [
    ("atomic", None, "f32"), ("sorted", None, "f32"), ("atomic", 1, "f32"), ("atomic", 2, "f32"),
    ("atomic", 2, "f16"), ("atomic", 3, "f32"), ("sorted", 0, "f32")])
def test_far_particles_touch_nothing(mode, coupled, storage):
    rng = np.random.default_rng(3)
    idx = np.stack(np.meshgrid(*[np.arange(7)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (12.0 + 0.5 * (idx + rng.uniform(0, 1, idx.shape))).astype(np.float32)
    got = []
    for extra in (0, len(FAR)):
        m = _solver(mode, pos, extra)
        if coupled is None:
            m.substep()
        else:
            lbm = LBMSolver3D(periodic_lbm(nx=N, ny=N, nz=N, initial_velocity=(1e-2, 2e-3, 1e-3),
                                           population_storage=storage))
            lbm.initialize(np.zeros((N, N, N), np.int32))
            m.desc.coupling_fold = coupled
            LBMMpmCoupler(CouplingConfig(gamma=0.1), lbm, m)._coupled_substep(1e-2, 0.1, True)
        got.append(m)
    plain, far = got
    n = len(pos)
    assert rel_l2(far.velocities_numpy()[:n], plain.velocities_numpy()) < 1e-5
    assert rel_l2(far.positions_numpy()[:n], plain.positions_numpy()) < 1e-6
    x, v = far.positions_numpy()[n:], far.velocities_numpy()[n:]
    np.testing.assert_array_equal(v, 0.0)
    d = far.desc
    want = np.clip(FAR, np.float32(d.clamp_lower), np.array(list(d.clamp_upper), np.float32))
    np.testing.assert_array_equal(x, want)


def test_base_cells_keep_the_cast():
    m = _solver("atomic", np.full((3, 3), 12.0, np.float32), len(FAR))
    cells = m.base_cells_numpy()
    assert cells[3][0] == 2 ** 31 - 1 and cells[7][0] == -(2 ** 31)
