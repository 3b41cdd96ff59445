"""The sorted scatter's tile scan where it can go wrong: one chunk of 1024 cell tiles, several, and more
than one launch sums by itself (64), with particles in the first and last tiles and between, over
substeps that reuse the counts. The order of every sum is the oracle's: equal, with no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

from fsi.config import MPMConfig
from fsi.mpm3d import MPMSolver3D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(20, 17, 23), (130, 131, 133), (2056, 130, 130)])
def test_tile_chunks_bit_exact(shape):
    rng = np.random.default_rng(shape[0])
    top = np.asarray(shape, float) - 1.6
    pos = np.concatenate([rng.uniform(0.6, 3, (150, 3)), rng.uniform(top - 2.5, top, (150, 3)),
                          rng.uniform(0.6, top, (300, 3)), top * 0.4 + rng.uniform(0, 2, (300, 3))])
    pos = pos[rng.permutation(len(pos))].astype(np.float32)
    vel = rng.normal(0, 1e-2, pos.shape).astype(np.float32)
    cfg = MPMConfig(nx=shape[0], ny=shape[1], nz=shape[2], max_particles=1000, dt=1e-2, youngs_modulus=100.0,
                    gravity=(0.0, -1e-3, 0.0), boundary_width=2, p2g_mode="sorted")
    g, o = MPMSolver3D(cfg), O.MPMSolver3D(cfg, polar="device", cell_order=True)
    for s in (g, o):
        s.initialize_particles_from_numpy(pos, vel, particle_volume=0.125)
    for _ in range(2):
        g.substep()
        o.substep()
        np.testing.assert_array_equal(g.velocities_numpy(), o.velocities_numpy())
        np.testing.assert_array_equal(g.positions_numpy(), o.positions_numpy())
