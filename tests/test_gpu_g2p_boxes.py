"""The gather's staged boxes where they can go wrong: a block that ends one body and begins the
next (cut in two boxes, at any thread, beside inactive particles), boxes just within and just past
the tile, three bodies in a block (straight from the grid), bodies at opposite faces.

The sorted scatter makes the grid bit for bit the oracle's, and the gather keeps the oracle's order
and rounding: the results are equal, with no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

from fsi.config import MPMConfig
from fsi.mpm3d import MPMSolver3D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _body(rng, lo, n, span=3.0):
    return np.asarray(lo) + rng.uniform(0, span, (n, 3))


def _positions(case, rng):
    kind, arg = case
    if kind == "cut":  # the second body's first particle is thread `arg` of the first block
        return np.concatenate([_body(rng, (4, 5, 6), arg), _body(rng, (28, 30, 31), 300)])
    if kind == "volume":  # one box of 16 x 16 x (arg / 256) nodes, touched at its corners
        lo, hi = np.array([3.6, 3.6, 3.6]), np.array([3.6 + 13, 3.6 + 13, 3.6 + arg // 256 - 3])
        return np.concatenate([lo + rng.uniform(0, 0.5, (2, 3)), hi + rng.uniform(0, 0.5, (2, 3)),
                               rng.uniform(lo, hi, (60, 3))])
    if kind == "faces":  # stencils that leave the grid on both sides
        return np.concatenate([_body(rng, (0.6, 0.6, 0.6), 100, 1.0), _body(rng, (38.2, 37.6, 38.0), 100, 1.3)])
    return np.concatenate([_body(rng, lo, 70) for lo in ((4, 5, 6), (28, 30, 31), (4, 30, 8))])  # three


@pytest.mark.parametrize("inactive", [0, 1])
@pytest.mark.parametrize("case", [("cut", 1), ("cut", 31), ("cut", 32), ("cut", 100), ("cut", 255), ("cut", 256),
                                  ("volume", 2048), ("volume", 2304), ("faces", 0), ("three", 0)])
def test_boxes_bit_exact(case, inactive):
    rng = np.random.default_rng(case[1] + inactive)
    pos = _positions(case, rng).astype(np.float32)
    vel = rng.normal(0, 1e-2, pos.shape).astype(np.float32)
    cfg = MPMConfig(nx=40, ny=40, nz=40, max_particles=1000, dt=1e-2, youngs_modulus=100.0,
                    gravity=(0.0, -1e-3, 0.0), boundary_width=2, p2g_mode="sorted")
    g, o = MPMSolver3D(cfg), O.MPMSolver3D(cfg, polar="device", cell_order=True)
    for s in (g, o):
        s.initialize_particles_from_numpy(pos, vel, particle_volume=0.125)
    if inactive:
        off = np.arange(len(pos)) % 5 == case[1] % 5  # the first thread past the cut among them
        g._active[:len(pos)][off.tolist()] = 0
        o.active[:len(pos)][off] = 0
    for _ in range(2):
        g.substep()
        o.substep()
        np.testing.assert_array_equal(g.velocities_numpy(), o.velocities_numpy())
        np.testing.assert_array_equal(g.positions_numpy(), o.positions_numpy())
