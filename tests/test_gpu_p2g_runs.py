"""P2G in runs (the atomic scatter's sort of a block's particles and its register sums) where
it can go wrong: block remainders, boxes that do and do not fit the sort, stencils that leave
the grid, crowded cells, gaps along a line, inactive particles.

Tolerance: one substep from C = 0, so the terms of a node are w m v alone. At most n = 600 of
them meet in a node here; the float32 sums of both sides are within n u = 600 * 6e-8 = 3.6e-5
of exact relative to the sum of magnitudes, and typical errors grow with its square root: 1e-5
on v covers both sides with a factor of four."""
from __future__ import annotations

import numpy as np
import pytest

from fsi.config import MPMConfig
from fsi.mpm3d import MPMSolver3D
from helpers import rel_l2
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _lattice(lo, shape):
    idx = np.stack(np.meshgrid(*[np.arange(n) for n in shape], indexing="ij"), -1).reshape(-1, 3)
    return np.asarray(lo) + 0.5 * idx


def _positions(case, rng):
    if case.startswith("count"):
        n = int(case[5:])
        side = int(np.ceil(n ** (1 / 3)))
        return (_lattice((6.0, 7.0, 8.0), (side,) * 3) + rng.uniform(0, 0.5, (side ** 3, 3)))[:n]
    if case == "scattered":  # a block's box has more cells than the sort counts
        return rng.uniform(1.0, 38.0, (700, 3))
    if case == "faces":  # stencils partly and wholly outside the grid
        return rng.uniform(-4.0, 43.0, (900, 3)) * np.array([1.0, 0.2, 0.2])
    if case == "crowded":
        return rng.uniform(9.6, 10.4, (600, 3))
    if case == "gaps":  # lines with empty base cells of one, two and more between
        z = np.concatenate([np.arange(4.0, 36.0, s) for s in (1.0, 2.0, 3.0, 5.0)])
        return np.concatenate([np.stack([np.full_like(z, 10.0 + i), np.full_like(z, 12.0), z], 1)
                               for i in range(8)]) + 0.3
    # two bodies in one block
    return np.concatenate([_lattice((4.0, 4.0, 4.0), (5, 5, 5)), _lattice((30.0, 31.0, 32.0), (5, 5, 5))])


@pytest.mark.parametrize("threads", [0, 128, 512])
@pytest.mark.parametrize("case", ["count1", "count31", "count255", "count256", "count257", "count600",
                                  "scattered", "faces", "crowded", "gaps", "two_bodies"])
def test_runs_against_oracle(case, threads):
    rng = np.random.default_rng(len(case) + threads)
    pos = _positions(case, rng).astype(np.float32)
    vel = rng.normal(0, 1e-2, pos.shape).astype(np.float32)
    cfg = MPMConfig(nx=40, ny=40, nz=40, max_particles=1000, dt=1e-2, youngs_modulus=100.0,
                    gravity=(0.0, -1e-3, 0.0), boundary_width=2)
    g, o = MPMSolver3D(cfg), O.MPMSolver3D(cfg, polar="device")
    for s in (g, o):
        s.initialize_particles_from_numpy(pos, vel, particle_volume=0.125)
    if len(pos) > 1:
        g._active[::7] = 0
        o.active[:len(pos):7] = 0
    g.desc.launch_threads = threads
    g.substep()
    o.substep()
    assert rel_l2(g.velocities_numpy(), o.velocities_numpy()) < 1e-5
    assert rel_l2(g.positions_numpy(), o.positions_numpy()) < 1e-6
    assert float(g._grid.abs().max()) == 0.0 and int(g._dirty.max()) == 0
    for _ in range(3):  # with C and F set, against noise amplified by the stress
        g.substep()
        o.substep()
    assert rel_l2(g.velocities_numpy(), o.velocities_numpy()) < 1e-3
    assert rel_l2(g.positions_numpy(), o.positions_numpy()) < 1e-6


@pytest.mark.parametrize("per_cell", [1, 10, 11, 12, 22, 23])
def test_sorted_chunks_and_triples_bit_exact(per_cell):
    """The sorted scatter's listed triples of cells at every place of a row of eight along z, with
    counts around the chunk that is staged at a time (11), bit for bit the oracle's cell order."""
    rng = np.random.default_rng(per_cell)
    cells = [(4, 5, z) for z in range(3, 22)] + [(6, 8, z) for z in (3, 5, 6, 9, 12, 14, 15)] + [(9, 9, 13)]
    pos = np.concatenate([np.asarray(c) + rng.uniform(0.55, 1.45, (per_cell, 3)) for c in cells])
    pos = pos[rng.permutation(len(pos))].astype(np.float32)
    vel = rng.normal(0, 1e-2, pos.shape).astype(np.float32)
    cfg = MPMConfig(nx=17, ny=18, nz=27, max_particles=1000, dt=1e-2, youngs_modulus=100.0,
                    gravity=(0.0, -1e-3, 0.0), boundary_width=2, p2g_mode="sorted")
    g, o = MPMSolver3D(cfg), O.MPMSolver3D(cfg, polar="device", cell_order=True)
    for s in (g, o):
        s.initialize_particles_from_numpy(pos, vel, particle_volume=0.125)
    for _ in range(3):
        g.substep()
        o.substep()
        np.testing.assert_array_equal(g.velocities_numpy(), o.velocities_numpy())
        np.testing.assert_array_equal(g.positions_numpy(), o.positions_numpy())
