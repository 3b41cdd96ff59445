"""The sums that feed a 16-bit lattice keep their order: every term rounded like the reference's, and
one addition per node and block of 256 particles into global memory, in batches and single scenes.

Exact, so no tolerance. Particles with no node in common: a node's sum is one term, the oracle's bits.
Two blocks of particles on one spot (weights 1/2, 1/2, 0), masses 1 and 2^-20: each block's sums are
exact in any order, and so is their sum 32 (1 + 2^-20); the second block's velocity 1 makes every
node's 2^-20 / (1 + 2^-20), which float32 holds as 2^-20 (1 - 2^-20). A block that adds its parts one
by one to the other's 32 loses them to rounding."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from fsi import _native as nat
from fsi.batch import SceneBatch
from fsi.config import CouplingConfig, MPMConfig, SimulationConfig
from fsi.coupling import LBMMpmCoupler
from fsi.lbm3d import LBMSolver3D
from fsi.mpm3d import MPMSolver3D
from helpers import periodic_lbm
from oracle import oracle as O

pytestmark = pytest.mark.gpu
N = 32


def _mpm(count):
    return MPMConfig(nx=N, ny=N, nz=N, max_particles=count, particles_per_cell=2, dx=1.0, dt=0.1,
                     density=1.0, youngs_modulus=0.05, poisson_ratio=0.3, gravity=(0.0, 0.0, 0.0),
                     boundary_width=2)


def _substep(where, storage, pos, set_state):
    """One MPM substep without coupling forces of each particle set; returns per scene x, v, C, F."""
    lbm = periodic_lbm(nx=N, ny=N, nz=N, population_storage=storage)
    coupling = CouplingConfig(gamma=0.0, mpm_substeps_per_lbm_step=10)
    if where == "batch":
        b = SceneBatch([SimulationConfig(num_steps=1, lbm_dt=1.0, lbm=lbm, mpm=_mpm(len(p)), coupling=coupling)
                        for p in pos])
        b.initialize([None] * len(pos), pos)
        views = [tuple(t[..., o:o + n] for t in (b._x, b._v, b._C, b._F, b._mass))
                 for o, n in zip(b.particle_offsets, b.particle_counts)]
        for i, v in enumerate(views):
            set_state(i, *v)
        nat.call("fsi_batch_mpm_substep", b.lattice._handle, b._parts, nat.ptr(b._grid), nat.ptr(b._dirty),
                 nat.stream_ptr())
        return [[t.cpu().numpy().T for t in v[:4]] for v in views]
    out = []
    for i, p in enumerate(pos):
        s = LBMSolver3D(lbm)
        s.initialize(np.zeros((N, N, N), np.int32))
        m = MPMSolver3D(_mpm(len(p)))
        m.initialize_particles_from_numpy(p)
        set_state(i, *(t[..., :len(p)] for t in (m._x, m._v, m._C, m._F, m._mass)))
        m.desc.coupling_fold = 2  # the kernels of large launches
        c = LBMMpmCoupler(coupling, s, m)
        if where == "single":
            c._coupled_substep(0.1, 0.1, False)
        else:  # the entry point that does not know the lattice's storage
            c._desc.gamma_eff, c._desc.dt_ratio, c._desc.build_fraction = 0.0, 0.1, 0
            m.desc.dt = 0.1
            nat.call("fsi_coupled_substep_tiled", c._desc, m.desc, m.particles, nat.ptr(s.macro), nat.ptr(s.flags),
                     nat.ptr(c._accum), nat.ptr(c._valid), nat.ptr(c._mask), nat.ptr(c._counters),
                     nat.ptr(m._grid), nat.ptr(m._dirty), nat.stream_ptr())
        out.append([t[..., :len(p)].cpu().numpy().T for t in (m._x, m._v, m._C, m._F)])
    return out


@pytest.mark.parametrize("where", ["batch", "single", "untold"])
@pytest.mark.parametrize("storage", ["f16", "bf16"])
def test_terms_are_rounded_one_by_one(where, storage):
    rng = np.random.default_rng(7)
    cells = np.stack(np.meshgrid(*[np.arange(2, N - 4, 4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = [(cells[:n] + rng.uniform(0.5, 1.5, (n, 3))).astype(np.float32) for n in (343, 100, 1)]
    vel = [rng.normal(0, 1e-2, p.shape).astype(np.float32) for p in pos]
    C = [rng.normal(0, 1e-2, (len(p), 9)).astype(np.float32) for p in pos]
    F = [(np.eye(3).reshape(9) + rng.normal(0, 5e-2, (len(p), 9))).astype(np.float32) for p in pos]

    def set_state(i, x, v, c, f, mass):
        for t, a in ((v, vel[i]), (c, C[i]), (f, F[i])):
            t.copy_(torch.from_numpy(np.ascontiguousarray(a.T)))

    got = _substep(where, storage, pos, set_state)
    for i, p in enumerate(pos):
        o = O.MPMSolver3D(_mpm(len(p)), polar="device")
        o.initialize_particles_from_numpy(p, vel[i])
        o.C[:len(p)] = C[i].reshape(o.C[:len(p)].shape)
        o.F[:len(p)] = F[i].reshape(o.F[:len(p)].shape)
        o.substep()
        for g, w in zip(got[i], (o.x, o.v, o.C, o.F)):
            np.testing.assert_array_equal(g, np.asarray(w[:len(p)]).reshape(g.shape))


@pytest.mark.parametrize("where", ["batch", "single", "untold"])
@pytest.mark.parametrize("storage", ["f16", "bf16"])
def test_a_block_adds_to_a_node_once(where, storage):
    spots = [(5.5, 6.5, 7.5), (20.5, 21.5, 9.5), (12.5, 5.5, 25.5), (25.5, 25.5, 25.5)]
    pos = [np.tile(np.float32(s), (512, 1)) for s in spots]

    def set_state(i, x, v, c, f, mass):
        mass[:256] = 1.0
        mass[256:] = 2.0 ** -20
        v[0, 256:] = 1.0

    for x, v, c, f in _substep(where, storage, pos, set_state):
        np.testing.assert_array_equal(v[:, 0], np.float32(2.0 ** -20 * (1 - 2.0 ** -20)))
        np.testing.assert_array_equal(v[:, 1:], 0.0)
