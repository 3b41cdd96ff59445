"""The work that programs have this framework do, as timed cases through its public entry points.

Kinds of case:

* ``lattice``: ``LBMSolver3D.step`` a few times, then the density and velocity field;
* ``solid``: ``MPMSolver3D.substep`` a few times;
* ``coupled``: ``FSISimulation.step`` with its diagnostics, or ``FSISimulation.advance``;
* ``batch``: ``SceneBatch.run`` of uneven coupled scenes;
* ``closure``: ``ClosureSimulation.step``, or the corrections of ``closure.infer``;
* ``training``: ``ClosureTrainer.fit`` for a few steps.

``exact`` gives the same quantities in float64 from plain torch.
"""
from __future__ import annotations

import dataclasses
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "taichi-mpm-lbm_gb300"))

from fsi import closure, scenes  # noqa: E402
from fsi.batch import SceneBatch  # noqa: E402
from fsi.config import BoundaryConfig, CouplingConfig, LBMConfig, MPMConfig, SimulationConfig  # noqa: E402
from fsi.lbm3d import LBMSolver3D  # noqa: E402
from fsi.mpm3d import MPMSolver3D  # noqa: E402
from fsi.simulation import FSISimulation  # noqa: E402

F64 = torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest lattice in use, a test-sized channel: the latency of a step
        {"name": "lattice_small_f32", "kind": "lattice", "nx": 48, "ny": 32, "nz": 32,
         "storage": "f32", "arithmetic": "auto", "faces": False, "fraction": 0.0, "tau": 0.6,
         "steps": 4},
        # an odd-sized inflow / outflow channel with obstacles on 16-bit populations
        {"name": "lattice_odd_bf16", "kind": "lattice", "nx": 211, "ny": 93, "nz": 107,
         "storage": "bf16", "arithmetic": "auto", "faces": True, "fraction": 0.05, "tau": 0.7,
         "steps": 4},
        # the standalone lattice at scale, in the default form and in half storage
        {"name": "lattice_256_f32", "kind": "lattice", "nx": 256, "ny": 256, "nz": 256,
         "storage": "f32", "arithmetic": "auto", "faces": False, "fraction": 0.1, "tau": 0.6,
         "steps": 4},
        {"name": "lattice_256_f16", "kind": "lattice", "nx": 256, "ny": 256, "nz": 256,
         "storage": "f16", "arithmetic": "auto", "faces": False, "fraction": 0.1, "tau": 0.6,
         "steps": 4},
        # a few small bodies alone: odd counts, launch- and latency-bound
        {"name": "solid_odd", "kind": "solid", "grid": 75, "cubes": 5, "edge": 9,
         "mode": "atomic", "model": "fixed_corotated", "substeps": 5},
        # the standalone solid at scale: 2,097,152 particles
        {"name": "solid_2m", "kind": "solid", "grid": 256, "cubes": 64, "edge": 16,
         "mode": "atomic", "model": "fixed_corotated", "substeps": 5},
        # the smoke workload: one cube in a force-driven channel, diagnostics every step
        {"name": "coupled_smoke", "kind": "coupled", "scene": "smoke", "nx": 48, "ny": 32,
         "nz": 32, "bodies": 1, "edge": 8, "mode": "atomic", "storage": "f32", "advance": 0},
        # a mid-sized inflow channel with the bit-reproducible scatter, no diagnostics
        {"name": "coupled_mid_sorted", "kind": "coupled", "scene": "bodies", "nx": 150, "ny": 78,
         "nz": 90, "bodies": 7, "edge": 11, "layout": 5, "mode": "sorted", "storage": "f32",
         "advance": 10},
        # the coupled step at scale with the runner's diagnostics
        {"name": "coupled_bodies", "kind": "coupled", "scene": "bodies", "nx": 384, "ny": 192,
         "nz": 192, "bodies": 48, "edge": 12, "layout": 3, "mode": "atomic", "storage": "f32",
         "advance": 0},
        # many uneven scenes at once, half-storage lattices
        {"name": "batch_64", "kind": "batch", "count": 64, "layout": 4, "storage": "f16", "steps": 8},
        # the learned closure: a corrected coarse step
        {"name": "closure_step", "kind": "closure", "nx": 192, "ny": 96, "nz": 96, "balls": 24,
         "fraction_feature": True, "what": "step"},
        # fitting the closure's network on mini-batches of the usual size
        {"name": "training", "kind": "training", "rows": 65536, "batch": 16384, "steps": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lattice", "lattice", "solid", "coupled", "coupled", "batch", "closure",
                       "training"])
    if kind == "lattice":
        n = [_log(rng, 16, 256) for _ in range(3)]
        storage = rng.choice(["f32", "f32", "f16", "bf16"])
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "storage": storage,
                "arithmetic": rng.choice(["auto", "auto", "fast"]),
                "faces": n[0] * n[1] * n[2] > 400_000 and rng.random() < 0.4,
                "fraction": rng.choice([0.0, 0.05, 0.1]), "tau": round(rng.uniform(0.6, 0.8), 3),
                "steps": rng.choice([3, 4])}
    if kind == "solid":
        grid = _log(rng, 48, 256)
        edge = rng.randint(6, 16)
        most = max(1, min(64, int((grid / (2.0 * edge + 2)) ** 3)))
        return {"kind": kind, "grid": grid, "cubes": _log(rng, 1, most) if most > 1 else 1,
                "edge": edge, "mode": rng.choice(["atomic", "sorted"]),
                "model": rng.choice(["fixed_corotated", "fixed_corotated", "neo_hookean"]),
                "substeps": 5}
    if kind == "coupled":
        if rng.random() < 0.4:
            return {"kind": kind, "scene": "smoke", "nx": rng.randint(40, 72),
                    "ny": rng.randint(28, 48), "nz": rng.randint(28, 48), "bodies": 1,
                    "edge": rng.randint(5, 12), "mode": rng.choice(["atomic", "sorted"]),
                    "storage": "f32", "advance": rng.choice([0, 10])}
        nx = _log(rng, 128, 320)
        return {"kind": kind, "scene": "bodies", "nx": nx, "ny": rng.randint(64, 160),
                "nz": rng.randint(64, 160), "bodies": max(2, nx // 24), "edge": rng.randint(8, 12),
                "layout": rng.randint(100, 999), "mode": rng.choice(["atomic", "atomic", "sorted"]),
                "storage": rng.choice(["f32", "f32", "f16"]), "advance": rng.choice([0, 10])}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 6, 60), "layout": rng.randint(100, 999),
                "storage": rng.choice(["f16", "f16", "f32"]), "steps": 8}
    if kind == "closure":
        return {"kind": kind, "nx": rng.randint(24, 180), "ny": rng.randint(12, 96),
                "nz": rng.randint(12, 96), "balls": rng.randint(2, 8),
                "fraction_feature": rng.random() < 0.7, "what": rng.choice(["step", "corrections"])}
    return {"kind": kind, "rows": 65536, "batch": 128 * _log(rng, 8, 128), "steps": 4}


# ------------------------------------------------------------------- inputs
def _obstacles(case, seed):
    """Walls in y and z, and balls of 4 to 12 cells (less in small channels) up to the fraction."""
    shape = (case["nx"], case["ny"], case["nz"])
    mask = np.zeros(shape, np.int32)
    if case["fraction"] > 0.0:
        top = min(12.0, min(shape) / 6.0)
        mask = scenes.sphere_packing(shape, case["fraction"], top / 3.0, top, seed)[0]
    return np.maximum(mask, scenes.wall_mask(*shape))


def _lattice_inputs(case, seed):
    rng = np.random.default_rng(seed)
    u0 = tuple(float(v) for v in rng.uniform([0.02, -0.005, -0.005], [0.05, 0.005, 0.005]))
    faces = dict(scenes.PERIODIC_FACES)
    if case["faces"]:
        faces["x_left"] = BoundaryConfig("velocity", velocity=(u0[0], 0.0, 0.0),
                                         velocity_update="simultaneous")
        faces["x_right"] = BoundaryConfig("pressure", rho=1.0)
    force = (0.0, 0.0, 0.0) if case["faces"] else (float(rng.uniform(1e-6, 2e-6)), 0.0, 0.0)
    cfg = LBMConfig(nx=case["nx"], ny=case["ny"], nz=case["nz"],
                    viscosity=scenes.viscosity_for_tau(case["tau"]), force=force,
                    initial_velocity=u0, population_storage=case["storage"],
                    collision_arithmetic=case["arithmetic"], **faces)
    return cfg, _obstacles(case, seed)


def _solid_inputs(case, seed):
    """Cubes of 8 jittered particles per cell, set moving: each has a velocity of its own that
    varies over the body, so it deforms from the first substep."""
    rng = np.random.default_rng(seed)
    pos = scenes.random_cubes(case["grid"], case["cubes"], case["edge"], seed)
    per = len(pos) // case["cubes"]
    vel = np.empty_like(pos)
    for b in range(case["cubes"]):
        p = pos[b * per:(b + 1) * per]
        vel[b * per:(b + 1) * per] = (rng.normal(0, 2e-3, 3)
                                      + (p - p.mean(0)) @ rng.normal(0, 1e-3, (3, 3)))
    cfg = MPMConfig(nx=case["grid"], ny=case["grid"], nz=case["grid"], max_particles=len(pos),
                    particles_per_cell=2, dx=1.0, dt=0.1, density=1.5, youngs_modulus=0.05,
                    poisson_ratio=0.3, gravity=(0.0, -2.0e-6, 0.0), boundary_width=3,
                    constitutive_model=case["model"], p2g_mode=case["mode"])
    return cfg, pos, vel.astype(np.float32)


def _coupled_inputs(case, seed):
    """(configuration, mask, positions, Young's modulus or None). The case's layout places the
    bodies; the seed moves them together by part of a cell and sets the inflow and stiffness."""
    if case["scene"] == "bodies":
        rng = np.random.default_rng(seed)
        cfg, mask, pos, young = scenes.coupled_bodies(
            case["nx"], case["ny"], case["nz"], bodies=case["bodies"], cube_edge=case["edge"],
            sphere_radius=case["edge"] / 2.0, inflow=float(rng.uniform(0.04, 0.05)),
            seed=case["layout"])
        pos = (pos + rng.uniform(0.0, 1.0, 3)).astype(np.float32)
        young = (young * rng.uniform(0.8, 1.2)).astype(np.float32)
        # the inlet that stays bounded on long runs
        inlet = dataclasses.replace(cfg.lbm.x_left, velocity_update="simultaneous")
        lbm = dataclasses.replace(cfg.lbm, x_left=inlet, population_storage=case["storage"])
    else:
        rng = np.random.default_rng(seed)
        e = case["edge"]
        lower = [int(rng.integers(6, 10)),
                 int(rng.integers(8, case["ny"] - e - 7)), int(rng.integers(8, case["nz"] - e - 7))]
        pos = scenes.cube_particles(lower, e, 2, rng)
        young = None
        mask = scenes.wall_mask(case["nx"], case["ny"], case["nz"])
        lbm = LBMConfig(nx=case["nx"], ny=case["ny"], nz=case["nz"],
                        viscosity=scenes.viscosity_for_tau(0.6), force=(1.0e-5, 0.0, 0.0),
                        initial_velocity=(float(rng.uniform(0.002, 0.004)), 0.0, 0.0),
                        population_storage=case["storage"], **scenes.PERIODIC_FACES)
        cfg = SimulationConfig(
            num_steps=1000, lbm_dt=1.0, lbm=lbm,
            mpm=MPMConfig(nx=case["nx"], ny=case["ny"], nz=case["nz"], max_particles=len(pos),
                          particles_per_cell=2, dx=1.0, dt=0.1, density=1.5, youngs_modulus=0.05,
                          poisson_ratio=0.3, gravity=(0.0, 0.0, 0.0), boundary_width=3),
            coupling=CouplingConfig(gamma=0.1, mpm_substeps_per_lbm_step=10))
    mpm = dataclasses.replace(cfg.mpm, p2g_mode=case["mode"])
    return dataclasses.replace(cfg, lbm=lbm, mpm=mpm), mask, pos, young


def _batch_inputs(case, seed):
    """Scenes placed by the case's layout; the seed sets their flow, stiffness and a shift."""
    rng = np.random.default_rng(seed)
    items = []
    for cfg, mask, pos, young in scenes.batch_scenes(case["count"], seed=case["layout"],
                                                     storage=case["storage"]):
        u0 = (float(rng.uniform(0.0, 0.02)), 0.0, 0.0)
        cfg = dataclasses.replace(cfg, lbm=dataclasses.replace(cfg.lbm, initial_velocity=u0))
        pos = (pos + rng.uniform(0.0, 0.5, 3)).astype(np.float32)
        items.append((cfg, mask, pos, (young * rng.uniform(0.8, 1.2)).astype(np.float32)))
    return items


def _closure_inputs(case, seed):
    """A fine channel with balls, and a network with the scales of a fitted one."""
    fine, mask, _ = scenes.closure_channel(seed, 2 * case["nx"], 2 * case["ny"], 2 * case["nz"],
                                           balls=case["balls"], rmin=3.0,
                                           rmax=min(12.0, case["ny"] / 4.0, case["nz"] / 4.0))
    rng = np.random.default_rng(seed)
    u0 = (float(rng.uniform(0.01, 0.03)), 0.0, 0.0)
    fine = dataclasses.replace(fine, initial_velocity=u0, force=(1.0e-6, 0.0, 0.0))
    net = closure.ClosureMLP(seed, use_fraction=case["fraction_feature"])
    net.pop_scale, net.force_scale, net.out_scale = 500.0, 2.5e5, 2.0e6
    return fine, mask, net


def _training_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((case["rows"], closure.FEATURES), generator=g, device="cuda")
    x[:, [c for c in range(closure.FEATURES) if c >= 27 * 24 or c % 24 == 23]] = 0.0
    mix = torch.randn((closure.FEATURES, closure.OUT), generator=g, device="cuda") / 25.0
    t = torch.tanh(x @ mix) + 0.1 * torch.randn((case["rows"], closure.OUT), generator=g, device="cuda")
    return x.to(torch.bfloat16), t.contiguous()


# A late, small learning rate: passes repeat on one network, and each has to fit the same one.
LR = 1e-6
WARM = 2  # steps before the measured ones: the flow has met the obstacles and the bodies move


def prepare(case, seed):
    kind = case["kind"]
    if kind == "lattice":
        cfg, mask = _lattice_inputs(case, seed)
        s = LBMSolver3D(cfg)
        s.initialize(mask)
        for _ in range(WARM):
            s.step()
        return {"case": case, "lbm": s}
    if kind == "solid":
        cfg, pos, vel = _solid_inputs(case, seed)
        s = MPMSolver3D(cfg)
        s.initialize_particles_from_numpy(pos, vel)
        return {"case": case, "mpm": s}
    if kind == "coupled":
        cfg, mask, pos, young = _coupled_inputs(case, seed)
        sim = FSISimulation(cfg)
        sim.initialize_lbm(mask)
        if young is None:
            sim.initialize_mpm_from_numpy(pos)
        else:
            sim.initialize_mpm_from_numpy(pos, youngs_modulus=young, poisson_ratio=0.3)
        for _ in range(WARM):
            sim.coupler.step(cfg.lbm_dt)
        return {"case": case, "sim": sim}
    if kind == "batch":
        items = _batch_inputs(case, seed)
        b = SceneBatch([i[0] for i in items])
        b.initialize([i[1] for i in items], [i[2] for i in items], [i[3] for i in items])
        return {"case": case, "batch": b}
    if kind == "closure":
        fine, mask, net = _closure_inputs(case, seed)
        sim = closure.ClosureSimulation(fine, mask, net)
        sim.coarse.step()
        return {"case": case, "sim": sim, "corr": None}
    x, t = _training_inputs(case, seed)
    trainer = closure.ClosureTrainer(closure.ClosureMLP(seed))
    trainer.x, trainer.t = x, t
    return {"case": case, "trainer": trainer}


# ------------------------------------------------------------------- a pass
def _solid_state(mpm):
    return {"x": mpm._x, "v": mpm._v, "C": mpm._C, "F": mpm._F}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "lattice":
        lbm = state["lbm"]
        for _ in range(case["steps"]):
            lbm.step()
        return {"macro": lbm.macro}
    if kind == "solid":
        mpm = state["mpm"]
        for _ in range(case["substeps"]):
            mpm.substep()
        return _solid_state(mpm)
    if kind == "coupled":
        sim = state["sim"]
        if case["advance"]:
            sim.advance(case["advance"])
            diag = {}
        else:
            diag = sim.step()
        return {"macro": sim.lbm.macro, "force": sim.lbm.force, "diag": diag,
                **_solid_state(sim.mpm)}
    if kind == "batch":
        b = state["batch"]
        b.run(case["steps"])
        return {"macro": b.lattice.macro, "x": b._x, "v": b._v, "C": b._C, "F": b._F}
    if kind == "closure":
        sim = state["sim"]
        if case["what"] == "step":
            sim.step()
            return {"macro": sim.coarse.macro}
        c = sim.coarse
        c.step()
        if state["corr"] is None:
            state["corr"] = torch.zeros((closure.OUT, c.n_cells), dtype=torch.float32, device="cuda")
        closure.infer(c, sim._weights, state["corr"], sim._rows, sim.net.err, sim._frac)
        return {"corr": state["corr"], "macro": c.macro}
    trainer = state["trainer"]
    loss = trainer.fit(steps=case["steps"], batch=case["batch"], lr=LR)
    return {"loss": np.array(loss, np.float32), "grads": trainer.net.grads, "params": trainer.net.params}


# ----------------------------------------------------- what a pass has to do
def _particles(case):
    """Particles and touched grid nodes, from the sizes alone (balls fill 0.52 of their cube)."""
    if case["kind"] == "solid":
        return 8 * case["cubes"] * case["edge"] ** 3, case["cubes"] * (case["edge"] + 3) ** 3
    share = 1.0 if case["scene"] == "smoke" else 0.76
    return (8 * share * case["bodies"] * case["edge"] ** 3,
            share * case["bodies"] * (case["edge"] + 3) ** 3)


def work(case):
    """Per lattice step and cell: 19 populations read and written, the force and the flags read,
    and (once a pass) rho and u written; about 500 operations. Per particle and substep: x, v, C,
    F read and written, mass, volume read; per touched node 32 bytes; about 2,500 operations."""
    kind = case["kind"]

    def lattice(cells, steps, storage):
        pop = 4 if storage == "f32" else 2
        return cells * (steps * (38 * pop + 12 + 4) + 16), cells * steps * 500.0

    def solid(p, nodes, substeps, coupled):
        per = 24 * 4 * 2 + 8 + (24 if coupled else 0)
        return substeps * (p * per + nodes * 32), substeps * p * (3500.0 if coupled else 2500.0)

    if kind == "lattice":
        cells = case["nx"] * case["ny"] * case["nz"] * (1.0 - case["fraction"])
        b, f = lattice(cells, case["steps"], case["storage"])
    elif kind == "solid":
        b, f = solid(*_particles(case), case["substeps"], False)
    elif kind == "coupled":
        steps = case["advance"] or 1
        b, f = lattice(case["nx"] * case["ny"] * case["nz"], steps, case["storage"])
        bs, fs = solid(*_particles(case), 10 * steps, True)
        b, f = b + bs, f + fs
    elif kind == "batch":
        # edges 32, 48, 64, 96 equally often; 2.5 bodies of 7 cells (balls have that radius)
        cells = case["count"] * (32 ** 3 + 48 ** 3 + 64 ** 3 + 96 ** 3) / 4.0
        b, f = lattice(cells, case["steps"], case["storage"])
        p = case["count"] * 2.5 * 8 * 1000.0
        bs, fs = solid(p, p / 4, 10 * case["steps"], True)
        b, f = b + bs, f + fs
    elif kind == "closure":
        cells = case["nx"] * case["ny"] * case["nz"]
        b, f = lattice(cells, 1, "f32")
        b, f = b + cells * 152, f + cells * 104448.0
    else:
        m, n = case["batch"], 656 * 64 + 2 * 64 * 64 + 64 * 32
        b = case["steps"] * (m * (656 * 2 + 19 * 4) + n * 28)
        f = case["steps"] * m * (6.0 * n - 2.0 * 656 * 64)
    return {"bytes": float(b), "flops": float(f)}


# -------------------------------------------------- the same in float64 torch
_E = torch.tensor([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
                   (1, 1, 0), (-1, -1, 0), (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1),
                   (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1)])
_OPP = [0] + [q + 1 if q % 2 else q - 1 for q in range(1, 19)]


class _Lattice:
    """D3Q19 multiple-relaxation-time lattice with Guo forcing, populations [19, nx, ny, nz]."""

    def __init__(self, cfg, mask):
        self.cfg = cfg
        dev = "cuda"
        self.e = _E.to(dev, F64)
        self.w = torch.tensor([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12, dtype=F64, device=dev)
        x, y, z = self.e.T
        c2 = (self.e ** 2).sum(1)
        # moments by their defining polynomials: density, energy, energy squared, momenta and heat
        # fluxes, normal stresses and their fourth-order companions, shear stresses, third order
        far = (c2 == 2).to(F64)
        near = (c2 == 1).to(F64)
        rest = (c2 == 0).to(F64)
        flux = far - 2.0 * near
        rows = [torch.ones_like(x), far - rest, rest - 2.0 * near + far, x, x * flux, y, y * flux, z,
                z * flux, 3 * x * x - c2, (3 * x * x - c2) * (far - near), y * y - z * z,
                (y * y - z * z) * (far - near), x * y, y * z, x * z, x * (y * y - z * z),
                y * (z * z - x * x), z * (x * x - y * y)]
        self.m = torch.stack(rows)
        self.inv = torch.linalg.inv(self.m)
        sv = 1.0 / (3.0 * cfg.viscosity + 0.5)
        so = 8.0 * (2.0 - sv) / (8.0 - sv)
        self.s = torch.tensor([0, sv, sv, 0, so, 0, so, 0, so, sv, sv, sv, sv, sv, sv, sv, so, so,
                               so], dtype=F64, device=dev).view(19, 1)
        self.solid = torch.from_numpy(np.asarray(mask) > 0).to(dev)
        self.shape = tuple(self.solid.shape)
        u0 = torch.tensor(np.float32(cfg.initial_velocity), device=dev).to(F64)
        self.u = (u0.view(3, 1, 1, 1) * (~self.solid)).contiguous()
        self.rho = torch.full(self.shape, float(cfg.rho0), dtype=F64, device=dev)
        self.f = self.equilibrium(self.rho, self.u)
        self.base = torch.tensor(np.float32(cfg.force), device=dev).to(F64).view(3, 1, 1, 1)
        self.force = (self.base * (~self.solid)).contiguous()

    def equilibrium(self, rho, u):
        eu = torch.tensordot(self.e, u, 1)
        w = self.w.view(19, *([1] * (u.dim() - 1)))
        return w * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * (u * u).sum(0))

    def collide(self):
        out = torch.empty_like(self.f)
        n = self.shape[0]
        for a in range(0, n, max(1, 2 ** 21 // (self.shape[1] * self.shape[2]))):
            b = min(n, a + max(1, 2 ** 21 // (self.shape[1] * self.shape[2])))
            f = self.f[:, a:b].reshape(19, -1)
            u = self.u[:, a:b].reshape(3, -1)
            g = self.force[:, a:b].reshape(3, -1)
            ug = (u * g).sum(0)
            eg = self.e @ g
            t = self.w.view(19, 1) * (eg - ug + (self.e @ u) * eg)
            m = self.m @ f
            eq = torch.zeros_like(m)
            ux, uy, uz = u
            eq[1] = ux * ux + uy * uy + uz * uz
            eq[9] = 2 * ux * ux - uy * uy - uz * uz
            eq[11] = uy * uy - uz * uz
            eq[13], eq[14], eq[15] = ux * uy, uy * uz, ux * uz
            m = m - self.s * (m - eq) * (self.s != 0) + (1 - 0.5 * self.s) * (self.m @ t)
            out[:, a:b] = (self.inv @ m).reshape(19, b - a, *self.shape[1:])
        return out

    def step(self):
        post = self.collide()
        new = torch.empty_like(post)
        for q in range(19):
            d = tuple(int(v) for v in _E[q])
            moved = torch.roll(post[q], d, (0, 1, 2))
            from_solid = torch.roll(self.solid, d, (0, 1, 2))
            new[q] = torch.where(from_solid, post[_OPP[q]], moved)
        self.f = torch.where(self.solid, self.f, new)
        for side, face in ((0, self.cfg.x_left), (self.shape[0] - 1, self.cfg.x_right)):
            if face.boundary_type == "periodic":
                continue
            old = self.f[:, side]
            if face.boundary_type == "pressure":
                inner = self.solid[side + 1 if side == 0 else side - 1]
                set_to = self.equilibrium(torch.full_like(self.rho[side], face.rho),
                                          self.u[:, side] * (~inner))
            else:
                v = torch.tensor(np.float32(face.velocity), device="cuda").to(F64).view(3, 1, 1)
                eq = self.equilibrium(torch.full_like(self.rho[side], float(self.cfg.rho0)),
                                      v.expand(3, *self.shape[1:]))
                set_to = eq + eq[_OPP] - old[_OPP]
            self.f[:, side] = torch.where(self.solid[side], old, set_to)
        self.refresh()

    def refresh(self):
        rho = self.f.sum(0)
        u = (torch.tensordot(self.e.T.contiguous(), self.f, 1) + 0.5 * self.force) / rho
        self.rho = torch.where(self.solid, torch.full_like(rho, float(self.cfg.rho0)), rho)
        self.u = torch.where(self.solid, torch.zeros_like(u), u)

    def macro(self):
        return torch.cat([self.u, self.rho[None]]).reshape(4, -1).T.contiguous()


def _rotation(F):
    """The rotation of F = R S by Newton's iteration (det F > 0)."""
    X = F.clone()
    for _ in range(30):
        X = 0.5 * (X + torch.linalg.inv(X).mT)
    return X


class _Solid:
    """MLS-MPM with APIC, particles [n, ...], optionally coupled to a _Lattice by a penalty force."""

    def __init__(self, cfg, pos, vel=None, young=None):
        dev = "cuda"
        self.cfg = cfg
        n = len(pos)
        self.x = torch.from_numpy(np.asarray(pos, np.float32)).to(dev, F64)
        self.v = (torch.zeros_like(self.x) if vel is None
                  else torch.from_numpy(np.asarray(vel, np.float32)).to(dev, F64))
        self.C = torch.zeros((n, 3, 3), dtype=F64, device=dev)
        self.F = torch.eye(3, dtype=F64, device=dev).expand(n, 3, 3).contiguous()
        self.vol = cfg.dx ** 3 / cfg.particles_per_cell ** 3
        self.mass = cfg.density * self.vol
        E = torch.full((n,), cfg.youngs_modulus, dtype=F64, device=dev)
        if young is not None:
            E = torch.from_numpy(np.asarray(young, np.float64)).to(dev)
        nu = cfg.poisson_ratio
        self.mu = (E / (2 * (1 + nu))).view(n, 1, 1)
        self.lam = (E * nu / ((1 + nu) * (1 - 2 * nu))).view(n, 1, 1)
        self.shape = (cfg.nx, cfg.ny, cfg.nz)
        self.fp = torch.zeros_like(self.x)

    def stencil(self):
        """Nodes [n, 27], whether inside, weights [n, 27] and offsets from the particle [n, 27, 3]."""
        g = self.x / self.cfg.dx
        base = torch.trunc(g - 0.5).to(torch.int64)
        fx = g - base
        w = torch.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2], 1)
        o = torch.tensor([(i, j, k) for i in range(3) for j in range(3) for k in range(3)],
                         device="cuda")
        wt = w[:, o[:, 0], 0] * w[:, o[:, 1], 1] * w[:, o[:, 2], 2]
        ijk = base[:, None] + o
        size = torch.tensor(self.shape, device="cuda")
        inside = ((ijk >= 0) & (ijk < size)).all(2)
        ijk = torch.minimum(ijk.clamp(min=0), size - 1)
        node = (ijk[..., 0] * self.shape[1] + ijk[..., 1]) * self.shape[2] + ijk[..., 2]
        return node, inside, wt * inside, o - fx[:, None]

    def couple(self, lat, gamma, ratio, accum, build):
        node, inside, w, _ = self.stencil()
        usable = inside & ~lat.solid.reshape(-1)[node]
        w = w * usable
        valid = w.sum(1)
        u = torch.stack([(w * lat.u[a].reshape(-1)[node]).sum(1) for a in range(3)], 1)
        ok = valid > 1e-6
        self.fp = torch.where(ok[:, None], gamma * self.mass * (u / valid[:, None] - self.v),
                              torch.zeros_like(u))
        nw = torch.where(ok[:, None], w / valid[:, None], torch.zeros_like(w))
        flat = node.reshape(-1)
        for a in range(3):
            accum[a].index_add_(0, flat, (-nw * self.fp[:, a:a + 1] * ratio).reshape(-1))
        if build:
            accum[3].index_add_(0, flat, (nw * self.vol).reshape(-1))

    def substep(self, dt):
        cfg = self.cfg
        eye = torch.eye(3, dtype=F64, device="cuda")
        self.F = (eye + dt * self.C) @ self.F
        J = torch.linalg.det(self.F).view(-1, 1, 1)
        if cfg.constitutive_model == "neo_hookean":
            tau = self.mu * (self.F @ self.F.mT - eye) + self.lam * torch.log(J) * eye
        else:
            tau = 2 * self.mu * (self.F - _rotation(self.F)) @ self.F.mT + self.lam * J * (J - 1) * eye
        A = -dt * self.vol * 4.0 / cfg.dx ** 2 * tau + self.mass * self.C
        node, inside, w, d = self.stencil()
        n = self.shape[0] * self.shape[1] * self.shape[2]
        flat = node.reshape(-1)
        gm = torch.zeros(n, dtype=F64, device="cuda").index_add_(0, flat, (w * self.mass).reshape(-1))
        gv = []
        for a in range(3):
            p = w * ((self.mass * self.v[:, a] + dt * self.fp[:, a])[:, None]
                     + cfg.dx * (d @ A[:, a, :, None])[..., 0])
            gv.append(torch.zeros_like(gm).index_add_(0, flat, p.reshape(-1)))
        gv = torch.stack(gv)
        live = gm > 0
        grav = torch.tensor(np.float32(cfg.gravity), device="cuda").to(F64).view(3, 1)
        gv = torch.where(live, gv / gm.clamp(min=1e-300) + dt * grav, gv)
        gv = gv.view(3, *self.shape)
        bw = cfg.boundary_width
        for a in range(3):
            lo, hi = gv[a].narrow(a, 0, bw), gv[a].narrow(a, self.shape[a] - bw, bw)
            lo.copy_(torch.where(lo < 0, -cfg.boundary_damping * lo, lo))
            hi.copy_(torch.where(hi > 0, -cfg.boundary_damping * hi, hi))
        got = torch.stack([gv[a].reshape(-1)[node] for a in range(3)], 2) * w[..., None]
        self.v = got.sum(1)
        self.C = 4.0 / cfg.dx * torch.einsum("pna,pnb->pab", got, d)
        if not cfg.apic:
            self.C = torch.zeros_like(self.C)
        top = torch.tensor([(s - 1.5) * cfg.dx for s in self.shape], dtype=F64, device="cuda")
        self.x = torch.minimum((self.x + dt * self.v).clamp(min=0.5 * cfg.dx), top)

    def state(self):
        n = len(self.x)
        return {"x": self.x.T.contiguous(), "v": self.v.T.contiguous(),
                "C": self.C.reshape(n, 9).T.contiguous(), "F": self.F.reshape(n, 9).T.contiguous()}


def _coupled_step(lat, sol, cfg):
    n = lat.solid.numel()
    accum = torch.zeros((4, n), dtype=F64, device="cuda")
    subs = cfg.coupling.mpm_substeps_per_lbm_step
    for s in range(subs):
        sol.couple(lat, cfg.coupling.gamma, 1.0 / subs, accum, s == 0)
        sol.substep(cfg.lbm_dt / subs)
    lat.force = ((lat.base + accum[:3].view(3, *lat.shape)) * (~lat.solid)).contiguous()
    lat.step()
    return accum


def _network(net, feats):
    """The network's outputs for features [n, 656] with the float32 parameters."""
    W1, b1, W2, b2, W3, b3, W4, b4 = (v.to(F64) for v in net.views)

    def act(z):
        return 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))

    h = act(act(act(feats @ W1.T + b1) @ W2.T + b2) @ W3.T + b3)
    return (h @ W4.T + b4)[:, :19]


def _corrections(lat, net, frac):
    """[19, N] corrections of a coarse lattice's state."""
    fluid = ~lat.solid
    rows = torch.zeros((*lat.shape, 24), dtype=F64, device="cuda")
    dev = (lat.f - (lat.w * float(lat.cfg.rho0)).view(19, 1, 1, 1)) * net.pop_scale * fluid
    rows[..., :19] = dev.permute(1, 2, 3, 0)
    rows[..., 19] = lat.solid.to(F64) if frac is None else frac.to(F64).view(lat.shape)
    rows[..., 20:23] = (lat.force * net.force_scale).permute(1, 2, 3, 0)
    out = torch.empty((19, *lat.shape), dtype=F64, device="cuda")
    for i in range(lat.shape[0]):
        planes = rows[[(i + d) % lat.shape[0] for d in (-1, 0, 1)]]
        cols = [torch.roll(planes[dx + 1], (-dy, -dz), (0, 1)).reshape(-1, 24)
                for dx in (-1, 0, 1) for dy in (-1, 0, 1) for dz in (-1, 0, 1)]
        feats = torch.cat(cols + [torch.zeros_like(cols[0][:, :8])], 1)
        out[:, i] = _network(net, feats).T.reshape(19, *lat.shape[1:]) / net.out_scale
    return out * fluid


def _fit(case, seed):
    x, t = _training_inputs(case, seed)
    net = closure.ClosureMLP(seed)
    params = net.params.to(F64).clone().requires_grad_(True)
    sizes = [tuple(v.shape) for v in net.views]
    m = torch.zeros_like(params)
    v = torch.zeros_like(params)
    g = torch.Generator(device="cpu").manual_seed(0)
    batch = max(128, min(case["batch"], case["rows"]) // 128 * 128)
    losses = []
    grads = None
    for it in range(case["steps"]):
        idx = torch.randint(0, case["rows"], (batch,), generator=g).cuda()
        parts, off = [], 0
        for s in sizes:
            k = math.prod(s)
            parts.append(params[off:off + k].view(s))
            off += k
        holder = type("N", (), {"views": parts})
        e = _network(holder, x[idx].to(F64)) - t[idx].to(F64)
        loss = (e * e).mean()
        (grads,) = torch.autograd.grad(loss, params)
        losses.append(loss.item())
        with torch.no_grad():
            m = 0.9 * m + 0.1 * grads
            v = 0.999 * v + 0.001 * grads * grads
            lr = LR * 0.5 ** (it / case["steps"] * 3.0)
            params -= lr * (m / (1 - 0.9 ** (it + 1))) / (torch.sqrt(v / (1 - 0.999 ** (it + 1))) + 1e-8)
    return {"loss": np.array(losses), "grads": grads.detach(), "params": params.detach()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "lattice":
        lat = _Lattice(*_lattice_inputs(case, seed))
        for _ in range(WARM + case["steps"]):
            lat.step()
        return {"macro": lat.macro()}
    if kind == "solid":
        cfg, pos, vel = _solid_inputs(case, seed)
        sol = _Solid(cfg, pos, vel)
        for _ in range(case["substeps"]):
            sol.substep(cfg.dt)
        return sol.state()
    if kind == "coupled":
        cfg, mask, pos, young = _coupled_inputs(case, seed)
        lat, sol = _Lattice(cfg.lbm, mask), _Solid(cfg.mpm, pos, young=young)
        accum = None
        for _ in range(WARM + (case["advance"] or 1)):
            accum = _coupled_step(lat, sol, cfg)
        diag = {}
        if not case["advance"]:
            fluid = ~lat.solid
            reaction = accum[:3] * fluid.reshape(-1)
            diag = {"lbm_total_mass": float(lat.rho[fluid].sum()),
                    "lbm_max_velocity_norm": float(torch.linalg.vector_norm(lat.u, dim=0).max()),
                    "mpm_center_of_mass": sol.x.mean(0),
                    "mpm_max_velocity_norm": float(torch.linalg.vector_norm(sol.v, dim=1).max()),
                    "total_particle_coupling_force": sol.fp.sum(0),
                    "total_fluid_coupling_force": reaction.sum(1)}
        return {"macro": lat.macro(), "force": lat.force.reshape(3, -1), "diag": diag,
                **sol.state()}
    if kind == "batch":
        items = _batch_inputs(case, seed)
        macro, parts = [], {k: [] for k in "xvCF"}
        for cfg, mask, pos, young in items:
            lat, sol = _Lattice(cfg.lbm, mask), _Solid(cfg.mpm, pos, young=young)
            for _ in range(case["steps"]):
                _coupled_step(lat, sol, cfg)
            macro.append(lat.macro())
            pad = -len(pos) % 256  # each scene's particles start at a multiple of 256
            for k, t in sol.state().items():
                parts[k].append(torch.nn.functional.pad(t, (0, pad)))
        return {"macro": torch.cat(macro), **{k: torch.cat(p, 1) for k, p in parts.items()}}
    if kind == "closure":
        fine, mask, net = _closure_inputs(case, seed)
        solid = np.asarray(mask) > 0
        share = solid.reshape(case["nx"], 2, case["ny"], 2, case["nz"], 2).mean((1, 3, 5))
        frac = torch.from_numpy(share).cuda() if case["fraction_feature"] else None
        cfg = dataclasses.replace(fine, nx=case["nx"], ny=case["ny"], nz=case["nz"],
                                  viscosity=fine.viscosity / 2,
                                  force=tuple(2.0 * g for g in fine.force))
        lat = _Lattice(cfg, (share >= 0.5).astype(np.int32))
        lat.step()
        lat.step()
        corr = _corrections(lat, net, frac)
        if case["what"] == "corrections":
            return {"corr": corr.reshape(19, -1), "macro": lat.macro()}
        lat.f += corr - lat.w.view(19, 1, 1, 1) * corr.sum(0)
        lat.refresh()
        return {"macro": lat.macro()}
    return _fit(case, seed)
