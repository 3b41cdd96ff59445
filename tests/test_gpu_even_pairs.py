"""The even step by pairs of neighbours in memory (fast forms, an even number of cells, aligned
arrays) against the even step by rows, which the same call takes when the force array starts in the
middle of a pair: every operation is rounded on its own in both, so the populations, and rho and u
where faces ask for them, are equal. Rows of odd and even length (pairs that straddle rows), one
block and several, solid cells on either side of a pair, faces, rho and u read and recomputed."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from fsi import _native as nat
from fsi.batch import LatticeBatch
from fsi.config import BoundaryConfig, LBMConfig
from fsi.lbm3d import LBMSolver3D
from helpers import PERIODIC

pytestmark = pytest.mark.gpu


SHAPES = [(6, 8, 10), (8, 5, 7), (16, 13, 33), (5, 6, 5)]


def _config(shape, storage, faces=False):
    kw = dict(PERIODIC)
    if faces:
        kw["x_left"] = BoundaryConfig("velocity", velocity=(1e-3, 0.0, 0.0))
        kw["x_right"] = BoundaryConfig("pressure", rho=1.0)
    return LBMConfig(nx=shape[0], ny=shape[1], nz=shape[2], viscosity=0.05, force=(1e-4, 2e-5, -1e-5),
                     initial_velocity=(1e-3, 0.0, 0.0), population_storage=storage,
                     collision_arithmetic="fast", **kw)


def _mid_pair(t):
    """A copy of t that starts four bytes after an 8-byte boundary."""
    out = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:]
    out.copy_(t.reshape(-1))
    assert out.data_ptr() % 8 == 4
    return out


def _both_ways(call, pops, macro, force, prev):
    """The state after an even step by pairs and by rows."""
    out = []
    for f in (force, _mid_pair(force)):
        p, m = pops.clone(), macro.clone()
        call(p, m, f, prev)
        out.append((p, m))
    return out


@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
def test_pairs_equal_rows(shape, storage, recompute):
    rng = np.random.default_rng(shape[2])
    faces = recompute
    lbm = LBMSolver3D(_config(shape, storage, faces))
    lbm.initialize((rng.uniform(size=shape) < 0.3).astype(np.int32))
    for _ in range(4):
        lbm.step()
    lbm._ensure_macro()
    force = lbm._force_buf[lbm._fcur]
    prev = force.clone() if recompute else None

    def call(p, m, f, fp):
        lbm._call("fsi_lbm_step", nat.ptr(p), nat.ptr(m), nat.ptr(f), nat.ptr(fp), nat.ptr(lbm._flags), 4,
                  nat.stream_ptr())

    (p0, m0), (p1, m1) = _both_ways(call, lbm._pops, lbm._macro, force, prev)
    assert not torch.equal(p0, lbm._pops)
    assert torch.equal(p0, p1) and torch.equal(m0, m1)


@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
def test_batch_pairs_equal_rows(storage, recompute):
    rng = np.random.default_rng(3)
    batch = LatticeBatch([_config(s, storage) for s in SHAPES])
    batch.initialize([(rng.uniform(size=s) < 0.3).astype(np.int32) for s in SHAPES])
    for _ in range(4):
        batch.step()
    batch._ensure_macro()
    force = batch._force_buf[batch._fcur]
    prev = force.clone() if recompute else None

    def call(p, m, f, fp):
        nat.call("fsi_batch_lbm_step", batch._handle, nat.ptr(p), nat.ptr(m), nat.ptr(f), nat.ptr(fp),
                 nat.ptr(batch._flags), 4, nat.stream_ptr())

    (p0, m0), (p1, m1) = _both_ways(call, batch._pops, batch._macro, force, prev)
    assert not torch.equal(p0, batch._pops)
    assert torch.equal(p0, p1) and torch.equal(m0, m1)


@pytest.mark.parametrize("steps", [4, 5])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
def test_macro_pairs_equal_cells(shape, storage, steps):
    """rho and u by pairs in both states of the populations; the diagnostic sums are float32 within a
    warp (32 terms of either path, 32 u = 2e-6) and float64 across warps."""
    rng = np.random.default_rng(shape[2])
    lbm = LBMSolver3D(_config(shape, storage))
    lbm.initialize((rng.uniform(size=shape) < 0.3).astype(np.int32))
    for _ in range(steps):
        lbm.step()
    force = lbm._force_buf[lbm._fcur]
    out = []
    for f in (force, _mid_pair(force)):
        m, diag = torch.full_like(lbm._macro, -1.0), torch.zeros(2, dtype=torch.float64, device="cuda")
        plain = m.clone()
        lbm._call("fsi_lbm_update_macro", nat.ptr(lbm._pops), nat.ptr(f), nat.ptr(lbm._flags), steps,
                  nat.ptr(plain), nat.stream_ptr())
        lbm._call("fsi_lbm_macro_diagnostics", nat.ptr(lbm._pops), nat.ptr(f), nat.ptr(lbm._flags), steps,
                  nat.ptr(m), nat.ptr(diag), nat.stream_ptr())
        assert torch.equal(m, plain)
        out.append((m, diag))
    (m0, d0), (m1, d1) = out
    assert torch.equal(m0, m1)
    assert d0[1] == d1[1] and abs(d0[0] / d1[0] - 1) < 4e-6


@pytest.mark.parametrize("steps", [4, 5])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
def test_batch_macro_pairs_equal_cells(storage, steps):
    rng = np.random.default_rng(3)
    batch = LatticeBatch([_config(s, storage) for s in SHAPES])
    batch.initialize([(rng.uniform(size=s) < 0.3).astype(np.int32) for s in SHAPES])
    for _ in range(steps):
        batch.step()
    force = batch._force_buf[batch._fcur]
    out = []
    for f in (force, _mid_pair(force)):
        m = torch.full_like(batch._macro, -1.0)
        diag = torch.zeros((len(SHAPES), 2), dtype=torch.float64, device="cuda")
        nat.call("fsi_batch_lbm_macro", batch._handle, nat.ptr(batch._pops), nat.ptr(f), nat.ptr(batch._flags),
                 steps, nat.ptr(m), nat.ptr(diag), nat.stream_ptr())
        out.append((m, diag))
    (m0, d0), (m1, d1) = out
    assert torch.equal(m0, m1)
    assert torch.equal(d0[:, 1], d1[:, 1]) and float((d0[:, 0] / d1[:, 0] - 1).abs().max()) < 4e-6
