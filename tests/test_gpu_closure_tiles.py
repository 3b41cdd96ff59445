"""The fused inference where its blocks' tiles can go wrong: fewer plane steps than blocks, one
column alone, blocks that cross columns after one, two and many plane steps (even and odd tiles are
issued by two threads and share the planes), ragged columns. Against the unfused passes, with the
tolerance of the small-lattice comparison (bfloat16 activations that round apart)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from fsi import closure as cl
from fsi.config import LBMConfig
from fsi.lbm3d import LBMSolver3D
from helpers import PERIODIC, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 12, 33), (40, 11, 32), (5, 122, 321), (160, 34, 63)])
def test_tiles_match_unfused_passes(shape):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx)
    lbm = LBMSolver3D(LBMConfig(nx=nx, ny=ny, nz=nz, viscosity=0.05, force=(1e-4, 2e-5, 0.0), **PERIODIC))
    lbm.initialize((rng.uniform(size=shape) < 0.1).astype(np.int32))
    for _ in range(3):
        lbm.step()
    net = cl.ClosureMLP(seed=3)
    net.pop_scale, net.force_scale, net.out_scale = 30.0, 1e3, 250.0
    corr = torch.zeros((19, lbm.n_cells), dtype=torch.float32, device="cuda")
    cl.infer(lbm, net.weights_struct(), corr, cl.rows_buffer(lbm), net.err)
    net.check()
    cells = np.sort(rng.choice(lbm.n_cells, min(lbm.n_cells, 65536), replace=False))
    ids = torch.from_numpy(cells.astype(np.int32)).cuda()
    x = cl.features(lbm, ids, net.pop_scale, net.force_scale)
    x = torch.cat([x, torch.zeros(((-len(cells)) % 128, 656), dtype=x.dtype, device="cuda")])
    y = net.predict(x)[:len(cells)] / net.out_scale
    solid = torch.from_numpy(lbm.solid_numpy().reshape(-1)[cells] > 0).cuda()
    got = corr[:, ids.long()].t()
    assert float(got[solid].abs().max()) == 0.0
    assert rel_l2(got[~solid].cpu().numpy(), y[~solid].cpu().numpy()) < 2e-3
