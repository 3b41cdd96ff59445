"""A tuner record stored for kernels whose variants meant something else is not applied (no GPU): the
cache key holds the launch set beside the GPU and the sizes."""
from __future__ import annotations

import hashlib
import json
from types import SimpleNamespace

from fsi import autotune


def test_records_of_an_earlier_launch_set_are_not_found(monkeypatch):
    monkeypatch.setattr(autotune.torch.cuda, "get_device_name", lambda *a: "GB300 (fake)")
    form = SimpleNamespace(population_storage="f16", resolved_arithmetic=lambda: "fast")
    batch = SimpleNamespace(configs=[form], shapes=[(8, 8, 8)])
    lbm = SimpleNamespace(nx=8, ny=8, nz=8, population_storage="f16")
    sim = SimpleNamespace(config=SimpleNamespace(lbm=lbm, mpm=SimpleNamespace(p2g_mode="atomic")),
                          mpm=SimpleNamespace(particle_count=lambda: 1))
    for sign, subject, without in (
            (autotune._signature, batch, ["GB300 (fake)", "f16", "fast", [(8, 8, 8)]]),
            (autotune.coupled_signature, sim, ["GB300 (fake)", "coupled", [8, 8, 8], 1, "atomic", "f16"])):
        key = sign(subject)
        assert key != hashlib.sha1(json.dumps(without).encode()).hexdigest()
        monkeypatch.setattr(autotune, "LAUNCH_SET", autotune.LAUNCH_SET + 1)
        assert sign(subject) != key
