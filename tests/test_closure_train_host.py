"""ClosureTrainer.fit refuses a data set that the training step, which reads rows by number on the
device, would read out of range or as another type (no GPU)."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

from fsi import closure as cl

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


@pytest.mark.parametrize("x,t,device,what", [
    ((256, 656, BF16), (255, 19, F32), "cpu", "targets"),
    ((256, 656, BF16), (256, 20, F32), "cpu", "targets"),
    ((256, 656, BF16), (256, 19, F64), "cpu", "targets"),
    ((256, 656, F32), (256, 19, F32), "cpu", "feature rows"),
    ((256, 648, BF16), (256, 19, F32), "cpu", "feature rows"),
    ((0, 656, BF16), (0, 19, F32), "cpu", "feature rows"),
    ((256, 656, BF16), (256, 19, F32), "meta", "the network on"),
])
def test_fit_rejects_rows_that_the_step_would_misread(x, t, device, what):
    trainer = cl.ClosureTrainer(SimpleNamespace(params=torch.empty(1, device=device)))
    trainer.x, trainer.t = torch.zeros(x[:2], dtype=x[2]), torch.zeros(t[:2], dtype=t[2])
    with pytest.raises(ValueError, match=what):
        trainer.fit(steps=1, batch=128)
