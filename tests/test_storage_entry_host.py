"""The coupled substep that is told the lattice's storage refuses one that is none (no GPU)."""
from __future__ import annotations

import pytest

from fsi import _native as nat


@pytest.mark.parametrize("storage", [-1, 3])
def test_unknown_storage_is_refused(storage):
    with pytest.raises(ValueError, match="unknown storage"):
        nat.call("fsi_coupled_substep_tiled_storage", storage, nat.CouplingDesc(), nat.MpmDesc(), nat.Particles(),
                 *[None] * 9)
