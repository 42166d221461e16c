"""Phase 4 run by itself depends on what the reference's check_v_vel reads (e_wpt, e_den, e_vel) and not
on the corner count that phase 1 leaves in v_mass: the state before it may be one a caller put together."""
import numpy as np
import pytest
from test_cycle_graph_gpu import _deck

from salec_b200 import capi, decks


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_phase_4_counts_the_void_corners(cuda_device, tmp_path, precision):
    path = decks.write_deck(_deck("base"), str(tmp_path))
    whole, alone = (capi.Simulation.from_deck(path, str(tmp_path), precision=precision) for _ in range(2))
    moved = 0
    for _ in range(12):
        for sim in (whole, alone):
            sim.step(3)
            sim.phases(0, 3)
        before, mass = whole.get_field("v_vel"), alone.get_field("v_mass")
        alone.set_field("v_mass", np.concatenate([mass[..., :1], np.zeros_like(mass[..., 1:])], axis=-1))
        for sim in (whole, alone):
            sim.phases(4, 4)
        after = whole.get_field("v_vel")
        assert np.array_equal(alone.get_field("v_vel"), after)
        moved += int((after != before).any(axis=-1).sum())
        alone.set_field("v_mass", mass)
        for sim in (whole, alone):
            sim.phases(5, 15)
    assert moved > 0   # phase 4 had vertices to correct
    whole.close()
    alone.close()
