"""A NaN density reaches the Tillotson cold-energy lookup as a NaN and not as an index out of its
range: the cycle completes, the result is non-finite where it has to be and the handle stays usable."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))
import make_golden  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_nan_density_stays_inside_the_cold_energy_curve(cuda_device, precision):
    import trajectory
    rec, _ = make_golden.load()
    sim = trajectory.simulation_from_record(rec, precision=precision)
    assert sim.check() == 0
    vof, den = sim.get_field("m_vof"), sim.get_field("m_den")
    j, i = np.argwhere(vof[2:-2, 2:-2, 1] > 0.5)[0] + 2
    den[j, i, 1] = np.nan
    sim.set_field("m_den", den)
    sim.step(2)
    assert sim.check() > 0
    assert np.isnan(sim.get_field("m_den")[j, i, 1])
    sim.close()
