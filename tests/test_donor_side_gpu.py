"""The side of a face that the cycle graph's remap takes the donor from is the side the flux left,
also where the material volumes do not all have its sign: a NaN fraction (NaN volumes beside finite
ones) and negative fractions that a caller wrote (volumes of both signs). Bit for bit against the
phase-by-phase path, which carries the donor in the face record."""
import numpy as np
import pytest
from test_cycle_graph_gpu import _deck, _phases, _same, _state

from salec_b200 import capi, decks


def _cut_cells(vof):
    """Interior cells with vacuum and material, in rows of the impact."""
    v0 = vof[3:-3, 3:-3, 0]
    return np.argwhere((v0 > 0.2) & (v0 < 0.8)) + 3


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("fraction", [float("nan"), -0.3, -0.05, -1.0e-17])
def test_donor_side_is_the_records(cuda_device, tmp_path, fraction, precision):
    path = decks.write_deck(_deck("two"), str(tmp_path))
    graph, phases = (capi.Simulation.from_deck(path, str(tmp_path), precision=precision) for _ in range(2))
    for sim in (graph, phases):
        _phases(sim, 30)
        vof = sim.get_field("m_vof")
        cells = _cut_cells(vof)
        assert len(cells) > 4
        for j, i in cells[::3] if np.isnan(fraction) else cells:
            vof[j, i, 1 + np.argmin(vof[j, i, 1:])] = fraction
        sim.set_field("m_vof", vof)
    # a NaN reaches velocities in its first cycle, and a face whose swept volume is NaN is written by both
    # of its cells
    for n in (1,) if np.isnan(fraction) else (1, 1, 2):
        graph.step(n)
        _phases(phases, n)
        _same(_state(graph), _state(phases), "after %d more cycles" % n)
    graph.close()
    phases.close()
