"""The quiet map of the cycle graph (vacuum tiles left out of the sweeps) is forgotten whatever comes
between a field write and the next graph cycle. A body is written into long-quiet vacuum after an odd
number of graph cycles, when the donor state lives in its second copy; then something runs that brings
it back to the first (phases, a profiled step, autotuning, the adjoint), and then the graph. Bit for
bit against a handle that runs phase by phase."""
import ctypes

import pytest
from test_cycle_graph_gpu import _phases, _same, _state

from salec_b200 import capi, decks


def _deck(kind):
    common = dict(npx=456, npy=470, radius_cells=12.0, velocity=-15000.0, oy=0.4)
    if kind == "adjoint":
        return decks.Deck(**{**decks.config5_deck(64, velocity=15000.0, cppr=12.0).__dict__, **common})
    return decks.Deck(damp_x=8, damp_y=8, **common)


def _tiles(sim):
    listed, total = ctypes.c_int(), ctypes.c_int()
    assert capi.lib().salec_internal_listed_tiles(sim.h, ctypes.byref(listed), ctypes.byref(total)) == 0
    return listed.value, total.value


def _place_body(sim):
    """A block of material in the vacuum far above the surface, moving up and to the right."""
    vof, den, eng, rho = (sim.get_field(n) for n in ("m_vof", "m_den", "m_eng", "e_den"))
    box = (slice(440, 446), slice(200, 208))
    assert (vof[box][..., 0] == 1.0).all()
    vof[box] = 0.0
    vof[box + (1,)] = 1.0
    den[box + (1,)] = 2700.0
    eng[box + (1,)] = 1.0e8
    rho[box] = 2700.0
    vel = sim.get_field("v_vel")
    vel[440:447, 200:209] = [300.0, 900.0]
    for n, a in (("m_vof", vof), ("m_den", den), ("m_eng", eng), ("e_den", rho), ("v_vel", vel)):
        sim.set_field(n, a)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("between", ["phases", "profile", "autotune", "adjoint", "nothing"])
def test_a_write_after_odd_cycles_reaches_every_tile(cuda_device, tmp_path, between, precision):
    if between == "adjoint" and precision:
        pytest.skip("the adjoint runs on the plain FP64 form")
    path = decks.write_deck(_deck(between), str(tmp_path))
    graph, phases = (capi.Simulation.from_deck(path, str(tmp_path), precision=precision) for _ in range(2))
    graph.step(41)
    _phases(phases, 41)
    listed, total = _tiles(graph)
    assert 0 < listed < total
    for sim in (graph, phases):
        _place_body(sim)
    assert _tiles(graph) == (total, total)
    if between == "phases":
        _phases(graph, 1)
        _phases(phases, 1)
    elif between == "profile":
        graph.profile(True)
        graph.step(1)
        graph.profile(False)
        _phases(phases, 1)
    elif between == "autotune":
        graph.autotune(cycles=1)
    elif between == "adjoint":
        graph.adjoint_reset()
    assert _tiles(graph) == (total, total)
    for n in (1, 2, 6):
        graph.step(n)
        _phases(phases, n)
        _same(_state(graph), _state(phases), "after %d more cycles" % n)
    graph.close()
    phases.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [float("nan"), float("inf"), 1.0e200])
def test_a_time_step_beyond_bounds_reaches_every_tile(cuda_device, tmp_path, dt):
    """0 * dt is NaN for such a time step, in vacuum too: what it leaves behind is the phase-by-phase
    path's, in the cycle itself and in those after it (whose CFL steps are then recounted)."""
    path = decks.write_deck(_deck("nothing"), str(tmp_path))
    graph, phases = (capi.Simulation.from_deck(path, str(tmp_path)) for _ in range(2))
    graph.step(40)
    _phases(phases, 40)
    listed, total = _tiles(graph)
    assert 0 < listed < total
    for sim in (graph, phases):
        sim.set_dt_schedule([1.0e-3, dt])
    for n in (2, 1, 1, 5):
        graph.step(n)
        _phases(phases, n)
        _same(_state(graph), _state(phases), "after %d more cycles" % n)
    graph.close()
    phases.close()
