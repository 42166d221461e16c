"""The cycle graph against the phase-by-phase path, bit for bit: the graph keeps two copies of the
donor state, stores face volumes instead of records and fuses sweeps, the phases work in place, one
sweep at a time. Both forms, with and without porosity, after odd and even numbers of cycles, and
with the two paths and field writes mixed on one handle."""
import numpy as np
import pytest

from salec_b200 import capi, decks, fields


def _deck(kind):
    if kind == "quiet":
        return decks.Deck(npx=456, npy=470, radius_cells=12.0, damp_x=8, damp_y=8, velocity=-15000.0, oy=0.4)
    common = dict(npx=45, npy=70, radius_cells=7.0, damp_x=5, damp_y=6, velocity=-9000.0)
    if kind == "pml3":
        return decks.Deck(damping="pml3", **common)
    if kind == "porous":
        return decks.Deck(materials=[decks.Material("basalt_", porosity="Wunnemann", alpha0=1.0 / 0.75, alphax=1.1,
                                                    epse0=-1.0e-5, kappa=0.98, chi=0.5)], damping="pml2", **common)
    if kind == "two":
        return decks.Deck(materials=[decks.Material("basalt_"), decks.Material("dunite_")], projectile="dunite_",
                          tensile_failure=1, **common)
    return decks.Deck(**common)


def _state(sim):
    nmat = sim.get_run().nmat
    out = {}
    for n in fields.STEP_FIELDS:
        a = sim.get_field(n)
        if n in ("bx_phi", "by_phi"):   # a face without flow has volumes only
            a = np.where((a[..., :nmat] != 0.0).any(axis=-1, keepdims=True), a, 0.0)
        out[n] = a
    out["tracers"] = sim.get_tracers()
    out["dt"], out["time"] = np.array(sim.scalar("dt")), np.array(sim.scalar("time"))
    return out


def _same(a, b, what):
    for n in a:
        assert np.array_equal(a[n], b[n], equal_nan=True), "%s: %s" % (what, n)


def _phases(sim, n):
    for _ in range(n):
        sim.phases(0, 15)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["base", "two", "porous", "pml3", "quiet"])
def test_cycle_graph_equals_the_phases(cuda_device, tmp_path, kind, precision):
    path = decks.write_deck(_deck(kind), str(tmp_path))
    graph, phases = (capi.Simulation.from_deck(path, str(tmp_path), precision=precision) for _ in range(2))
    for n in (1, 2, 30, 25):
        graph.step(n)
        _phases(phases, n)
        _same(_state(graph), _state(phases), "after %d more cycles" % n)
    # an odd number of graph cycles, then phases, then the graph again
    graph.step(1)
    _phases(graph, 2)
    graph.step(2)
    _phases(phases, 5)
    _same(_state(graph), _state(phases), "paths mixed")
    # a body placed in the vacuum far above the surface, moving up
    for sim in (graph, phases):
        vof, den, eng, rho = (sim.get_field(n) for n in ("m_vof", "m_den", "m_eng", "e_den"))
        top = sim.get_run().ny - 12
        box = (slice(top, top + 5), slice(20, 26))
        vof[box] = 0.0
        vof[box + (1,)] = 1.0
        den[box + (1,)] = 2700.0
        eng[box + (1,)] = 1.0e8
        rho[box] = 2700.0
        for n, a in (("m_vof", vof), ("m_den", den), ("m_eng", eng), ("e_den", rho)):
            sim.set_field(n, a)
        vel = sim.get_field("v_vel")
        vel[top:top + 6, 20:27] = [50.0, 900.0]
        sim.set_field("v_vel", vel)
    graph.step(9)
    _phases(phases, 9)
    _same(_state(graph), _state(phases), "after the body")
    graph.close()
    phases.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cycles", [1, 2])
def test_adjoint_fields_after_graph_cycles(cuda_device, tmp_path, cycles):
    """An adjoint field read after forward cycles is the one that was set: the forward donor state may
    then live in its second copy, the adjoint planes have one place."""
    deck = decks.config5_deck(64, velocity=1000.0, cppr=8.0)
    sim = capi.Simulation.from_deck(decks.write_deck(deck, str(tmp_path)), str(tmp_path))
    sim.adjoint_reset()
    bar = np.random.default_rng(3).standard_normal(sim.shape("m_den"))
    sim.step(cycles)
    sim.adjoint_set("m_den", bar)
    sim.step(cycles)
    assert np.array_equal(sim.adjoint_get("m_den"), bar)
    sim.close()
