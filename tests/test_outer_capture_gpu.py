"""Phases that a caller captures into a CUDA graph of its own on the handle's stream: the replays go on
where the handle was, also when the cycle graph ran before (an odd or an even number of cycles) and
runs between and after them, with field writes in between. Bit for bit against a handle that runs
phase by phase."""
import pytest
from test_cycle_graph_gpu import _phases, _same, _state
from test_quiet_map_gpu import _deck, _place_body

from salec_b200 import capi, decks


@pytest.mark.gpu
@pytest.mark.parametrize("cycles,how", [(0, "phases"), (0, "step"), (40, "phases"), (41, "phases")])
def test_replays_of_a_callers_graph(cuda_device, tmp_path, cycles, how):
    import torch
    path = decks.write_deck(_deck("nothing"), str(tmp_path))
    mixed, phases = (capi.Simulation.from_deck(path, str(tmp_path)) for _ in range(2))
    stream = torch.cuda.ExternalStream(mixed.stream())
    mixed.step(cycles)
    _phases(phases, cycles)
    mixed.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        if how == "phases":
            mixed.phases(0, 15)
        else:
            mixed.step(1)
        graph.capture_end()
    done = 0

    def both(run, n):
        nonlocal done
        run(n)
        _phases(phases, n)
        done += n
        _same(_state(mixed), _state(phases), "%d cycles after the capture" % done)

    def replay(n):
        with torch.cuda.stream(stream):
            for _ in range(n):
                graph.replay()

    both(replay, 3)
    both(mixed.step, 5)
    for sim in (mixed, phases):
        _place_body(sim)
    both(replay, 2)
    both(mixed.step, 3)
    both(replay, 1)
    del graph
    mixed.close()
    phases.close()
