"""The second copy of the donor state is optional: when the device is out of memory for something a
caller asks for, it is taken from the handle itself and then from the others, also while another thread
steps one of them. Nothing is refused that fits without the copies, and no result changes."""
import threading

import pytest
from test_cycle_graph_gpu import _same, _state

from salec_b200 import capi, decks

N = 512


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.gpu
def test_spare_copies_are_given_up(cuda_device, tmp_path):
    import torch
    path = decks.write_deck(decks.Deck(npx=N, npy=N, radius_cells=12.0, damp_x=8, damp_y=8, velocity=-15000.0),
                            str(tmp_path))

    def new():
        return capi.Simulation.from_deck(path, str(tmp_path))

    control = new()
    want = {}
    for n in (6, 21, 30, 121):
        control.step(n - int(control.scalar("i_step")))
        want[n] = _state(control)
    control.close()
    before = _free()
    others = [new() for _ in range(8)]
    each = (before - _free()) // len(others)
    for sim in others:
        sim.step(21)
        sim.sync()
    # room for 0.6 of a handle: its field planes alone take 0.8 of it
    fill = torch.empty(_free() - int(0.6 * each), dtype=torch.uint8, device="cuda")
    try:
        busy = threading.Thread(target=lambda: [others[0].step(1) for _ in range(100)])
        busy.start()
        late = new()
        late.step(6)
        _same(_state(late), want[6], "created with the others' memory")
        busy.join()
        # what a handle asks for later comes from the copies as well
        others[2].write_output(str(tmp_path), "late", 0)
        others[3].conservation()
        others[4].set_tracers(others[4].get_tracers())
    finally:
        del fill
        torch.cuda.empty_cache()
    for sim in others[1:]:
        _same(_state(sim), want[21], "after the others asked")
        sim.step(9)
        _same(_state(sim), want[30], "nine cycles on")
    _same(_state(others[0]), want[121], "stepped meanwhile")
    for sim in [late] + others:
        sim.close()
