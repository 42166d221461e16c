"""The workloads whose speed is followed, each through the public entry points a program calls.

Every case but the first is an impact simulation that is created from a deck, tuned where a
program for a single large mesh would tune it, and already some cycles into its run. One pass
advances it by a stretch of cycles the way a host loop does and reads back the snapshot fields
into page-locked buffers, so a pass is "the cycles between two outputs". The states go on from
pass to pass, as a run does.

The ranges: meshes from 40 to 2048 cells per axis, square and not, odd sizes included; one to
three materials beside vacuum; Tillotson and tabulated equations of state; the plain FP64 and the
mixed form; PML and PML2 damping, porosity, acoustic fluidisation and tensile failure; single
runs, ensembles of uneven meshes and the adjoint window; and the stand-alone CFL time step.
"""
from __future__ import annotations

import concurrent.futures
import math
import os
import random
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "salec-2d-public_b200"))
from salec_b200 import capi, decks  # noqa: E402

# what a host program reads back at an output cycle
SNAPSHOT = ["v_vel", "e_den", "e_pre", "e_tem", "e_ste", "e_dam", "m_vof", "m_eng"]
FORMS = {"fp64": capi.PRECISION_FP64, "mixed": capi.PRECISION_MIXED}
# interior cells x cycles of the largest listed case; drawn cases stay below it
LARGEST = 2048 * 2048 * 100


def listed():
    return [
        # the allocation-free CFL step that a host code with its own device planes calls once per
        # cycle: the smallest call of all, one reduction
        {"name": "cfl_dt_1021x1533", "kind": "cfl", "nx": 1021, "ny": 1533},
        # a coarse scoping run whose host loop looks at dt, time and the surface after every
        # cycle: launches and synchronisations count, not bytes
        {"name": "basalt_64x80_report", "kind": "basalt", "nx": 64, "ny": 80, "form": "fp64", "cycles": 32,
         "before": 40, "report": True, "tune": False},
        # the reference's own CPU-runnable configuration, 200 x 400 cells
        {"name": "basalt_200x400", "kind": "basalt", "nx": 200, "ny": 400, "form": "fp64", "cycles": 50,
         "before": 60, "report": False, "tune": False},
        # two materials with the optional physics on (PML2, acoustic fluidisation, tensile
        # failure), odd mesh
        {"name": "options_333x217", "kind": "options", "nx": 333, "ny": 217, "form": "fp64", "cycles": 50,
         "before": 60, "report": False, "tune": False},
        # ice on granite with the tabulated EOS: the benchmark's deck, from a quarter of its
        # width to its full 2048 x 2048
        {"name": "impact_517x771_mixed", "kind": "impact", "nx": 517, "ny": 771, "form": "mixed", "cycles": 60,
         "before": 100, "report": True, "tune": False},
        {"name": "impact_1024", "kind": "impact", "nx": 1024, "ny": 1024, "form": "fp64", "cycles": 100,
         "before": 200, "report": False, "tune": True},
        {"name": "impact_1536_mixed", "kind": "impact", "nx": 1536, "ny": 1536, "form": "mixed", "cycles": 100,
         "before": 100, "report": False, "tune": True},
        {"name": "impact_2048", "kind": "impact", "nx": 2048, "ny": 2048, "form": "fp64", "cycles": 100,
         "before": 100, "report": False, "tune": True},
        # porous regolith over basalt over dunite with seeded density noise: every cell moves and
        # every face carries a full record
        {"name": "layered_1024", "kind": "layered", "nx": 1024, "ny": 1024, "form": "fp64", "cycles": 40,
         "before": 20, "report": False, "tune": True},
        {"name": "layered_600x450_mixed", "kind": "layered", "nx": 600, "ny": 450, "form": "mixed", "cycles": 60,
         "before": 20, "report": False, "tune": False},
        # a parameter study: uneven small meshes stepped together
        {"name": "ensemble_12_mixed", "kind": "ensemble", "members": 12, "nmin": 128, "nmax": 512, "form": "mixed",
         "cycles": 32},
        # the backward direction: gradients of the surface misfit over a window of cycles
        {"name": "adjoint_256", "kind": "adjoint", "nx": 256, "ny": 256, "cycles": 40, "every": 20},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["cfl", "basalt", "basalt", "options", "impact", "impact", "layered", "ensemble", "adjoint"])
    if kind == "cfl":
        return {"kind": "cfl", "nx": _log_int(rng, 40, 4000), "ny": _log_int(rng, 40, 4000)}
    if kind == "ensemble":
        nmin = _log_int(rng, 100, 200)
        return {"kind": "ensemble", "members": rng.randint(3, 16), "nmin": nmin, "nmax": rng.randint(nmin + 50, 600),
                "form": rng.choice(["fp64", "mixed"]), "cycles": rng.randint(8, 40)}
    if kind == "adjoint":
        return {"kind": "adjoint", "nx": _log_int(rng, 64, 384), "ny": _log_int(rng, 64, 384),
                "cycles": rng.randint(8, 40), "every": rng.randint(4, 20)}
    lo, hi = {"basalt": (40, 900), "options": (60, 700), "impact": (200, 1600), "layered": (150, 900)}[kind]
    nx = _log_int(rng, lo, hi)
    ny = max(lo, min(hi, int(nx * math.exp(rng.uniform(-0.7, 0.7)))))
    return {"kind": kind, "nx": nx, "ny": ny, "form": rng.choice(["fp64", "fp64", "mixed"]),
            "cycles": min(rng.randint(16, 80), LARGEST // (nx * ny)), "before": rng.randint(10, 80),
            "report": rng.random() < 0.4, "tune": nx * ny > 500000}


# ---------------------------------------------------------------- decks
_eos_dir = None


def _folder() -> str:
    """The program's folder of decks and EOS files (the table is written once, as on a user's disk)."""
    global _eos_dir
    if _eos_dir is None:
        _eos_dir = tempfile.TemporaryDirectory(prefix="salec_cases_")
    return _eos_dir.name


def _deck(case, seed: int):
    """The deck of one case: sizes from the case, speed, cohesion and friction from the seed."""
    rng = np.random.default_rng(seed)
    nx, ny, kind = case["nx"], case["ny"], case["kind"]
    small = min(nx, ny)
    damp = max(4, min(30, small // 6))
    cohesion, friction = float(10.0 ** rng.uniform(6.5, 7.5)), float(rng.uniform(0.8, 1.4))
    rock = dict(yint0=cohesion, yintfri=friction)
    if kind == "impact":
        d = decks.config2_deck(nx)
        d.npx, d.npy, d.damp_x, d.damp_y = nx, ny, damp, damp
        d.radius_cells = float(min(40, small // 6))
        d.velocity = -float(rng.uniform(12000.0, 18000.0))
        d.materials[0].yint0, d.materials[0].yintfri = cohesion, friction
        return d
    if kind == "layered":
        d = decks.config3_deck(nx, regolith=50.0 * (ny // 24), basalt=50.0 * (ny // 6), side_layers=damp,
                               base_layers=damp, cppr=float(min(30, small // 8)))
        d.npx, d.npy = nx, ny
        d.velocity = -float(rng.uniform(8000.0, 12000.0))
        return d
    common = dict(npx=nx, npy=ny, dx=50.0, dy=50.0, radius_cells=float(min(20, small // 6)), damp_x=damp, damp_y=damp,
                  gravity=-1.62, dt0=1.0e-3, maxdt=0.05)
    if kind == "options":
        mats = [decks.Material("basalt_", toff=16.0, block_size=200.0, **rock), decks.Material("dunite_", **rock)]
        return decks.Deck(materials=mats, projectile="dunite_", velocity=-float(rng.uniform(6000.0, 10000.0)),
                          damping="pml2", tensile_failure=1, right="outflow", **common)
    if kind == "adjoint":
        return decks.Deck(**{**decks.config5_deck(64, cohesion=cohesion, friction=friction,
                                                  velocity=float(rng.uniform(6000.0, 9000.0)),
                                                  cppr=float(min(20, small // 6))).__dict__, "npx": nx, "npy": ny})
    return decks.Deck(materials=[decks.Material("basalt_", **rock)], velocity=-float(rng.uniform(5000.0, 12000.0)),
                      **common)


def _simulation(path: str, form: str):
    sim = capi.Simulation.from_deck(path, _folder(), precision=FORMS[form])
    os.unlink(path)
    return sim


def _pinned(sim, names):
    """Page-locked numpy buffers for the fields a program reads back. torch's pinned allocations
    are freed when the arrays are."""
    return {n: torch.empty(sim.shape(n), dtype=torch.float64, pin_memory=True).numpy() for n in names}


_count = [0]


def prepare(case, seed):
    _count[0] += 1
    stem = "case_%d_%d" % (os.getpid(), _count[0])
    kind = case["kind"]
    if kind == "cfl":
        return _prepare_cfl(case, seed)
    if kind == "ensemble":
        # the meshes of a study are the case's, the impacts on them the seed's
        members = decks.ensemble_decks(case["members"], nmin=case["nmin"], nmax=case["nmax"])
        rng = np.random.default_rng(seed)
        for d in members:
            d.velocity = -float(rng.uniform(5000.0, 20000.0))
            d.materials[0].yint0 = float(10.0 ** rng.uniform(6.0, 8.0))
            d.materials[0].yintfri = float(rng.uniform(0.6, 1.4))
        paths = [decks.write_deck(d, _folder(), "%s_%d" % (stem, k)) for k, d in enumerate(members)]
        with concurrent.futures.ThreadPoolExecutor(8) as ex:
            sims = list(ex.map(lambda p: _simulation(p, case["form"]), paths))
        capi.step_many(sims, 16)
        for s in sims:
            s.sync()
        return {"case": case, "sims": sims, "out": [_pinned(s, ["e_den", "e_pre", "v_vel"]) for s in sims]}
    sim = _simulation(decks.write_deck(_deck(case, seed), _folder(), stem), case.get("form", "fp64"))
    if kind == "layered":
        md, ed = decks.density_noise(sim.get_field("m_den"), sim.get_field("e_den"), seed=seed)
        sim.set_field("m_den", md)
        sim.set_field("e_den", ed)
    if kind == "adjoint":
        vof, pos = sim.get_field("m_vof"), sim.get_field("e_pos")
        heights = ((1.0 - vof[2:-2, 2:-2, 0]) * pos[2:-2, 2:-2, 3]).sum(axis=0)
        return {"case": case, "sim": sim, "target": decks.target_profile(heights, 50.0, seed=seed)}
    if case["tune"]:
        sim.autotune(cycles=2)
    sim.step(case["before"])
    sim.sync()
    state = {"case": case, "sim": sim, "out": _pinned(sim, SNAPSHOT)}
    state["profile"] = _pinned(sim, ["y_profile"])["y_profile"]
    return state


def run(state):
    case = state["case"]
    kind, cycles = case["kind"], case.get("cycles", 0)
    if kind == "cfl":
        p = state["planes"]
        capi.cfl_dt_noalloc(case["nx"], case["ny"], *[p[k].data_ptr() for k in CFL_PLANES], state["dt_prev"],
                            state["max_dt"], state["dt"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"dt": state["dt"]}
    if kind == "ensemble":
        capi.step_many(state["sims"], cycles)
        for s, out in zip(state["sims"], state["out"]):
            for n, a in out.items():
                s.get_field(n, a)
        return {n: [out[n] for out in state["out"]] for n in ("e_den", "e_pre", "v_vel")}
    sim = state["sim"]
    if kind == "adjoint":
        misfit, d_params, d_velocity, d_density = sim.adjoint_window(cycles, case["every"], state["target"])
        return {"misfit": misfit, "d_params": d_params, "d_velocity": d_velocity, "d_density": d_density}
    if case["report"]:
        # the host loop of the reference: dt, time and the surface after every cycle
        for _ in range(cycles):
            dt, time = sim.step_report(1, state["profile"])
    else:
        sim.step(cycles)
        dt, time = sim.step_report(0, state["profile"])
    for n, a in state["out"].items():
        sim.get_field(n, a)
    return {"dt": dt, "time": time, "y_profile": state["profile"], **state["out"]}


# ---------------------------------------------------------------- the CFL step
CFL_PLANES = ["vel_r", "vel_z", "csd", "scale_r", "scale_z", "vof_vacuum"]


def _prepare_cfl(case, seed):
    nx, ny = case["nx"], case["ny"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    shape = (ny + 4, nx + 4)

    def uniform(lo, hi):
        return lo + (hi - lo) * torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)

    planes = {"vel_r": uniform(-9e3, 9e3), "vel_z": uniform(-9e3, 9e3), "csd": uniform(1e3, 9e3),
              "scale_r": torch.full(shape, 50.0, device="cuda", dtype=torch.float64),
              "scale_z": torch.full(shape, 50.0, device="cuda", dtype=torch.float64)}
    # vacuum above the surface, rock below it, cut cells at the surface
    level = (torch.arange(ny + 4, device="cuda") / (ny + 3.0)).reshape(-1, 1).double()
    planes["vof_vacuum"] = ((level - 0.5) * ny + uniform(-1.0, 1.0)).clamp(0.0, 1.0)
    return {"case": case, "planes": planes, "dt_prev": 1.0, "max_dt": 0.05,
            "dt": torch.zeros(1, device="cuda", dtype=torch.float64)}


# ---------------------------------------------------------------- what a pass cannot do without
def _cycle_doubles(nmat: int, damping: str, porous: bool, mixed: bool) -> float:
    """Bytes per cell and cycle: every persistent field read once and written once, read-only
    fields once; the conserved fields in FP64, the others in the form's own type."""
    e_alpha = 2 if damping in ("pml", "pml2") else 0
    v_alpha = 2 if damping == "pml2" else 0
    exact = 2 * 3 * nmat + (3 * nmat if porous else 0)
    relaxed = 2 * (4 + 2 + 12 + 4 + 2 + e_alpha + 8 + v_alpha) + 1 + (7 if e_alpha else 0)
    return 8.0 * exact + (4.0 if mixed else 8.0) * relaxed


def work(case):
    kind = case["kind"]
    if kind == "cfl":
        cells = (case["nx"]) * (case["ny"])
        return {"bytes": 8.0 * 6 * cells, "flops": 6.0 * cells}
    mixed = case.get("form") == "mixed"
    if kind == "ensemble":
        mean = 0.5 * (case["nmin"] + case["nmax"])
        cells = case["members"] * mean * mean
        return {"bytes": cells * (case["cycles"] * _cycle_doubles(2, "pml", False, mixed) + 8.0 * 4),
                "flops": 900.0 * cells * case["cycles"]}
    cells = case["nx"] * case["ny"]
    if kind == "adjoint":
        # a forward cycle and its reverse, which reads the forward state again and reads and
        # writes the adjoint state
        one = _cycle_doubles(2, "none", False, False)
        return {"bytes": cells * case["cycles"] * 2.5 * one, "flops": 4000.0 * cells * case["cycles"]}
    nmat = {"basalt": 2, "options": 3, "impact": 3, "layered": 4}[kind]
    one = _cycle_doubles(nmat, "pml2" if kind == "options" else "pml", kind == "layered", mixed)
    return {"bytes": cells * (case["cycles"] * one + 8.0 * (10 + 2 * nmat)),
            "flops": (500.0 + 200.0 * nmat) * cells * case["cycles"]}


def exact(case, seed):
    """The CFL step in 64 bits with numpy; a simulation's cycles have no short independent form."""
    if case["kind"] != "cfl":
        return None
    state = _prepare_cfl(case, seed)
    p = {k: v.cpu().numpy()[2:-2, 2:-2] for k, v in state["planes"].items()}
    dt_r = p["scale_r"] / (np.abs(p["vel_r"]) + p["csd"])
    dt_z = p["scale_z"] / (np.abs(p["vel_z"]) + p["csd"])
    cand = (0.2 * np.minimum(dt_r, dt_z))[~(p["vof_vacuum"] > 1.0 - 1e-6)]
    best = min([1.1 * state["dt_prev"]] + ([float(cand.min())] if cand.size else []))
    return {"dt": np.array([min(state["max_dt"], best)])}
