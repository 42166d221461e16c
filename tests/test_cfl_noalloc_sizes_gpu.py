"""salec_cfl_dt_noalloc at the edges of its blocks (1024 cells up to 8.4 million cells, 4096 beyond),
against numpy's fold of the same candidates in traversal order, bit for bit: with no NaN, a NaN in the
middle, a NaN last, and all vacuum."""
import numpy as np
import pytest

from salec_b200 import capi

PLANES = ("vr", "vz", "csd", "sr", "sz", "vof")


def _expected(p, dt_prev, max_dt):
    a = {k: v[2:-2, 2:-2].ravel() for k, v in p.items()}
    dt_r, dt_z = a["sr"] / (np.abs(a["vr"]) + a["csd"]), a["sz"] / (np.abs(a["vz"]) + a["csd"])
    cand = (0.2 * np.where(dt_r < dt_z, dt_r, dt_z))[~(a["vof"] > 1.0 - 1e-6)]
    nans = np.flatnonzero(np.isnan(cand))
    if nans.size:
        cand = cand[nans[-1] + 1:]
        best = cand.min() if cand.size else np.nan
    else:
        best = min([1.1 * dt_prev] + ([cand.min()] if cand.size else []))
    return max_dt if max_dt < best else best


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 341), (255, 4), (257, 4), (1024, 1), (1, 1025), (2048, 4096), (2897, 2897)])
def test_cfl_sizes(cuda_device, nx, ny):
    import torch
    rng = np.random.default_rng(nx * 7919 + ny)
    shape = (ny + 4, nx + 4)
    p = {"vr": rng.uniform(-9e3, 9e3, shape), "vz": rng.uniform(-9e3, 9e3, shape), "csd": rng.uniform(1e3, 9e3, shape),
         "sr": rng.uniform(10.0, 50.0, shape), "sz": rng.uniform(10.0, 50.0, shape),
         "vof": (rng.random(shape) < 0.3).astype(float)}
    p["vof"][ny + 1, nx + 1] = 0.0   # the last cell of the traversal counts
    out = torch.zeros(1, device="cuda", dtype=torch.float64)
    for case in ("none", "middle", "last", "vacuum"):
        q = {k: v.copy() for k, v in p.items()}
        if case == "middle":
            q["csd"][2 + ny // 2, 2 + nx // 2] = np.nan
            q["vof"][2 + ny // 2, 2 + nx // 2] = 0.0
        elif case == "last":
            q["csd"][ny + 1, nx + 1] = np.nan
        elif case == "vacuum":
            q["vof"][:] = 1.0
        dev = [torch.from_numpy(q[k]).cuda() for k in PLANES]
        capi.cfl_dt_noalloc(nx, ny, *[d.data_ptr() for d in dev], 1.0, 0.05, out.data_ptr(),
                            torch.cuda.current_stream().cuda_stream)
        got, want = float(out.cpu()[0]), float(_expected(q, 1.0, 0.05))
        assert got == want or (np.isnan(got) and np.isnan(want)), (case, got, want)
