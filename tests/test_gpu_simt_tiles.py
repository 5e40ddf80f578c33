"""The FP32 forward at every tile size it picks (16 x 4, 5, 6 and 8 voxels per axis), at the edges of its
tiles and spot chunks, and in a batch of fields of different sizes (one tile size for all)."""
import importlib

import numpy as np
import pytest

from oracle import engine_ref as er

pytestmark = pytest.mark.gpu

TOL = 1e-6   # the FP32 dose's bound, of the largest dose


@pytest.fixture(scope="module")
def pb():
    return importlib.import_module("gpu-proton-dose-engine_b200")


def _problem(pb, nx, ny, nz, nsx, nsy, nl, seed=0):
    rng = np.random.default_rng(seed)
    grid = pb.model.DoseGrid(nx, ny, nz, 0.2, 0.17, 0.2, -0.1 * nx, -0.08 * ny, 0.0)
    lat = pb.model.SpotLattice(nsx, nsy, nl, 0.25, 0.3, 0.03, -0.02,
                               weights=rng.uniform(0.1, 1.0, (nl, nsy, nsx)))
    idd = rng.uniform(0.5, 2.0, (nl, nz))
    idd[rng.uniform(size=idd.shape) < 0.3] = 0.0
    return pb.model.PBProblem(grid, lat, idd, rng.uniform(0.25, 0.8, (nl, nz)))


def _ref(p):
    g, L = p.grid, p.lattice
    return er.separable_f64(g.x, g.y, L.spot_x, L.spot_y, np.float32(L.weights), p.idd, p.sigma)


@pytest.mark.parametrize("shape", [
    (64, 65, 3, 64, 65, 3),         # 4 x 5 groups of 16; one whole chunk, two chunks
    (80, 81, 3, 17, 16, 3),         # 5 x 6
    (96, 97, 3, 33, 48, 3),         # 6 x 8
    (128, 129, 3, 49, 3, 3),        # 8 x 5 (two tiles)
    (160, 257, 2, 81, 129, 2),      # 5 (two tiles) x 6 (three tiles); chunks of 44 and less
    (1, 3, 2, 1, 1, 1),
])
def test_fp32_tiles_vs_oracle(pb, shape):
    p = _problem(pb, *shape)
    got = pb.engines.torch_separable(p, "cuda", precision="fp32").cpu().numpy()
    ref = _ref(p)
    assert np.max(np.abs(got - ref)) <= TOL * np.max(np.abs(ref))


def test_fp32_batch_of_uneven_grids(pb):
    import torch
    lib = pb._lib
    probs = [_problem(pb, 70, 130, 3, 9, 30, 2, 1), _problem(pb, 128, 60, 4, 70, 7, 3, 2), _problem(pb, 20, 20, 2, 3, 3, 1, 3)]
    jobs, keep, doses = (lib.Job * 3)(), [], []
    for k, p in enumerate(probs):
        w = torch.as_tensor(np.float32(p.lattice.weights), device="cuda")
        i, s = (torch.as_tensor(a, device="cuda") for a in (p.idd, p.sigma))
        d = torch.empty(p.grid.shape, dtype=torch.float32, device="cuda")
        jobs[k] = lib.Job(field=lib.field_of(p), w=lib.ptr(w), idd=lib.ptr(i), sigma=lib.ptr(s), dose=lib.ptr(d))
        keep += [w, i, s]
        doses.append(d)
    prec = lib.PREC["fp32"]
    ws = torch.empty(lib.query("pbd_forward_batch_workspace", jobs, 3, prec), dtype=torch.uint8, device="cuda")
    lib.call("pbd_forward_batch", jobs, 3, prec, lib.ptr(ws), ws.numel(), lib.stream_handle())
    for p, d in zip(probs, doses):
        ref = _ref(p)
        assert np.max(np.abs(d.cpu().numpy() - ref)) <= TOL * np.max(np.abs(ref))
