"""The FP64 forward at the edges of its tiles and spot chunks, and its exponential.

Oracle: the reference's float64 engine (oracle.engine_ref.separable_f64)."""
import importlib

import numpy as np
import pytest

from oracle import engine_ref as er

pytestmark = pytest.mark.gpu


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


# Products and sums of n_sx + n_sy + layers terms, all positive: (4 + 63 + 81 + 130) 2^-53 of a voxel's
# dose from them, and the exponent's two roundings times its size, at most ~40 where a voxel
# still has 1e-17 of the largest dose: 80 2^-53 twice.  Against the largest dose 1e-13 holds with
# room.
@pytest.mark.parametrize("shape", [
    (64, 128, 3, 41, 41, 3),        # one whole 128-row tile
    (65, 129, 2, 4, 5, 2),          # one voxel past the tiles: 64-row tiles (129-192 rows)
    (1, 1, 1, 1, 1, 1),
    (63, 64, 5, 44, 45, 4),         # 64-row tile, chunk of 48
    (100, 193, 2, 64, 64, 2),       # the largest whole chunk
    (70, 70, 2, 65, 81, 130),       # chunked spots (64 + 1, 64 + 17), layers past one batch
])
def test_f64_dose_vs_oracle(pb, shape):
    import torch
    p = _problem(pb, *shape)
    g, L = p.grid, p.lattice
    ref = er.separable_f64(g.x, g.y, L.spot_x, L.spot_y, L.weights, p.idd, p.sigma)
    got = pb.engines.torch_separable(p, "cuda", dtype=torch.float64)
    err = np.max(np.abs(got.cpu().numpy() - ref)) / max(np.max(np.abs(ref)), 1e-300)
    assert err <= 1e-13


def test_f64_exponential_relative(pb):
    """One spot, one layer: a voxel is a product of two exponentials, held to its own size down
    to 1e-300.  d carries 2 roundings, d^2 k2 3 more, so the exponent x is off by 8 |x| 2^-53 at most
    per axis; 16 2^-53 for the exponentials and products themselves."""
    import torch
    n = 127
    grid = pb.model.DoseGrid(n, n, 1, 0.1, 0.1, 0.1, -6.3, -6.3, 0.0)
    lat = pb.model.SpotLattice(1, 1, 1, 0.25, 0.25, 0.013, -0.007, weights=np.ones((1, 1, 1)))
    sig = np.array([[0.25]])
    p = pb.model.PBProblem(grid, lat, np.array([[1.0]]), sig)
    got = pb.engines.torch_separable(p, "cuda", dtype=torch.float64).cpu().numpy()[0]
    ref = er.separable_f64(grid.x, grid.y, lat.spot_x, lat.spot_y, lat.weights, p.idd, sig)[0]
    x = ((grid.y[:, None] - lat.spot_y[0]) ** 2 + (grid.x[None, :] - lat.spot_x[0]) ** 2) / (2 * 0.25**2)
    ok = x < 690.0
    assert ok.sum() > 10000
    assert np.all(np.abs(got[ok] - ref[ok]) <= (16 + 16 * x[ok]) * 2.0**-53 * ref[ok])
    assert np.all(got[~ok] <= 1e-290)
