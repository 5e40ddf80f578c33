"""The tensor-core adjoint from beams below a voxel to ones far wider than the grid, for dL/dD of one sign,
of random sign and in one voxel, on one and two row tiles and several column tiles.

Oracle: the matrix products Gy G Gx^T / (2 pi s^2) in float64."""
import numpy as np
import pytest

from conftest import has_gpu, load_pkg

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]

VOX = 0.2
# Of the largest sum of |dL/dD| terms.  Truncating accumulators take up to 1.2 units (of 2^-24) per k-step:
# 8 + 8 of them on one tile, 16 + 8 on two row tiles, and 2 more; the kernel gives back 2 + 0.75 per k-step at
# most, so 14 (20) units are left either way.  Three operands split to 2^-22 (4 units each, averaged over
# the sums): 6 more, 10 with two tiles' sums.  20 and 30 units.
TOL = {1: 1.2e-6, 2: 1.8e-6}
WIDTHS = (0.3, 1.0, 4.0, 7.0, 10.0, 14.0, 20.0, 40.0, 100.0, 1000.0)      # voxels


def _maps(ny, nx, rng):
    one = np.zeros((ny, nx))
    one[ny // 2, nx // 3] = 1.0
    group = np.zeros((ny, nx))
    group[ny // 2:ny // 2 + 5, nx // 3:nx // 3 + 5] = rng.uniform(0.5, 1.0, (5, 5))
    return np.stack([np.ones((ny, nx)), rng.uniform(0.2, 1.0, (ny, nx)), rng.uniform(-1.0, 1.0, (ny, nx)), one, group])


def _check(nx, ny, nsx, nsy, widths, x0, precision="auto"):
    import torch
    pb = load_pkg()
    rng = np.random.default_rng(nx + ny)
    g = _maps(ny, nx, rng).astype(np.float32)
    nk, nl = len(g), len(g) * len(widths)
    grid = pb.model.DoseGrid(nx, ny, nk, VOX, VOX, VOX, -(nx - 1) * VOX / 2, -(ny - 1) * VOX / 2, 0.0)
    lat = pb.model.SpotLattice(nsx, nsy, nl, 0.25, 0.25, x0, x0, weights=rng.uniform(0.1, 1.0, (nl, nsy, nsx)))
    # layer a * nk + k: width a, active on slice k only
    idd = np.tile(np.eye(nk), (len(widths), 1))
    sig = np.repeat(np.asarray(widths) * VOX, nk)[:, None] * np.ones((1, nk))
    plan = pb.engines.DosePlan(pb.model.PBProblem(grid, lat, idd, sig), tables="problem", precision=precision)
    z = torch.zeros(nl, nk, dtype=torch.float64, device="cuda")
    gw, _ = plan.adjoint(torch.as_tensor(g, device="cuda"), didd=z, dsig=z)
    plan.check("adj")
    gw = gw.double().cpu().numpy()
    tol = TOL[1 if ny <= 128 else 2]
    for a, width in enumerate(widths):
        s = width * VOX
        gx = np.exp(-(grid.x[None, :] - np.asarray(lat.spot_x)[:, None]) ** 2 / (2 * s * s))
        gy = np.exp(-(grid.y[None, :] - np.asarray(lat.spot_y)[:, None]) ** 2 / (2 * s * s))
        for k in range(nk):
            want = gy @ g[k].astype(np.float64) @ gx.T / (2 * np.pi * s * s)
            size = gy @ np.abs(g[k]).astype(np.float64) @ gx.T / (2 * np.pi * s * s)
            # and the split's absolute step, 2^-25 of operands scaled to 2^14 and more: where only the
            # Gaussians' tails reach a dL/dD, three factors of 2^-39 each (8 widths out: exactly 0)
            floor = 2.0 ** -37 * np.sum(np.abs(g[k]), dtype=np.float64) / (2 * np.pi * s * s)
            err = np.max(np.abs(gw[a * nk + k] - want))
            assert err <= tol * np.max(size) + floor, (width, k, err / np.max(size))


@pytest.mark.parametrize("shape", [(128, 128, 41, 41), (117, 93, 37, 29), (64, 48, 17, 21), (32, 20, 9, 9),
                                   (200, 200, 61, 61), (130, 256, 64, 64), (300, 40, 33, 5)])
@pytest.mark.parametrize("x0", [0.0, 0.037])
def test_adjoint_at_any_width(shape, x0):
    _check(*shape, WIDTHS, x0)


def test_more_than_64_layers_on_several_tiles():
    _check(260, 140, 19, 23, tuple(0.5 * 1.35 ** k for k in range(15)), 0.02)       # 75 layers


def test_widths_far_past_the_grid():
    """Flat beams: Y's scale is bounded by the grid's rows, not by the width; no dose, no gradient in the limit."""
    _check(64, 48, 17, 21, (1e4, 1e6, 1e9, 1e12), 0.02)
    _check(150, 140, 17, 21, (1e4, 1e6, 1e9, 1e12), 0.02)


@pytest.mark.parametrize("width", [1e45, 1e160, np.inf])
def test_infinite_widths_give_zero(width):
    import torch
    pb = load_pkg()
    rng = np.random.default_rng(0)
    grid = pb.model.DoseGrid(40, 33, 2, VOX, VOX, VOX, -4.0, -3.0, 0.0)
    lat = pb.model.SpotLattice(9, 7, 3, 0.25, 0.25, 0.0, 0.0, weights=rng.uniform(0.1, 1.0, (3, 7, 9)))
    sig = np.full((3, 2), 0.4)
    sig[1] = width
    plan = pb.engines.DosePlan(pb.model.PBProblem(grid, lat, np.ones((3, 2)), sig), tables="problem")
    g = torch.as_tensor(rng.uniform(-0.4, 1.0, grid.shape).astype(np.float32), device="cuda")
    one = torch.ones(3, 2, dtype=torch.float64, device="cuda")
    gw, gr = plan.adjoint(g, didd=one, dsig=one)
    assert bool((gw[1] == 0).all()) and float(gr[1]) == 0.0
    assert bool((gw[0] != 0).any()) and bool(torch.isfinite(gr).all())
