"""The tensor-core adjoint at the edges of its tiles, groups and lattices: one and two 128-row tiles,
several column tiles, ragged last groups, lattices at the padding's edges, symmetric and not.

Oracle: float64 autograd through the reference's batched-matmul engine
(oracle.engine_ref.separable_torch)."""
import importlib

import numpy as np
import pytest

from oracle import engine_ref as er

pytestmark = pytest.mark.gpu

# Of the largest gradient.  Truncating FP32 accumulators: at most 8 k-steps per stage and two row tiles,
# 2^-24 each on average, 24 * 6e-8 = 1.4e-6 if nothing were given back; operands to 22 bits and the
# exponentials to 2^-22: 3 * 2.4e-7, averaged over the sums.
TOL = 2e-6


@pytest.fixture(scope="module")
def pb():
    return importlib.import_module("gpu-proton-dose-engine_b200")


def _problem(pb, nx, ny, nz, nsx, nsy, nl, dx=0.2, dy=0.2, px=0.25, py=0.25, x0=0.03, y0=-0.02, seed=0):
    rng = np.random.default_rng(seed)
    grid = pb.model.DoseGrid(nx, ny, nz, dx, dy, 0.2, -(nx - 1) * dx / 2, -(ny - 1) * dy / 2, 0.0)
    lat = pb.model.SpotLattice(nsx, nsy, nl, px, py, x0, y0, weights=rng.uniform(0.1, 1.0, (nl, nsy, nsx)))
    idd = rng.uniform(0.5, 2.0, (nl, nz))
    idd[rng.uniform(size=idd.shape) < 0.3] = 0.0
    return pb.model.PBProblem(grid, lat, idd, rng.uniform(0.25, 0.8, (nl, nz)))


def _grads(pb, p, g, didd, dsig):
    import torch
    plan = pb.engines.DosePlan(p, tables="problem")
    t = [torch.as_tensor(a, device="cuda") for a in (didd, dsig)]
    gw, gr = plan.adjoint(torch.as_tensor(g, device="cuda"), didd=t[0], dsig=t[1])
    plan.check("adj")
    return gw.cpu().numpy().astype(np.float64), gr.cpu().numpy().astype(np.float64)


@pytest.mark.parametrize("shape", [
    (128, 128, 3, 64, 64, 2),       # whole tile, the largest lattice, symmetric but for its offsets
    (129, 128, 3, 17, 16, 2),       # a column tile of one column
    (128, 129, 3, 16, 17, 2),       # a row tile of one row
    (150, 256, 2, 64, 64, 2),       # both, two whole row tiles
    (300, 200, 2, 31, 60, 2),       # three column tiles
    (33, 15, 4, 1, 1, 3),           # one spot, less than one group of rows
    (100, 37, 4, 48, 3, 2),
])
def test_adjoint_tiles_vs_autograd(pb, shape):
    import torch
    p = _problem(pb, *shape)
    g_, L = p.grid, p.lattice
    rng = np.random.default_rng(1)
    g = (rng.uniform(-0.4, 1.0, g_.shape) * 1e-3).astype(np.float32)
    didd, dsig = rng.uniform(-1.0, 1.0, p.idd.shape), rng.uniform(-0.1, 0.1, p.idd.shape)
    gw, gr = _grads(pb, p, g, didd, dsig)
    w = torch.tensor(L.weights.astype(np.float32).astype(np.float64), requires_grad=True)
    idd = torch.tensor(p.idd, requires_grad=True)
    sig = torch.tensor(p.sigma, requires_grad=True)
    d = er.separable_torch(g_.x, g_.y, L.spot_x, L.spot_y, w, idd, sig)
    (d * torch.as_tensor(g.astype(np.float64))).sum().backward()
    on = p.idd != 0
    rw = w.grad.numpy()
    rr = (np.where(on, idd.grad.numpy() * didd, 0.0) + sig.grad.numpy() * dsig).sum(1)
    # dL/dR sums terms of both signs: held to the sum of their sizes
    size = (np.where(on, np.abs(idd.grad.numpy() * didd), 0.0) + np.abs(sig.grad.numpy() * dsig)).sum(1)
    assert np.max(np.abs(gw - rw)) <= TOL * np.max(np.abs(rw))
    assert np.max(np.abs(gr - rr)) <= TOL * np.max(size)


def test_adjoint_symmetric_equals_general_path(pb):
    """A symmetric field takes B from A's rows; moved by nothing but a sign of zero it does not differ,
    so the same field with its y spacing a bit off (the general path) stays within that change."""
    rng = np.random.default_rng(2)
    a = _problem(pb, 96, 96, 4, 33, 33, 3, x0=0.0, y0=0.0)
    b = _problem(pb, 96, 96, 4, 33, 33, 3, x0=0.0, y0=1e-9)
    g = rng.uniform(-0.5, 1.0, a.grid.shape).astype(np.float32)
    z = np.zeros(a.idd.shape)
    ga, _ = _grads(pb, a, g, z, z)
    gb, _ = _grads(pb, b, g, z, z)
    assert np.max(np.abs(ga - gb)) <= 1e-6 * np.max(np.abs(ga))


def test_adjoint_off_grid_lattice_and_non_finite(pb):
    p = _problem(pb, 64, 64, 3, 9, 9, 2, x0=100.0)
    g = np.ones(p.grid.shape, dtype=np.float32)
    z = np.zeros(p.idd.shape)
    gw, gr = _grads(pb, p, g, z, z)
    assert np.all(gw == 0.0) and np.all(gr == 0.0)
    for bad in (np.nan, np.inf):
        p = _problem(pb, 64, 64, 3, 9, 9, 2)
        p.idd[:] = 1.0
        g = np.ones(p.grid.shape, dtype=np.float32)
        g[1, 3, 5] = bad
        gw, _ = _grads(pb, p, g, z, z)
        assert np.all(np.isnan(gw))


@pytest.mark.parametrize("scale", [1e-30, 1e-12, 1e12, 1e30])
def test_adjoint_scales_with_grad_dose(pb, scale):
    """dL/dD of any size: the slice is scaled by a power of two, so a power of two changes no bit."""
    p = _problem(pb, 80, 70, 3, 21, 13, 2)
    rng = np.random.default_rng(3)
    g = rng.uniform(-0.4, 1.0, p.grid.shape).astype(np.float32)
    s = np.float32(2.0 ** round(np.log2(scale)))
    z = np.zeros(p.idd.shape)
    a, _ = _grads(pb, p, g, z, z)
    b, _ = _grads(pb, p, g * s, z, z)
    assert np.array_equal(a.astype(np.float32) * s, b.astype(np.float32))
