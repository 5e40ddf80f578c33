"""The FP64 forward with depth doses and widths at the ends of float64's range, on lattices that do not fill
the kernel's groups of four spots.

A width whose square overflows spreads its dose to zero; an infinite depth dose gives an infinite dose at
every voxel the spots reach."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pb():
    return importlib.import_module("gpu-proton-dose-engine_b200")


def _problem(pb, nsx, nsy, nx=70, ny=66):
    rng = np.random.default_rng(nsx)
    grid = pb.model.DoseGrid(nx, ny, 3, 0.2, 0.2, 0.2, -0.1 * nx, -0.1 * ny, 0.0)
    lat = pb.model.SpotLattice(nsx, nsy, 2, 0.25, 0.25, 0.0, 0.0, weights=rng.uniform(0.1, 1.0, (2, nsy, nsx)))
    return pb.model.PBProblem(grid, lat, rng.uniform(0.5, 2.0, (2, 3)), rng.uniform(0.4, 0.8, (2, 3)))


def _dose(pb, p):
    import torch
    return pb.engines.torch_separable(p, "cuda", dtype=torch.float64).cpu().numpy()


@pytest.mark.parametrize("lattice", [(9, 7), (65, 3), (5, 66), (8, 4)])
@pytest.mark.parametrize("width", [1e200, np.inf])
def test_overflowing_width_gives_no_dose(pb, lattice, width):
    p = _problem(pb, *lattice)
    p.sigma[1, 2] = width
    got = _dose(pb, p)
    p.idd[1, 2], p.sigma[1, 2] = 0.0, 1.0
    assert np.array_equal(got, _dose(pb, p))


@pytest.mark.parametrize("lattice", [(9, 7), (65, 3), (5, 66), (8, 4)])
def test_infinite_depth_dose_is_infinite(pb, lattice):
    p = _problem(pb, *lattice, nx=40, ny=36)
    plain = _dose(pb, p)
    p.idd[1, 2] = np.inf
    got = _dose(pb, p)
    assert np.all(np.isposinf(got[2]))
    assert np.array_equal(got[:2], plain[:2])
