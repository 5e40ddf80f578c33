"""The heterogeneous dose at the edges of its kernels: lateral maps of one and several tiles with rows
that allow 32-byte stores and rows that do not, the smallest and largest lattices, weights over six
orders of magnitude; voxel counts that are no multiple of a block, more layers than the combine stages
at once, water-equivalent depths below 0 and beyond every curve; the ray trace past one pass of depths.

Tolerances: the dose's 1e-6 of the largest (the module's TF32x3 bound); WED 1e-13 of max."""
import numpy as np
import pytest

from conftest import has_gpu, load_pkg
from oracle import hetero_ref as hr
from oracle import physics_ref as pr

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]


@pytest.fixture(scope="module")
def pb():
    return load_pkg()


def _problem(pb, nx, ny, nz, nsx, nsy, nl, seed):
    rng = np.random.default_rng(seed)
    grid = pb.model.DoseGrid(nx, ny, nz, 0.2, 0.2, 0.4, -0.1 * nx, -0.1 * ny, 0.0)
    en = pr.layer_energies(nl, 1.5, 1.5 + 0.5 * nz * 0.4)
    w = 10.0 ** rng.uniform(-6.0, 0.0, (nl, nsy, nsx))
    lat = pb.model.SpotLattice(nsx, nsy, nl, 0.4, 0.4, 0.0, 0.0, energies=en, weights=w)
    zc = grid.oz + np.arange(nz) * grid.dz
    idd, sig = pr.layer_luts(zc, en)
    rho = rng.uniform(0.4, 1.6, (nz, ny, nx)).astype(np.float32)
    return pb.model.PBProblem(grid, lat, idd, sig), en, sig, rho


@pytest.mark.parametrize("shape", [
    (128, 128, 7, 16, 16, 4),       # one whole tile, symmetric, 32-byte stores
    (136, 129, 5, 64, 33, 3),       # 2 x 2 tiles, the largest lattice along x
    (131, 40, 6, 17, 64, 3),        # rows of odd length: scalar stores
    (36, 1, 9, 1, 1, 2),            # rows of 4 (no 32-byte stores), one spot, one row
    (24, 17, 5, 3, 5, 131),         # layers over the staged 128
])
@pytest.mark.parametrize("prec", ["tf32x3", "fp16x3"])
def test_dose_vs_oracle(pb, shape, prec):
    prob, en, sig, rho = _problem(pb, *shape, seed=sum(shape))
    g = prob.grid
    wed = hr.wed_ref(rho, g.oz, g.dz)
    wed[0, 0, 0], wed[-1, -1, -1] = -0.3, 1e6       # inside no curve
    L = prob.lattice
    want = hr.dose_ref(g.x, g.y, L.spot_x, L.spot_y, np.float32(L.weights), en, sig, wed)
    assert want[0, 0, 0] == 0.0 and want[-1, -1, -1] == 0.0
    got = pb.hetero.WedPlan(prob, precision=prec).forward(wed).cpu().numpy()
    assert np.max(np.abs(got - want)) <= 1e-6 * np.max(np.abs(want))


@pytest.mark.parametrize("shape", [(37, 50, 6, 17, 33, 3), (128, 5, 4, 3, 2, 131)])
def test_gradients_vs_oracle(pb, shape):
    """dL/dW and dL/dR with water-equivalent depths inside no curve, on the curves' far ends and over 128
    layers; 1e-5 of the largest (the adjoint's split FP16 is good to some 1e-6)."""
    import torch
    prob, en, sig, rho = _problem(pb, *shape, seed=sum(shape))
    g, L = prob.grid, prob.lattice
    wed = hr.wed_ref(rho, g.oz, g.dz)
    wed[0, 0, 0], wed[-1, -1, -1], wed[1, 0, 0] = -0.3, 1e6, 0.0
    grad = np.random.default_rng(2).standard_normal(wed.shape).astype(np.float32)
    w = np.float32(L.weights)
    want = hr.grad_w_ref(g.x, g.y, L.spot_x, L.spot_y, w, en, sig, wed, grad.astype(np.float64))
    plan = pb.hetero.WedPlan(prob)
    gw, gr = plan.adjoint(torch.as_tensor(grad, device="cuda"), torch.as_tensor(wed), with_range=True)
    assert np.max(np.abs(gw.cpu().numpy() - want)) <= 1e-5 * np.max(np.abs(want))
    assert torch.equal(gw, plan.adjoint(torch.as_tensor(grad, device="cuda"), torch.as_tensor(wed)))
    zc = g.oz + np.arange(g.nz) * g.dz
    want_r = hr.grad_range_ref(g.x, g.y, L.spot_x, L.spot_y, w, en, zc, wed, grad.astype(np.float64), plan.fd_step)
    assert np.max(np.abs(gr.cpu().numpy() - want_r)) <= 1e-4 * np.max(np.abs(want_r))


@pytest.mark.parametrize("shape", [(1, 1, 1), (128, 3, 33), (129, 5, 31), (257, 2, 40)])
@pytest.mark.parametrize("oz", [0.0, -1.3, 2.1])
def test_raytrace_vs_oracle(pb, shape, oz):
    rho = np.random.default_rng(1).uniform(0.0, 2.0, shape).astype(np.float32)
    grid = {"nz": shape[0], "ny": shape[1], "nx": shape[2], "oz": oz, "dz": 0.11}
    got = pb.hetero.wed_raytrace(rho, grid).cpu().numpy()
    want = hr.wed_ref(rho, oz, 0.11)
    assert np.max(np.abs(got - want)) <= 1e-13 * np.max(np.abs(want))
