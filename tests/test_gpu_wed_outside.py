"""dL/dW in a medium with a gradient that is not finite beyond every depth curve (or above the surface):
such voxels hold no dose, so they add nothing, whatever their dL/dD."""
import numpy as np
import pytest

from conftest import has_gpu, load_pkg

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]


@pytest.mark.parametrize("prec", ["fp32", "tf32x3", "bf16", "fp16x3"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_gradient_outside_the_curves_is_not_read(prec, bad):
    import torch
    pb = load_pkg()
    nx, ny, nz, nl = 48, 40, 12, 4
    rng = np.random.default_rng(0)
    grid = pb.model.DoseGrid(nx, ny, nz, 0.2, 0.2, 0.2, -0.1 * nx, -0.1 * ny, 0.0)
    en = pb.model.clinical_layer_energies(nl, 1.5, 3.0)
    lat = pb.model.SpotLattice(9, 7, nl, 0.25, 0.25, 0.03, -0.02, energies=en, weights=rng.uniform(0.1, 1.0, (nl, 7, 9)))
    wed = pb.hetero.wed_raytrace(rng.uniform(0.5, 1.5, (nz, ny, nx)).astype(np.float32), grid)
    out = [(9, 3, 4), (5, 20, 20), (2, 39, 47)]
    wed[out[0]], wed[out[1]], wed[out[2]] = 50.0, np.inf, -0.5
    g = torch.as_tensor(rng.standard_normal((nz, ny, nx)).astype(np.float32), device="cuda")
    for v in out:
        g[v] = 0.0
    plan = pb.hetero.WedPlan(pb.model.PBProblem(grid, lat, None, None), precision=prec)
    want = plan.adjoint(g, wed).clone()
    assert bool(torch.isfinite(want).all()) and float(want.abs().max()) > 0
    for v in out:
        g[v] = bad
    assert torch.equal(plan.adjoint(g, wed), want)
    assert torch.equal(plan.adjoint(g, wed, with_range=True)[0], want)
