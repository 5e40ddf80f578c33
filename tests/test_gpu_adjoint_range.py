"""The tensor-core adjoint over FP32's exponent range: weights and dL/dD are scaled by powers of two on the way, so
a power of two on either changes no bit of what it multiplies."""
import numpy as np
import pytest

from conftest import has_gpu, load_pkg

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]


def _grads(nx, ny, w_exp, g_exp, precision):
    import torch
    pb = load_pkg()
    rng = np.random.default_rng(4)
    grid = pb.model.DoseGrid(nx, ny, 3, 0.2, 0.2, 0.2, -0.1 * (nx - 1), -0.1 * (ny - 1), 0.0)
    w = (rng.uniform(0.1, 1.0, (2, 7, 9)).astype(np.float32) * np.float32(2.0) ** w_exp).astype(np.float32)
    lat = pb.model.SpotLattice(9, 7, 2, 0.25, 0.25, 0.03, -0.02, weights=w)
    plan = pb.engines.DosePlan(pb.model.PBProblem(grid, lat, rng.uniform(0.5, 2.0, (2, 3)), rng.uniform(0.3, 0.6, (2, 3))),
                               tables="problem", precision=precision)
    g = rng.uniform(0.4, 1.0, grid.shape).astype(np.float32) * np.float32(2.0) ** g_exp
    one = torch.ones(2, 3, dtype=torch.float64, device="cuda")
    gw, gr = plan.adjoint(torch.as_tensor(g, device="cuda"), didd=one, dsig=one)
    return gw.double().cpu().numpy(), gr.double().cpu().numpy()


@pytest.mark.parametrize("precision", ["fp16x3", "tf32", "bf16"])
@pytest.mark.parametrize("nx, ny", [(40, 33), (150, 140)])
@pytest.mark.parametrize("w_exp, g_exp", [(110, 0), (-60, 0), (0, -110), (0, 110), (60, -118), (-100, 100)])
def test_powers_of_two_change_no_bit(precision, nx, ny, w_exp, g_exp):
    gw0, gr0 = _grads(nx, ny, 0, 0, precision)
    gw, gr = _grads(nx, ny, w_exp, g_exp, precision)
    assert np.array_equal(gw, gw0 * 2.0 ** g_exp)
    assert np.array_equal(gr, gr0 * 2.0 ** (w_exp + g_exp))
