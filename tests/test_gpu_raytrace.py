"""Water-equivalent depth for every number of runs the kernel takes, at the edges of their depths: a few
columns (up to 16 runs), 16,000 (4) and 100,000 (1), grids that start above, at and below depth 0.

Oracle: the path sums in float64."""
import numpy as np
import pytest

from conftest import has_gpu, load_pkg

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]


@pytest.mark.parametrize("ny, nx, depths", [
    (5, 7, (1, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 300)),
    (127, 126, (1, 8, 9, 32, 33, 70)), (125, 129, (1, 8, 9, 32, 33, 70)), (317, 316, (1, 8, 9, 33)),
    (400, 251, (1, 8, 9, 33))])
@pytest.mark.parametrize("oz", [0.0, -0.75, 1.3])
def test_raytrace_at_every_run_count(ny, nx, depths, oz):
    import torch
    pb = load_pkg()
    rng = np.random.default_rng(nx)
    for nz in depths:
        dz = 0.25
        rho = rng.uniform(0.0, 3.0, (nz, ny, nx)).astype(np.float32)
        g = dict(nz=nz, ny=ny, nx=nx, oz=oz, dz=dz)
        z = oz + np.arange(nz) * dz
        lo, mid, hi = (np.maximum(z + s, 0.0)[:, None, None] for s in (-0.5 * dz, 0.0, 0.5 * dz))
        r = rho.astype(np.float64)
        through = r * (hi - lo)
        want = max(oz - 0.5 * dz, 0.0) + np.cumsum(through, axis=0) - through + r * (mid - lo)
        got = pb.hetero.wed_raytrace(rho, g).cpu().numpy()
        # nz + 1 additions of positive terms, each rounded, in another order than the oracle's
        assert np.max(np.abs(got - want)) <= 2 * (nz + 2) * 2.0 ** -53 * np.max(want) + 1e-300
        assert got.dtype == np.float64 and torch.cuda.is_available()
