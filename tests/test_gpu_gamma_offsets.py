"""The gamma index with every offset of the largest radius inside the distance to agreement (13^3 of
them: the kernel's largest shared memory) and with the sizes just below.

Bar: the oracle's map bit for bit."""
import numpy as np
import pytest

from conftest import has_gpu, load_pkg
from oracle import gamma_ref as gr

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dta_mm", [3.0, 2.58, 2.5])       # at 0.25 mm: all 2197 offsets, all but the corners, fewer
def test_gamma_with_the_largest_radius(dtype, dta_mm):
    pb = load_pkg()
    rng = np.random.default_rng(4)
    shape = (7, 9, 35)
    ref = rng.uniform(0.5, 2.0, shape).astype(dtype)
    ev = (ref * rng.normal(1.0, 0.05, shape)).astype(dtype)
    kw = dict(spacing=(0.025,) * 3, dose_crit_pct=0.5, dta_mm=dta_mm)
    want = gr.gamma_index(ref.astype(np.float64), ev.astype(np.float64), **kw)
    assert (want["n_dta_offsets"] == 13 ** 3) == (dta_mm == 3.0)
    got = pb.gamma.gamma_index(ref, ev, **kw)
    assert got["n_dta_offsets"] == want["n_dta_offsets"]
    assert np.array_equal(got["gamma"], want["gamma"]) and np.array_equal(got["mask"], want["mask"])
