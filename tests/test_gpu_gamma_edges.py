"""The gamma kernel where its screen cannot decide (equal sums, magnitudes outside its range, infinities
and NaN), at ragged brick edges and the largest radius, and the percentile select with most keys equal or
nearly equal (candidates of one block and of many).

Bar: map, mask, counts, maximum and percentiles bit for bit the oracle's; the mean within 1e-13."""
import warnings

import numpy as np
import pytest

from conftest import has_gpu, load_pkg
from oracle import gamma_ref as gr

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]

EXACT = ("pass_rate", "gamma_max", "gamma_p95", "gamma_p99", "n_eval", "n_pass", "ref_max",
         "n_dta_offsets")


@pytest.fixture(scope="module")
def pb():
    return load_pkg()


def _doses(case, shape, dtype):
    rng = np.random.default_rng(len(case) + sum(shape))
    z, y, x = (np.arange(n) - (n - 1) / 2 for n in shape)
    bump = np.exp(-(x[None, None] ** 2 + y[None, :, None] ** 2 + z[:, None, None] ** 2) / 60.0)
    ref = (2.0 * bump).astype(dtype)
    if case == "same":                      # every key equal
        ev = ref.copy()
    elif case == "symmetric":               # pairs of offsets with equal sums on the centre planes
        ev = (2.1 * bump ** 1.1).astype(dtype)
    elif case == "scaled":                  # local criterion: keys equal up to rounding
        ev = (ref * dtype(1.02)).astype(dtype)
    elif case == "noise":
        ev = (ref + rng.normal(0, 0.05, shape)).astype(dtype)
    elif case == "wild":                    # beyond the screen's magnitudes, finite
        ev = (ref + rng.normal(0, 0.05, shape)).astype(dtype)
        ev[0, 0, 0], ev[-1, -1, -1] = 3e38, -2e33
    elif case == "nan":
        ev = (ref + rng.normal(0, 0.05, shape)).astype(dtype)
        ev[shape[0] // 2, 0, -1], ev[0, -1, 0] = np.nan, np.inf
    elif case == "tiny":                    # criterion below the screen's range
        ref = (ref * dtype(1e-30)).astype(dtype)
        ev = (ref * dtype(1.01)).astype(dtype)
    return ref, ev


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("case,shape,spacing,kw", [
    ("same", (9, 17, 33), 0.2, {}),
    ("symmetric", (9, 17, 33), 0.1, {}),
    ("symmetric", (13, 9, 7), 0.05, {"dta_mm": 3.0, "max_vox": 6}),      # radius 6 on every axis
    ("scaled", (24, 40, 40), 0.2, {"normalization": "local", "threshold_pct": 0.0}),
    ("noise", (5, 8, 64), 0.2, {"dose_crit_pct": 2.0, "dta_mm": 2.0}),
    ("noise", (4, 7, 31), 0.25, {"dta_mm": 2.0}),                        # no offset but the centre
    ("wild", (8, 16, 40), 0.15, {}),
    ("nan", (8, 16, 40), 0.15, {}),
    ("tiny", (6, 10, 34), 0.15, {}),
])
def test_gamma_edges(pb, case, shape, spacing, kw, dtype):
    ref, ev = _doses(case, shape, dtype)
    sp = (spacing,) * 3
    with warnings.catch_warnings(), np.errstate(all="ignore"):
        warnings.simplefilter("ignore")
        want = gr.gamma_index(ref.astype(np.float64), ev.astype(np.float64), spacing=sp, **kw)
    got = pb.gamma.gamma_index(ref, ev, spacing=sp, **kw)
    assert np.array_equal(got["mask"], want["mask"])
    assert np.array_equal(got["gamma"], want["gamma"], equal_nan=True)
    for k in EXACT:
        assert got[k] == want[k] or (got[k] != got[k] and want[k] != want[k]), (k, got[k], want[k])
    a, b = got["gamma_mean"], want["gamma_mean"]
    assert (a != a and b != b) or a == b or abs(a - b) <= 1e-13 * abs(b)
