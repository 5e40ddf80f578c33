"""Depth tables at the sizes where the table builder changes its way: fewer depths than a block
holds, whole and ragged blocks, and both sides of the line between summing two curve points per
depth and building the whole curve (4 nz against n_fine)."""
import importlib

import numpy as np
import pytest

from oracle import physics_ref as pr

pytestmark = pytest.mark.gpu

# Sums of at most 2 * 600 products: 1200 * 2^-53 = 1.4e-13 of the largest term, and the last bits of
# log, exp and of the range table's searches, steepest at the range's end (100 MeV/cm and more).
TOL = 1e-11


@pytest.fixture(scope="module")
def pb():
    return importlib.import_module("gpu-proton-dose-engine_b200")


@pytest.mark.parametrize("model", ["bohr", "none"])
@pytest.mark.parametrize("nz", [1, 7, 8, 9, 149, 150])
def test_tables_vs_oracle(pb, nz, model):
    n_fine = 600
    spread = 0.0033 if model == "bohr" else 0.0        # "none": no straggling at all
    en = pr.layer_energies(3, 4.0, 9.0)
    z = 0.3 + np.arange(nz) * (11.0 / max(nz, 8))      # the last depths lie past every range
    idd_model = pb.physics.IDDModel(straggling_model=model, energy_spread=spread, n_fine=n_fine)
    idd, sig = pb.physics.layer_luts(z, en, idd_model=idd_model)
    ri = np.stack([pr.idd_fluence(z, e, energy_spread=spread, n_fine=n_fine, model=model) for e in en])
    rs = np.stack([pr.fermi_eyges_sigma(z, e, sigma_x0=0.30) for e in en])
    assert np.max(np.abs(idd - ri)) <= TOL * np.max(np.abs(ri))
    assert np.max(np.abs(sig - rs)) <= TOL * np.max(rs)
