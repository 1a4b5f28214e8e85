"""Isotope scattering on the device against the oracle: columns (q2, b2) around the edge of
the kernel's 2048-column tile, the three smearings, one to five atoms."""
import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Options, Problem, QLists, ScatteringRates

pytestmark = pytest.mark.gpu


# 192, 2058, 3750 and 4320 columns: part of a tile, one full tile and 10 columns, odd sizes
@pytest.mark.parametrize("name,mesh", [("fcc", 4), ("rocksalt", 7), ("fluorite", 5), ("perovskite", 5), ("l12", 6)])
@pytest.mark.parametrize("it", [1, 2, 6])
def test_isotope_rows_match_the_oracle(configs, name, mesh, it):
    prob = Problem.load(configs[name], (mesh,) * 3)
    prob.mass_disorder = 1e-4 * (1.0 + np.arange(prob.n_atom))
    opts = Options(integrationtype=it, sigma=0.7, thirdorder=False)
    lists = QLists.per_irreducible(prob)
    sr = ScatteringRates(prob)
    lw, xi = sr.generate(opts, lists), sr.Xi
    sr.close()
    gamma, xi_ref, _ = orc.scattering(prob, opts, lists)
    lw_ref, _, _ = orc.finish(prob, opts, lists, gamma, xi_ref)
    # The exponent, at most 32, carries 4 roundings: 1.5e-14 of a term; the strength, the
    # factors and the orbit means of these non-negative terms a few more. 1e-12 leaves a
    # margin of 50.
    np.testing.assert_allclose(lw, lw_ref, rtol=1e-12, atol=0)
    np.testing.assert_allclose(xi, xi_ref, rtol=1e-12, atol=0)
