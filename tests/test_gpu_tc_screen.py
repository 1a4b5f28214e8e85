"""The screen of the tensor-core three-phonon kernel at every mode count it is built for: windows
that hold nearly all, few, or no mode triplets, and the width type that is not screened, against
FP64."""
import numpy as np
import pytest

from tdep_gb300 import Options, Problem, QLists, ScatteringRates

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,mesh", [("fluorite", 4), ("l12", 4), ("perovskite", 4)])
@pytest.mark.parametrize("it,sigma", [(1, 2.0), (1, 1e-6), (2, 1.0), (2, 0.1), (6, 1.0)])
def test_rows_match_fp64(configs, name, mesh, it, sigma):
    prob = Problem.load(configs[name], (mesh,) * 3)
    o64 = Options(integrationtype=it, sigma=sigma, isotopescattering=False, seed=3)
    lists = QLists.monte_carlo(prob, o64)
    sr = ScatteringRates(prob)
    lw64 = sr.generate(o64, lists)
    lw = sr.generate(Options(**{**o64.__dict__, "precision": "mixed"}), lists)
    assert sr.last_path() == 1
    sr.close()
    # BF16 pairs 1e-5 a product, FP32 weights 4e-6
    np.testing.assert_allclose(lw, lw64, rtol=1e-4, atol=1e-5 * max(np.abs(lw64).max(), 1e-300))
