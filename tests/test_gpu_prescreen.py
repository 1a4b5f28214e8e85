"""Three-phonon rows where the q-triplets without a survivor are left out before the fused kernel
(3 and 6 modes, 16 384 q-triplets or more), against the oracle: adaptive and fixed widths, one
that nothing survives, sampled rows."""
import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Options, Problem, QLists, ScatteringRates

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,mesh,it,sigma,qg", [("rocksalt", 12, 2, 1.0, None), ("rocksalt", 12, 1, 0.5, None),
                                                   ("rocksalt", 12, 1, 1e-7, None), ("rocksalt", 14, 2, 0.3, (8, 8, 8)),
                                                   ("fcc", 14, 2, 1.0, None), ("fcc", 14, 1, 1.0, None)])
def test_rows_match_the_oracle(configs, name, mesh, it, sigma, qg):
    prob = Problem.load(configs[name], (mesh,) * 3)
    kw = {} if qg is None else {"qg3ph": qg}
    opts = Options(integrationtype=it, sigma=sigma, isotopescattering=False, seed=3, **kw)
    lists = QLists.monte_carlo(prob, opts)
    sr = ScatteringRates(prob)
    lw = sr.generate(opts, lists)
    assert sr.stats["triplets"] >= 16384
    lw32 = sr.generate(Options(**{**opts.__dict__, "precision": "mixed"}), lists)
    sr.close()
    gamma, xi, _ = orc.scattering(prob, opts, lists)
    ref, _, _ = orc.finish(prob, opts, lists, gamma, xi)
    # sums of like terms over a few thousand points: 1e-10 covers the order of summation; FP32
    # products and weights 1e-6 of a term, Gaussians with exponents up to 32 amplify to 4e-6
    np.testing.assert_allclose(lw, ref, rtol=1e-10, atol=1e-14 * max(np.abs(ref).max(), 1e-300))
    np.testing.assert_allclose(lw32, ref, rtol=1e-4, atol=1e-5 * max(np.abs(ref).max(), 1e-300))
