"""The gradient slices of the mixed adjoint: triplet counts that are and are not a multiple of
four (the tensor-core slices hold quads), and the Xi row terms' cotangents as FP32 pairs,
against the FP64 adjoint."""
import numpy as np
import pytest

from tdep_gb300 import Options, Problem, QLists, ScatteringRates

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,mesh", [("fluorite", (4, 4, 4)), ("l12", (4, 4, 4)), ("perovskite", (4, 4, 4))])
@pytest.mark.parametrize("iterative", [False, True])
def test_mixed_gradient_matches_fp64(configs, name, mesh, iterative):
    # 195, 220 and 1115 force-constant triplets
    prob = Problem.load(configs[name], mesh)
    out = {}
    for precision in ("fp64", "mixed"):
        opts = Options(integrationtype=2, isotopescattering=False, seed=3, precision=precision)
        lists = QLists.monte_carlo(prob, opts)
        sr = ScatteringRates(prob)
        sr.generate(opts, lists)
        assert (sr.last_path() == 1) == (precision == "mixed")
        if iterative:
            sr.kappa(opts)
            lw_bar = sr.kappa_iter_vjp(opts, np.eye(3))
        else:
            lw_bar = np.random.default_rng(4).normal(size=(prob.n_irr, prob.n_mode))
        out[precision] = sr.adjoint_fc3(opts, lw_bar)
        sr.close()
    # BF16 pairs through six contractions: 1e-4 of the gradient's norm, times the condition of
    # the iterated solution where the cotangents come from it
    d = np.linalg.norm(out["mixed"] - out["fp64"])
    assert d <= 1e-3 * np.linalg.norm(out["fp64"])
