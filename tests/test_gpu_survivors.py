"""The screened contraction of the SIMT three-phonon kernel against the oracle: every mode
count it is built for, few survivors (adaptive widths), nearly all of them (a broad fixed
width), none at all (a width below every mismatch), second and third stages in one and in
several passes over b1, and its adjoint."""
import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Options, Problem, QLists, ScatteringRates, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def crystal18(tmp_path_factory, built):
    """Six atoms (18 modes): three rocksalt cells in a row."""
    def config(seed=1):
        cell, pot, cutoff = synth.config_rocksalt(seed=seed)
        return synth.supercell(cell, (3, 1, 1)), pot, cutoff

    synth.CONFIGS["rocksalt_row"] = config
    return synth.write_config("rocksalt_row", tmp_path_factory.mktemp("row") / "row", seed=1)


def _case(configs, crystal18, name, mesh):
    prob = Problem.load(crystal18 if name == "row" else configs[name], mesh)
    opts = dict(isotopescattering=False, seed=3)
    return prob, opts


CELLS = [("fcc", (5, 5, 5)), ("rocksalt", (5, 5, 5)), ("fluorite", (4, 4, 4)), ("l12", (3, 3, 3)),
         ("perovskite", (3, 3, 3)), ("row", (2, 3, 3))]


@pytest.mark.parametrize("name,mesh", CELLS)
@pytest.mark.parametrize("it,sigma", [(1, 2.0), (1, 1e-6), (2, 1.0), (6, 1.0)])
def test_fp64_rows_match_the_oracle(configs, crystal18, name, mesh, it, sigma):
    prob, kw = _case(configs, crystal18, name, mesh)
    opts = Options(integrationtype=it, sigma=sigma, **kw)
    lists = QLists.monte_carlo(prob, opts)
    sr = ScatteringRates(prob)
    lw = sr.generate(opts, lists)
    assert sr.last_path() == 0
    sr.close()
    gamma, xi, _ = orc.scattering(prob, opts, lists)
    ref, _, _ = orc.finish(prob, opts, lists, gamma, xi)
    # sums of like terms over at most 125 points and n^2 modes, n^3 products each: 1e-10
    # covers the order of summation in both
    np.testing.assert_allclose(lw, ref, rtol=1e-10, atol=1e-14 * max(np.abs(ref).max(), 1e-300))


@pytest.mark.parametrize("name,mesh", CELLS)
@pytest.mark.parametrize("it", [1, 2, 6])
def test_mixed_rows_match_fp64(configs, crystal18, name, mesh, it):
    prob, kw = _case(configs, crystal18, name, mesh)
    o64 = Options(integrationtype=it, sigma=1.0, **kw)
    o32 = Options(**{**o64.__dict__, "precision": "mixed", "tensor_cores": 2})
    lists = QLists.monte_carlo(prob, o64)
    sr = ScatteringRates(prob)
    lw64, lw32 = sr.generate(o64, lists), sr.generate(o32, lists)
    assert sr.last_path() == 0
    sr.close()
    # FP32 products and weights: 1e-6 of a term, Gaussians with exponents up to 32 amplify the
    # rounding of their argument to 4e-6
    np.testing.assert_allclose(lw32, lw64, rtol=1e-4, atol=1e-5 * np.abs(lw64).max())


@pytest.mark.parametrize("name,mesh", CELLS)
@pytest.mark.parametrize("it", [1, 2, 6])
def test_fp64_adjoint_matches_the_oracle(configs, crystal18, name, mesh, it):
    prob, kw = _case(configs, crystal18, name, mesh)
    opts = Options(integrationtype=it, sigma=1.0, **kw)
    lists = QLists.monte_carlo(prob, opts)
    lw_bar = np.random.default_rng(1).normal(size=(prob.n_irr, prob.n_mode))
    sr = ScatteringRates(prob)
    sr.generate(opts, lists)
    grad = sr.adjoint_fc3(opts, lw_bar)
    sr.close()
    ref = orc.adjoint_fc3(prob, opts, lists, lw_bar)
    np.testing.assert_allclose(grad, ref, rtol=1e-9, atol=1e-10 * np.abs(ref).max())
