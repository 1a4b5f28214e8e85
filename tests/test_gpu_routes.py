"""Which form the rules on sizes choose, so that the tests of each form are known to reach it, and
the forms that take a context from one to another."""
import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Options, Problem, QLists, ScatteringRates
from tdep_gb300 import _native as N

pytestmark = pytest.mark.gpu


# the cases of test_gpu_bte_sparse.py, and a mesh below its 128 MB of columns
@pytest.mark.parametrize("name,mesh,it,sigma,form", [("rocksalt", 19, 2, 1.0, 2), ("rocksalt", 18, 1, 3.0, 1),
                                                     ("fcc", 28, 2, 1.0, 2), ("rocksalt", 18, 2, 0.2, 2),
                                                     ("rocksalt", 8, 2, 1.0, 1)])
def test_products_of_the_iterative_solution(configs, name, mesh, it, sigma, form):
    prob = Problem.load(configs[name], (mesh,) * 3)
    opts = Options(integrationtype=it, sigma=sigma, isotopescattering=False, precision="mixed", itermaxsteps=2)
    sr = ScatteringRates(prob)
    sr.generate(opts, QLists.monte_carlo(prob, opts))
    sr.kappa(opts)
    assert sr.last_routes()["bte_products"] == form
    sr.close()


def test_one_context_from_sparse_to_dense_products_and_back(configs):
    prob = Problem.load(configs["rocksalt"], (18,) * 3)
    few = Options(integrationtype=2, isotopescattering=False, precision="mixed", itertol=1e-6, itermaxsteps=25)
    many = Options(**{**few.__dict__, "integrationtype": 1, "sigma": 3.0})
    lists = QLists.monte_carlo(prob, few)
    shared = ScatteringRates(prob)
    for opts, form in ((few, 2), (many, 1), (few, 2), (many, 1)):
        own = ScatteringRates(prob)
        own.generate(opts, lists)
        ref = own.kappa(opts)
        own.close()
        shared.generate(opts, lists)
        got = shared.kappa(opts)
        assert shared.last_routes()["bte_products"] == form
        again = shared.kappa(opts)  # from the second solution on a recorded graph
        for a, b, c in zip(got, again, ref):
            np.testing.assert_array_equal(a, b)
            # Xi is summed in no fixed order
            np.testing.assert_allclose(a, c, rtol=1e-9, atol=1e-9 * np.abs(c).max())
    shared.close()


# 16 384 q-triplets and more at 6 modes, fixed and adaptive widths; fewer; width type 6; a million and
# more at 3 modes, adaptive widths; fewer; one width; 9 modes
@pytest.mark.parametrize("name,mesh,it,taken", [("rocksalt", 12, 2, 1), ("rocksalt", 12, 1, 1), ("rocksalt", 6, 2, 0),
                                                ("rocksalt", 12, 6, 0), ("fcc", 23, 2, 1), ("fcc", 14, 2, 0),
                                                ("fcc", 23, 1, 0), ("fluorite", 12, 2, 0)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_triplets_left_out_before_the_fused_kernel(configs, name, mesh, it, taken, precision):
    prob = Problem.load(configs[name], (mesh,) * 3)
    opts = Options(integrationtype=it, isotopescattering=False, precision=precision)
    sr = ScatteringRates(prob)
    sr.generate(opts, QLists.monte_carlo(prob, opts))
    routes = sr.last_routes()
    assert routes["prescreen"] == taken
    assert 0 < routes["live_triplets"] < sr.stats["triplets"] if taken else routes["live_triplets"] == -1
    sr.close()


@pytest.mark.parametrize("counts,parts", [(1, None), (0, 1)])
def test_samples_merged_in_parts(configs, counts, parts):
    """Rows with samples of their own, points repeated, against the oracle: all at once and a q1 at
    a time."""
    prob = Problem.load(configs["rocksalt"], (6, 6, 6))
    opts = Options(isotopescattering=False, qg3ph=(5, 5, 5), seed=2)
    lists = QLists.monte_carlo(prob, opts)
    sr = ScatteringRates(prob)
    N.check(N.lib().tdg_check_union_counts(sr._ctx, counts), "tdg_check_union_counts")
    lw = sr.generate(opts, lists)
    xi = sr.Xi
    assert sr.last_routes()["sample_parts"] == (parts or prob.n_irr)
    sr.close()
    gamma, xi_ref, _ = orc.scattering(prob, opts, lists)
    ref, _, _ = orc.finish(prob, opts, lists, gamma, xi_ref)
    # FP64 sums of a few thousand terms in another order
    np.testing.assert_allclose(lw, ref, rtol=1e-10, atol=1e-13 * np.abs(ref).max())
    assert (np.abs(xi - xi_ref) <= 1e-9 * np.abs(xi_ref).max()).all()


def test_three_modes_with_triplets_left_out_match_the_oracle(configs):
    prob = Problem.load(configs["fcc"], (23, 23, 23))
    opts = Options(isotopescattering=False)
    lists = QLists.monte_carlo(prob, opts)
    sr = ScatteringRates(prob)
    lw = sr.generate(opts, lists)
    lw32 = sr.generate(Options(**{**opts.__dict__, "precision": "mixed"}), lists)
    assert sr.last_routes()["prescreen"] == 1
    sr.close()
    # the rows of six points over the zone; a point's linewidths are averaged over degenerate
    # modes, which leaves their sum
    for q1 in np.linspace(2, prob.n_irr, 6).astype(int):
        rows = np.nonzero(lists.row_q1 == q1)[0]
        gamma, _, _ = orc.scattering(prob, opts, lists, rows=(rows[0], rows[-1] + 1))
        np.testing.assert_allclose(lw[q1 - 1].sum(), gamma.sum(), rtol=1e-10)
        # FP32 products and weights 1e-6 of a term, exponents of up to 32 amplify to 4e-6
        np.testing.assert_allclose(lw32[q1 - 1].sum(), gamma.sum(), rtol=1e-4)
