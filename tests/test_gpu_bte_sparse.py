"""The iterative BTE where the compacted scattering matrix is large enough for the sparse form:
few non-zero elements (adaptive widths: the form is taken) and many (a wide fixed one: it is
not), rows with none at all, against the oracle's iteration on the device's own matrix."""
import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Options, Problem, QLists, ScatteringRates

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,mesh,it,sigma", [("rocksalt", 19, 2, 1.0), ("rocksalt", 18, 1, 3.0), ("fcc", 28, 2, 1.0),
                                                ("rocksalt", 18, 2, 0.2)])
def test_iterative_solution_matches_the_oracle(configs, name, mesh, it, sigma):
    prob = Problem.load(configs[name], (mesh,) * 3)
    opts = Options(integrationtype=it, sigma=sigma, isotopescattering=False, itertol=1e-6, itermaxsteps=25,
                   precision="mixed")
    lists = QLists.monte_carlo(prob, opts)
    sr = ScatteringRates(prob)
    lw = sr.generate(opts, lists)
    ks, ki = sr.kappa(opts)
    xi, qs = sr.Xi, 2.0 * lw
    v = prob.vel[prob.irr_full - 1]
    with np.errstate(divide="ignore", invalid="ignore"):
        f0 = np.where(lw[..., None] > 1e-9, v / qs[..., None], 0.0)
    ks_ref, ki_ref, n_iter = orc.kappa(prob, opts, lists, xi, qs.ravel(), np.ascontiguousarray(f0).ravel(),
                                       opts.itermaxsteps, opts.itertol)
    assert sr.n_iter == n_iter
    # double-float products: 2^-44 of a row's sum of magnitudes, over at most 25 iterations
    for got, ref in ((ks, ks_ref), (ki, ki_ref)):
        np.testing.assert_allclose(got, ref, rtol=1e-10, atol=1e-10 * np.abs(ref).max())
    again = sr.kappa(opts)[1]  # a replayed graph, from F0 again
    np.testing.assert_array_equal(again, ki)
    # another matrix in the same context, and the first one again
    hot = Options(**{**opts.__dict__, "temperature": 600.0})
    sr.generate(hot, lists)
    sr.kappa(hot)
    sr.generate(opts, lists)
    np.testing.assert_allclose(sr.kappa(opts)[1], ki, rtol=1e-9, atol=1e-9 * np.abs(ki).max())
    sr.close()
