"""Iterative BTE on the device against the oracle where its kernels can go wrong: degenerate
sets of one to three modes, sets that overlap without being equal (each mode's set is the
caller's), fewer modes than a warp and more than one."""
import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Options, Problem, QLists, ScatteringRates

pytestmark = pytest.mark.gpu


def _overlapping(prob):
    """Modes 1-2, 1-2-3 and 2-3 averaged together, and a set listed out of order."""
    dg, dm = np.ones_like(prob.degen), np.zeros_like(prob.degen_mode)
    dm[:, :, 0] = np.arange(1, prob.n_mode + 1)
    for b, members in ((0, (1, 2)), (1, (3, 1, 2)), (2, (3, 2))):
        dg[:, b] = len(members)
        dm[:, b, :len(members)] = members
    prob.degen, prob.degen_mode = dg, dm


# 3 to 30 modes; meshes on which operations of a point's little group leave the mesh (unequal
# dimensions); the identity alone and rows in two items (30 modes); columns of one
# and of many chunks, even and odd in number
@pytest.mark.parametrize("name,mesh,overlap", [
    ("fcc", (5, 5, 5), False), ("fcc", (6, 6, 6), True), ("fcc", (3, 4, 5), False), ("fcc", (16, 16, 16), False),
    ("rocksalt", (6, 6, 6), False), ("rocksalt", (5, 5, 5), True), ("rocksalt", (6, 6, 4), False),
    ("rocksalt", (13, 13, 13), False), ("fluorite", (5, 5, 5), False), ("l12", (4, 4, 4), False),
    ("perovskite", (4, 4, 4), False), ("perovskite", (4, 4, 3), True), ("supercell", (3, 3, 3), False)])
def test_iterative_solution_matches_the_oracle(configs, name, mesh, overlap):
    prob = Problem.load(configs[name], mesh)
    if overlap:
        _overlapping(prob)
    opts = Options(integrationtype=2, isotopescattering=False, itertol=1e-7, itermaxsteps=60,
                   precision="mixed" if prob.n_mode > 18 else "fp64")
    lists = QLists.monte_carlo(prob, opts)
    sr = ScatteringRates(prob)
    lw = sr.generate(opts, lists)
    ks, ki = sr.kappa(opts)
    # the oracle's solution on the device's own linewidths and scattering matrix: what is
    # compared is the iteration
    xi, qs = sr.Xi, 2.0 * lw
    v = prob.vel[prob.irr_full - 1]
    with np.errstate(divide="ignore", invalid="ignore"):
        f0 = np.where(lw[..., None] > 1e-9, v / qs[..., None], 0.0)
    ks_ref, ki_ref, n_iter = orc.kappa(prob, opts, lists, xi, qs.ravel(), np.ascontiguousarray(f0).ravel(),
                                       opts.itermaxsteps, opts.itertol)
    assert sr.n_iter == n_iter
    # double-float products: 2^-44 of a row's sum of magnitudes, over at most 60 iterations
    for got, ref in ((ks, ks_ref), (ki, ki_ref)):
        np.testing.assert_allclose(got, ref, rtol=1e-10, atol=1e-10 * np.abs(ref).max())
    again = sr.kappa(opts)[1]  # a replayed graph, from F0 again
    np.testing.assert_array_equal(again, ki)
    sr.close()
