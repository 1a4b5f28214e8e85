"""The delta kernel of the large-cell path at every number of columns a lane can have (30, 45,
75 and 105 modes: one to four), all width types, windows that hold few, all or no mode pairs:
linewidths and adjoint against the oracle where its n^6 products are affordable, beyond that
linewidths and adjoint against each other (linewidths are homogeneous of degree two in the
force constants)."""
import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Options, Problem, QLists, ScatteringRates, synth

pytestmark = pytest.mark.gpu

MESH = {2: (1, 3, 1), 3: (1, 1, 3), 5: (1, 1, 3), 7: (1, 3, 1)}


@pytest.fixture(scope="module")
def row_of_cells(tmp_path_factory, built):
    base = tmp_path_factory.mktemp("rows")
    made = {}

    def get(k):
        if k not in made:
            made[k] = synth.write_config("perovskite_supercell", base / str(k), seed=1, reps=(k, 1, 1))
        return Problem.load(made[k], MESH[k])

    return get


@pytest.mark.parametrize("k,it,sigma", [(2, 1, 1.0), (2, 1, 1e-6), (2, 2, 1.0), (2, 6, 1.0), (3, 2, 1.0), (3, 6, 1.0)])
def test_linewidths_and_adjoint_match_the_oracle(row_of_cells, k, it, sigma):
    prob = row_of_cells(k)
    opts = Options(integrationtype=it, sigma=sigma, isotopescattering=False, seed=3, precision="mixed")
    lists = QLists.monte_carlo(prob, opts)
    lw_bar = np.random.default_rng(5).normal(size=(prob.n_irr, prob.n_mode))
    sr = ScatteringRates(prob)
    lw = sr.generate(opts, lists)
    assert sr.last_path() == 2
    g = sr.adjoint_fc3(opts, lw_bar)
    sr.close()
    gamma, xi, _ = orc.scattering(prob, opts, lists)
    ref, _, _ = orc.finish(prob, opts, lists, gamma, xi)
    # three contractions of BF16 pairs (2^-16 an operand) and FP32 weights: 1e-4 of a linewidth
    # that is not itself a small rest of the sums
    np.testing.assert_allclose(lw, ref, rtol=1e-4, atol=1e-5 * max(np.abs(ref).max(), 1e-300))
    gref = orc.adjoint_fc3(prob, opts, lists, lw_bar)
    assert np.linalg.norm(g - gref) <= 1e-3 * np.linalg.norm(gref)


@pytest.mark.parametrize("k", [2, 5, 7])
@pytest.mark.parametrize("it", [1, 2, 6])
def test_adjoint_and_linewidths_agree(row_of_cells, k, it):
    prob = row_of_cells(k)
    opts = Options(integrationtype=it, isotopescattering=False, seed=3, precision="mixed")
    lists = QLists.monte_carlo(prob, opts)
    lw_bar = np.random.default_rng(5).uniform(0.5, 1.5, size=(prob.n_irr, prob.n_mode))
    sr = ScatteringRates(prob)
    lw = sr.generate(opts, lists)
    g = sr.adjoint_fc3(opts, lw_bar)
    sr.close()
    # Euler: <d L / d Phi, Phi> = 2 L; both sides within 1e-4 of the FP64 value
    left, right = np.vdot(g, prob.fc3_mwm.reshape(g.shape)), 2.0 * np.vdot(lw_bar, lw)
    assert right > 0 and abs(left - right) <= 3e-4 * right
