"""The screened four-phonon kernel against the oracle: every mode count it is built for (b1 in
batches or one at a time, a thread per output or per column), few survivors, nearly all and
none, in FP64, and the mixed path against FP64."""
import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Options, Problem, QLists, ScatteringRates, synth

pytestmark = pytest.mark.gpu

CELLS = [("fcc_morse", 6), ("rocksalt", 5), ("fluorite", 4), ("l12", 3), ("perovskite", 3)]


@pytest.fixture(scope="module")
def crystals(tmp_path_factory, built):
    base = tmp_path_factory.mktemp("fourth")
    return {name: synth.write_config(name, base / name, seed=1, order4=True) for name, _ in CELLS}


def _pairs(prob, k):
    rng = np.random.default_rng(4)
    pts = np.arange(1, prob.n_full + 1)
    draw = lambda: np.sort(rng.choice(pts, size=min(k, prob.n_full), replace=False)).astype(np.int32)  # noqa: E731
    return QLists.per_irreducible(prob, samples4={q: (draw(), draw()) for q in range(1, prob.n_irr + 1)})


@pytest.mark.parametrize("name,mesh", CELLS)
@pytest.mark.parametrize("it,sigma", [(1, 1.0), (1, 1e-6), (2, 1.0), (6, 1.0)])
def test_rows_match_the_oracle(crystals, name, mesh, it, sigma):
    prob = Problem.load(crystals[name], (mesh,) * 3, fourthorder=True)
    # the oracle costs n^8 per row and q-quartet
    lists = _pairs(prob, {3: 12, 6: 6, 9: 4, 12: 3, 15: 2}[prob.n_mode])
    o64 = Options(integrationtype=it, sigma=sigma, isotopescattering=False, thirdorder=False, fourthorder=True)
    o32 = Options(**{**o64.__dict__, "precision": "mixed"})
    sr = ScatteringRates(prob)
    lw, lw32 = sr.generate(o64, lists), None
    xi = sr.Xi
    lw32 = sr.generate(o32, lists)
    sr.close()
    gamma, xi_ref, _ = orc.scattering(prob, o64, lists)
    ref, _, _ = orc.finish(prob, o64, lists, gamma, xi_ref)
    scale = max(np.abs(ref).max(), 1e-300)
    # sums of at most n^3 terms, n^4 products each, in another order
    np.testing.assert_allclose(lw, ref, rtol=1e-10, atol=1e-13 * scale)
    # an entry of analytically zero sum may enter an orbit's average on one side only
    far = np.abs(xi - xi_ref) > 1e-9 * max(np.abs(xi_ref).max(), 1e-300)
    assert far.mean() < 1e-3
    # FP32 weights and Psi; 1e-6 a term, 4e-6 from exponents of up to 32
    np.testing.assert_allclose(lw32, lw, rtol=1e-4, atol=1e-5 * scale)
