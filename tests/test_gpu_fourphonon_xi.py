"""Every element of the four-phonon scattering matrix against the oracle, without exception: with
little groups of the identity alone no orbit is averaged, so that no element of analytically
zero sum decides by its rounding over a mean."""
import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Options, Problem, QLists, ScatteringRates, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,mesh,points", [("fcc_morse", 6, 12), ("rocksalt", 5, 6), ("fluorite", 4, 4), ("l12", 3, 3),
                                              ("perovskite", 3, 2)])
@pytest.mark.parametrize("it", [1, 2, 6])
def test_elements_match_the_oracle(tmp_path, built, name, mesh, points, it):
    prob = Problem.load(synth.write_config(name, tmp_path / name, seed=1, order4=True), (mesh,) * 3, fourthorder=True)
    assert (prob.irr_ops[:, 0] == 1).all()  # the identity
    prob.irr_nop = np.ones_like(prob.irr_nop)
    rng = np.random.default_rng(6)
    draw = lambda: np.sort(rng.choice(prob.n_full, points, replace=False)).astype(np.int32) + 1  # noqa: E731
    lists = QLists.per_irreducible(prob, samples4={q: (draw(), draw()) for q in range(1, prob.n_irr + 1)})
    opts = Options(integrationtype=it, isotopescattering=False, thirdorder=False, fourthorder=True)
    sr = ScatteringRates(prob)
    sr.generate(opts, lists)
    xi = sr.Xi
    sr.generate(Options(**{**opts.__dict__, "precision": "mixed"}), lists)
    xi32 = sr.Xi
    sr.close()
    gamma, ref, _ = orc.scattering(prob, opts, lists)
    orc.finish(prob, opts, lists, gamma, ref)
    top = np.abs(ref).max()
    assert top > 0
    # up to n^3 = 3375 terms an element, each right to some 2e-14 of its size (contraction of 4 n
    # products, exponent up to 32), of the size of the largest element at most
    assert np.abs(xi - ref).max() <= 1e-10 * top
    # 4e-6 a term in FP32, of either sign
    assert np.abs(xi32 - ref).max() <= 1e-4 * top
