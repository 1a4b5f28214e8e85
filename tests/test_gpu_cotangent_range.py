"""The tensor-core adjoint with cotangents beyond the range of its FP32 pairs: the gradient is linear
in them, so a power of two on the cotangent is the same power of two on the gradient."""
import numpy as np
import pytest

from tdep_gb300 import Options, Problem, QLists, ScatteringRates

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["fluorite", "l12", "perovskite"])
@pytest.mark.parametrize("iterated", [False, True])
def test_gradient_is_linear_in_the_cotangent(configs, name, iterated):
    prob = Problem.load(configs[name], (4, 4, 4))
    opts = Options(precision="mixed", isotopescattering=False)
    sr = ScatteringRates(prob)
    lw = sr.generate(opts, QLists.monte_carlo(prob, opts))
    assert sr.last_path() == 1
    sr.kappa(opts)
    bar = np.eye(3) + 0.25 * (np.ones((3, 3)) - np.eye(3))
    direct = np.random.default_rng(4).normal(size=lw.shape)

    def gradient(power):
        # iterated: the scattering matrix has a cotangent as well (kappa_iter_vjp)
        lw_bar = sr.kappa_iter_vjp(opts, np.ldexp(bar, power)) if iterated else np.ldexp(direct, power)
        return sr.adjoint_fc3(opts, lw_bar)

    ref = gradient(0)
    assert np.isfinite(ref).all() and np.abs(ref).max() > 0
    for power in (-140, -61, 61, 140):
        got = np.ldexp(gradient(power), -power)
        # the same FP32 operations, but for what the smallest terms lose below 2^-126
        np.testing.assert_allclose(got, ref, rtol=1e-6, atol=1e-6 * np.abs(ref).max())
    sr.close()
