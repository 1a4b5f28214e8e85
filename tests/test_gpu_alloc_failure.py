"""Calls on a context whose earlier call ran out of device memory (tdg_check_alloc_failure)."""
import numpy as np
import pytest

from tdep_gb300 import Options, Problem, QLists, ScatteringRates
from tdep_gb300 import _native as N

pytestmark = pytest.mark.gpu


def test_the_next_call_does_not_find_the_error_again(configs):
    prob = Problem.load(configs["fcc"], (4, 4, 4))
    opts = Options(isotopescattering=False)
    lists = QLists.monte_carlo(prob, opts)
    sr = ScatteringRates(prob)
    ref = sr.generate(opts, lists)
    sr.close()
    sr = ScatteringRates(prob)
    N.lib().tdg_check_alloc_failure(0)
    try:
        with pytest.raises(N.TdgError) as e:
            sr.generate(opts, lists)
        assert e.value.code == 8
    finally:
        N.lib().tdg_check_alloc_failure(-1)
    got = sr.generate(opts, lists)
    sr.close()
    # the same non-negative sums in the order in which the device adds them
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=0)
