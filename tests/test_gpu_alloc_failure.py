"""Calls on a context whose earlier call ran out of device memory (tdg_check_alloc_failure)."""
from itertools import count

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


def run(sr, opts, lists):
    return {"linewidth": sr.generate(opts, lists), "xi": sr.Xi}


def every_failure(prob, opts, lists, steps=run):
    """Fails allocation 0, 1, 2, ... of the calls in `steps`, each on a new context, until none is
    left, and compares the same calls made again with those of a context without a failure.
    Returns how many failed."""
    sr = ScatteringRates(prob)
    ref = steps(sr, opts, lists)
    sr.close()
    assert all(np.abs(v).max() > 0 for v in ref.values())
    for after in count():
        N.lib().tdg_release_cached_memory(0)  # the context before holds these calls' values in its blocks
        sr = ScatteringRates(prob)
        N.lib().tdg_check_alloc_failure(after)
        try:
            steps(sr, opts, lists)
            failed = False
        except N.TdgError as e:
            assert e.code == 8
            failed = True
        finally:
            N.lib().tdg_check_alloc_failure(-1)
        if not failed:
            sr.close()
            return after
        got = steps(sr, opts, lists)
        sr.close()
        for k, v in ref.items():
            # FP64 sums of up to 1e4 terms in the order in which the device adds them; gradients
            # are summed in FP32
            tol = 1e-5 if k == "grad" else 1e-9
            np.testing.assert_allclose(got[k], v, rtol=tol, atol=1e-2 * tol * np.abs(v).max(),
                                       err_msg=f"{k}, allocation {after}")


# samples that go up as they are (fcc 4^3), and one per q1 (more than 65 536 entries: fcc 10^3)
@pytest.mark.parametrize("name,mesh,precision", [("fcc", 4, "fp64"), ("fcc", 10, "fp64"), ("rocksalt", 4, "mixed"),
                                                 ("fluorite", 4, "mixed")])
def test_generate_after_a_failed_allocation(configs, name, mesh, precision):
    prob = Problem.load(configs[name], (mesh,) * 3)
    opts = Options(precision=precision, isotopescattering=False)
    assert every_failure(prob, opts, QLists.monte_carlo(prob, opts)) > 10


def test_isotopes_after_a_failed_allocation(configs):
    prob = Problem.load(configs["rocksalt"], (4, 4, 4))
    prob.mass_disorder = 1e-4 * (1.0 + np.arange(prob.n_atom))
    opts = Options(thirdorder=False)
    assert every_failure(prob, opts, QLists.per_irreducible(prob)) > 5


def solve(sr, opts, lists):
    out = run(sr, opts, lists)
    out["kappa_sma"], out["kappa_iter"] = sr.kappa(opts)
    out["kappa_offdiag"] = sr.kappa_offdiag(opts)
    return out


@pytest.mark.parametrize("name", ["fcc", "rocksalt"])
def test_solve_after_a_failed_allocation(configs, name):
    prob = Problem.load(configs[name], (4, 4, 4))
    opts = Options(precision="mixed")
    assert every_failure(prob, opts, QLists.monte_carlo(prob, opts), solve) > 40


def fit(sr, opts, lists):
    lw = sr.generate(opts, lists)
    return {"linewidth": lw, "xi": sr.Xi, "grad": sr.adjoint_fc3(opts, np.ones_like(lw))}


# the fused kernels and, without symmetry, the large-cell path with padded operand planes
@pytest.mark.parametrize("name,mesh", [("rocksalt", 4), ("fluorite", 4), ("supercell", 3)])
def test_gradient_after_a_failed_allocation(configs, name, mesh):
    prob = Problem.load(configs[name], (mesh,) * 3)
    opts = Options(precision="mixed", isotopescattering=False)
    assert every_failure(prob, opts, QLists.monte_carlo(prob, opts), fit) > 20


def test_gradient_of_the_scattering_before_a_failed_one(configs):
    """Until a call replaces what the last one left, its gradient stays; from then on there is none
    to ask for, whatever the call comes to."""
    prob = Problem.load(configs["fluorite"], (4, 4, 4))
    opts = Options(precision="mixed", isotopescattering=False)
    few = QLists.per_irreducible(prob, samples3={q: np.array([1, 5, 9]) for q in range(1, prob.n_irr + 1)})
    many = QLists.monte_carlo(prob, opts)
    wrong = QLists.per_irreducible(prob, samples3={q: np.array([1, 5, 9]) for q in range(1, prob.n_irr + 1)})
    wrong.list3[-1] = prob.n_full + 1
    refused = kept = 0
    for after in count():
        sr = ScatteringRates(prob)
        bar = np.ones_like(sr.generate(opts, few))
        ref = sr.adjoint_fc3(opts, bar)
        with pytest.raises(N.TdgError) as e:
            sr.generate(opts, wrong)
        assert e.value.code == 5
        np.testing.assert_array_equal(sr.adjoint_fc3(opts, bar), ref)
        N.lib().tdg_check_alloc_failure(after)
        try:
            sr.generate(opts, many)
            failed = False
        except N.TdgError as x:
            assert x.code == 8
            failed = True
        finally:
            N.lib().tdg_check_alloc_failure(-1)
        if failed:
            try:
                np.testing.assert_array_equal(sr.adjoint_fc3(opts, bar), ref)
                kept += 1
            except N.TdgError as x:
                assert x.code == 5
                refused += 1
        sr.close()
        if not failed:
            break
    assert refused > 3 and kept > 0
