"""Enumeration of the irreducible q-triplets against the oracle where its kernels change over:
little groups of one thread's size and of one and two warps of operations, operations that
leave the mesh, repeated sample points, samples below, at and above a scan block of 2048."""
import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Options, Problem, QLists, ScatteringRates
from tdep_gb300._native import TdgError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,mesh", [("fcc", (13, 13, 13)), ("rocksalt", (6, 6, 4)), ("perovskite", (4, 6, 4)),
                                       ("supercell", (3, 4, 5)), ("fcc", (1, 1, 1))])
def test_triplets_bit_exact(configs, name, mesh):
    prob = Problem.load(configs[name], mesh)
    sr = ScatteringRates(prob)
    rng = np.random.default_rng(3)
    full = np.arange(1, prob.n_full + 1, dtype=np.int32)
    samples = [full, rng.integers(1, prob.n_full + 1, size=2048).astype(np.int32),
               rng.integers(1, prob.n_full + 1, size=33).astype(np.int32)]
    # the zone centre and the points with the largest and the smallest little groups
    order = np.argsort(prob.irr_nop, kind="stable")
    for q1 in {1, *(int(i) + 1 for i in order[:3]), *(int(i) + 1 for i in order[-4:])}:
        for sample in samples:
            assert sr.triplets(q1, sample) == orc.triplets(prob, q1, sample)
    sr.close()


def _own_lists(prob, size, seed):
    """Another sample for every row, with repeated points."""
    rng = np.random.default_rng(seed)
    lists = QLists.per_irreducible(prob, samples3={q: np.zeros(size, np.int32) for q in range(1, prob.n_irr + 1)})
    lists.list3 = rng.integers(1, prob.n_full + 1, size=lists.list3.size).astype(np.int32)
    return lists


# short lists, merged without a comparison, and lists long enough to be compared first
@pytest.mark.parametrize("mesh,size", [((5, 5, 5), 40), ((8, 8, 8), 400)])
def test_samples_of_their_own_match_the_oracle(configs, mesh, size):
    prob = Problem.load(configs["rocksalt"], mesh)
    opts = Options(isotopescattering=False)
    lists = _own_lists(prob, size, 5)
    sr = ScatteringRates(prob)
    lw = sr.generate(opts, lists)
    gamma, xi, _ = orc.scattering(prob, opts, lists)
    ref, _, _ = orc.finish(prob, opts, lists, gamma, xi)
    np.testing.assert_allclose(lw, ref, rtol=1e-10, atol=1e-14 * np.abs(ref).max())
    # a point off the mesh is refused, and the last scattering stays
    ks = sr.kappa(opts)[1]
    lists.list3[-1] = prob.n_full + 1
    with pytest.raises(TdgError) as err:
        sr.generate(opts, lists)
    assert err.value.code == 5 and "out of range" in str(err.value)
    np.testing.assert_array_equal(sr.kappa(opts)[1], ks)
    sr.close()


def test_one_sample_per_point_by_both_routes(configs):
    """The same sample for all rows of a point: long lists go up once per point, short ones are
    merged from all rows."""
    prob = Problem.load(configs["fcc"], (12, 12, 12))
    opts = Options(isotopescattering=False)
    rng = np.random.default_rng(6)
    every = {q: rng.permutation(prob.n_full).astype(np.int32) + 1 for q in range(1, prob.n_irr + 1)}
    sr = ScatteringRates(prob)
    for take in (prob.n_full, 300):
        lists = QLists.per_irreducible(prob, samples3={q: s[:take] for q, s in every.items()})
        assert (lists.list3.size > 1 << 16) == (take == prob.n_full)
        lw = sr.generate(opts, lists)
        gamma, xi, _ = orc.scattering(prob, opts, lists)
        ref, _, _ = orc.finish(prob, opts, lists, gamma, xi)
        np.testing.assert_allclose(lw, ref, rtol=1e-10, atol=1e-14 * np.abs(ref).max())
    sr.close()
