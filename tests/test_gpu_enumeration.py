"""Enumeration of the irreducible q-triplets against the oracle where its kernels change over:
little groups of one thread's size and of one and two warps of operations, operations that
leave the mesh, repeated sample points, samples below, at and above a scan block of 2048."""
import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Problem, ScatteringRates

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
