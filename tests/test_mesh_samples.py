"""Monte-Carlo samples on a grid that is the mesh: whole rows taken from the stream unseen, with the
rows that hold a small draw, and the stream after them, as point-by-point drawing gives them."""
import ctypes as C

import numpy as np
import pytest

from oracle import binding as orc
from tdep_gb300 import Options, Problem
from tdep_gb300 import _native as N

ALL = 2 ** 64 - 1  # every row point by point


def samples(grid, rows, low, seed=1):
    n = int(np.prod(grid))
    out, nxt = np.zeros((rows, n), np.int32), np.zeros(8, np.uint64)
    g = np.array(grid, np.int32)
    N.check(N.lib().tdg_check_mesh_samples(N.ptr(g, C.c_int32), seed, rows, low, N.ptr(out, C.c_int32),
                                           N.ptr(nxt, C.c_uint64)), "tdg_check_mesh_samples")
    return out, nxt


# 104 points take exactly one block of 312 words, 52 half of one, 60 and 27 no whole share; 40 000
# points more rows than one batch holds
@pytest.mark.parametrize("grid,rows", [((4, 26, 1), 40), ((13, 2, 2), 31), ((3, 4, 5), 50), ((3, 3, 3), 64),
                                       ((1, 1, 1), 700), ((40, 40, 25), 7)])
def test_rows_with_small_draws(built, grid, rows):
    plain, after = samples(grid, rows, ALL)
    np.testing.assert_array_equal(plain, np.arange(1, plain.shape[1] + 1)[None].repeat(rows, 0))
    n = plain.shape[1]
    # from no row to nearly all with a draw below it
    for share in (0.0, 0.05, 0.5, 0.95):
        low = int(2.0 ** 64 * (1.0 - (1.0 - share) ** (1.0 / (3 * n))))
        got, then = samples(grid, rows, low)
        np.testing.assert_array_equal(got, plain)
        np.testing.assert_array_equal(then, after)


def test_the_stream_is_the_generator_s(built):
    """Without rows the words are the seeded generator's; a row takes three per point."""
    _, first = samples((3, 4, 5), 0, ALL, seed=4)
    ref = orc.mt_sequence(8 + 180 * 3, seed=4)
    np.testing.assert_array_equal(first, ref[:8])
    for low in (0, ALL):
        np.testing.assert_array_equal(samples((3, 4, 5), 3, low, seed=4)[1], ref[540:548])


def test_lists_match_the_oracle(configs):
    prob = Problem.load(configs["fcc"], (5, 4, 3))
    opts = Options(seed=7)
    want = orc.mc_qlists(prob, opts)
    for low in (0, 2 ** 58, ALL):
        got, _ = samples((5, 4, 3), want.n_row, low, seed=7)
        np.testing.assert_array_equal(got.ravel(), want.list3)
