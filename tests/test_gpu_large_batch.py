"""A batch of more pairs than the y extent of a CUDA grid (65,535), with tile tables (strand 2 over 64)
among them: accepted, and every score that of the pair alone."""
import numpy as np
import pytest

from bpmax_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_wide_pairs_in_a_batch_over_65535(oracle_mod):
    from bpmax_b200 import Engine

    one = (np.array([1], np.int32), np.array([2], np.int32))
    wide = [W.pair(3, 65, 1), W.pair(2, 130, 2)]
    pairs = [wide[0]] + [one] * 65_536 + [wide[1]]
    e = Engine(0)
    try:
        e.set_weights(W.INTEGER_WEIGHTS)
        got = e.score_batch(pairs)
    finally:
        e.close()
    exp = [oracle_mod.score(oracle_mod.fill(a, b, W.INTEGER_WEIGHTS)[0], len(a), len(b)) for a, b in (*wide, one)]
    assert got[0] == exp[0] and got[-1] == exp[1]
    assert np.all(got[1:-1] == exp[2])
