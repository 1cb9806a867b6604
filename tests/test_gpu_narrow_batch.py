"""Batches of very many cells of strand 2 up to 16: the finalize with one warp per cell, bit for bit
against the oracle and in proportion to the next width's."""
import numpy as np
import pytest

from bpmax_b200 import workloads as W

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


@pytest.fixture()
def eng():
    from bpmax_b200 import Engine

    e = Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("N", [1, 4, 5, 7, 8, 9, 13, 15, 16])
def test_narrow_batch_vs_oracle(eng, oracle_mod, N):
    """7 * 120 cells on the first diagonal, fewer than three per SM on the last ones."""
    rng = np.random.default_rng(N)
    pairs = [(W.random_sequence(7, rng), W.random_sequence(N, rng)) for _ in range(120)]
    w = W.random_weights(N)
    eng.set_weights(w)
    eng.score_batch(pairs)
    iu, ju = np.triu_indices(7)
    for p, (a, b) in enumerate(pairs):
        F = oracle_mod.fill(a, b, w)[0]
        assert np.array_equal(bits(eng.read_cells(p, 0, 7, 0, 7, N)[iu, ju]), bits(F)), p


def test_narrow_finalize_time(eng):
    """The finalizes of 30,000 cells of width 8 take well under half the time of those of width 24 (0.23 with
    one warp per cell, 0.56 with four)."""
    rng = np.random.default_rng(1)

    def finalize_ms(n):
        eng.score_batch([(W.random_sequence(3, rng), W.random_sequence(n, rng)) for _ in range(10_000)])
        return min(eng.profile_kernels()["finalize"][0] for _ in range(5))

    assert finalize_ms(8) < 0.4 * finalize_ms(24)
