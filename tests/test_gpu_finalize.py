"""The finalize of tables up to width 64 bit for bit against the oracle: strand-2 lengths around its
8x8 blocks and at the ends of every width class, and launches of enough cells for the
form with fewer threads per cell."""
import numpy as np
import pytest

from bpmax_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from bpmax_b200 import Engine

    e = Engine(0)
    yield e
    e.close()


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


@pytest.mark.parametrize("N", [1, 2, 4, 5, 6, 8, 9, 10, 11, 15, 16, 17, 20, 21, 25, 26, 31, 32, 33, 34, 40, 47, 51, 56, 61, 63, 64])
def test_batches_vs_oracle(eng, oracle_mod, N):
    M = 7  # SW1 starts at outer diagonal 4
    s1, s2 = W.pair(M, N, 2000 + N)
    for w in (W.INTEGER_WEIGHTS, W.random_weights(N)):
        eng.set_weights(w)
        F, score = eng.fill_compact(s1, s2)
        Fo, _, _ = oracle_mod.fill(s1, s2, w)
        assert np.array_equal(bits(F), bits(Fo))
        assert score == oracle_mod.score(Fo, M, N)


@pytest.mark.parametrize("N", [8, 16, 24, 40, 48, 64])
def test_bulk_launches_vs_oracle(eng, oracle_mod, N):
    rng = np.random.default_rng(N)
    pairs = [(W.random_sequence(8, rng), W.random_sequence(N - p % 3, rng)) for p in range(160)]
    eng.set_weights(W.REFERENCE_WEIGHTS)
    got = eng.score_batch(pairs)
    exp = [oracle_mod.score(oracle_mod.fill(a, b, W.REFERENCE_WEIGHTS)[0], len(a), len(b)) for a, b in pairs]
    assert np.array_equal(bits(got), bits(np.array(exp, dtype=np.float32)))


@pytest.mark.parametrize("N", [65, 66, 71, 72, 73, 96, 127, 128, 129, 137, 192, 193, 255, 320, 321, 385])
def test_tile_tables_vs_oracle(eng, oracle_mod, N):
    """Tables of 64x64 tiles: strand-2 lengths around whole tiles and whole 8x8 blocks, and fewer outer
    diagonals than tile diagonals."""
    M = 6
    s1, s2 = W.pair(M, N, 3000 + N)
    w = W.random_weights(N) if N % 2 else W.INTEGER_WEIGHTS
    eng.set_weights(w)
    F, score = eng.fill_compact(s1, s2)
    Fo, _, _ = oracle_mod.fill(s1, s2, w)
    assert np.array_equal(bits(F), bits(Fo))
    assert score == oracle_mod.score(Fo, M, N)


@pytest.mark.parametrize("lo,hi", [(65, 128), (129, 192), (193, 200)])
def test_tile_tables_of_many_cells_vs_oracle(eng, oracle_mod, lo, hi):
    """Many tiles of several outer diagonals, tile diagonals and pairs in one step."""
    rng = np.random.default_rng(lo)
    pairs = [(W.random_sequence(5, rng), W.random_sequence(int(rng.integers(lo, hi + 1)), rng)) for _ in range(40)]
    eng.set_weights(W.INTEGER_WEIGHTS)
    got = eng.score_batch(pairs)
    tables = [oracle_mod.fill(a, b, W.INTEGER_WEIGHTS)[0] for a, b in pairs]
    exp = [oracle_mod.score(F, len(a), len(b)) for F, (a, b) in zip(tables, pairs)]
    assert np.array_equal(bits(got), bits(np.array(exp, dtype=np.float32)))
    for p in (0, 39):
        win = eng.read_cells(p, 0, 5, 0, 5, len(pairs[p][1]))
        iu, ju = np.triu_indices(5)
        assert np.array_equal(bits(win[iu, ju]), bits(tables[p]))
