"""The strip product kernel (bpmax_strip.cuh) bit for bit against the oracle: every width class it
has, strand-1 lengths around its groups of T diagonals, ragged strand-2 lengths, more jobs than CTAs
with the pair changing from job to job, and the R0-only mode. The strips are forced on every diagonal
that has offsets for them; every F value is an exact maximum, so nothing may differ."""
import numpy as np
import pytest

from bpmax_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture()
def eng():
    from bpmax_b200 import Engine

    e = Engine(0)
    e.set_tuning("strip_tasks", 0)
    yield e
    e.close()


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


@pytest.mark.parametrize("N", [9, 16, 17, 24, 31, 40, 41, 48, 49, 56, 57, 64])
@pytest.mark.parametrize("M", [3, 4, 5, 7, 8, 9, 10, 21])
def test_strip_tables_vs_oracle(eng, oracle_mod, M, N):
    s1, s2 = W.pair(M, N, 1000 + 70 * M + N)
    w = W.random_weights(N) if (M + N) % 2 else W.INTEGER_WEIGHTS
    eng.set_weights(w)
    F, score = eng.fill_compact(s1, s2)
    Fo, _, _ = oracle_mod.fill(s1, s2, w)
    assert np.array_equal(bits(F), bits(Fo))
    assert score == oracle_mod.score(Fo, M, N)


@pytest.mark.parametrize("widths", [(57, 64), (49, 56), (33, 48), (9, 64)])
def test_strip_batches_vs_oracle(eng, oracle_mod, widths):
    """More strips than SMs, so every CTA walks several jobs of different pairs."""
    rng = np.random.default_rng(widths[0])
    pairs = [(W.random_sequence(int(rng.integers(18, 34)), rng), W.random_sequence(int(rng.integers(widths[0], widths[1] + 1)), rng))
             for _ in range(14)]
    eng.set_weights(W.INTEGER_WEIGHTS)
    eng.set_tuning("r0_pairs_per_job", 2)
    got = eng.score_batch(pairs)
    tables = [oracle_mod.fill(a, b, W.INTEGER_WEIGHTS)[0] for a, b in pairs]
    exp = np.array([oracle_mod.score(F, len(a), len(b)) for F, (a, b) in zip(tables, pairs)], dtype=np.float32)
    assert np.array_equal(bits(got), bits(exp))
    for p in (0, 7, 13):
        M, N = len(pairs[p][0]), len(pairs[p][1])
        win = eng.read_cells(p, 0, M, 0, M, N)
        iu, ju = np.triu_indices(M)
        assert np.array_equal(bits(win[iu, ju]), bits(tables[p]))


@pytest.mark.parametrize("M,N", [(11, 40), (9, 64), (14, 20)])
def test_strip_r0_only_vs_oracle(eng, oracle_mod, M, N):
    rng = np.random.default_rng(M)
    s1, s2 = rng.integers(0, 1000, M), rng.integers(0, 1000, N)
    F, _ = eng.r0_only(s1, s2)
    assert np.array_equal(bits(F), bits(oracle_mod.r0only(s1, s2)))


def test_strip_wait_timeout_is_reported(eng, oracle_mod):
    """The test mode issues no copies: every wait runs out, the call returns BPMAX_ETIMEOUT and the
    next call is right."""
    from bpmax_b200 import BpmaxError

    s1, s2 = W.pair(12, 60, 5)
    eng.set_weights(W.INTEGER_WEIGHTS)
    eng.set_tuning("wait_limit_us", 2000)
    eng.set_tuning("inject_wait_timeout", 1)
    with pytest.raises(BpmaxError) as e:
        eng.score(s1, s2)
    assert e.value.status == 5
    eng.set_tuning("wait_limit_us", 4_000_000)
    assert eng.score(s1, s2) == oracle_mod.score(oracle_mod.fill(s1, s2, W.INTEGER_WEIGHTS)[0], 12, 60)
