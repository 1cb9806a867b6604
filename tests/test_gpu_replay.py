"""Every form of a plan's launches: the first run is launched as it is, the second captures the graph and
launches it, the others replay it. Each run has other sequences of the same shape, and every table and score
is compared bit for bit with the oracle's."""
import numpy as np
import pytest
import torch

from bpmax_b200 import workloads as W

pytestmark = pytest.mark.gpu
RUNS = 4  # eager, capture and first launch, two replays


@pytest.fixture()
def eng():
    from bpmax_b200 import Engine

    e = Engine(0)
    yield e
    e.close()


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


@pytest.mark.parametrize("strips", [False, True])
@pytest.mark.parametrize("M,N", [(1, 5), (12, 8), (21, 16), (13, 31), (40, 23), (15, 48), (13, 56), (14, 64)])
def test_narrow_tables(eng, oracle_mod, M, N, strips):
    if strips:
        eng.set_tuning("strip_tasks", 0)
    w = W.random_weights(M)
    eng.set_weights(w)
    for r in range(RUNS):
        s1, s2 = W.pair(M, N, 100 * r + M)
        F, score = eng.fill_compact(s1, s2)
        Fo = oracle_mod.fill(s1, s2, w)[0]
        assert np.array_equal(bits(F), bits(Fo)), r
        assert score == oracle_mod.score(Fo, M, N)


@pytest.mark.parametrize("M,N", [(1, 65), (3, 200), (9, 70), (7, 130), (5, 321), (3, 400)])
def test_tile_tables(eng, oracle_mod, M, N):
    w = W.random_weights(N)
    eng.set_weights(w)
    for r in range(RUNS):
        s1, s2 = W.pair(M, N, 100 * r + N)
        F, score = eng.fill_compact(s1, s2)
        Fo = oracle_mod.fill(s1, s2, w)[0]
        assert np.array_equal(bits(F), bits(Fo)), r
        assert score == oracle_mod.score(Fo, M, N)


@pytest.mark.parametrize("streams", [1, 0])
@pytest.mark.parametrize("strips", [False, True])
def test_batches_of_several_widths(eng, oracle_mod, streams, strips):
    """Width classes on streams of their own, and in one chain."""
    rng = np.random.default_rng(5)
    shapes = [(int(rng.integers(1, 22)), int(rng.integers(1, 140))) for _ in range(24)] + [(3, 330), (16, 64), (16, 40)]
    eng.set_tuning("class_streams", streams)
    if strips:
        eng.set_tuning("strip_tasks", 0)
    eng.set_weights(W.INTEGER_WEIGHTS)
    for r in range(RUNS):
        pairs = [W.pair(m, n, 1000 * r + k) for k, (m, n) in enumerate(shapes)]
        got = eng.score_batch(pairs)
        for p, (a, b) in enumerate(pairs):
            Fo = oracle_mod.fill(a, b, W.INTEGER_WEIGHTS)[0]
            assert got[p] == oracle_mod.score(Fo, len(a), len(b)), (r, p)
            if p % 5 == 0:
                iu, ju = np.triu_indices(len(a))
                assert np.array_equal(bits(eng.read_cells(p, 0, len(a), 0, len(a), len(b))[iu, ju]), bits(Fo)), (r, p)


@pytest.mark.parametrize("M,N", [(14, 40), (9, 64), (5, 130)])
def test_r0_only(eng, oracle_mod, M, N):
    rng = np.random.default_rng(M)
    for r in range(RUNS):
        s1, s2 = rng.integers(0, 1000, M), rng.integers(0, 1000, N)
        F, _ = eng.r0_only(s1, s2)
        assert np.array_equal(bits(F), bits(oracle_mod.r0only(s1, s2))), r


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("M,N,T", [(21, 64, 32), (8, 17, 8), (17, 40, 12), (9, 150, 64)])
def test_reference_layout(eng, oracle_mod, M, N, T, pinned):
    """Written by the finalize (pinned, up to width 64) or converted per outer diagonal or row, each copied out
    while the fill runs; the buffer is cleared before every call."""
    buf = torch.empty(eng.reference_size(M, N, T), dtype=torch.float32, pin_memory=pinned)
    mask = oracle_mod.reference_written_mask(M, N, T)
    w = W.random_weights(T)
    eng.set_weights(w)
    for r in range(RUNS):
        buf.fill_(float("nan"))
        s1, s2 = W.pair(M, N, 100 * r + T)
        F, score = eng.fill(s1, s2, T, out=buf.numpy())
        Fo = oracle_mod.fill(s1, s2, w)[0]
        assert np.array_equal(bits(F[mask]), bits(oracle_mod.to_reference_layout(Fo, M, N, T)[mask])), r
        assert score == oracle_mod.score(Fo, M, N)


@pytest.mark.parametrize("mode", [1, 2])
def test_persistent_fill(eng, oracle_mod, mode):
    rng = np.random.default_rng(3)
    shapes = [(int(rng.integers(1, 30)), int(rng.integers(1, 65))) for _ in range(20)]
    eng.set_tuning("persistent", mode)
    eng.set_weights(W.REFERENCE_WEIGHTS)
    for r in range(RUNS):
        pairs = [W.pair(m, n, 1000 * r + k) for k, (m, n) in enumerate(shapes)]
        exp = [oracle_mod.score(oracle_mod.fill(a, b, W.REFERENCE_WEIGHTS)[0], len(a), len(b)) for a, b in pairs]
        assert np.array_equal(bits(eng.score_batch(pairs)), bits(np.array(exp, np.float32))), r


def test_weights_between_runs(eng, oracle_mod):
    """New weights between the runs of one plan: its graph holds the old ones and is captured again."""
    s1, s2 = W.pair(18, 30, 4)
    for r in range(6):
        w = W.random_weights(50 + r // 2)
        if r % 2 == 0:
            eng.set_weights(w)
        assert eng.score(s1, s2) == oracle_mod.score(oracle_mod.fill(s1, s2, w)[0], 18, 30), r
