"""The rule that takes a batch to the strip product kernel: where it does, the fill is no slower than without
strips (the rest of the tests compare tables bit for bit with strips forced everywhere)."""
import numpy as np
import pytest

from bpmax_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs,M,N", [(1000, 16, 16), (400, 30, 16), (1000, 16, 24), (400, 30, 32), (1000, 16, 48), (1000, 8, 64)])
def test_short_strands_no_slower_than_without_strips(pairs, M, N):
    from bpmax_b200 import Engine

    rng = np.random.default_rng(M + N)
    batch = [(W.random_sequence(M, rng), W.random_sequence(N, rng)) for _ in range(pairs)]
    engines, times, scores = {}, {}, {}
    try:
        for tasks in (None, 1 << 40):  # the rule, no strips
            engines[tasks] = e = Engine(0)
            if tasks is not None:
                e.set_tuning("strip_tasks", tasks)
            e.set_weights(W.INTEGER_WEIGHTS)
        for _ in range(8):  # in turn
            for tasks, e in engines.items():
                scores[tasks] = e.score_batch(batch)
                times.setdefault(tasks, []).append(e.last_timing()[0])
    finally:
        for e in engines.values():
            e.close()
    ms = {tasks: min(t[2:]) for tasks, t in times.items()}
    assert np.array_equal(scores[None], scores[1 << 40])
    assert ms[None] < 1.04 * ms[1 << 40], ms
