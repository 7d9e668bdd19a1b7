"""Which instances a batch steps in packed one-CTA-per-trotter launches: those of at least
the caller's limit, or without one those of 64 spins (128 in batches of more than 152)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies,limit,least", [(1, None, 64), (51, None, 128), (51, 65, 65), (1, 1024, 1024),
                                                (1, 0, None)])
def test_packed_count(copies, limit, least):
    import sqaod_gb300 as sq
    from sqaod_gb300.batch import DenseBatchAnnealer
    sizes = [(63, 4), (64, 4), (127, 1), (128, 4)] * copies if copies == 1 else [(127, 4), (128, 4), (64, 4)] * copies
    b = DenseBatchAnnealer()
    problems = {}
    for N, m in sizes:
        if N not in problems:
            W = np.random.default_rng(N).uniform(-1, 1, (N, N))
            problems[N] = (W + W.T).astype(np.float32)
        b.add(problems[N], m, sq.minimize, 1)
    b.set_schedule(np.array([1.0], np.float32), 20.0)
    if limit is not None:
        b.set_multicta_min_n(limit)
    b.prepare()
    assert b.packed_count() == sum(1 for N, m in sizes if least is not None and N >= least and m >= 2)
