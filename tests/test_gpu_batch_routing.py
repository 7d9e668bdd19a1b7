"""Which instances a batch steps in packed one-CTA-per-trotter launches: those of at least
the caller's limit; without one, small ones where they are few or have few trotters, and
none of them where their packed launches, one after another, would take longer than the
persistent kernel, which runs all at once (measured for each of these: 2 to 20 times)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ALL = [(64, 4), (65, 4), (100, 4)]


@pytest.mark.parametrize("sizes,limit,packed", [
    (ALL, None, 3), (ALL * 60, None, 180), ([(64, 256)] * 4, None, 4),
    ([(64, 256)] * 60, None, 0), ([(64, 64)] * 150, None, 0), ([(64, 64)] * 150 + [(2000, 8)], None, 1),
    ([(63, 4), (64, 1), (128, 4)], None, 1),
    ([(64, 256)] * 60, 64, 60), (ALL, 65, 2), (ALL, 1024, 0), (ALL, 0, 0)])
def test_packed_count(sizes, limit, packed):
    import sqaod_gb300 as sq
    from sqaod_gb300.batch import DenseBatchAnnealer
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
    assert b.packed_count() == packed
