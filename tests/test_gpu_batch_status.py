"""A bounded device wait of the batch that ran out is reported by every call that returns
results of it (the status words are written from the host)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sym(rng, N):
    W = rng.uniform(-1, 1, (N, N))
    return (np.triu(W) + np.triu(W, 1).T).astype(np.float32)


def test_timeouts_are_raised():
    import sqaod_gb300 as sq
    from sqaod_gb300.batch import DenseBatchAnnealer
    rng = np.random.default_rng(1)
    b = DenseBatchAnnealer()
    for i, (N, m) in enumerate([(1030, 4), (40, 2), (1100, 3)]):
        b.add(_sym(rng, N), m, sq.minimize, i)
    b.set_schedule(np.geomspace(3, 0.1, 10).astype(np.float32), 20.0)

    def run():
        b.prepare()
        b.anneal(10)
        return [(b.get_E64(i), b.get_q(i)) for i in range(3)]

    def inject(which):
        b._call("inject_status", ctypes.c_int(which), ctypes.c_int(1))
    first = run()
    inject(1)  # the energies: once
    with pytest.raises(RuntimeError, match="timed out"):
        b.get_E64(2)
    for i in range(3):
        assert np.array_equal(b.get_E64(i), first[i][0])
    inject(0)  # the sweeps and refreshes: until the next prepare
    for call in (b.sync, lambda: b.get_E64(1), lambda: b.get_q(0), lambda: b.get_E64(0)):
        with pytest.raises(RuntimeError, match="timed out"):
            call()
    for (E, q), (E1, q1) in zip(run(), first):
        assert np.array_equal(E, E1) and np.array_equal(q, q1)
    with pytest.raises(RuntimeError):
        inject(2)
