"""Bipartite searches in which every x1 reaches the minimum (nonnegative couplings, no
biases): all of them are searched state by state, spread over the CTAs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_few_x1_within_reach_of_many_x0():
    """Few blocks of x1 over many x0, split between the CTAs: the minimum is x0 = 0 with any x1."""
    import sqaod_gb300 as sq
    N0, N1 = 25, 6
    rng = np.random.default_rng(2)
    W = rng.integers(0, 3, (N1, N0)).astype(np.float32)
    s = sq.cuda.bipartite_graph_bf_searcher(np.ones(N0, np.float32), np.zeros(N1, np.float32), W, sq.minimize,
                                            np.float32)
    s.search()
    pack = lambda v: int(np.asarray(v, np.int64) @ (1 << np.arange(len(v) - 1, -1, -1, dtype=np.int64)))
    assert [(pack(a), pack(b)) for a, b in s.get_x()] == [(0, x1) for x1 in range(1 << N1)]
    assert s.get_E()[0] == 0.0


@pytest.mark.parametrize("N0,N1", [(3, 13), (5, 14), (4, 16), (12, 13)])
def test_every_x1_within_reach(N0, N1):
    import sqaod_gb300 as sq
    rng = np.random.default_rng(N0 + N1)
    W = rng.integers(1, 4, (N1, N0)).astype(np.float32)  # E = 0 exactly where x0 = 0 or x1 = 0
    s = sq.cuda.bipartite_graph_bf_searcher(np.zeros(N0, np.float32), np.zeros(N1, np.float32), W, sq.minimize,
                                            np.float32)
    s.set_preferences(tile_size_0=1 << 16, tile_size_1=1 << 16)
    s.search()
    pack = lambda v: int(np.asarray(v, np.int64) @ (1 << np.arange(len(v) - 1, -1, -1, dtype=np.int64)))
    got = [(pack(a), pack(b)) for a, b in s.get_x()]
    want = [(0, x1) for x1 in range(1 << N1)] + [(x0, 0) for x0 in range(1, 1 << N0)]
    assert got == want[:len(got)] and len(got) >= min(len(want), (1 << N1) + (1 << min(N0, 13)))
    assert s.get_E()[0] == 0.0
