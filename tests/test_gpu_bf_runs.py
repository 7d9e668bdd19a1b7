"""Brute-force searches around the run kernel's edges (2^20 states a run) and the
bipartite minimum over all x0, against the FP64 energies of every state."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(x, n):
    return ((x[:, None] >> np.arange(n - 1, -1, -1)) & 1).astype(np.float64)


def _dense(rng, N, kind):
    W = rng.integers(-3, 4, (N, N)) if kind == "integer" else rng.uniform(-1, 1, (N, N))
    W = np.triu(W)
    return (W + np.triu(W, 1).T).astype(np.float64 if kind == "real64" else np.float32)


@pytest.mark.parametrize("kind", ["integer", "real", "real64"])
@pytest.mark.parametrize("N,begin,end", [(20, 0, 1 << 20), (21, 5, (1 << 21) - 3), (22, (1 << 20) - 1, 1 << 22),
                                         (22, 1 << 20, (3 << 20) + 1), (21, 1 << 20, (1 << 21) - (1 << 14))])
def test_dense_runs(N, begin, end, kind):
    import sqaod_gb300 as sq
    rng = np.random.default_rng(N + begin % 97 + end % 89)
    W = _dense(rng, N, kind)
    s = sq.cuda.dense_graph_bf_searcher(W, sq.minimize, W.dtype.type)
    s.prepare()
    s.search_subrange(begin, end)
    s.make_solution()
    W64 = W.astype(np.float64)
    E = np.empty(end - begin)
    for b in range(begin, end, 1 << 18):
        e = min(b + (1 << 18), end)
        x = _bits(np.arange(b, e), N)
        E[b - begin:e - begin] = ((x @ W64) * x).sum(1)
    best = E.min()
    # FP64 energies of distinct states differ by far more than 1e-10 (real couplings)
    want = begin + np.flatnonzero(E <= best + 1e-10)
    got = np.array(s.get_x(), np.int64) @ (1 << np.arange(N - 1, -1, -1, dtype=np.int64))
    assert np.array_equal(got, want)
    assert abs(s.get_E64() - best) <= 1e-12 * max(1.0, abs(best))


@pytest.mark.parametrize("kind", ["integer", "real", "real64"])
@pytest.mark.parametrize("N0,N1", [(1, 1), (3, 14), (8, 4), (15, 6), (7, 13)])
def test_bipartite_minimum(N0, N1, kind):
    import sqaod_gb300 as sq
    rng = np.random.default_rng(31 * N0 + N1)
    draw = (lambda *s: rng.integers(-2, 3, s)) if kind == "integer" else (lambda *s: rng.uniform(-1, 1, s))
    b0, b1, W = (v.astype(np.float64 if kind == "real64" else np.float32) for v in (draw(N0), draw(N1), draw(N1, N0)))
    s = sq.cuda.bipartite_graph_bf_searcher(b0, b1, W, sq.minimize, W.dtype.type)
    s.search()
    x0, x1 = _bits(np.arange(1 << N0), N0), _bits(np.arange(1 << N1), N1)
    E = (x0 @ b0.astype(np.float64))[:, None] + x1 @ b1.astype(np.float64) + x0 @ W.T.astype(np.float64) @ x1.T
    best = E.min()
    want = np.argwhere(E <= best + 1e-10)  # ascending (x0, x1)
    got = s.get_x()
    pack = lambda v: int(np.asarray(v, np.int64) @ (1 << np.arange(len(v) - 1, -1, -1, dtype=np.int64)))
    assert [(pack(a), pack(b)) for a, b in got] == [tuple(w) for w in want.tolist()][:len(got)]
    assert len(got) == min(len(want), 8192 * 2 if min(N0, N1) > 13 else (1 << min(N0, 13)) + (1 << min(N1, 13)))
    assert abs(s.get_E()[0] - best) <= 1e-6 * max(1.0, abs(best))


def test_bipartite_minimum_many_x0():
    """More x0 variables than a warp has lanes: the minimiser is each negative D[j]."""
    import sqaod_gb300 as sq
    rng = np.random.default_rng(5)
    N0, N1 = 33, 2
    b0, b1, W = (rng.uniform(-1, 1, s).astype(np.float32) for s in (N0, N1, (N1, N0)))
    s = sq.cuda.bipartite_graph_bf_searcher(b0, b1, W, sq.minimize, np.float32)
    s.search()
    x1 = _bits(np.arange(4), N1)
    D = b0.astype(np.float64) + x1 @ W.astype(np.float64)
    E = x1 @ b1.astype(np.float64) + np.minimum(D, 0).sum(1)
    k = int(E.argmin())
    (a, b), = s.get_x()
    assert np.array_equal(a, (D[k] < 0).astype(np.int8)) and np.array_equal(b, x1[k].astype(np.int8))
    assert abs(s.get_E()[0] - E[k]) <= 1e-6 * abs(E[k])
