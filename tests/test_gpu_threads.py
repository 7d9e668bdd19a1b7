"""Host threads with solvers of their own share the kernels' shared memory limits: while
other threads search, or ask for the capacity of, small problems, the launches of a larger
one must not fail."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sym(rng, N):
    W = rng.uniform(-1, 1, (N, N))
    return (np.triu(W) + np.triu(W, 1).T).astype(np.float32)


def _searcher(N):
    import sqaod_gb300 as sq
    a = sq.cuda.dense_graph_bf_searcher(_sym(np.random.default_rng(N), N))
    return lambda: (a.search(), np.array(a.get_x()))[1]


def _annealer(N):
    import sqaod_gb300 as sq
    a = sq.cuda.dense_graph_annealer(_sym(np.random.default_rng(N), N), n_trotters=4)
    G = np.array([3.0, 0.1], np.float32)

    def run():
        a.seed(1)
        a.prepare()
        a.randomize_spin()
        a.anneal(G, 20.0)
        return np.array(a.get_q())
    return run


def _capacities():
    from sqaod_gb300 import _lib
    L = _lib.lib()
    return lambda: [L.sq103_dense_multicta_capacity(N) for N in (64, 65)]


def test_capacity_does_not_depend_on_the_order_of_questions():
    from sqaod_gb300 import _lib
    L = _lib.lib()
    sizes = [64, 3000, 5000, 64, 20000, 5000, 3000]
    got = [L.sq103_dense_multicta_capacity(N) for N in sizes]
    assert got[0] == got[3] and got[1] == got[6] and got[2] == got[5]
    assert L.sq103_dense_multicta_capacity(1 << 20) == 0


@pytest.mark.parametrize("large,small,repeats", [(lambda: _searcher(27), lambda: _searcher(20), 300),
                                                 (lambda: _annealer(2100), _capacities, 300)],
                         ids=["search", "anneal"])
def test_threads_of_different_sizes(large, small, repeats):
    run = large()
    expected = run()
    others = [small() for _ in range(3)]
    stop, errors = threading.Event(), []

    def work(f):
        try:
            while not stop.is_set():
                f()
        except BaseException as e:
            errors.append(repr(e))
    threads = [threading.Thread(target=work, args=(f,)) for f in others]
    for t in threads:
        t.start()
    try:
        for _ in range(repeats):
            assert np.array_equal(run(), expected)
    finally:
        stop.set()
        for t in threads:
            t.join()
    assert not errors, errors
