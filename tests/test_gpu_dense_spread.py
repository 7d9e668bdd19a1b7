"""Dense anneals of couplings with one far above the rest, at sizes whose fields come from
the tensor cores: where the digits would be too coarse for the decisions' tolerance the
fields stay in fp32, in the single solver, the batch and the server alike, and every
decision replays in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

G = np.geomspace(5, 0.05, 17).astype(np.float32)


def _problem(N, outlier):
    W = np.random.default_rng(N).uniform(-1, 1, (N, N))
    W = np.triu(W) + np.triu(W, 1).T
    W[3, 70] = W[70, 3] = outlier
    return W.astype(np.float32)


@pytest.mark.parametrize("N,m,algo,outlier", [(1100, 12, "coloring", 1e7), (1100, 9, "sa_naive", 1e9),
                                              (1025, 12, "coloring", 1e5), (1030, 12, "sa_naive", 30.0)])
def test_one_large_coupling_replays(orc, N, m, algo, outlier):
    import sqaod_gb300 as sq
    code = {"coloring": orc.ALGO_COLORING, "sa_naive": orc.ALGO_SA_NAIVE}[algo]
    a = sq.cuda.dense_graph_annealer(_problem(N, outlier), n_trotters=m, algorithm=algo)
    h, J, _ = a.get_hamiltonian()
    a.seed(3)
    a.prepare()
    a.randomize_spin()
    q = np.array(a.get_q())
    a.set_trace(True)
    _, step0 = a.get_rng_state()
    a.anneal(G, 30.0)
    nw = (N * m + 31) // 32
    trace = np.array(a.get_trace(nw * len(G)), np.uint32).reshape(len(G), nw)
    for s in range(len(G)):
        q, st = orc.dg_replay(h, J, m, code, 3, step0 + s, float(G[s]), 30.0, q, trace[s], 1e-6)
        assert st["n_mismatch"] == st["n_mismatch_small"], (s, st)
    assert np.array_equal(np.array(a.get_q()), q)


def test_batch_and_server_hold_the_same_fields():
    import sqaod_gb300 as sq
    from sqaod_gb300.batch import DenseBatchAnnealer
    from sqaod_gb300.serve import AnnealServer
    problems = [(_problem(1100, 1e8), 6), (_problem(1030, 1.0), 5), (_problem(1200, 1e6), 7)]
    b = DenseBatchAnnealer()
    srv = AnnealServer(budget_bytes=1 << 30)
    ids = []
    for i, (W, m) in enumerate(problems):
        b.add(W, m, sq.minimize, 20 + i)
        ids.append(srv.submit_dense(W, m, G, 30.0, seed=20 + i))
    b.set_schedule(G, 30.0)
    b.prepare()
    b.anneal(len(G))
    srv.run()
    for i, (W, m) in enumerate(problems):
        a = sq.cuda.dense_graph_annealer(W, n_trotters=m)
        a.seed(20 + i)
        a.prepare()
        a.randomize_spin()
        a.anneal(G, 30.0)
        q, E = np.array(a.get_q()), a.get_E64()
        assert np.array_equal(q, b.get_q(i)) and np.array_equal(E, b.get_E64(i))
        E1, q1 = srv.result(ids[i])
        assert np.array_equal(q, q1) and np.array_equal(E, E1)
