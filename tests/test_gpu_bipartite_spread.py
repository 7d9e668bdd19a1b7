"""Bipartite anneals of couplings with one far above the rest, as the penalty terms of
QUBOs give: every decision replays in FP64, on the shapes whose half-step fields come from
the tensor cores always (the trials' tolerance covers the digits' rounding), and on those
where they do only when the digits are as fine as fp32 for every spin; and a served
request ends with the spins of the single-instance solver."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MARGIN_TOL = 1e-6


def _problem(N0, N1, outlier, integer):
    rng = np.random.default_rng(N0 + 2 * N1)

    def values(*shape):
        v = rng.integers(-8, 9, shape) * 4 if integer else rng.uniform(-1, 1, shape)
        return v.astype(np.float32)
    b0, b1, W = values(N0), values(N1), values(N1, N0)
    W[7, N0 - 5] = outlier
    return b0, b1, W


@pytest.mark.parametrize("N0,N1,m,algo,outlier,integer", [
    (1100, 2900, 20, "coloring", 1e5, False), (1100, 2900, 20, "coloring", -1e6, True),
    (2900, 1100, 20, "sa_coloring", 1e6, False), (1100, 2900, 20, "coloring", 20.0, False),
    (1030, 1100, 400, "coloring", 1e5, False), (1030, 1100, 400, "sa_coloring", 1e4, False),
    (1030, 1100, 400, "coloring", 1e9, False)])
def test_one_large_coupling_replays(orc, N0, N1, m, algo, outlier, integer):
    import sqaod_gb300 as sq
    b0, b1, W = _problem(N0, N1, outlier, integer)
    a = sq.cuda.bipartite_graph_annealer(b0, b1, W, n_trotters=m, algorithm=algo)
    h0, h1, J, _ = a.get_hamiltonian()
    a.seed(11)
    a.prepare()
    a.randomize_spin()
    pairs = a.get_q()
    q0, q1 = np.array([p[0] for p in pairs]), np.array([p[1] for p in pairs])
    a.set_trace(True)
    code = {"coloring": orc.ALGO_COLORING, "sa_coloring": orc.ALGO_SA_COLORING}[algo]
    for G, beta in [(3.0, 10.0), (0.3, 50.0)]:
        _, step = a.get_rng_state()
        a.anneal_one_step(G, beta)
        trace = a.get_trace((m * (N0 + N1) + 31) // 32)
        q0, q1, st = orc.bg_replay(h0, h1, J, m, code, 11, step, G, beta, q0, q1, trace, MARGIN_TOL)
        pairs = a.get_q()
        assert np.array_equal(np.array([p[0] for p in pairs]), q0)
        assert np.array_equal(np.array([p[1] for p in pairs]), q1)
        assert st["n_mismatch"] == st["n_mismatch_small"], (G, beta, st)


@pytest.mark.parametrize("N0,N1,m", [(1100, 2900, 20), (1030, 1100, 400)])
def test_served_equals_single_with_one_large_coupling(N0, N1, m):
    import sqaod_gb300 as sq
    from sqaod_gb300.serve import AnnealServer
    b0, b1, W = _problem(N0, N1, 1e6, False)
    G = np.geomspace(3.0, 0.1, 12).astype(np.float32)
    s = AnnealServer(budget_bytes=2 << 30)
    rid = s.submit_bipartite(b0, b1, W, m, G, 20.0, seed=4)
    s.run()
    E, (q0, q1) = s.result(rid)
    a = sq.cuda.bipartite_graph_annealer(b0, b1, W, n_trotters=m)
    a.seed(4)
    a.prepare()
    a.randomize_spin()
    a.anneal(G, 20.0)
    pairs = a.get_q()
    assert np.array_equal(np.array([p[0] for p in pairs]), q0)
    assert np.array_equal(np.array([p[1] for p in pairs]), q1)
    assert np.array_equal(a.get_E64(), E)
