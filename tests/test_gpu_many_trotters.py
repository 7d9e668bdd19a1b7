"""The one-CTA-per-trotter sweep with more trotters than two CTAs per SM hold
(the four-per-SM instances): replayed against FP64, and bit-identical to the
one-CTA kernel, around the sizes where the instance changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MARGIN_TOL = 1e-6


def _sym(rng, N):
    W = rng.uniform(-1, 1, (N, N))
    return (np.triu(W) + np.triu(W, 1).T).astype(np.float32)


@pytest.mark.parametrize("N,m,algo", [(64, 305, "coloring"), (130, 608, "coloring"), (1025, 455, "coloring"),
                                      (97, 500, "sa_naive")])
def test_many_trotters_replay(orc, N, m, algo):
    import sqaod_gb300 as sq
    from sqaod_gb300 import _lib
    import torch
    code = {"coloring": orc.ALGO_COLORING, "sa_naive": orc.ALGO_SA_NAIVE}[algo]
    assert _lib.lib().sq103_dense_multicta_ok(N, m, code) == 1
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert 2 * sms < m <= _lib.lib().sq103_dense_multicta_capacity(N)
    rng = np.random.default_rng(N + m)
    a = sq.cuda.dense_graph_annealer(_sym(rng, N), n_trotters=m, algorithm=algo)
    h, J, c = a.get_hamiltonian()
    a.seed(3)
    a.prepare()
    a.randomize_spin()
    q = np.array(a.get_q())
    a.set_trace(True)
    _, step0 = a.get_rng_state()
    G = np.array([3.0, 0.3, 0.03], np.float32)
    a.anneal(G, 40.0)
    nw = (N * m + 31) // 32
    trace = np.array(a.get_trace(nw * len(G)), np.uint32).reshape(len(G), nw)
    for s in range(len(G)):
        q, st = orc.dg_replay(h, J, m, code, 3, step0 + s, float(G[s]), 40.0, q, trace[s], MARGIN_TOL)
        assert st["n_mismatch"] == st["n_mismatch_small"], (s, st)
    assert np.array_equal(np.array(a.get_q()), q)


def test_many_trotters_equal_one_cta():
    import sqaod_gb300 as sq
    N, m = 100, 401
    W = _sym(np.random.default_rng(8), N)
    out = []
    for flags in (1, 2):
        a = sq.cuda.dense_graph_annealer(W, n_trotters=m)
        a.set_kernel(flags)
        a.seed(4)
        a.prepare()
        a.randomize_spin()
        a.anneal(np.geomspace(5, 0.05, 10).astype(np.float32), 30.0)
        out.append((np.array(a.get_q()), a.get_E64()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
