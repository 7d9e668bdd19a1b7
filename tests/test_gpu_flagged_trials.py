"""Trials the fp32 Metropolis test flags, decided from the exact local field.

With couplings of some 1e3 to 1e4 every trial near its threshold is flagged
(the flag's tolerance scales with the field), hundreds per half-step, so the
replay checks the exact decisions of the bipartite flip kernels: rows and
columns of J, ragged sizes around a warp's and a block's multiples, float and
double problems, SQA and SA.  A decision may differ from the FP64 host replay
only where the FP64 acceptance margin is below 1e-6 (counted by the replay).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MARGIN_TOL = 1e-6


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("N0,N1,m,algo", [(31, 33, 3, "coloring"), (257, 64, 17, "coloring"),
                                          (40, 515, 200, "coloring"), (129, 95, 7, "sa_coloring")])
def test_bipartite_flagged_trials_replay(orc, N0, N1, m, algo, dtype):
    import sqaod_gb300 as sq
    rng = np.random.default_rng(N0 + 3 * N1 + m)
    scale = 4e3
    b0, b1 = (scale * rng.uniform(-1, 1, n).astype(dtype) for n in (N0, N1))
    W = (scale * rng.uniform(-1, 1, (N1, N0))).astype(dtype)
    a = sq.cuda.bipartite_graph_annealer(b0, b1, W, dtype=dtype, n_trotters=m, algorithm=algo)
    h0, h1, J, _ = a.get_hamiltonian()
    a.seed(11)
    a.prepare()
    a.randomize_spin()
    pairs = a.get_q()
    q0, q1 = np.array([p[0] for p in pairs]), np.array([p[1] for p in pairs])
    a.set_trace(True)
    code = {"coloring": orc.ALGO_COLORING, "sa_coloring": orc.ALGO_SA_COLORING}[algo]
    for G, beta in [(3e4, 1e-3), (3e3, 2e-3), (3e2, 5e-3)]:
        _, step = a.get_rng_state()
        a.anneal_one_step(G, beta)
        trace = a.get_trace((m * (N0 + N1) + 31) // 32)
        q0, q1, st = orc.bg_replay(h0, h1, J, m, code, 11, step, G, beta, q0, q1, trace, MARGIN_TOL)
        pairs = a.get_q()
        assert np.array_equal(np.array([p[0] for p in pairs]), q0)
        assert np.array_equal(np.array([p[1] for p in pairs]), q1)
        assert st["n_mismatch"] == st["n_mismatch_small"], (G, beta, st)
