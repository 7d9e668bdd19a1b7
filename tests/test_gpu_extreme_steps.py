"""Steps and couplings outside the fp32 form of the decisions (temperature zero, an
infinite beta, couplings near the float range): the one-CTA-per-trotter sweep ends, and
takes the decisions of the one-CTA kernel.  tests/cpp/rounds.cpp shows on the host that
its rounds end for every such step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INF = float("inf")


def _anneal(W, m, algo, G, beta, kernel):
    import sqaod_gb300 as sq
    a = sq.cuda.dense_graph_annealer(W, n_trotters=m, algorithm=algo)
    a.set_kernel(kernel)
    a.seed(5)
    a.prepare()
    a.randomize_spin()
    a.anneal(np.array(G, np.float32), beta)
    return np.array(a.get_q())


@pytest.mark.parametrize("N,m,algo,G,beta,coupling", [
    (64, 2, "sa_naive", [1.0, 0.0, 0.0], 1.0, None),
    (200, 7, "sa_naive", [2.0, 1e-39, 0.0], 1.0, None),
    (100, 320, "sa_naive", [0.5, 0.0], 1.0, None),
    (1030, 3, "sa_naive", [0.0], 1.0, None),
    (130, 5, "coloring", [1.0, 0.1], INF, None),
    (130, 6, "coloring", [1.0, 0.0], 20.0, None),
    (64, 2, "coloring", [1.0, 0.5], 3e38, None),
    (96, 4, "coloring", [3.0, 0.3], 10.0, 3e38),
    (96, 4, "sa_naive", [3.0, 0.0], 10.0, 3e38),
    (96, 4, "coloring", [3.0, 0.3], 10.0, INF),
    # few couplings a spin: an fp32 dE of zero where the exact one is not
    (175, 31, "sa_naive", [4.8, 3.2, 1.6, 0.0], 1.0, "sparse"),
    (246, 121, "sa_naive", [2.3, 0.0], 1.0, "sparse"),
    (198, 8, "coloring", [1.2, 0.8, 0.4, 0.0], INF, "sparse"),
    (81, 88, "sa_naive", [4.5, 0.0], 1.0, "sparse"),
    (113, 224, "coloring", [5.0, 0.5, 0.05], INF, "sparse"),
    (196, 23, "coloring", [3.0, 1.0, 0.0], 1e30, 1e20),
    (82, 24, "coloring", [5.0, 1.0, 0.3, 0.1, 0.03, 0.01], 1e30, 1e22),
    (75, 7, "coloring", [5.0, 1.0, 0.3, 0.1, 0.03, 0.01], 1e30, 1e27),
])
def test_extreme_steps_equal_the_one_cta_kernel(N, m, algo, G, beta, coupling):
    rng = np.random.default_rng(N + m)
    W = rng.uniform(-1, 1, (N, N)).astype(np.float32)
    W = np.triu(W) + np.triu(W, 1).T
    if coupling == "sparse":
        mask = np.triu(rng.random((N, N)) < 0.05)
        W = W * (mask | mask.T)
    elif coupling is not None:
        W[3, 70] = W[70, 3] = coupling
    assert np.array_equal(_anneal(W, m, algo, G, beta, 2), _anneal(W, m, algo, G, beta, 1))
