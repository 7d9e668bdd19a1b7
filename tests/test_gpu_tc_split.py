"""The tensor-core field refresh with K split over a cluster, and a half-step that
takes it: tile edges, remainders of K, the smallest and largest splits.  The
digits' integer sums are exact, so each field is the fp32 rounding of the
31-bit-quantised product whatever the split."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,K,m", [(64, 64, 1), (65, 1000, 127), (1024, 1024, 64), (129, 4097, 129), (2047, 513, 200),
                                   (1000, 300, 3)])
def test_split_refresh_is_exact(R, K, m):
    torch = pytest.importorskip("torch")
    from sqaod_gb300 import _lib
    L = _lib.lib()
    L.sq103_tc_digits_bytes.restype = ctypes.c_ulonglong
    L.sq103_tc_spins_bytes.restype = ctypes.c_ulonglong
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    g = torch.Generator(device="cuda").manual_seed(R + K + m)
    # multiples of 2^-20 below 1: exact in the 31-bit digits, every partial sum exact in FP64
    J = (torch.randint(-(1 << 20), 1 << 20, (R, K), device="cuda", generator=g).double() * 2.0**-20).float()
    q = (torch.randint(0, 2, (m, K), device="cuda", generator=g) * 2 - 1).to(torch.int8)
    D = torch.empty(int(L.sq103_tc_digits_bytes(R, K)), dtype=torch.uint8, device="cuda")
    A = torch.empty(int(L.sq103_tc_spins_bytes(m, K)), dtype=torch.uint8, device="cuda")
    F = torch.full((m, R + 3), -7.0, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert L.sq103_tc_make_digits(P(J), K, R, K, 0, P(D), s) == 0
    assert L.sq103_tc_refresh(P(D), R, K, P(q), K, m, P(A), P(F), R + 3, 0, P(status), s) == 0
    torch.cuda.synchronize()
    assert status.item() == 0
    assert torch.equal(F[:, :R], (q.double() @ J.double().T).float())
    assert (F[:, R:] == -7.0).all()


def test_half_steps_on_tensor_cores_replay(orc):
    """A problem the annealer takes to the tensor cores by its products per half-step."""
    import sqaod_gb300 as sq
    N0, N1, m = 1100, 1030, 65
    rng = np.random.default_rng(9)
    b0, b1 = rng.uniform(-1, 1, N0).astype(np.float32), rng.uniform(-1, 1, N1).astype(np.float32)
    W = rng.uniform(-1, 1, (N1, N0)).astype(np.float32)
    a = sq.cuda.bipartite_graph_annealer(b0, b1, W, n_trotters=m)
    h0, h1, J, _ = a.get_hamiltonian()
    a.seed(2)
    a.prepare()
    a.randomize_spin()
    pairs = a.get_q()
    q0, q1 = np.array([p[0] for p in pairs]), np.array([p[1] for p in pairs])
    a.set_trace(True)
    for G, beta in [(3.0, 10.0), (0.05, 50.0)]:
        _, step = a.get_rng_state()
        a.anneal_one_step(G, beta)
        trace = a.get_trace((m * (N0 + N1) + 31) // 32)
        q0, q1, st = orc.bg_replay(h0, h1, J, m, orc.ALGO_COLORING, 2, step, G, beta, q0, q1, trace, 1e-6)
        pairs = a.get_q()
        assert np.array_equal(np.array([p[0] for p in pairs]), q0)
        assert np.array_equal(np.array([p[1] for p in pairs]), q1)
        assert st["n_mismatch"] == st["n_mismatch_small"], st


@pytest.mark.parametrize("N,m,spread", [(1024, 1, 0.0), (1025, 130, 3.0), (1501, 63, 0.0)])
def test_dense_energies_on_tensor_cores(orc, N, m, spread):
    """FP64 energies from the exact digit sums, couplings of one and of many magnitudes."""
    import sqaod_gb300 as sq
    rng = np.random.default_rng(N + m)
    W = rng.uniform(-1, 1, (N, N)) * np.exp(spread * rng.standard_normal((N, N)))
    W = (np.triu(W) + np.triu(W, 1).T).astype(np.float32)
    for opt, sign in ((sq.minimize, 1.0), (sq.maximize, -1.0)):
        a = sq.cuda.dense_graph_annealer(W, opt, n_trotters=m)
        a.seed(1)
        a.prepare()
        a.randomize_spin()
        a.make_solution()
        q = np.array(a.get_q()).astype(np.float64)
        h, J, _ = a.get_hamiltonian()
        J64 = J.astype(np.float64)
        W64 = sign * W.astype(np.float64)
        c = -0.25 * (W64.sum() + np.trace(W64))
        ref = sign * (-c - q @ h.astype(np.float64) - ((q @ J64) * q).sum(1))
        scale = np.abs(J64).sum()
        # one FP64 rounding per row sum and the final sums: a few ulp of the total magnitude
        assert np.max(np.abs(a.get_E64() - ref)) <= 2.0**-50 * scale


def test_bipartite_energies_on_tensor_cores():
    import sqaod_gb300 as sq
    N0, N1, m = 1200, 1030, 70
    rng = np.random.default_rng(4)
    b0, b1, W = (rng.uniform(-1, 1, s).astype(np.float32) for s in (N0, N1, (N1, N0)))
    a = sq.cuda.bipartite_graph_annealer(b0, b1, W, n_trotters=m)
    a.seed(1)
    a.prepare()
    a.randomize_spin()
    a.make_solution()
    q = a.get_q()
    q0, q1 = np.array([p[0] for p in q]).astype(np.float64), np.array([p[1] for p in q]).astype(np.float64)
    h0, h1, J, _ = (np.asarray(v, np.float64) for v in a.get_hamiltonian())
    c = -0.25 * W.astype(np.float64).sum() - 0.5 * (b0.astype(np.float64).sum() + b1.astype(np.float64).sum())
    ref = -c - q0 @ h0 - q1 @ h1 - ((q0 @ J.T) * q1).sum(1)
    assert np.max(np.abs(a.get_E64() - ref)) <= 2.0**-50 * np.abs(J).sum()
