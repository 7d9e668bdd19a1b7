"""The low digit planes of the tensor-core energies: without device memory for them the
energies come from the sums that need none, and planes above the size that a problem keeps
are freed after each call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _annealer(N, m, seed):
    import sqaod_gb300 as sq
    W = np.random.default_rng(seed).uniform(-1, 1, (N, N)).astype(np.float32)
    i, j = np.tril_indices(N, -1)
    W[i, j] = W[j, i]
    a = sq.cuda.dense_graph_annealer(W, n_trotters=m)
    a.seed(1)
    a.prepare()
    a.randomize_spin()
    return a, W


def _exact(a, W):
    """FP64 Ising energies of the current spins from the h and J that the solver holds."""
    q = np.array(a.get_q()).astype(np.float64)
    h, J, _ = a.get_hamiltonian()
    J = J.astype(np.float64)
    W = W.astype(np.float64)
    c = -0.25 * (W.sum() + np.trace(W))
    return -c - q @ h.astype(np.float64) - ((q @ J) * q).sum(1), np.abs(J).sum()


def test_energies_without_memory_for_the_planes():
    torch = pytest.importorskip("torch")
    N, m = 2048, 5
    _annealer(100, 4, 0)[0].get_E64()  # the kernels of the other sums are loaded
    a, W = _annealer(N, m, 1)
    planes = 8 * N * N
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - planes // 2, dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < planes
        E = np.array(a.get_E64())
    finally:
        del hold
        torch.cuda.empty_cache()
    ref, scale = _exact(a, W)
    assert np.max(np.abs(E - ref)) <= 2.0**-44 * scale  # double-float sums of fp32 products
    a.calculate_E()
    assert np.max(np.abs(a.get_E64() - ref)) <= 2.0**-50 * scale


def test_large_planes_are_freed_after_the_call():
    torch = pytest.importorskip("torch")
    N = 11600
    a, W = _annealer(N, 2, 2)
    E = np.array(a.get_E64())
    used = torch.cuda.mem_get_info()[0]
    a.calculate_E()
    assert np.array_equal(E, a.get_E64())
    assert torch.cuda.mem_get_info()[0] == used
    q = np.array(a.get_q())
    x = ((q + 1) // 2).astype(np.float64)
    ref = np.array([(v[v > 0] @ W[v > 0][:, v > 0].astype(np.float64)).sum() for v in x])
    # h is held in fp32: N roundings of values up to its largest
    assert np.max(np.abs(E - ref)) <= 2.0**-24 * np.abs(W.astype(np.float64).sum(1)).sum()
