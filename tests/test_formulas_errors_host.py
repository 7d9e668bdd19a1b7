"""Matrices that the dense formulas refuse, before any device work: of several errors the
matrix's comes first, and a NaN on its diagonal is refused."""
import numpy as np
import pytest

from sqaod_gb300.cuda import formulas


def _W(N=5):
    W = np.random.default_rng(N).uniform(-1, 1, (N, N))
    return W + W.T


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_refused_matrices(dtype):
    h, x, q = np.zeros(5), np.zeros((2, 5), np.int8), np.ones((2, 5), np.int8)
    bad = _W()
    bad[1, 3] += 1
    nan = _W()
    nan[2, 2] = np.nan
    for W in (bad, nan):
        if W is nan:
            with pytest.raises(RuntimeError, match="not triangular nor symmetric"):
                formulas.dense_graph_calculate_hamiltonian(W, dtype)
            with pytest.raises(RuntimeError, match="not triangular nor symmetric"):
                formulas.dense_graph_batch_calculate_E(W, x, dtype)
            with pytest.raises(RuntimeError, match="not triangular nor symmetric"):
                formulas.dense_graph_batch_calculate_E_from_spin(h, W, 0., q, dtype)
        # with a second error
        with pytest.raises(RuntimeError, match="not triangular nor symmetric"):
            formulas.dense_graph_batch_calculate_E(W, x[:, :4], dtype)
        with pytest.raises(RuntimeError, match="not triangular nor symmetric"):
            formulas.dense_graph_batch_calculate_E_from_spin(h[:4], W, 0., q, dtype)
        with pytest.raises(RuntimeError, match="not triangular nor symmetric"):
            formulas.dense_graph_batch_calculate_E_from_spin(h, W, h, q, dtype)
    with pytest.raises(RuntimeError, match="dimension mismatch"):
        formulas.dense_graph_batch_calculate_E(_W(), x[:, :4], dtype)
    with pytest.raises(RuntimeError, match="not a scalar"):
        formulas.dense_graph_batch_calculate_E_from_spin(h, _W(), h, q, dtype)
