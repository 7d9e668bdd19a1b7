"""Matrices that the dense formulas refuse: of several errors the matrix's comes first, and a
NaN on its diagonal is refused."""
import numpy as np
import pytest

from sqaod_gb300.cuda import formulas


def _W(N=5):
    W = np.random.default_rng(N).uniform(-1, 1, (N, N))
    return W + W.T


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_refused_matrices_on_a_device(dtype):
    h, x, q = np.zeros(5), np.zeros((2, 5), np.int8), np.ones((2, 5), np.int8)
    W = _W()
    W[2, 2] = np.nan
    with pytest.raises(RuntimeError, match="not triangular nor symmetric"):
        formulas.dense_graph_calculate_hamiltonian(W, dtype)
    with pytest.raises(RuntimeError, match="not triangular nor symmetric"):
        formulas.dense_graph_batch_calculate_E_from_spin(h, W, 0., q, dtype)
    # bits that select nothing of the NaN's row, and a triangular matrix, as symmetrize takes it
    with pytest.raises(RuntimeError, match="not triangular nor symmetric"):
        formulas.dense_graph_batch_calculate_E(W, x, dtype)
    with pytest.raises(RuntimeError, match="not triangular nor symmetric"):
        formulas.dense_graph_batch_calculate_E(W, np.full((3, 5), 2, np.int8), dtype)
    U = np.triu(W)
    assert np.isnan(formulas.dense_graph_batch_calculate_E(U, np.ones((1, 5), np.int8), dtype)).all()
    assert np.isnan(formulas.dense_graph_calculate_hamiltonian(U, dtype)[2])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_refused_matrices(dtype):
    h, x, q = np.zeros(5), np.zeros((2, 5), np.int8), np.ones((2, 5), np.int8)
    bad = _W()
    bad[1, 3] += 1
    nan = _W()
    nan[2, 2] = np.nan
    for W in (bad, nan):
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
