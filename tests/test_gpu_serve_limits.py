"""The server's memory budget covers the scratch of the tensor-core energies; a request
whose scratch does not fit takes the energies that need none; and requests beyond the
light limits, which step in the persistent kernels on the side streams beside the
others, end as alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _sym(rng, N):
    W = rng.uniform(-1, 1, (N, N))
    return (np.triu(W) + np.triu(W, 1).T).astype(np.float32)


def _bip(rng, N0, N1):
    return tuple(rng.uniform(-1, 1, s).astype(np.float32) for s in (N0, N1, (N1, N0)))


def _single(problem, m, G, beta, seed):
    import sqaod_gb300 as sq
    make = sq.cuda.dense_graph_annealer if len(problem) == 1 else sq.cuda.bipartite_graph_annealer
    a = make(*problem, n_trotters=m)
    a.seed(seed)
    a.prepare()
    a.randomize_spin()
    a.anneal(G, beta)
    q = a.get_q()
    if len(problem) == 3:
        q = (np.array([p[0] for p in q]), np.array([p[1] for p in q]))
    else:
        q = (np.array(q),)
    return a.get_E64(), q


def _submit(srv, problem, m, G, beta, seed):
    f = srv.submit_dense if len(problem) == 1 else srv.submit_bipartite
    return f(*problem, m, G, beta, seed=seed)


def _spins(q):
    return q if isinstance(q, tuple) else (q,)


@pytest.mark.parametrize("shape,m,planes,budget", [
    ((1100,), 4, 1, 64 * MB), ((1100,), 4, 1, 21 * MB),
    # steps on the fp32 fields: the digits for the energies are scratch too
    ((1100, 2900), 20, 2, 128 * MB), ((1100, 2900), 20, 2, 40 * MB)])
def test_energy_scratch_is_in_the_budget(shape, m, planes, budget):
    from sqaod_gb300.serve import AnnealServer
    rng = np.random.default_rng(sum(shape))
    problems = [(_sym(rng, *shape),) if len(shape) == 1 else _bip(rng, *shape) for _ in range(2)]
    G = np.geomspace(3.0, 0.1, 20).astype(np.float32)
    srv = AnnealServer(budget_bytes=budget)
    ids = [_submit(srv, p, m, G, 20.0, 7 + i) for i, p in enumerate(problems)]
    srv.tick()
    N1, N0 = shape[-1], shape[0]
    digits = planes * 8 * N1 * N0  # at least: four bf16 planes each
    tight = budget < 100 * MB and budget != 64 * MB
    in_use = srv.stats()["bytes_in_use"]
    assert in_use <= budget
    if not tight:
        assert in_use >= 2 * 4 * N0 * N1 + digits
    srv.run()
    assert srv.stats()["bytes_in_use"] == 0
    for i, p in enumerate(problems):
        E, q = srv.result(ids[i])
        E1, q1 = _single(p, m, G, 20.0, 7 + i)
        for a, b in zip(_spins(q), q1):
            assert np.array_equal(a, b)
        if tight:  # FP64 sums of other order: 2^-44 of the largest partial sum and less
            assert np.max(np.abs(E - E1)) <= 2.0**-40 * np.sum(np.abs(p[-1]))
        else:
            assert np.array_equal(E, E1)


def test_requests_beyond_the_light_limits():
    from sqaod_gb300.serve import AnnealServer
    rng = np.random.default_rng(3)
    G = np.geomspace(3.0, 0.1, 11).astype(np.float32)
    srv = AnnealServer(budget_bytes=2 << 30)
    sizes = [(64 + k % 40,) for k in range(70)] + [(40 + k, 90 - k) for k in range(40)] + [(1100,), (300,)]
    problems = [((_sym(rng, *s),) if len(s) == 1 else _bip(rng, *s), 3 + k % 6) for k, s in enumerate(sizes)]
    ids = [_submit(srv, p, m, G, 20.0, k) for k, (p, m) in enumerate(problems)]
    srv.run()
    for k, (p, m) in enumerate(problems):
        E, q = srv.result(ids[k])
        E1, q1 = _single(p, m, G, 20.0, k)
        assert all(np.array_equal(a, b) for a, b in zip(_spins(q), q1)), sizes[k]
        assert np.array_equal(E, E1), sizes[k]
