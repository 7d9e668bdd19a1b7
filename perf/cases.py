"""Performance cases of sqaod_gb300: the work its users have it do, through the Python API.

A case is a dict of plain values.  `prepare` makes the problem (couplings uniform in
[-1, 1], the distribution of the reference's generators and of bench.py) and the solver
object a program keeps, `run` is one solve as such a program writes it: seed, random
spins, the schedule, the energies and the spins.  Anneals run a geometric schedule from
G = 5 to G = 0.01 at beta = 50, the shape of the reference's 619-step schedule, in fewer
steps, so that a pass sees high and low acceptance alike.
"""
import math

import numpy as np
import torch

import sqaod_gb300 as sq
from sqaod_gb300.batch import DenseBatchAnnealer
from sqaod_gb300.cuda import formulas
from sqaod_gb300.serve import AnnealServer

BETA = 50.0
DTYPES = {"f32": np.float32, "f64": np.float64}


def listed():
    return [
        # the reference's own benchmark case and its anneal() loop: one annealOneStep call per
        # step, the smallest calls, where latency counts
        {"name": "dense_small_loop", "kind": "dense", "N": 128, "m": 16, "steps": 64, "loop": True},
        # an ordinary problem with the default number of trotters (N / 4), one call for the schedule
        {"name": "dense_default_m", "kind": "dense", "N": 1000, "m": 250, "steps": 64},
        # default trotters on a larger problem: more replicas than one per SM
        {"name": "dense_many_trotters", "kind": "dense", "N": 2000, "m": 500, "steps": 8},
        # the headline configuration of bench.py, the largest couplings in regular use
        {"name": "dense_headline", "kind": "dense", "N": 4096, "m": 256, "steps": 64},
        # simulated annealing, maximising, with an odd size and trotter count
        {"name": "dense_sa", "kind": "dense", "N": 1501, "m": 63, "steps": 64, "algorithm": "sa_naive",
         "maximize": True},
        # double precision, the default dtype of the reference's factories, in its step loop
        {"name": "dense_double_loop", "kind": "dense", "N": 512, "m": 128, "steps": 64, "dtype": "f64", "loop": True},
        # bench.py's bipartite configuration
        {"name": "bipartite", "kind": "bipartite", "N0": 1024, "N1": 1024, "m": 64, "steps": 64},
        # a large ragged bipartite problem
        {"name": "bipartite_large", "kind": "bipartite", "N0": 3001, "N1": 2047, "m": 200, "steps": 32},
        # exhaustive search with real couplings, the check a user runs beside an annealer
        {"name": "bf_dense", "kind": "bf", "N": 31},
        # scoring a set of given bit vectors, host arrays in and out
        {"name": "energies", "kind": "energies", "N": 1000, "m": 256, "dtype": "f32"},
        # many uneven problems at once, a slice of bench.py's batched workload
        {"name": "batch", "kind": "batch", "count": 128, "lo": 64, "hi": 2048, "steps": 16},
        # a mixed set of requests through the server, sizes of bench.py's served stream
        {"name": "server", "kind": "server", "count": 24, "lo": 32, "hi": 2048, "steps": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dense", "dense", "dense", "dense", "bipartite", "bipartite", "bf", "bip_bf", "energies",
                       "batch", "server"])
    if kind == "dense":
        N = _log_int(rng, 100, 4096)
        m = rng.choice([rng.randint(2, 32), rng.randint(33, 256), max(2, N // 4)])
        steps = rng.choice([16, 24, 32, 64])
        if m > 256:  # default trotters of large problems: short schedules
            N, m, steps = min(N, 2000), min(m, 500), 8
        c = {"kind": kind, "N": N, "m": m, "steps": steps}
        if rng.random() < 0.25:
            c["algorithm"] = "sa_naive"
        if rng.random() < 0.25:
            c["maximize"] = True
        if N <= 1200 and rng.random() < 0.3:
            c["dtype"] = "f64"
        if rng.random() < 0.4:
            c["loop"] = True
        return c
    if kind == "bipartite":
        c = {"kind": kind, "N0": _log_int(rng, 64, 3000), "N1": _log_int(rng, 64, 3000), "m": rng.randint(2, 200),
             "steps": rng.choice([16, 32])}
        if rng.random() < 0.25:
            c["algorithm"] = "sa_coloring"
        if rng.random() < 0.25:
            c["maximize"] = True
        if c["N0"] * c["N1"] <= 1 << 19 and rng.random() < 0.3:
            c["dtype"] = "f64"
        if rng.random() < 0.4:
            c["loop"] = True
        return c
    if kind == "bf":
        return {"kind": kind, "N": rng.randint(16, 31), "dtype": rng.choice(["f32", "f64"]),
                "integer": rng.random() < 0.5, "maximize": rng.random() < 0.25}
    if kind == "bip_bf":
        return {"kind": kind, "N0": rng.randint(6, 15), "N1": rng.randint(6, 15), "dtype": rng.choice(["f32", "f64"]),
                "integer": rng.random() < 0.5}
    if kind == "energies":
        return {"kind": kind, "N": _log_int(rng, 64, 2048), "m": _log_int(rng, 1, 512),
                "dtype": rng.choice(["f32", "f64"])}
    lo = rng.randint(32, 100)
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 8, 100), "lo": lo, "hi": _log_int(rng, 200, 2048), "steps": 16}
    return {"kind": kind, "count": rng.randint(4, 20), "lo": lo, "hi": _log_int(rng, 200, 2048), "steps": 32}


# ------------------------------------------------------------------------ problems

def _symmetric(rng, N, dtype, integer=False):
    W = rng.integers(-4096, 4097, (N, N)) if integer else rng.uniform(-1.0, 1.0, (N, N))
    W = np.triu(W)
    W += np.triu(W, 1).T
    return W.astype(dtype)


def _bipartite(rng, N0, N1, dtype, integer=False):
    def values(*shape):
        v = rng.integers(-4096, 4097, shape) if integer else rng.uniform(-1.0, 1.0, shape)
        return v.astype(dtype)
    return values(N0), values(N1), values(N1, N0)


def _dtype(case):
    return DTYPES[case.get("dtype", "f32")]


def _optimize(case):
    return sq.maximize if case.get("maximize") else sq.minimize


def _schedule(steps):
    return np.geomspace(5.0, 0.01, steps).astype(np.float32)


def _mixed_sizes(case):
    """Sizes of a batch or a set of requests: N log-uniform, a few trotter counts (bench.py's workloads)."""
    rng = np.random.default_rng(case["count"])
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    out = []
    for i in range(case["count"]):
        dense = case["kind"] == "batch" or rng.random() < 0.7
        m = int(rng.choice([8, 16, 32, 64, 128] if case["kind"] == "batch" else [16, 64, 256]))
        out.append(tuple(int(round(math.exp(rng.uniform(lo, hi)))) for _ in range(1 if dense else 2)) + (m, ))
    return out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind, dtype = case["kind"], _dtype(case)
    st = {"case": case, "seed": seed}
    if kind == "dense":
        W = _symmetric(rng, case["N"], dtype)
        st["solver"] = sq.cuda.dense_graph_annealer(W, _optimize(case), dtype, n_trotters=case["m"],
                                                    algorithm=case.get("algorithm", "coloring"))
        st["solver"].seed(seed)
        st["solver"].prepare()
    elif kind == "bipartite":
        b0, b1, W = _bipartite(rng, case["N0"], case["N1"], dtype)
        st["solver"] = sq.cuda.bipartite_graph_annealer(b0, b1, W, _optimize(case), dtype, n_trotters=case["m"],
                                                        algorithm=case.get("algorithm", "coloring"))
        st["solver"].seed(seed)
        st["solver"].prepare()
    elif kind == "bf":
        W = _symmetric(rng, case["N"], dtype, case.get("integer"))
        st["solver"] = sq.cuda.dense_graph_bf_searcher(W, _optimize(case), dtype)
    elif kind == "bip_bf":
        b0, b1, W = _bipartite(rng, case["N0"], case["N1"], dtype, case.get("integer"))
        st["solver"] = sq.cuda.bipartite_graph_bf_searcher(b0, b1, W, sq.minimize, dtype)
    elif kind == "energies":
        st["W"] = _symmetric(rng, case["N"], dtype)
        st["x"] = rng.integers(0, 2, (case["m"], case["N"])).astype(np.int8)
    elif kind == "batch":
        st["solver"] = DenseBatchAnnealer()
        for i, (N, m) in enumerate(_mixed_sizes(case)):
            st["solver"].add(_symmetric(rng, N, np.float32), m, sq.minimize, seed * 1000 + i)
    else:
        st["solver"] = AnnealServer(budget_bytes=32 << 30)
        st["requests"] = []
        for size in _mixed_sizes(case):
            m = size[-1]
            if len(size) == 2:
                st["requests"].append((m, (_symmetric(rng, size[0], np.float32), )))
            else:
                st["requests"].append((m, _bipartite(rng, size[0], size[1], np.float32)))
    if kind in ("dense", "bipartite", "batch", "server"):
        st["G"] = _schedule(case["steps"])
    torch.cuda.synchronize()
    return st


def run(st):
    case, a = st["case"], st.get("solver")
    kind = case["kind"]
    if kind in ("dense", "bipartite"):
        a.seed(st["seed"])
        a.randomize_spin()
        if case.get("loop"):
            for G in st["G"]:
                a.anneal_one_step(float(G), BETA)
        else:
            a.anneal(st["G"], BETA)
        a.make_solution()
        q = a.get_q()
        if kind == "dense":
            return {"E": a.get_E64(), "q": np.array(q)}
        return {"E": a.get_E64(), "q0": np.array([p[0] for p in q]), "q1": np.array([p[1] for p in q])}
    if kind == "bf":
        a.search()
        return {"E": a.get_E(), "x": np.array(a.get_x())}
    if kind == "bip_bf":
        a.search()
        x = a.get_x()
        return {"E": a.get_E(), "x0": np.array([p[0] for p in x]), "x1": np.array([p[1] for p in x])}
    if kind == "energies":
        dtype = _dtype(case)
        E = formulas.dense_graph_batch_calculate_E(st["W"], st["x"], dtype)
        h, J, c = formulas.dense_graph_calculate_hamiltonian(st["W"], dtype)
        return {"E": E, "h": h, "J": J, "c": c}
    if kind == "batch":
        a.set_schedule(st["G"], BETA)
        a.prepare()
        a.anneal(len(st["G"]))
        n = case["count"]
        return {"E": np.concatenate([a.get_E64(i) for i in range(n)]),
                "q": np.concatenate([a.get_q(i).ravel() for i in range(n)])}
    ids = []
    for i, (m, problem) in enumerate(st["requests"]):
        submit = a.submit_dense if len(problem) == 1 else a.submit_bipartite
        ids.append(submit(*problem, m, st["G"], BETA, seed=st["seed"] * 1000 + i))
    a.run()
    out = [a.result(i) for i in ids]
    spins = [v.ravel() for E, q in out for v in (q if isinstance(q, tuple) else (q, ))]
    return {"E": np.concatenate([E for E, q in out]), "q": np.concatenate(spins)}


def work(case):
    """Couplings read and results written once; a trial's decision (its draw, dE and test, about
    100 operations) and one field contraction for the random start and one for the energies."""
    kind, real = case["kind"], np.dtype(_dtype(case)).itemsize
    if kind == "dense":
        N, m = case["N"], case["m"]
        return {"bytes": real * N * N + N * m + 8 * m, "flops": 100 * N * m * case["steps"] + 4 * N * N * m}
    if kind == "bipartite":
        N0, N1, m = case["N0"], case["N1"], case["m"]
        return {"bytes": real * N0 * N1 + (N0 + N1) * m + 8 * m,
                "flops": case["steps"] * (4 * N0 * N1 + 100 * (N0 + N1)) * m + 2 * N0 * N1 * m}
    if kind == "bf":  # an addition and a comparison for each state
        return {"bytes": real * case["N"]**2 + 64, "flops": 2 * 2**case["N"]}
    if kind == "bip_bf":
        return {"bytes": real * case["N0"] * case["N1"] + 64, "flops": 2 * 2**(case["N0"] + case["N1"])}
    if kind == "energies":
        N, m = case["N"], case["m"]
        return {"bytes": real * (2 * N * N + N + m) + N * m, "flops": 2 * N * N * m + 3 * N * N}
    # a batch or a set of requests: mean sizes of the ranges
    lo, hi, n = case["lo"], case["hi"], case["count"]
    N, N2 = (hi - lo) / math.log(hi / lo), (hi * hi - lo * lo) / (2 * math.log(hi / lo))
    m = 50 if kind == "batch" else 112
    return {"bytes": n * (4 * N2 + N * m), "flops": n * m * (100 * N * case["steps"] + 4 * N2)}


# ------------------------------------------------------- the same results in 64 bits

def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) over arrays of counters."""
    mask, m0, m1 = np.uint64(0xFFFFFFFF), np.uint64(0xD2511F53), np.uint64(0xCD9E8D57)
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    c = [np.asarray(v, np.uint64) for v in np.broadcast_arrays(c0, c1, c2, c3)]
    for _ in range(10):
        p0, p1 = m0 * c[0], m1 * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & mask,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _random_spins(N, m, seed, step, side=0):
    w = _philox(np.arange((N + 127) // 128)[None, :], np.arange(m)[:, None], step, 0x21 | side << 8, seed)
    bits = (np.stack(w, -1)[..., None] >> np.arange(32, dtype=np.uint64)) & np.uint64(1)
    return np.where(bits.reshape(m, -1)[:, :N] > 0, 1.0, -1.0)


def _uniform(w):
    return (w >> np.uint64(8)).astype(np.float64) * 2.0**-24


def _accepts(dE, rate, u):
    return (dE < 0) | (np.exp(-np.maximum(dE, 0) * rate) > u)


def _phases(m):
    """The trotters of each colour phase: the even ones, the last when m is odd, the odd ones."""
    e = m // 2 * 2
    return [p for p in (np.arange(0, e, 2), np.arange(e, m), np.arange(1, e, 2)) if len(p)]


def _exact_dense(case, seed):
    N, m, sa = case["N"], case["m"], case.get("algorithm") == "sa_naive"
    W = _symmetric(np.random.default_rng(seed), N, _dtype(case)).astype(np.float64)
    sign = -1.0 if case.get("maximize") else 1.0
    h, J = -0.5 * sign * W.sum(1), -0.25 * sign * W
    c = J.sum() + np.trace(J)
    if case.get("dtype") != "f64":  # the float solver's h is a float
        h = h.astype(np.float32).astype(np.float64)
    np.fill_diagonal(J, 0.0)
    q = _random_spins(N, m, seed, 0)
    F = q @ J
    everyone = np.arange(m)
    for s, G in enumerate(_schedule(case["steps"]).astype(np.float64)):
        words = _philox(np.arange(N)[:, None], everyone[None, :], s + 1, 0x12 if sa else 0x11, seed)
        sites, us = ((words[0] * np.uint64(N)) >> np.uint64(32)).astype(np.int64), _uniform(words[1])
        coef = 0.0 if sa else math.log(math.tanh(G * BETA / m)) / BETA
        for k in range(N):
            for ys in [everyone] if sa else _phases(m):
                x, u = sites[k, ys], us[k, ys]
                v = q[ys, x]
                t = h[x] + 2 * F[ys, x]
                if sa:
                    acc = _accepts(2 * v * t, 1 / G, u)
                else:
                    acc = _accepts(2.0 / m * v * t - v * (q[(ys + m - 1) % m, x] + q[(ys + 1) % m, x]) * coef, BETA, u)
                for y, i in zip(ys[acc], x[acc]):
                    F[y] -= 2 * q[y, i] * J[i]
                    q[y, i] = -q[y, i]
    return {"E": sign * (-c - q @ h - ((q @ J) * q).sum(1)), "q": None}


def _exact_bipartite(case, seed):
    N0, N1, m, sa = case["N0"], case["N1"], case["m"], case.get("algorithm") == "sa_coloring"
    b0, b1, W = (v.astype(np.float64) for v in _bipartite(np.random.default_rng(seed), N0, N1, _dtype(case)))
    sign = -1.0 if case.get("maximize") else 1.0
    J = -0.25 * sign * W
    h = [J.sum(0) - 0.5 * sign * b0, J.sum(1) - 0.5 * sign * b1]
    c = J.sum() - 0.5 * sign * (b0.sum() + b1.sum())
    if case.get("dtype") != "f64":
        h = [v.astype(np.float32).astype(np.float64) for v in h]
    q = [_random_spins(N0, m, seed, 0, 0), _random_spins(N1, m, seed, 0, 1)]
    for s, G in enumerate(_schedule(case["steps"]).astype(np.float64)):
        coef = 0.0 if sa else math.log(math.tanh(G * BETA / m)) / BETA
        for side in (1, 0):
            v, F = q[side], q[1 - side] @ (J if side == 0 else J.T)
            u = _uniform(_philox(np.arange(v.shape[1])[None, :], np.arange(m)[:, None], s + 1,
                                 (0x32 if sa else 0x31) | side << 8, seed)[1])
            for ys in [np.arange(m)] if sa else _phases(m):
                a, t = v[ys], h[side] + F[ys]
                if sa:
                    acc = _accepts(2 * a * t, 1 / G, u[ys])
                else:
                    acc = _accepts(2.0 / m * a * t - a * (v[(ys + m - 1) % m] + v[(ys + 1) % m]) * coef, BETA, u[ys])
                v[ys] = np.where(acc, -a, a)
    return {"E": sign * (-c - q[0] @ h[0] - q[1] @ h[1] - ((q[1] @ J) * q[0]).sum(1)), "q0": None, "q1": None}


def _bits(lo, hi, n):
    return ((np.arange(lo, hi)[:, None] >> np.arange(n - 1, -1, -1)) & 1).astype(np.float64)


def _lowest(energies, total):
    """Least value of energies(lo, hi) over the packed states [0, total), and how many states share it."""
    best, count = math.inf, 0
    for lo in range(0, total, 1 << 16):
        E = energies(lo, min(lo + (1 << 16), total))
        e = E.min()
        if e < best - 1e-9:
            best, count = e, 0
        if e < best + 1e-9:
            count += int((E < best + 1e-9).sum())
    return best, count


def exact(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    if kind == "dense":
        return _exact_dense(case, seed) if case["N"] * case["steps"] * case["m"] <= 1 << 23 else None
    if kind == "bipartite":
        return _exact_bipartite(case, seed) if case["steps"] * case["m"] * case["N0"] * case["N1"] <= 1 << 33 else None
    if kind == "bf":
        if case["N"] > 21:
            return None
        W = _symmetric(rng, case["N"], _dtype(case), case.get("integer")).astype(np.float64)
        sign = -1.0 if case.get("maximize") else 1.0

        def energies(lo, hi):
            x = _bits(lo, hi, case["N"])
            return sign * ((x @ W) * x).sum(1)
        best, count = _lowest(energies, 1 << case["N"])
        return {"E": np.full(count, sign * best), "x": None}
    if kind == "bip_bf":
        if case["N0"] + case["N1"] > 22:
            return None
        b0, b1, W = (v.astype(np.float64)
                     for v in _bipartite(rng, case["N0"], case["N1"], _dtype(case), case.get("integer")))
        x0 = _bits(0, 1 << case["N0"], case["N0"])

        def energies(lo, hi):
            # states are packed as (x1, x0), whole x0 ranges at a time
            n0 = 1 << case["N0"]
            x1 = _bits(lo // n0, -(-hi // n0), case["N1"])
            return ((x1 @ b1)[:, None] + x0 @ b0 + x1 @ W @ x0.T).ravel()[lo % n0:lo % n0 + hi - lo]
        best, count = _lowest(energies, 1 << (case["N0"] + case["N1"]))
        return {"E": np.full(count, best), "x0": None, "x1": None}
    if kind == "energies":
        W = _symmetric(rng, case["N"], _dtype(case)).astype(np.float64)
        x = rng.integers(0, 2, (case["m"], case["N"])).astype(np.float64)
        J = -0.25 * W
        c = J.sum() + np.trace(J)
        np.fill_diagonal(J, 0.0)
        return {"E": ((x @ W) * x).sum(1), "h": -0.5 * W.sum(1), "J": J, "c": c}
    return None
