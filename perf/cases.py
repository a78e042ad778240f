"""The work that a user of egsolver_b200 has it do, as cases that can be timed.

Every case goes through the package's public entry points:

  solve     `egsolver_b200.solve`: host arrays in, host credits out, one call.  What the reference's command line
            does for one game: upload, preprocessing, lifting, read-back.
  resident  `ResidentGame.solve` and `.credits`: the game is in device memory, a solve is started from f = 0 and
            the credits are read back.
  batch     `Batch.solve` and `.credits`: many uneven games at K mean-payoff thresholds each, planned beforehand.
  serve     `Server.submit`, `.wait` and `.result`: threshold queries on registered games, all in flight at once.
  csr2csc   the stand-alone stable transpose of host arrays.

Games are the seeded ones of the benchmark's workloads (`egsolver_b200.workloads`): random 4-regular ("regular"),
power-law out-degrees ("power"), complete digraphs ("clique"), uniform out-degrees 2..16 ("uniform") and geometric
out-degrees ("geometric"), at sizes from tens of vertices, where a call is launches and latency, to millions of edges.
Credits are whole numbers, equal for every schedule of lifts.
"""
from __future__ import annotations

import numpy as np

import egsolver_b200 as eg

# generator kind, largest out-degree (None: n - 1), largest |weight|, generator parameter
GRAPHS = {
    "regular": (1, 4, 10, 0),
    "power": (2, 4096, 1000, 0),
    "clique": (3, None, 500, 0),
    "uniform": (4, 16, 100, 2),
    "geometric": (5, 256, 1000, 6),
}
MEAN_DEGREE = {"regular": 4.0, "power": 7.9, "uniform": 9.0, "geometric": 6.0}


def listed():
    return [
        # a toy game of the size of the reference's shipped examples: what is left is launches and allocations
        {"name": "solve_tiny", "api": "solve", "graph": "regular", "n": 101, "bits": 64},
        # the smallest benchmark configuration: a game that a CPU solves too, 32-bit credits
        {"name": "solve_1k_i32", "api": "solve", "graph": "regular", "n": 1000, "bits": 32},
        # an application's game of a few thousand vertices, odd size, solved once from host memory
        {"name": "solve_geometric_4k", "api": "solve", "graph": "geometric", "n": 4099, "bits": 64},
        # skewed out-degrees (1 to thousands), 64-bit credits: the large sparse configuration scaled to 6 K vertices
        {"name": "power_6k", "api": "resident", "graph": "power", "n": 6007, "bits": 64},
        # the dense configuration: complete digraph of 2,000 vertices, 32-bit credits, 4 M edges
        {"name": "clique_2000_i32", "api": "resident", "graph": "clique", "n": 2000, "bits": 32},
        # one mean-payoff threshold on a game of ordinary size
        {"name": "threshold_16k", "api": "resident", "graph": "uniform", "n": 16381, "bits": 64, "p": -100, "d": 8},
        # the largest single game: 131 K vertices and 1.2 M edges that do not fit one SM
        {"name": "uniform_131k", "api": "resident", "graph": "uniform", "n": 131072, "bits": 64},
        # a batch of uneven games at eight thresholds each, as a search over thresholds asks for them
        {"name": "batch_32x8", "api": "batch", "graph": "uniform", "games": 32, "n_lo": 1024, "n_hi": 16384,
         "k": 8, "d": 8, "p_max": 400},
        # threshold queries in flight together on games that stay registered
        {"name": "serve_12", "api": "serve", "graph": "uniform", "games": 6, "queries": 12, "n_lo": 1000, "n_hi": 8000,
         "k": 6, "d": 8, "p_max": 400},
        # the transpose alone, small and large
        {"name": "csr2csc_8k", "api": "csr2csc", "rows": 1013, "cols": 997, "nnz": 8191},
        {"name": "csr2csc_6m", "api": "csr2csc", "rows": 800_003, "cols": 1_000_000, "nnz": 6_300_001},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    api = rng.choice(["solve", "solve", "resident", "resident", "resident", "batch", "serve", "csr2csc"])
    if api == "solve":
        graph = rng.choice(["regular", "uniform", "geometric"])
        return {"api": api, "graph": graph, "n": _log_int(rng, 64, 4096), "bits": rng.choice([32, 64])}
    if api == "resident":
        graph = rng.choice(["power", "clique", "uniform", "uniform", "geometric"])
        hi = {"power": 6000, "clique": 2000, "uniform": 120000, "geometric": 13000}[graph]
        case = {"api": api, "graph": graph, "n": _log_int(rng, 300, hi), "bits": 32 if graph == "clique" else 64}
        if graph == "uniform" and rng.random() < 0.5:
            case.update(p=rng.randrange(-400, 401), d=8)
        return case
    if api == "batch":
        return {"api": api, "graph": "uniform", "games": rng.randrange(4, 33), "n_lo": 1024,
                "n_hi": _log_int(rng, 2048, 16384), "k": rng.choice([1, 3, 5, 8]), "d": 8, "p_max": rng.randrange(100, 401)}
    if api == "serve":
        return {"api": api, "graph": "uniform", "games": rng.randrange(2, 7), "queries": rng.randrange(4, 13),
                "n_lo": 1000, "n_hi": _log_int(rng, 2000, 8000), "k": rng.choice([4, 5, 6]), "d": 8,
                "p_max": rng.randrange(100, 401)}
    nnz = _log_int(rng, 5000, 6_000_000)
    return {"api": api, "rows": max(1, int(nnz * rng.uniform(0.05, 0.5))), "cols": max(1, int(nnz * rng.uniform(0.05, 0.5))),
            "nnz": nnz}


def _game(graph, n, seed):
    kind, deg, wmax, param = GRAPHS[graph]
    return eg.generate(kind, n, n - 1 if deg is None else min(deg, n - 1), wmax, seed, param=param)


def _sizes(case):
    """Vertices of the case's games: spread evenly over the logarithm of [n_lo, n_hi]."""
    lo, hi, num = case["n_lo"], case["n_hi"], case["games"]
    return [int(round(lo * (hi / lo) ** ((i + 0.5) / num))) for i in range(num)]


class _Serving:
    """A server with its registered games, closed with its last user."""

    def __init__(self, games):
        self.server = eg.Server()
        self.ids = [self.server.add_game(g) for g in games]

    def __del__(self):
        self.server.close()


def _csr(case, seed):
    rng = np.random.default_rng(seed)
    rows, cols, nnz = case["rows"], case["cols"], case["nnz"]
    row_ptr = np.concatenate([[0], np.cumsum(np.bincount(rng.integers(0, rows, nnz), minlength=rows))]).astype(np.int64)
    return (rows, cols, row_ptr, rng.integers(0, cols, nnz, dtype=np.int32),
            rng.integers(-1000, 1001, nnz, dtype=np.int32))


def _single(case, seed):
    g = _game(case["graph"], case["n"], seed)
    return eg.threshold_game(g, case["p"], case["d"]) if "p" in case else g


def prepare(case, seed):
    api = case["api"]
    state = {"case": case}
    if api == "csr2csc":
        state["csr"] = _csr(case, seed)
        return state
    if api in ("solve", "resident"):
        g = _single(case, seed)
        state["game"] = g if api == "solve" else eg.ResidentGame(g)
        return state
    rng = np.random.default_rng(seed)
    games = [_game(case["graph"], n, seed * 1_000_003 + i) for i, n in enumerate(_sizes(case))]
    if api == "batch":
        b = eg.Batch(games, case["k"], scale=case["d"])
        b.set_thresholds(rng.integers(-case["p_max"], case["p_max"] + 1, size=(len(games), case["k"])))
        state["batch"] = b
    else:
        state["serving"] = _Serving(games)
        state["queries"] = [(i % len(games), rng.integers(-case["p_max"], case["p_max"] + 1, size=case["k"]).astype(np.int32))
                            for i in range(case["queries"])]
    return state


def run(state):
    case = state["case"]
    api = case["api"]
    if api == "solve":
        return eg.solve(state["game"], credit_bits=case["bits"])[0]
    if api == "resident":
        state["game"].solve(credit_bits=case["bits"])
        return state["game"].credits(case["bits"])
    if api == "batch":
        state["batch"].solve()
        return [state["batch"].credits(i) for i in range(case["games"])]
    if api == "serve":
        sv = state["serving"]
        qids = [sv.server.submit(sv.ids[g], p, case["d"]) for g, p in state["queries"]]
        out = []
        for q in qids:
            sv.server.wait(q)
            out.append(sv.server.result(q)[0])
        return out
    return eg.csr2csc(*state["csr"])


def _edges(case, n):
    return n * (n - 1) if case["graph"] == "clique" else int(n * MEAN_DEGREE[case["graph"]])


def work(case):
    """Bytes: the inputs read once (row offsets 8 B, successor and weight 4 B each) and the outputs written once.
    Operations: a subtraction and a comparison for every edge, once per threshold."""
    if case["api"] == "csr2csc":
        return {"bytes": 8 * (case["rows"] + case["cols"] + 2) + 16 * case["nnz"], "flops": 0}
    if case["api"] in ("solve", "resident"):
        n, m = case["n"], _edges(case, case["n"])
        return {"bytes": 8 * (n + 1) + 8 * m + case["bits"] // 8 * n, "flops": 2 * m}
    sizes = _sizes(case)
    n = sum(sizes)
    m = n * MEAN_DEGREE[case["graph"]]
    if case["api"] == "serve":
        solved = case["k"] * sum(sizes[i % len(sizes)] for i in range(case["queries"]))
    else:
        solved = case["k"] * n
    return {"bytes": 8 * n + 8 * m + 8 * solved, "flops": 2 * solved * MEAN_DEGREE[case["graph"]]}


def _values(game, sweeps_max=20000):
    """Least fixed point of the lifting operator by numpy value iteration; None when it takes too many sweeps."""
    top = np.iinfo(np.int64).max
    rp, succ, w, own = game.row_ptr[:-1], game.succ, game.weight.astype(np.int64), game.owners()
    mg = int(np.maximum(0, -np.minimum.reduceat(w, rp)).sum())
    f = np.zeros(game.num_nodes, np.int64)
    for _ in range(sweeps_max):
        a = f[succ]
        d = np.where(a == top, 0, a) - w
        v = np.where((a == top) | (d > mg), top, np.maximum(d, 0))
        new = np.maximum(f, np.where(own == 0, np.minimum.reduceat(v, rp), np.maximum.reduceat(v, rp)))
        if np.array_equal(new, f):
            return f
        f = new
    return None


def exact(case, seed):
    if case["api"] == "csr2csc":
        rows, cols, row_ptr, col, val = _csr(case, seed)
        order = np.argsort(col, kind="stable")
        ptr = np.concatenate([[0], np.cumsum(np.bincount(col, minlength=cols))]).astype(np.int64)
        src = np.repeat(np.arange(rows, dtype=np.int32), np.diff(row_ptr))
        return ptr, src[order], val[order]
    if case["api"] in ("solve", "resident") and (case["n"] <= 1000 or case["graph"] == "clique"):
        f = _values(_single(case, seed))
        if f is None or case["bits"] == 64:
            return f
        return np.where(f == np.iinfo(np.int64).max, np.iinfo(np.int32).max, f).astype(np.int32)
    return None
