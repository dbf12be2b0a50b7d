"""The searches and planner steps that the engine's speed is judged by.

Every case goes through the package's public entry points from a graph on the
host, as `multigpubfs_b200.bfs` and `run_graph` do: a handle is created,
planned, run, read and destroyed in each pass (`bfs`), a sweep is created, run
and read (`sweep`), the shards of a split search are reset and run (`sharded`),
and the planner network takes one forward and backward pass (`planner`).  The
seed picks the start state of a search (its orbit, and so its cost, stays the
same), the generators of a sweep, and the rows of a training step.
"""
import math

import numpy as np

from multigpubfs_b200 import GraphDefinition, planner, sharded, workloads
from multigpubfs_b200.batch import BatchSweep
from multigpubfs_b200.engine import NativeGraph

PRIMES = tuple(p for p in range(29, 212) if all(p % q for q in range(2, 15)))
DEPTH = 256  # columns of a sweep's table of layer sizes, past the deepest of these graphs


def listed():
    return [
        # The smallest search a user calls graph.bfs() on: 40,320 states, all latency.
        {"name": "s8-lrx", "kind": "bfs", "family": "lrx", "n": 8, "visited": "auto"},
        # The reference's own GPU example: adjacent transpositions of 10 symbols.
        {"name": "s10-coxeter", "kind": "bfs", "family": "coxeter", "n": 10, "visited": "auto"},
        # The exact-key hash that a user picks where a rank bitmap would not fit.
        {"name": "s11-lrx-hash", "kind": "bfs", "family": "lrx", "n": 11, "visited": "hash"},
        # The headline: 6,227,020,800 states under three generators.
        {"name": "s13-lrx", "kind": "bfs", "family": "lrx", "n": 13, "visited": "auto"},
        # The same group under twelve generators, the largest search here.
        {"name": "s13-coxeter", "kind": "bfs", "family": "coxeter", "n": 13, "visited": "auto"},
        # A puzzle with repeated labels: four of each of four colours on 16 positions.
        {"name": "multiset-16", "kind": "bfs", "family": "multiset", "n": 16, "labels": 4, "visited": "auto"},
        # 0/1 strings of 24 positions, the wide states of more than 16 positions.
        {"name": "binary-24", "kind": "bfs", "family": "multiset", "n": 24, "labels": 2, "visited": "auto"},
        # A matrix group over a prime field: 1,972,681,200 states, six generators.
        {"name": "gl2-211", "kind": "bfs", "family": "gl2", "n": 211, "visited": "auto"},
        # The batched sweep over small random graphs, directed and inverse-closed.
        {"name": "sweep-512", "kind": "sweep", "family": "mixed", "count": 512},
        # A batch of large random graphs: 12 symbols, two to four generators and their inverses.
        {"name": "sweep-s12", "kind": "sweep", "family": "planner", "count": 8, "n": 12},
        # One search split by state ownership, both ranks' shards on this GPU.
        # Stopped past its largest layer, as a search with a layer limit is.
        {"name": "sharded-s12", "kind": "sharded", "family": "lrx", "n": 12, "world": 2, "layers": 52},
        # One training pass of the planner network over the rows of a sweep's layer tables.
        {"name": "planner-train", "kind": "planner", "rows": 6568},
    ]


def draw(rng):
    kind = rng.choice(["family", "random", "random", "hash", "hash", "multiset", "binary", "gl2", "sweep", "planner-sweep", "sharded",
                       "planner"])
    if kind == "family":
        family, n = rng.choice([(f, n) for f in ("lrx", "coxeter") for n in range(7, 13)
                                if (f, n) not in (("lrx", 8), ("coxeter", 10))])
        return {"kind": "bfs", "family": family, "n": n, "visited": "auto"}
    if kind == "random":
        return {"kind": "bfs", "family": "random", "n": rng.randint(7, 12), "gens": rng.randint(2, 4),
                "closed": rng.random() < 0.5, "graph": rng.randrange(1 << 30), "visited": "auto"}
    if kind == "hash":
        return {"kind": "bfs", "family": "random", "n": rng.randint(8, 11), "gens": rng.randint(2, 4),
                "closed": rng.random() < 0.5, "graph": rng.randrange(1 << 30), "visited": "hash"}
    if kind == "multiset":
        return {"kind": "bfs", "family": "multiset", "n": rng.randint(8, 15), "labels": rng.randint(3, 5),
                "visited": "auto"}
    if kind == "binary":
        return {"kind": "bfs", "family": "multiset", "n": rng.choice([17, 18, 19, 20, 21, 22, 23, 25]), "labels": 2,
                "visited": "auto"}
    if kind == "gl2":
        return {"kind": "bfs", "family": "gl2", "n": rng.choice(PRIMES[:-1]), "visited": "auto"}
    if kind == "sweep":
        return {"kind": "sweep", "family": "mixed", "count": 2 * int(round(math.exp(rng.uniform(0.0, math.log(255.0)))))}
    if kind == "planner-sweep":
        return {"kind": "sweep", "family": "planner", "count": rng.randint(1, 9), "n": rng.choice([10, 11])}
    if kind == "sharded":
        n = rng.randint(8, 11)
        return {"kind": "sharded", "family": rng.choice(["lrx", "coxeter"]), "n": n, "world": rng.randint(1, 5),
                "layers": rng.randint(n, n * (n - 1) // 2 - n)}
    return {"kind": "planner", "rows": int(round(math.exp(rng.uniform(math.log(100.0), math.log(20000.0)))))}


def _start(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    if case["family"] == "gl2":
        while True:
            m = [int(x) for x in rng.integers(0, n, 4)]
            if (m[0] * m[3] - m[1] * m[2]) % n:
                return m
    if case["family"] == "multiset":
        names = [int(x) for x in rng.choice(1000, case["labels"], replace=False)]
        return [names[i % case["labels"]] for i in range(n)]
    return [int(x) for x in rng.permutation(n)]


def _graph(case, seed):
    start = _start(case, seed)
    if case["family"] == "gl2":
        graph = workloads.gl2_graph(case["n"])
        graph["start"] = start
        return GraphDefinition.from_dict(graph)
    if case["family"] == "random":
        rng = np.random.default_rng(case["graph"])
        gens = [[int(x) for x in rng.permutation(case["n"])] for _ in range(case["gens"])]
        gens = workloads.with_inverses(gens) if case["closed"] else gens
    else:
        gens = workloads.coxeter(case["n"]) if case["family"] == "coxeter" else workloads.lrx(case["n"])
    return GraphDefinition.permutation(gens, start)


def _sweep_graphs(case, seed):
    if case["family"] == "mixed":
        return workloads.sweep(case["count"], seed_base=1_000_000 * (seed % 1000) + 20261203)
    return [workloads.planner_instance(i, case["n"], seed_base=1_000_000 * (seed % 1000) + 20261204)
            for i in range(case["count"])]


def _rows(case, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(0.0, 1.0, (case["rows"], planner.INPUTS)).astype(np.float32)
    t = np.column_stack([rng.normal(0.3, 0.6, case["rows"]), rng.uniform(0.0, 1.0, case["rows"])])
    return x, t.astype(np.float32)


def prepare(case, seed):
    if case["kind"] == "bfs":
        return {"case": case, "graph": _graph(case, seed)}
    if case["kind"] == "sweep":
        return {"case": case, "graphs": _sweep_graphs(case, seed)}
    if case["kind"] == "sharded":
        graph = _graph(case, seed)
        # A quarter of the rank's states holds its part of any layer of these graphs.
        room = sharded.geometry(case["n"], case["world"]).slice_bits // 4 + 4096
        shards = [sharded.DeviceShard(graph, r, case["world"], "cuda:0", frontier_capacity=room)
                  for r in range(case["world"])]
        return {"case": case, "shards": shards}
    x, t = _rows(case, seed)
    return {"case": case, "net": planner.PlannerNet(0, seed=seed % 65536), "x": x, "t": t}


def run(state):
    case = state["case"]
    if case["kind"] == "bfs":
        with NativeGraph(state["graph"]) as engine:
            engine.plan(visited=case["visited"])
            result = engine.run()
            out = {"layer_sizes": np.asarray(result.layer_sizes, dtype=np.int64),
                   "complete": np.asarray([result.complete], dtype=np.int64),
                   "previous_small": np.asarray(engine.sample(1), dtype=np.int64)}
            current = engine.sample(0)
            if result.layer_sizes[-1] <= 1000:  # of a larger layer, any 1000 of its states are the sample
                out["current"] = np.asarray(current, dtype=np.int64)
            return out
    if case["kind"] == "sweep":
        with BatchSweep(state["graphs"]) as sweep:
            sweep.run()
            tables = np.zeros((case["count"], DEPTH), dtype=np.int64)
            for row, table in zip(tables, sweep.layer_tables()):
                row[:len(table)] = table
            return tables
    if case["kind"] == "sharded":
        for shard in state["shards"]:
            shard.reset()
        bfs = sharded.ShardedBfs(state["shards"], sharded.LocalExchange(case["world"]))
        sizes = bfs.run(max_layers=case["layers"])
        return {"layer_sizes": np.asarray(sizes, dtype=np.int64), "visited": [s.slice for s in state["shards"]]}
    loss, grad = state["net"].loss_and_grad(state["x"], state["t"])
    return {"loss": np.asarray([loss], dtype=np.float32), "grad": grad}


def _states(case):
    """(states settled, generators) of one search."""
    n = case["n"]
    if case["family"] == "gl2":
        return (n * n - 1) * (n * n - n), 6
    if case["family"] == "multiset":
        ways = math.factorial(n)
        for c in range(case["labels"]):
            ways //= math.factorial(len(range(c, n, case["labels"])))
        return ways, 3
    graph = _graph(case, 0).to_dict()
    return int(planner.batch_statics([graph])[1][0]), len(graph["action"]["generators"])


def work(case):
    """A search on a rank domain marks each state once and expands it once, one
    bit written and one bit read; a hash or wide search writes and reads each
    key.  One operation per edge.  A training pass reads its rows and parameters
    and writes the gradient; forward and backward are six operations per weight
    and row."""
    if case["kind"] == "planner":
        weights = 64 * planner.INPUTS + 64 * 64 + 2 * 64
        return {"bytes": 4 * (case["rows"] * (planner.INPUTS + 2) + 2 * (weights + 130)),
                "flops": 6 * case["rows"] * weights}
    if case["kind"] == "sweep":
        graphs = _sweep_graphs(case, 0)
        sizes = [int(s) for s in planner.batch_statics(graphs)[1]]
        return {"bytes": sum(s // 4 + 1 for s in sizes),
                "flops": sum(s * len(g["action"]["generators"]) for s, g in zip(sizes, graphs))}
    states, gens = _states(case)
    key = 8 if case.get("visited") == "hash" else (8 * ((4 * case["n"] + 63) // 64) if case["family"] == "multiset"
                                                   and case["n"] > 16 else 0)
    return {"bytes": 2 * key * states if key else states // 4 + 1, "flops": gens * states}


def exact(case, seed):
    if case["kind"] != "planner":
        return None  # every output is a whole number
    x, t = (a.astype(np.float64) for a in _rows(case, seed))
    rng = np.random.default_rng(seed % 65536)
    w = []
    for rows, cols in ((64, planner.INPUTS), (64, 64), (2, 64)):
        w.append(rng.normal(0.0, math.sqrt(2.0 / cols), rows * cols).astype(np.float32).astype(np.float64)
                 .reshape(rows, cols))
    z1 = x @ w[0].T
    h1 = np.maximum(z1, 0.0)
    z2 = h1 @ w[1].T
    h2 = np.maximum(z2, 0.0)
    d = h2 @ w[2].T - t
    loss = (d * d).sum() / len(x)
    dy = 2.0 * d / len(x)
    d2 = (dy @ w[2]) * (z2 > 0)
    d1 = (d2 @ w[1]) * (z1 > 0)
    grad = np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), (dy.T @ h2).ravel(),
                           dy.sum(0)])
    return {"loss": np.asarray([loss]), "grad": grad}
