"""Timed cases of the subgraph-matching paths.

A user's program keeps a data graph resident on the GPU and an engine (or a
server) beside it, and sends it queries it has not sent before. So a state
holds the resident graph, the engine and a set of queries drawn from the
seed; a pass answers all of them through the public Python API, host work
included. The graphs are the seeded generators' data sets
(psm_benchmark_b200/gen.py), one per configuration.

Kinds of a case:
  match    one call per query (match), the whole GPU for each: interactive use
  batch    all queries in one call (match_batch)
  serve    all queries submitted to a server, results drained
  inspect  one run per query, its candidates, tables and order read back
  join     one call per query of the decomposition + hash-join path

Counts, candidate sets, table rows and orders are whole numbers.
"""
from __future__ import annotations

from functools import lru_cache

import numpy as np

from psm_benchmark_b200 import api, gen

CAP = 10**9  # embedding cap of the R-MAT workloads


def _case(name, kind, graph, scale, edge_factor, labels, zipf, queries, lo, hi, method, cap):
    """graph: "rmat" (2^scale vertices) or "chung_lu" (9,460 vertices; scale
    and edge_factor 0). Query sizes are spread evenly over [lo, hi]."""
    c = {"kind": kind, "graph": graph, "scale": scale, "edge_factor": edge_factor, "labels": labels, "zipf": zipf,
         "queries": queries, "lo": lo, "hi": hi, "method": method, "cap": cap}
    return {"name": name, **c} if name else c


def listed():
    return [
        # The smallest calls: 4- to 6-vertex queries on a graph the size of a
        # protein-interaction network (gen.plain_small), counted in full.
        # Latency and launches.
        _case("match_small", "match", "chung_lu", 0, 0, 307, 1.1, 8, 4, 6, "GQL_GQL_GQL", 0),
        # The same data set queried in one call: gen.plain_small's 200 queries
        # of 8 vertices.
        _case("batch_small", "batch", "chung_lu", 0, 0, 307, 1.1, 200, 8, 8, "GQL_GQL_GQL", 0),
        # Odd-sized small queries on a mid-sized graph, GQL filter and order.
        _case("match_gql", "match", "rmat", 17, 8, 32, 0.0, 7, 5, 11, "GQL_GQL_EXPLORE", CAP),
        # The benchmark's queries (gen.plain_rmat), one call each: 12 vertices ...
        _case("match_12", "match", "rmat", 20, 8, 32, 0.0, 16, 12, 12, "CFL_CFL_EXPLORE", CAP),
        # ... and 16 vertices.
        _case("match_16", "match", "rmat", 20, 8, 32, 0.0, 16, 16, 16, "CFL_CFL_EXPLORE", CAP),
        # The largest queries the interface takes.
        _case("match_32", "match", "rmat", 20, 8, 32, 0.0, 9, 24, 32, "CFL_CFL_EXPLORE", CAP),
        # A small batch and a large one of mixed sizes (gen.batched).
        _case("batch_mixed", "batch", "rmat", 20, 8, 32, 0.0, 48, 4, 32, "CFL_CFL_EXPLORE", CAP),
        _case("batch_large", "batch", "rmat", 20, 8, 32, 0.0, 160, 4, 32, "CFL_CFL_EXPLORE", CAP),
        # Requests arriving faster than they are answered, mostly small ones.
        _case("serve", "serve", "rmat", 20, 8, 32, 0.0, 96, 4, 16, "CFL_CFL_EXPLORE", CAP),
        # Filtering and tables alone matter: candidates, tables and order are
        # read back, the enumeration stops early.
        _case("inspect_cfl", "inspect", "rmat", 20, 8, 32, 0.0, 3, 10, 16, "CFL_CFL_EXPLORE", 10**5),
        _case("inspect_gql", "inspect", "rmat", 18, 8, 32, 0.0, 3, 9, 13, "GQL_GQL_GQL", 10**5),
        # Decomposition and hash joins, counted in full.
        _case("join", "join", "chung_lu", 0, 0, 307, 1.1, 16, 7, 9, "CFL_CFL_EXPLORE", 0),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["match", "match", "batch", "batch", "serve", "inspect", "join"])
    if kind == "join" or (kind in ("match", "batch") and rng.random() < 0.25):
        lo = rng.randint(4, 8)
        n = rng.randint(1, 24) if kind == "join" else _log_int(rng, 1, 240)
        method = rng.choice(["GQL_GQL_GQL", "CFL_CFL_EXPLORE", "CFL_GQL_LFTJ", "NLF_GQL_LFTJ"])
        return _case(None, kind, "chung_lu", 0, 0, 307, 1.1, n, lo, rng.randint(lo, 8), method, 0)
    # On the smaller graphs (a few thousand vertices of a label) a large query
    # may have few embeddings and a search of minutes: they get small queries.
    scale = rng.randint(16, 20)
    most_vertices = {16: 8, 17: 10, 18: 12, 19: 20, 20: 32}[scale]
    lo = rng.randint(4, min(20, most_vertices))
    hi = rng.randint(lo, min(most_vertices, lo + 12))
    method = rng.choice(["CFL_CFL_EXPLORE", "CFL_CFL_EXPLORE", "GQL_GQL_EXPLORE", "CFL_GQL_LFTJ"])
    most = {"match": 12, "batch": 100, "serve": 80, "inspect": 4}[kind]
    return _case(None, kind, "rmat", scale, 8, rng.choice([16, 32, 32]), 0.0, _log_int(rng, 1, most), lo, hi, method,
                 10**5 if kind == "inspect" else CAP)


@lru_cache(maxsize=3)
def _graph(kind, scale, edge_factor, labels, zipf):
    if kind == "chung_lu":
        return gen.make_graph("chung_lu", 1, n=9460, num_labels=labels, zipf_s=zipf)
    return gen.make_graph("rmat", 2, scale=scale, edge_factor=edge_factor, num_labels=labels, zipf_s=zipf)


def prepare(case, seed):
    g = _graph(case["graph"], case["scale"], case["edge_factor"], case["labels"], case["zipf"])
    sizes = np.linspace(case["lo"], case["hi"], case["queries"]).round().astype(int)
    # gen.make_queries takes query j from seed ^ j: the seed stays clear of j's bits
    queries = gen.make_queries(g, sizes, (gen.BASE_SEED + seed) << 12)
    data = api.DataGraph.from_graph(g)
    state = {"case": case, "queries": queries, "data": data}
    if case["kind"] == "serve":
        state["server"] = api.Server(data, case["method"], cap=case["cap"], lanes=2, max_batch=64)
    else:
        state["engine"] = api.Engine()
    return state


def _place(out, at, values):
    out[at: at + len(values)] = values
    return at + len(values)


def _inspect(engine, data, query, method, cap):
    """What a run holds, in buffers of one size for every query."""
    cand = np.zeros(1 << 21, np.uint32)
    tables = np.zeros(1 << 23, np.uint32)
    plan = np.zeros((2, 32), np.uint32)
    with api.Run(engine, data, query, method, cap=cap) as r:
        at = 0
        for u in range(query.num_vertices):
            at = _place(cand, at, r.candidates(u))
        at = 0
        for a, b in query.edge_list():
            for t in (*r.table(int(a), int(b)), *r.table(int(b), int(a))):
                at = _place(tables, at, t)
        order, pivot = r.order()
        plan[0, : len(order)] = order
        plan[1, 1: len(pivot)] = pivot[1:]  # the first vertex has no pivot
        return {"count": r.result.count, "candidates": cand, "tables": tables, "plan": plan}


def run(state):
    case, data, queries = state["case"], state["data"], state["queries"]
    method, cap, kind = case["method"], case["cap"], case["kind"]
    if kind == "serve":
        server = state["server"]
        place = {server.submit(q): i for i, q in enumerate(queries)}
        counts = np.zeros(len(queries), np.int64)
        for r in server.drain(len(queries)):
            counts[place[r.ticket]] = r.count
        return counts
    engine = state["engine"]
    if kind == "inspect":
        return [_inspect(engine, data, q, method, cap) for q in queries]
    if kind == "join":
        got = [api.match_join(engine, data, q, method, max_unit_vertices=4) for q in queries]
        rows = np.zeros((2, len(got), 32), np.int64)
        for i, r in enumerate(got):
            _place(rows[0, i], 0, r.unit_rows)
            _place(rows[1, i], 0, r.join_rows)
        return {"count": np.array([r.count for r in got], np.int64), "unit_rows": rows[0], "join_rows": rows[1]}
    if kind == "batch":
        got = api.match_batch(engine, data, queries, method, cap=cap)
    else:
        got = [api.match(engine, data, q, method, cap=cap) for q in queries]
    return {"count": np.array([r.count for r in got], np.int64),
            "table_entries": np.array([r.table_entries for r in got], np.int64)}


def work(case):
    """Every query vertex's filter reads its label's vertices (offsets and
    rows) once; what the search below needs depends on the data."""
    if case["graph"] == "chung_lu":
        vertices, degree = 9460, 7.8
    else:
        vertices, degree = 2 ** case["scale"], 2 * case["edge_factor"]
    per_vertex = vertices / case["labels"] * (8 + 4 * degree)
    size = (case["lo"] + case["hi"]) / 2
    return {"bytes": case["queries"] * size * per_vertex, "flops": 0}
