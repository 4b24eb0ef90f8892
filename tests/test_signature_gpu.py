"""Neighbour-label signatures in the NLF filter: candidates equal the oracle's
around 32 labels (up to which a signature bit is one label) and for neighbour
labels needed once, twice and three times (the signature counts to two)."""
import numpy as np
import pytest

from oracle.oracle import OracleGraph
from psm_benchmark_b200 import api, gen
from psm_benchmark_b200.graphs import Graph

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    with api.Engine(arena_bytes=1 << 30) as e:
        yield e


@pytest.mark.parametrize("labels", [1, 2, 31, 32, 33, 64, 70])
def test_nlf_candidates_match_oracle(engine, labels):
    g = gen.make_graph("rmat", 80 + labels, scale=10, edge_factor=8, num_labels=labels)
    og, dg = OracleGraph(g), api.DataGraph.from_graph(g)
    top = labels - 1
    queries = gen.make_queries(g, [4, 6, 9], 0x77)
    for need in (1, 2, 3):  # a centre with `need` neighbours of the last label, and one of label 0
        lab = np.array([top // 2] + [top] * need + [0])
        queries.append(Graph.from_edges(need + 2, lab, [(0, i) for i in range(1, need + 2)]))
    # a label that hashes to label 0's bit, and one past the graph's labels
    queries.append(Graph.from_edges(3, np.array([0, 32 % labels, top]), [(0, 1), (0, 2)]))
    queries.append(Graph.from_edges(2, np.array([0, labels + 31]), [(0, 1)]))
    for q in queries:
        for f in ("NLF", "GQL", "CFL"):
            ref = og.run(q, f, "GQL", cap=1000, want_tables=False)
            with api.Run(engine, dg, q, f"{f}_GQL_LFTJ", cap=1000) as run:
                assert run.result.count == ref.count, (f, q.labels)
                if ref.filter_ok:
                    for u in range(q.num_vertices):
                        assert np.array_equal(run.candidates(u), ref.candidates[u]), (f, u)
    dg.close()
