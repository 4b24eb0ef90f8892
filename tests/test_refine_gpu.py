"""GQL refinement on rows around the 128 entries that a warp holds at once:
candidates equal the oracle's for centres with 30 to 400 neighbours whose
matching needs one or several neighbours of a label, some of them shared."""
import numpy as np
import pytest

from oracle.oracle import OracleGraph
from psm_benchmark_b200 import api
from psm_benchmark_b200.graphs import Graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("labels", [2, 3, 4])
def test_refined_candidates_match_oracle(labels):
    rng = np.random.default_rng(9 + labels)
    degrees = [30, 32, 33, 127, 128, 129, 130, 160, 255, 256, 257, 400]
    leaves = 500
    n = len(degrees) + leaves
    lab = np.concatenate([np.zeros(len(degrees), int), rng.integers(1, labels, leaves) if labels > 2 else
                          np.ones(leaves, int)])
    edges = [(i, len(degrees) + int(x)) for i, d in enumerate(degrees) for x in rng.choice(leaves, d, replace=False)]
    edges += [(len(degrees) + int(a), len(degrees) + int(b)) for a, b in rng.integers(0, leaves, (150, 2)) if a != b]
    g = Graph.from_edges(n, lab, edges)
    og, dg = OracleGraph(g), api.DataGraph.from_graph(g)
    a, b = 1, labels - 1
    queries = [Graph.from_edges(4, [0, a, b, a], [(0, 1), (0, 2), (0, 3), (1, 2)]),
               Graph.from_edges(5, [0, a, a, b, b], [(0, 1), (0, 2), (0, 3), (0, 4), (1, 2), (3, 4)]),
               Graph.from_edges(8, [0] + [a] * 7, [(0, i) for i in range(1, 8)] + [(1, 2), (3, 4)])]
    with api.Engine(arena_bytes=1 << 30) as eng:
        for q in queries:
            ref = og.run(q, "GQL", "GQL", cap=1000, want_tables=False)
            with api.Run(eng, dg, q, "GQL_GQL_GQL", cap=1000) as run:
                assert run.result.count == ref.count
                if ref.filter_ok:
                    for u in range(q.num_vertices):
                        assert np.array_equal(run.candidates(u), ref.candidates[u]), u
    dg.close()
