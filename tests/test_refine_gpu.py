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


@pytest.mark.parametrize("run", [31, 32, 95, 96, 97, 127, 128, 129, 224, 225, 600])
def test_label_runs_around_the_warp_walk(run):
    """Marking and table passes walk label runs above 96 entries with a whole
    warp, 128 entries a round: candidates and tables equal the oracle's for
    centres whose run of one label has `run` entries (all or every third of
    them candidates), beside short ones."""
    rng = np.random.default_rng(run)
    leaves = 700
    centres = 6
    lab = np.concatenate([np.zeros(centres, int), np.ones(leaves, int), np.full(leaves // 3 + 1, 2)])
    edges = []
    for c in range(centres):
        d = run if c % 2 == 0 else 5
        edges += [(c, centres + int(x)) for x in rng.choice(leaves, d, replace=False)]
    edges += [(centres + 3 * i, centres + leaves + i) for i in range(leaves // 3)]  # every third leaf
    g = Graph.from_edges(len(lab), lab, edges)
    og, dg = OracleGraph(g), api.DataGraph.from_graph(g)
    queries = [Graph.from_edges(3, [1, 0, 1], [(0, 1), (1, 2)]),
               Graph.from_edges(4, [2, 1, 0, 1], [(0, 1), (1, 2), (2, 3)])]
    with api.Engine(arena_bytes=1 << 30) as eng:
        for q in queries:
            for f, m in (("CFL", "CFL_CFL_EXPLORE"), ("GQL", "GQL_GQL_GQL")):
                ref = og.run(q, f, f, cap=10**6)
                with api.Run(eng, dg, q, m, cap=10**6) as r:
                    assert r.result.count == ref.count
                    for u in range(q.num_vertices):
                        assert np.array_equal(r.candidates(u), ref.candidates[u]), (m, u)
                    for (a, b), (off, adj) in ref.tables.items():
                        got = r.table(a, b)
                        assert np.array_equal(got[0], off) and np.array_equal(got[1], adj), (m, a, b)
                batch = api.match_batch(eng, dg, [q, q], m, cap=10**6)
                assert [x.count for x in batch] == [ref.count] * 2
    dg.close()
