"""Preparation team of a batch: the rule's counts equal both teams' around the
batch size where it changes, and a batch whose clusters' buffers do not fit the
arena is prepared with a block per query."""
import pytest

from psm_benchmark_b200 import api, gen

pytestmark = pytest.mark.gpu

METHOD, CAP = "CFL_CFL_EXPLORE", 10**5


def counts(engine, dg, queries, team):
    engine.set_batch_tuning(team=team)
    return [r.count for r in api.match_batch(engine, dg, queries, METHOD, cap=CAP)]


@pytest.mark.parametrize("queries", [1, 29, 31, 60, 200])
def test_teams_count_alike(queries):
    g = gen.make_graph("rmat", 90, scale=14, edge_factor=8, num_labels=32)
    qs = gen.make_queries(g, [4 + i % 6 for i in range(queries)], 0x99)
    with api.Engine(arena_bytes=1 << 30) as e:
        dg = api.DataGraph.from_graph(g)
        rule = counts(e, dg, qs, "RULE")
        assert rule == counts(e, dg, qs, "BLOCK") == counts(e, dg, qs, "CLUSTER")
        dg.close()


def test_batch_that_only_fits_with_blocks():
    g = gen.make_graph("rmat", 91, scale=18, edge_factor=8, num_labels=32)
    qs = gen.make_queries(g, [6] * 60, 0x9A)
    dg = api.DataGraph.from_graph(g)
    found = False
    for mb in range(60, 400, 12):
        with api.Engine(arena_bytes=mb << 20) as e:
            try:
                want = counts(e, dg, qs, "BLOCK")
            except Exception:
                continue  # too small for blocks
            try:
                counts(e, dg, qs, "CLUSTER")
            except Exception:
                assert counts(e, dg, qs, "RULE") == want
                found = True
            break
    assert found
    dg.close()
