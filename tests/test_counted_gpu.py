"""Counted vertices (query vertices without later neighbours in the matching
order, which multiply a weight instead of being branched on): counts and
algorithmic bytes equal the oracle's on random queries of few and many labels
(a counted vertex sharing its label with walked vertices before and after it,
several counted vertices, multi-row ones, counts of zero), with and without
the enumerator's caches, plain and batched; products beyond 64 bits."""
import os

import numpy as np
import pytest

from oracle.oracle import OracleGraph
from psm_benchmark_b200 import api, gen
from psm_benchmark_b200.graphs import Graph
from psm_benchmark_b200.native import PSM_ERR_TIMEOUT, PSM_OK

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engines():
    with api.Engine(arena_bytes=1 << 30) as eng:
        os.environ["PSM_ENUM_CACHE"] = "0"
        try:
            plain = api.Engine(arena_bytes=1 << 30)
        finally:
            del os.environ["PSM_ENUM_CACHE"]
        yield eng, plain
        plain.close()


@pytest.mark.parametrize("labels,size", [(2, 5), (3, 6), (4, 7), (6, 8), (8, 9), (8, 12), (16, 10), (16, 16), (40, 14),
                                         (40, 24), (40, 32)])
def test_counts_and_bytes_match_oracle(engines, labels, size):
    g = gen.make_graph("rmat", 60 + labels, scale=8 if labels < 16 else 9, edge_factor=4, num_labels=labels)
    queries = gen.make_queries(g, [size] * 12, 0x51 + (size << 8))
    og, dg = OracleGraph(g), api.DataGraph.from_graph(g)
    limit = 20_000_000
    checked = 0
    for f, m in (("CFL", "CFL_CFL_EXPLORE"), ("GQL", "GQL_GQL_GQL")):
        refs = [og.run(q, f, f, cap=limit, want_tables=False) for q in queries]
        batch = api.match_batch(engines[0], dg, queries, m, cap=limit)
        for q, r, b in zip(queries, refs, batch):
            assert b.count == min(r.count, limit)
            for e in engines:
                got = api.match(e, dg, q, m, cap=limit)
                assert got.count == min(r.count, limit)
                if r.count < limit:
                    assert got.alg_bytes == int(r.depth_bytes.sum())
                    checked += 1
    assert checked >= 1 or size >= 24
    dg.close()


def test_products_beyond_64_bits(engines):
    """A hub with 4,096 neighbours of each of eight labels: a star of eight
    leaves has 2^96 embeddings. A capped count is the cap, an uncapped one
    ends as partial, and the context serves the next query."""
    k, per = 8, 4096
    leaves = np.arange(1, k * per + 1)
    labels = np.concatenate([[0], (leaves - 1) // per + 1])
    g = Graph.from_edges(len(labels), labels, np.stack([np.zeros(len(leaves), np.int64), leaves], axis=1))
    star = Graph.from_edges(k + 1, np.arange(k + 1), [(0, i) for i in range(1, k + 1)])
    small = Graph.from_edges(5, np.arange(5), [(0, i) for i in range(1, 5)])
    dg = api.DataGraph.from_graph(g)
    for e in engines:
        for cap in (10**9, 2**63 + 7, 2**64 - 1):
            r = api.match(e, dg, star, "CFL_CFL_EXPLORE", cap=cap)
            assert r.count == cap and r.status == PSM_OK and r.overtime == 0
        r = api.match(e, dg, star, "CFL_CFL_EXPLORE", cap=0, time_limit=20.0)
        assert r.status == PSM_ERR_TIMEOUT and r.overtime == 1 and r.count > 0
        r = api.match(e, dg, small, "CFL_CFL_EXPLORE", cap=0)
        assert r.count == per**4 and r.status == PSM_OK
    dg.close()
