"""Device hash join at the sizes where its launches change: probe sides around
one and two scan tiles (4,096 and 8,192 rows), build sides around a power of
two, one heavy key, empty sides; rows equal the oracle's."""
import numpy as np
import pytest

from oracle.join_oracle import hash_join
from psm_benchmark_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("build,probe", [(0, 5), (1, 0), (1, 1), (31, 33), (32, 4095), (33, 4096), (1024, 4097),
                                         (1025, 8191), (2048, 8192), (3000, 8193), (5000, 20000)])
def test_join_rows(build, probe):
    rng = np.random.default_rng(build * 31 + probe)
    r = rng.integers(0, 500, (build, 3)).astype(np.uint32)
    s = rng.integers(0, 500, (probe, 2)).astype(np.uint32)
    if build:
        r[: build // 8, 0] = 7  # one heavy key
    rows, vert = None, None
    with api.Engine(arena_bytes=1 << 30) as e:
        rows, vert = api.hash_join(e, r, [0, 1, 2], s, [0, 3])
        assert api.hash_join(e, r, [0, 1, 2], s, [0, 3], count_only=True) == len(rows)
    want, wv = hash_join(r, [0, 1, 2], s, [0, 3])
    order = [list(vert).index(v) for v in wv] if len(rows) else []
    got = rows[:, order] if len(rows) else np.empty((0, len(wv)), np.uint32)
    key = lambda a: a[np.lexsort(a.T[::-1])] if len(a) else a  # noqa: E731
    assert np.array_equal(key(got), key(np.asarray(want, np.uint32).reshape(-1, len(wv))))
