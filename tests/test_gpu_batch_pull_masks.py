"""Pull rounds of BFS batches on vertex masks, whatever the out-degrees (graphs
of out-degrees up to 64 take the pair frontier otherwise, which has no pull
rounds): units of one edge, so that most vertices share their words between
several units, and many units a warp."""
from __future__ import annotations

import numpy as np
import pytest

from vertexapi2_gb300 import GASBatch
from vertexapi2_gb300._lib import PROGRAM_BFS

pytestmark = pytest.mark.gpu

DEGREES = (0, 1, 2, 31, 32, 33, 63, 64, 65)


@pytest.mark.parametrize("nv,nq,chunk", [(12000, 255, 1), (12000, 31, 1), (12000, 64, 3), (3000, 256, 33),
                                         (50, 65, 1)])
def test_bfs_pull_matches_oracle(gpu, port, nv, nq, chunk):
    rng = np.random.default_rng(nv + nq + chunk)
    deg = np.where(rng.random(nv) < 0.5, rng.integers(0, 4, nv), rng.choice(DEGREES, nv))
    d = np.repeat(np.arange(nv, dtype=np.int32), deg)
    s = rng.integers(0, nv, d.size, dtype=np.int32)
    sources = rng.integers(0, nv, nq).astype(np.int32)
    with GASBatch() as b:
        b.set_graph(nv, s, d, None)
        b.set_frontier(0)
        b.set_config(chunk, 0, False)
        b.set_policy(1 << 20)  # pull while anything changes
        got, _ = b.run(PROGRAM_BFS, sources)
    for q in sorted({0, *range(0, nq, max(1, nq // 40)), nq - 1}):
        assert np.array_equal(got[q], port.bfs(nv, s, d, int(sources[q]))[0]), f"query {q}"
