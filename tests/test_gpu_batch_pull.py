"""Pull rounds of BFS batches at the edges of their units (64 edges a step,
256 a unit, 32 units a look-up) and of their mask words, a vertex's units with
it alone or shared, against single-source oracle depths."""
from __future__ import annotations

import numpy as np
import pytest

from vertexapi2_gb300 import GASBatch
from vertexapi2_gb300._lib import PROGRAM_BFS

pytestmark = pytest.mark.gpu

DEGREES = (0, 1, 2, 31, 32, 33, 63, 64, 65, 96, 127, 129, 255, 256, 257, 511, 513, 1025)


@pytest.mark.parametrize("nv,nq,chunk", [(5, 1, 256), (40, 31, 256), (900, 33, 256), (900, 64, 64),
                                         (900, 65, 32), (2500, 129, 256), (2500, 256, 2048),
                                         (12000, 255, 1)])
def test_bfs_pull_matches_oracle(gpu, port, nv, nq, chunk):
    rng = np.random.default_rng(nv + nq + chunk)
    some = np.array(DEGREES if nv < 10000 else DEGREES[:9])
    deg = np.where(rng.random(nv) < 0.5, rng.integers(0, 4, nv), rng.choice(some, nv))
    d = np.repeat(np.arange(nv, dtype=np.int32), deg)
    s = rng.integers(0, nv, d.size, dtype=np.int32)
    sources = rng.integers(0, nv, nq).astype(np.int32)
    with GASBatch() as b:
        b.set_graph(nv, s, d, None)
        b.set_config(chunk, 0, False)
        b.set_policy(1 << 20)  # pull while anything changes
        got, _ = b.run(PROGRAM_BFS, sources)
    for q in range(0, nq, max(1, nq // 40)):
        ref, _ = port.bfs(nv, s, d, int(sources[q]))
        assert np.array_equal(got[q], ref), f"query {q}"
    assert np.array_equal(got[nq - 1], port.bfs(nv, s, d, int(sources[nq - 1]))[0])
