"""Pair-frontier batches where their mask walk and lists can go wrong: masks
of a few words and of several passes, every width, out-degrees up to the
limit of 64, SSSP buckets, BFS on both sides of the switch to lists."""
from __future__ import annotations

import numpy as np
import pytest

from vertexapi2_gb300 import GASBatch
from vertexapi2_gb300._lib import PROGRAM_BFS, PROGRAM_SSSP

pytestmark = pytest.mark.gpu


def shallow(nv, fan, seed):
    """A tree of `fan` children a vertex plus a back edge each: few rounds,
    out-degree at most fan + 1."""
    rng = np.random.default_rng(seed)
    child = np.arange(1, nv, dtype=np.int32)
    parent = ((child - 1) // fan).astype(np.int32)
    s = np.concatenate([parent, child])
    d = np.concatenate([child, rng.integers(0, nv, nv - 1).astype(np.int32)])
    return s, d, rng.integers(1, 90, s.size, dtype=np.int32)


@pytest.mark.parametrize("nv,fan,nq,delta", [(2, 1, 1, 0), (31, 2, 32, 0), (33, 3, 33, 64), (5000, 63, 64, 0),
                                             (70001, 4, 100, 128), (300007, 7, 129, 0), (300007, 63, 256, 64)])
def test_pairs_match_oracle(gpu, port, nv, fan, nq, delta):
    s, d, w = shallow(nv, fan, seed=nv + nq)
    sources = np.random.default_rng(nq).integers(0, nv, nq).astype(np.int32)
    with GASBatch() as b:
        b.set_graph(nv, s, d, w)
        b.set_delta(delta)
        bfs, _ = b.run(PROGRAM_BFS, sources)
        sssp, _ = b.run(PROGRAM_SSSP, sources)
        again, _ = b.run(PROGRAM_SSSP, sources[::-1].copy())
    assert np.array_equal(again[::-1], sssp)  # masks are clean again after a run
    for q in sorted({0, nq // 2, nq - 1}):
        assert np.array_equal(bfs[q], port.bfs(nv, s, d, int(sources[q]))[0])
        assert np.array_equal(sssp[q], port.sssp(nv, s, d, w, int(sources[q]))[0])
