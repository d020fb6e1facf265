"""Batched personalised PageRank over every class of row width, with
in-degrees around the long units' thresholds, the ring's stages and the hub
chunks: the FP32 reference loop's bits where no in-degree exceeds 4096, and
sums of left-folded 4096-edge chunks above it."""
from __future__ import annotations

import numpy as np
import pytest

from vertexapi2_gb300 import GASBatch
from vertexapi2_gb300._lib import PROGRAM_PPR

pytestmark = pytest.mark.gpu

DEGREES = (1, 7, 8, 31, 32, 33, 255, 256, 257, 263, 289, 1023, 1024, 1025, 4095, 4096)


def edges(nv, degrees, seed):
    rng = np.random.default_rng(seed)
    d = np.concatenate([np.full(k, i, np.int32) for i, k in enumerate(degrees)]
                       + [rng.integers(len(degrees), nv, 3000).astype(np.int32)])
    return rng.integers(0, nv, d.size).astype(np.int32), d


def chunked_ppr(nv, s, d, source, iters=20):
    """The batched sums in FP32: each 4096-edge chunk of a vertex's in-edges a
    left fold from 0 in edge order, the chunks added in order."""
    into = [s[d == v] for v in range(nv)]
    deg = np.bincount(s, minlength=nv).astype(np.float32)
    alpha = np.float32(0.15)
    damp = np.float32(1) - alpha
    rank = np.zeros(nv, np.float32)
    rank[source] = 1
    tele = np.zeros(nv, np.float32)
    tele[source] = alpha
    fold = lambda x: np.cumsum(x, dtype=np.float32)[-1] if x.size else np.float32(0)
    for _ in range(iters):
        c = np.divide(rank, deg, out=np.zeros_like(rank), where=deg > 0)
        total = np.array([fold(np.array([fold(c[u[k:k + 4096]]) for k in range(0, u.size, 4096)], np.float32))
                          for u in into], np.float32)
        rank = tele + damp * total
    return rank


def batch(nv, s, d, sources):
    with GASBatch() as b:
        b.set_graph(nv, s, d)
        return b.run(PROGRAM_PPR, sources)[0]


@pytest.mark.parametrize("nq", [1, 2, 3, 4, 16, 31, 33, 40, 64, 65, 100, 129, 255])
def test_row_widths(gpu, port, nq):
    nv = 700
    sources = np.random.default_rng(nq).integers(0, nv, nq).astype(np.int32)
    s, d = edges(nv, DEGREES, seed=nq)
    got = batch(nv, s, d, sources)
    for q in sorted({0, nq // 2, nq - 1}):
        assert np.array_equal(got[q], port.ppr(nv, s, d, int(sources[q]))[0])
    s, d = edges(nv, DEGREES + (4097, 9000), seed=nq + 1000)
    got = batch(nv, s, d, sources)
    assert np.array_equal(got[-1], chunked_ppr(nv, s, d, int(sources[-1])))
    one = batch(nv, s, d, sources[-1:])
    assert np.array_equal(one[0].view(np.int32), got[-1].view(np.int32))
