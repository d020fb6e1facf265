"""The leading dense rounds' kernel (pull.cuh) at the edges of its degree
classes, in both forms (few and many work units), with and without hot
sources: minima against the oracle, PageRank bit for bit against the same
rounds run by the main kernel's pull pass, which folds in the same order."""
from __future__ import annotations

import numpy as np
import pytest

from vertexapi2_gb300 import GASEngine
from vertexapi2_gb300 import programs as P
from vertexapi2_gb300._lib import PROGRAM_CC, PROGRAM_PAGERANK, PROGRAM_SSSP

pytestmark = pytest.mark.gpu

EDGES = (0, 1, 3, 4, 7, 8, 9, 10, 31, 32, 33, 63, 64, 65, 66, 127, 129, 511, 1023, 1024, 1025, 2047, 2049)


def degree_graph(nv, degrees, hot_share, seed):
    """Vertex v has in-degree degrees[v % len]; `hot_share` of the sources
    are among 50 vertices."""
    rng = np.random.default_rng(seed)
    deg = np.array([degrees[v % len(degrees)] for v in rng.permutation(nv)], np.int64)
    d = np.repeat(np.arange(nv, dtype=np.int32), deg)
    s = rng.integers(0, nv, d.size, dtype=np.int32)
    hot = rng.random(d.size) < hot_share
    s[hot] = rng.integers(0, 50, int(hot.sum()), dtype=np.int32)
    w = rng.integers(1, 60, d.size, dtype=np.int32)
    p = rng.permutation(d.size)
    return s[p], d[p], w[p]


def run(program, nv, s, d, vd, w=None, max_iters=0, blocks=0):
    vd = vd.copy()
    with GASEngine(program) as e:
        e.set_graph(nv, vd, s, d, w)
        if blocks:  # a launch shape of its own leaves every round to the main kernel
            e.set_launch_config(True, blocks)
        e.set_dense_policy(1 << 20)  # dense while any vertex returned true
        e.set_active(0, nv)
        rounds = e.run(max_iters)
        st = e.round_stats()
        e.get_results()
    return vd, rounds, st


# (vertices, in-degrees, share of edges from 50 sources): the wide form, the
# narrow one (over 8,512 slices), one without a hot source
GRAPHS = [(900, EDGES, 0.6), (70000, (9, 64, 65, 66, 3, 0), 0.5), (70000, (1, 2, 1), 0.0)]


@pytest.mark.parametrize("nv,degrees,hot", GRAPHS)
def test_minima_match_oracle(gpu, port, nv, degrees, hot):
    s, d, w = degree_graph(nv, degrees, hot, seed=nv + len(degrees))
    ref, st = port.cc(nv, s, d, stats_cap=4096)
    got, rounds, gst = run(PROGRAM_CC, nv, s, d, P.cc_init(nv))
    assert np.array_equal(got, ref) and rounds == st["iterations"]
    for k in ("active", "gathered", "ret", "scattered"):
        assert np.array_equal(gst[k], st[k])
    ref, st = port.sssp(nv, s, d, w, int(s[0]), stats_cap=4096)
    got, rounds, gst = run(PROGRAM_SSSP, nv, s, d, P.sssp_init(nv, int(s[0])), w)
    assert np.array_equal(got, ref) and rounds == st["iterations"]
    assert np.array_equal(gst["active"], st["active"])


@pytest.mark.parametrize("nv,degrees,hot", GRAPHS)
def test_pagerank_order_is_the_pull_pass_order(gpu, nv, degrees, hot):
    s, d, _ = degree_graph(nv, degrees, hot, seed=nv)
    init = P.pagerank_init(nv, s)
    a, ra, sa = run(PROGRAM_PAGERANK, nv, s, d, init, max_iters=15)
    b, rb, sb = run(PROGRAM_PAGERANK, nv, s, d, init, max_iters=15, blocks=4)
    assert ra == rb
    assert np.array_equal(a["rank"].view(np.int32), b["rank"].view(np.int32))
    for k in sa:
        assert np.array_equal(sa[k], sb[k])
