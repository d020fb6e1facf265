"""The device graph builder at the edges of its sort tiles, on edge lists in
every order, and on an engine whose graph is replaced by a larger or smaller
one: CSC order (the batched PPR's ranks equal the FP32 left fold bit for
bit), CSR, weights and degree bins against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from vertexapi2_gb300 import GASBatch, GASEngine
from vertexapi2_gb300 import programs as P
from vertexapi2_gb300._lib import PROGRAM_CC, PROGRAM_PPR, PROGRAM_SSSP

pytestmark = pytest.mark.gpu


def make_edges(nv, ne, order, seed, hubs=()):
    """Random edges (duplicates and ties kept); the first targets get
    `hubs[k]` extra in-edges."""
    rng = np.random.default_rng(seed)
    s = rng.integers(0, nv, ne, dtype=np.int32)
    d = rng.integers(0, nv, ne, dtype=np.int32)
    at = 0
    for k, n in enumerate(hubs):
        d[at:at + n] = k
        at += n
    w = rng.integers(1, 100, ne, dtype=np.int32)
    if order in ("src", "both"):
        p = np.lexsort((d, s)) if order == "both" else np.argsort(s, kind="stable")
    elif order == "dst":
        p = np.argsort(d, kind="stable")
    else:
        p = rng.permutation(ne)
    return s[p], d[p], w[p]


def check_engine(e, port, nv, s, d, w):
    vd = P.sssp_init(nv, int(s[0]))
    e.set_graph(nv, vd, s, d, w)
    e.set_active(0, nv)
    rounds = e.run()
    st = e.round_stats()
    e.get_results()
    ref, rst = port.sssp(nv, s, d, w, int(s[0]), stats_cap=4096)
    assert np.array_equal(vd, ref) and rounds == rst["iterations"]
    assert np.array_equal(st["gathered"], rst["gathered"])
    assert np.array_equal(st["scattered"], rst["scattered"])


@pytest.mark.parametrize("order", ["random", "src", "dst", "both"])
@pytest.mark.parametrize("nv,ne", [(1, 1), (2, 3), (300, 4095), (257, 4096), (65537, 4097),
                                   (9000, 70001)])
def test_orders_and_tile_edges(gpu, port, nv, ne, order):
    hubs = (1024, 1025, 2049) if ne > 60000 else ()
    s, d, w = make_edges(nv, ne, order, seed=ne, hubs=hubs)
    with GASEngine(PROGRAM_SSSP) as e:
        check_engine(e, port, nv, s, d, w)
    src = np.array([int(s[0]), int(d[0])], np.int32)
    with GASBatch() as b:
        b.set_graph(nv, s, d, w)
        got, _ = b.run(PROGRAM_PPR, src)
    for q, x in enumerate(src):
        assert np.array_equal(got[q], port.ppr(nv, s, d, int(x))[0])


def test_graph_replaced(gpu, port):
    with GASEngine(PROGRAM_SSSP) as e:
        for nv, ne, order in ((500, 5000, "random"), (20000, 90000, "src"), (40, 60, "dst"),
                              (19000, 80000, "random")):
            check_engine(e, port, nv, *make_edges(nv, ne, order, seed=nv))
        with pytest.raises(Exception):
            e.set_graph(5, None, np.array([0, 7], np.int32), np.array([1, 2], np.int32),
                        np.array([1, 1], np.int32))
        check_engine(e, port, 700, *make_edges(700, 9000, "both", seed=3))
    with GASEngine(PROGRAM_CC) as e:
        z = np.zeros(0, np.int32)
        vd = P.cc_init(6)
        e.set_graph(6, vd, z, z)
        e.set_active(0, 6)
        assert e.run() == 1
        e.get_results()
        assert vd.tolist() == list(range(6))
