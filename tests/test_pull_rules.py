"""Which kernel runs the leading dense rounds: the shapes on which each of the
three was measured to be the fastest, or as fast."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

from vertexapi2_gb300 import graphs

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

# (any order, messages, bytes of a value, slices carry the edge data)
CC, SSSP, PAGERANK = (1, 1, 4, 1), (1, 0, 4, 1), (0, 1, 4, 1)
PLAIN, LARGE, EDGES8 = (0, 0, 8, 1), (0, 0, 256, 1), (0, 0, 8, 0)


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("pull_rules") / "pull_rules")
    r = subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O1",
                        "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "cpp", "pull_rules.cu"),
                        "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]

    def run(program, nv, s, d):
        deg = np.bincount(d, minlength=nv)
        hub = deg > 1024
        chunks = int(((deg[hub] + 1023) // 1024).sum())
        mid, small = int(((deg > 64) & ~hub).sum()), int(((deg > 8) & (deg <= 64)).sum())
        tiny = (int((deg <= 8).sum()) + 31) // 32
        shape = (*program, nv, len(s), int(np.bincount(s, minlength=nv).max()), chunks + mid // 4 + small // 32,
                 chunks + (mid + 3) // 4 + (small + 31) // 32 + tiny, chunks + mid + (small + 3) // 4 + tiny)
        out = subprocess.run([exe], input=" ".join(map(str, shape)), capture_output=True, text=True, check=True)
        return out.stdout.strip()

    return run


def even(nv, degree):
    rng = np.random.default_rng(nv + degree)
    return nv, rng.integers(0, nv, nv * degree, dtype=np.int32), rng.integers(0, nv, nv * degree, dtype=np.int32)


def lattice(side):
    g = graphs.grid(side, side, 0.15, seed=7)
    return g.n_vertices, g.srcs, g.dsts


def rmat(scale, symmetric):
    g = graphs.rmat(scale, 16, seed=7, symmetrize=symmetric)
    return g.n_vertices, g.srcs, g.dsts


@pytest.mark.parametrize("graph,expected", [
    ((rmat, 14, True), {CC: "wide", SSSP: "wide", PAGERANK: "wide", PLAIN: "wide", LARGE: "csc", EDGES8: "wide"}),
    ((rmat, 16, False), {CC: "wide", PAGERANK: "wide", PLAIN: "wide", EDGES8: "csc"}),
    ((rmat, 19, True), {CC: "narrow", SSSP: "narrow", PAGERANK: "narrow", PLAIN: "csc", LARGE: "csc", EDGES8: "csc"}),
    ((lattice, 200), {CC: "wide", PAGERANK: "wide", PLAIN: "wide", EDGES8: "wide"}),
    ((lattice, 1000), {CC: "wide", SSSP: "csc", PAGERANK: "wide", PLAIN: "csc", EDGES8: "csc"}),
    ((lattice, 1700), {CC: "csc", PAGERANK: "wide", PLAIN: "csc"}),
    ((even, 20000, 16), {CC: "wide", PAGERANK: "wide"}),
    ((even, 100000, 16), {CC: "narrow", SSSP: "narrow", PAGERANK: "narrow", PLAIN: "csc"}),
    ((even, 1000000, 3), {CC: "wide", SSSP: "csc", PAGERANK: "wide"}),
    ((even, 2000000, 8), {CC: "narrow", SSSP: "narrow", PAGERANK: "narrow"}),
], ids=str)
def test_choice(choose, graph, expected):
    make, *size = graph
    g = make(*size)
    assert {p: choose(p, *g) for p in expected} == expected
