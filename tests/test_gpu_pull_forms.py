"""The leading dense rounds' kernels: results equal, bit for bit, those of the
same rounds run by the main kernel's pull pass.  256-byte vertex data with more
sources of 65,535 and more out-edges than the table of hot sources holds;
Programs that declare nothing, with vertex data and edge data of 8 bytes, on
small graphs (the sliced layout, wide) and on large ones (the CSC kernel);
PageRank's messages on a graph of enough work units for the narrow form (two
for each warp of the chip), where a lane walks eight or four lanes' shares of
a vertex one after the other."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

from vertexapi2_gb300 import GASEngine
from vertexapi2_gb300 import programs as P
from vertexapi2_gb300._lib import PROGRAM_PAGERANK

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def driver(gpu, tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("pull_forms") / "pull_forms")
    lib = os.path.join(ROOT, "vertexapi2_gb300", "_build")
    r = subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-fmad=false",
                        "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "cpp", "pull_forms.cu"),
                        "-L", lib, "-lgas_gb300", "-Xlinker", f"-rpath={lib}", "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return exe


def both(exe, tmp_path, nv, s, d, which, words):
    """Rounds and vertex data of the two runs."""
    inp, out = tmp_path / "in.bin", tmp_path / "out.bin"
    with open(inp, "wb") as f:
        np.array([nv, s.size, which, 0], np.int32).tofile(f)
        s.astype(np.int32).tofile(f)
        d.astype(np.int32).tofile(f)
    r = subprocess.run([exe, str(inp), str(out)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
    data = np.fromfile(out, np.int32).reshape(2, 2 + nv * words)
    os.remove(inp)
    os.remove(out)
    assert data[:, 0].tolist() == [0, 0]
    return data[0, 1:], data[1, 1:]


@pytest.mark.parametrize("which", [0, 3])  # undeclared, minima in any order
@pytest.mark.parametrize("hubs,low,high", [(600, 66000, 80000), (200, 60000, 70000), (600, 300, 900)])
def test_large_vertex_data_hot_sources(driver, tmp_path, hubs, low, high, which):
    nv = 40000
    rng = np.random.default_rng(hubs + low)
    s = np.repeat(rng.choice(nv, hubs, False), rng.integers(low, high, hubs)).astype(np.int32)
    s = np.concatenate([s, rng.integers(0, nv, 200000, dtype=np.int32)])
    d = rng.integers(0, nv, s.size, dtype=np.int32)
    a, b = both(driver, tmp_path, nv, s, d, which, 64)
    assert a[0] > 2 and np.array_equal(a, b)


DEGREES = (0, 1, 3, 4, 7, 8, 9, 10, 31, 32, 33, 63, 64, 65, 66, 127, 129, 511, 1023, 1024, 1025, 2047, 2049)


def narrow_graph(hot_share, seed):
    """Every degree class and its edges, mostly vertices of 65 and 66
    in-edges; `hot_share` of the edges leave 50 vertices."""
    nv = 70000
    rng = np.random.default_rng(seed)
    deg = rng.choice([65, 66, 67, 70], nv)
    some = rng.choice(nv, 20000, False)
    deg[some] = rng.choice(DEGREES[:17], some.size)
    deg[some[:400]] = rng.choice(DEGREES, 400)
    assert (deg > 64).sum() // 4 + ((deg > 8) & (deg <= 64)).sum() // 32 > 2 * 152 * 28 + 2000
    d = np.repeat(np.arange(nv, dtype=np.int32), deg)
    s = rng.integers(0, nv, d.size, dtype=np.int32)
    hot = rng.random(d.size) < hot_share
    s[hot] = rng.integers(0, 50, int(hot.sum()), dtype=np.int32)
    p = rng.permutation(d.size)
    return nv, s[p], d[p]


@pytest.mark.parametrize("hot", [0.0, 0.5])
@pytest.mark.parametrize("which", [1, 2])
def test_undeclared_programs_on_a_large_graph(driver, tmp_path, which, hot):
    nv, s, d = narrow_graph(hot, which)
    a, b = both(driver, tmp_path, nv, s, d, which, 2)
    assert a[0] > 2 and np.array_equal(a, b)


@pytest.mark.parametrize("which", [1, 2])
@pytest.mark.parametrize("nv", [1, 33, 700, 3000])
def test_undeclared_programs_on_a_small_graph(driver, tmp_path, nv, which):
    rng = np.random.default_rng(nv + which)
    deg = rng.choice(DEGREES, nv) if nv > 1 else np.array([5])
    d = np.repeat(np.arange(nv, dtype=np.int32), deg)
    s = rng.integers(0, nv, d.size, dtype=np.int32)
    s[rng.random(d.size) < 0.3] = nv // 2
    p = rng.permutation(d.size)
    a, b = both(driver, tmp_path, nv, s[p], d[p], which, 2)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("hot", [0.0, 0.5])
def test_narrow_form_of_messages(gpu, hot):
    nv, s, d = narrow_graph(hot, 3)
    out = []
    for blocks in (0, 4):  # 4: a launch shape of its own, every round in the main kernel
        vd = P.pagerank_init(nv, s)
        with GASEngine(PROGRAM_PAGERANK) as e:
            e.set_graph(nv, vd, s, d)
            if blocks:
                e.set_launch_config(True, blocks)
            e.set_dense_policy(1 << 20)
            e.set_active(0, nv)
            rounds = e.run(12)
            st = e.round_stats()
            e.get_results()
        out.append((rounds, vd["rank"].view(np.int32).copy(), st))
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
    for k in out[0][2]:
        assert np.array_equal(out[0][2][k], out[1][2][k])
