"""The leading dense rounds' kernel for Programs that declare nothing: their
results equal, bit for bit, those of the same rounds run by the main kernel's
pull pass.  256-byte vertex data with more sources of 65,535 and more
out-edges than its table of hot sources holds."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

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


@pytest.mark.parametrize("hubs,low,high", [(600, 66000, 80000), (200, 60000, 70000), (600, 300, 900)])
def test_large_vertex_data_hot_sources(driver, tmp_path, hubs, low, high):
    nv = 40000
    rng = np.random.default_rng(hubs + low)
    s = np.repeat(rng.choice(nv, hubs, False), rng.integers(low, high, hubs)).astype(np.int32)
    s = np.concatenate([s, rng.integers(0, nv, 200000, dtype=np.int32)])
    d = rng.integers(0, nv, s.size, dtype=np.int32)
    a, b = both(driver, tmp_path, nv, s, d, 0, 64)
    assert a[0] > 2 and np.array_equal(a, b)
