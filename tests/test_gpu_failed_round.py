"""getResults after a failed round: the error, and the caller's vertex data as it
was."""
from __future__ import annotations

import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

STATE = 5  # GAS_ERR_STATE


def test_download_leaves_the_array_on_error(gpu, tmp_path):
    exe, lib = str(tmp_path / "failed_round"), os.path.join(ROOT, "vertexapi2_gb300", "_build")
    r = subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2",
                        "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "failed_round.cu"),
                        "-L", lib, "-lgas_gb300", "-Xlinker", f"-rpath={lib}", "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.stdout, r.stderr[-500:])
    first, touched, second, wrong, run, after = map(int, r.stdout.split())
    assert (first, touched) == (STATE, 0)
    assert (second, wrong) == (0, 0)
    assert (run, after) == (STATE, 0)
