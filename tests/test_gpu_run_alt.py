"""A run kernel compiled into a user's binary may leave the vertex data in the
alternate buffer (gas_run_args::vcurOut): the library brings it back."""
from __future__ import annotations

import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_result_in_the_alternate_buffer(gpu, tmp_path):
    exe, lib = str(tmp_path / "run_alt"), os.path.join(ROOT, "vertexapi2_gb300", "_build")
    r = subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2",
                        "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "run_alt.cu"),
                        "-L", lib, "-lgas_gb300", "-Xlinker", f"-rpath={lib}", "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.stdout, r.stderr[-500:])
