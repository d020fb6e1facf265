"""The hot sources of the leading dense rounds: the listed ones are exactly
those of out-degree >= minOut, which is how the kernel tells them, and fit the
table, also where degrees pass the 16 bits of the sort's keys."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("hot_cut") / "hot_cut")
    r = subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O1",
                        "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "cpp", "hot_cut.cu"),
                        "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]

    def run(deg, most, least):
        text = f"{len(deg)} {most} {least}\n" + " ".join(map(str, deg))
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split()
        return int(out[0]), [int(v) for v in out[1:]]

    return run


def degrees(case):
    rng = np.random.default_rng(len(case))
    low = rng.integers(0, 300, 2000)
    if case == "above the cap":  # more than the table holds
        low[rng.choice(2000, 600, False)] = rng.integers(66000, 80000, 600)
    elif case == "few above the cap":
        low[rng.choice(2000, 100, False)] = rng.integers(65000, 80000, 100)
    elif case == "one class too many":
        low[:600] = 70
    elif case == "at the cap":
        low[:512] = 65535
    elif case == "next to the cap":
        low[:300], low[300:700] = 65535, 65534
    elif case == "few vertices":
        low = low[:40]
    return low


@pytest.mark.parametrize("least", [1, 64])
@pytest.mark.parametrize("case", ["ordinary", "above the cap", "few above the cap", "one class too many",
                                  "at the cap", "next to the cap", "few vertices"])
def test_listed_are_those_of_min_degree(cut, case, least):
    deg = degrees(case)
    for most in (127, 511, 512, 2047):
        min_out, listed = cut(deg, most, least)
        assert len(listed) <= most and min_out >= least
        assert sorted(listed) == np.flatnonzero(deg >= min_out).tolist()
        if case == "few above the cap" and most >= 511:
            assert len(listed) >= 100
