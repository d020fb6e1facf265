"""gas_run_args is read by kernels in the user's binary: the fields that such a
binary may have been compiled with keep their places."""
from __future__ import annotations

import os
import subprocess

from conftest import ROOT

# offsets in bytes on a 64-bit target
PLACES = {
    "g": 0, "outDests": 272, "vertexBytes": 280, "maxGatherTiles": 284, "frontL": 288,
    "scatL": 384, "mark": 480, "stats": 488, "maxStatRounds": 496, "cur": 500, "sidx": 504,
    "maxRounds": 508, "epochBase": 512, "stampBase": 516, "barrier": 520, "roundsOut": 528,
    "vertexAlt": 536, "retBits": 544, "bitWords": 568, "frontBits": 576, "denseCnt": 600,
    "denseAlpha": 608, "allActive": 612, "vcurOut": 616, "binMid": 624, "binSmall": 632,
    "binTiny": 640, "nMid": 648, "nSmall": 652, "nTiny": 656, "chunkVertex": 664,
    "chunkBegin": 672, "chunkFirst": 680, "chunkCount": 688, "chunkSlot": 696, "nChunks": 704,
    "nChunkVertices": 708, "chunkArrive": 712, "chunkVal": 720, "chunkFlags": 728,
    "edgeScatter": 736, "csr2csc": 744, "fused": 752, "ellIn": 760, "ellOut": 768, "ellEd": 776,
    "ellWidth": 784, "fusedCells": 792, "denseFirst": 800, "resume": 808, "denseEndOut": 816,
}


def test_fields_keep_their_places(tmp_path):
    src, exe = tmp_path / "places.c", tmp_path / "places"
    src.write_text('#include <stddef.h>\n#include <stdio.h>\n#include "gas_gb300_core.h"\nint main(void) {\n'
                   + "".join(f'  printf("{n} %zu\\n", offsetof(gas_run_args, {n}));\n' for n in PLACES)
                   + "  return 0;\n}\n")
    r = subprocess.run(["gcc", "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    got = {n: int(o) for n, o in (line.split() for line in out.splitlines())}
    assert got == PLACES
