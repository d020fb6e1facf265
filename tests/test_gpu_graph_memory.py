"""set_graph near the end of device memory: a graph that fits on its own is
taken, whatever an engine keeps from its last graph, whether or not the layout
of the leading dense rounds would fit beside it, and with no more than its own
arrays or its adjacency and the build's working memory."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from vertexapi2_gb300 import GASEngine
from vertexapi2_gb300 import programs as P
from vertexapi2_gb300._lib import PROGRAM_BFS, PROGRAM_CC, load

pytestmark = pytest.mark.gpu

MB = 1 << 20
SLACK = 16 * MB  # the device allocates in blocks of 2 MB
LEFT = 4096 * MB


class Memory:
    """Leaves a chosen number of free bytes."""

    def __init__(self, torch):
        self.torch = torch
        torch.zeros(1, device="cuda")
        torch.cuda.synchronize()
        self.fine = None
        self.coarse = self.block(self.free() - LEFT)

    def free(self):
        return self.torch.cuda.mem_get_info(0)[0]

    def block(self, n):
        return self.torch.empty(max(n, 1) // (2 * MB) * 2 * MB, dtype=self.torch.uint8, device="cuda")

    def leave(self, n):
        self.release()
        self.fine = self.block(self.free() - n)
        assert abs(self.free() - n) <= 4 * MB

    def release(self):
        self.fine = None
        self.torch.cuda.empty_cache()


@pytest.fixture
def memory(gpu):
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info(0)[0] < LEFT + 64 * MB:
        pytest.skip("device memory in use")
    m = Memory(torch)
    yield m
    m.coarse = None
    m.release()


def i32(a):
    return a.ctypes.data_as(C.POINTER(C.c_int32))


def bare_set_graph(nv, s, d, vertex_bytes=4, entry=0, flags=0):
    """Status of set_graph on an engine of source values of `entry` bytes (0:
    it keeps no layout), and the bytes it holds then."""
    import torch
    lib, core = load(), C.c_void_p()
    assert lib.gas_core_create(0, None, C.byref(core)) == 0
    assert lib.gas_core_set_pull_entry(core, entry, flags) == 0
    free = torch.cuda.mem_get_info(0)[0]
    st = lib.gas_core_set_graph(core, nv, s.size, i32(s), i32(d), None, 0, vertex_bytes, 4)
    held = free - torch.cuda.mem_get_info(0)[0]
    lib.gas_core_destroy(core)
    return st, held


def least_free(memory, nv, s, d):
    """Free bytes (to 2 MB) in which the graph fits without the layout."""
    lo, hi = 0, LEFT // (2 * MB)
    while lo + 1 < hi:
        mid = (lo + hi) // 2
        memory.leave(mid * 2 * MB)
        if bare_set_graph(nv, s, d)[0] == 0:
            hi = mid
        else:
            lo = mid
    memory.release()
    return hi * 2 * MB


def random_graph(nv, ne, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(0, nv, ne, dtype=np.int32), rng.integers(0, nv, ne, dtype=np.int32)


def ring(nv):
    """Degrees of 2: a graph of the fused rounds."""
    v = np.arange(nv, dtype=np.int32)
    n = np.roll(v, -1)
    return np.concatenate([v, n]), np.concatenate([n, v])


def labels(e, nv, s, d):
    vd = P.cc_init(nv)
    e.set_graph(nv, vd, s, d)
    e.set_active(0, nv)
    e.run(4)
    e.get_results()
    return vd


@pytest.mark.parametrize("kind", ["random", "ring"])
@pytest.mark.parametrize("before", ["new engine", "other graph before"])
def test_a_graph_that_fits_is_taken(memory, kind, before):
    nv, (s, d) = (1 << 20, random_graph(1 << 20, 1 << 24, 1)) if kind == "random" else (3 << 19, ring(3 << 19))
    other = random_graph(1 << 19, 3 << 21, 2)
    with GASEngine(PROGRAM_CC) as e:
        ref = labels(e, nv, s, d)
    least = least_free(memory, nv, s, d)
    with GASEngine(PROGRAM_CC) as e:
        held = memory.free()
        if before != "new engine":
            labels(e, 1 << 19, *other)
        held -= memory.free()
        memory.leave(least + SLACK - held)
        assert np.array_equal(labels(e, nv, s, d), ref)
        assert np.array_equal(labels(e, nv, s, d), ref)
        memory.release()
        assert np.array_equal(labels(e, nv, s, d), ref)


def test_state_may_take_the_build_memory(memory):
    nv = 1 << 20
    s, d = random_graph(nv, 1 << 24, 3)
    st, held = bare_set_graph(nv, s, d, 256)
    assert st == 0
    memory.leave(held + SLACK)
    assert bare_set_graph(nv, s, d, 256)[0] == 0


@pytest.mark.parametrize("kind", ["random", "ring"])
def test_a_second_engine_still_fits(memory, kind):
    nv, (s, d) = (1 << 20, random_graph(1 << 20, 1 << 24, 5)) if kind == "random" else (3 << 19, ring(3 << 19))
    own = bare_set_graph(nv, s, d)[1]
    least = least_free(memory, nv, s, d)
    with GASEngine(PROGRAM_CC) as a, GASEngine(PROGRAM_CC) as b:
        ref = labels(a, nv, s, d)
        before = memory.free()
        a.set_graph(0, None, s[:0], d[:0])
        held = memory.free() - before
        assert held > own + 16 * MB  # with its layout, where there is room
        memory.leave(own + least + SLACK)  # two graphs, the second one's build
        assert np.array_equal(labels(a, nv, s, d), ref)
        assert np.array_equal(labels(b, nv, s, d), ref)
        assert np.array_equal(labels(a, nv, s, d), ref)


def held_by(program, *graphs):
    """Bytes an engine holds after setting the graphs in turn."""
    import torch
    with GASEngine(program) as e:
        free = torch.cuda.mem_get_info(0)[0]
        for nv, s, d in graphs:
            e.set_graph(nv, None, s, d)
        return free - torch.cuda.mem_get_info(0)[0]


def test_no_layout_without_a_gather(gpu):
    pytest.importorskip("torch")
    nv = 1 << 20
    s, d = random_graph(nv, 1 << 24, 4)
    bare = bare_set_graph(nv, s, d)[1]
    assert held_by(PROGRAM_BFS, (nv, s, d)) <= bare + 8 * MB
    assert held_by(PROGRAM_CC, (nv, s, d)) > bare + 64 * MB


@pytest.mark.parametrize("kind", ["random", "ring"])
def test_smaller_graph_gives_memory_back(gpu, kind):
    pytest.importorskip("torch")
    if kind == "random":
        big, small = [(nv, *random_graph(nv, 16 * nv, nv)) for nv in (1 << 20, 1 << 19)]
    else:
        big, small = [(nv, *ring(nv)) for nv in (4 << 20, 2 << 20)]
    own = held_by(PROGRAM_CC, small)
    assert held_by(PROGRAM_CC, big, small) <= own * 4 // 3 + 12 * MB
    assert held_by(PROGRAM_CC, small, big) <= held_by(PROGRAM_CC, big) + 12 * MB


def test_layout_only_where_it_pays(gpu):
    """Programs that declare nothing keep no layout on large graphs, where the
    kernel that reads the CSC is the faster one."""
    pytest.importorskip("torch")
    nv = 1 << 20
    s, d = random_graph(nv, 1 << 24, 6)
    bare = bare_set_graph(nv, s, d, 8)[1]
    assert bare_set_graph(nv, s, d, 8, 8, 0)[1] <= bare + 8 * MB
    for declared in (2, 4):  # any order, messages
        assert bare_set_graph(nv, s, d, 8, 8, declared)[1] > bare + 64 * MB
    nv = 100000  # 3,125 slices
    s, d = ring(nv)
    bare = bare_set_graph(nv, s, d)[1]
    assert bare_set_graph(nv, s, d, 4, 4, 0)[1] > bare
    assert bare_set_graph(nv, s, d, 4, 64, 0)[1] <= bare  # too large a value for a lane
