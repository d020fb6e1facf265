"""What the engine's users run, as timed cases: a graph resident on the device
(or a host edge list, where the build is the work) and one call sequence
through the public API.

Graphs are drawn on the GPU from the seed alone: R-MAT with the parameters of
the repository's benchmark (edge factor 16 by default, 0.57 / 0.19 / 0.19 /
0.05, self-loops and duplicates removed), cut to any number of vertices, and
4-neighbour lattices with 15 % of the edges deleted, queried from crossings of
their largest component.  Initial vertex data and results live in page-locked
host memory, as a program that runs traversal after traversal on one graph
keeps them.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from vertexapi2_gb300 import (GASEngine, GASServer, PROGRAM_BFS, PROGRAM_CC, PROGRAM_PAGERANK,
                              PROGRAM_PPR, PROGRAM_SSSP, load)
from vertexapi2_gb300._lib import check

PROGRAMS = {"bfs": PROGRAM_BFS, "sssp": PROGRAM_SSSP, "cc": PROGRAM_CC,
            "pagerank": PROGRAM_PAGERANK, "ppr": PROGRAM_PPR}
UNREACHED = 2**31 - 1 - 100000  # the SSSP program's distance of an unreached vertex
PPR_ROUNDS = 20
PR_DTYPE = np.dtype([("rank", np.float32), ("numOutEdges", np.int32)])


def listed():
    return [
        # the headline workload: shortest paths over a road-like network of
        # a million crossings, thousands of small rounds
        {"name": "sssp_lattice_1024", "kind": "run", "program": "sssp", "graph": "lattice",
         "rows": 1024, "cols": 1024, "w_lo": 1, "w_hi": 100},
        # a neighbourhood of a road network, driven round by round as the
        # reference's own drivers do: call and launch latency alone
        {"name": "sssp_lattice_small_steps", "kind": "steps", "program": "sssp", "graph": "lattice",
         "rows": 61, "cols": 47, "w_lo": 1, "w_hi": 100},
        # one traversal of a small social graph: six rounds of latency
        {"name": "bfs_rmat_small", "kind": "run", "program": "bfs", "graph": "rmat",
         "vertices": 9001, "edge_factor": 16, "symmetric": True},
        # the same on a large one, where most rounds are bound by memory
        {"name": "bfs_rmat_large", "kind": "run", "program": "bfs", "graph": "rmat",
         "vertices": 2097152, "edge_factor": 16, "symmetric": True},
        # weighted shortest paths on a power-law graph: list rounds with hubs
        {"name": "sssp_rmat", "kind": "run", "program": "sssp", "graph": "rmat",
         "vertices": 262144, "edge_factor": 16, "symmetric": True, "w_lo": 1, "w_hi": 255},
        # component labelling of the largest graph the benchmark names
        {"name": "cc_rmat_large", "kind": "run", "program": "cc", "graph": "rmat",
         "vertices": 4194304, "edge_factor": 16, "symmetric": True},
        # page ranking of a web-like directed graph, up to 50 rounds
        {"name": "pagerank_rmat_large", "kind": "run", "program": "pagerank", "graph": "rmat",
         "vertices": 4000003, "edge_factor": 16, "symmetric": False, "rounds": 50},
        # a distance table: many sources at once over a road network
        {"name": "batch_sssp_lattice", "kind": "batch", "program": "sssp", "graph": "lattice",
         "rows": 512, "cols": 500, "w_lo": 1, "w_hi": 100, "queries": 64, "delta": 512},
        # hop counts from 256 members of a social graph, one full batch
        {"name": "batch_bfs_rmat", "kind": "batch", "program": "bfs", "graph": "rmat",
         "vertices": 262144, "edge_factor": 16, "symmetric": True, "queries": 256, "delta": 0},
        # recommendations for 100 users: personalised ranks, 20 rounds
        {"name": "batch_ppr_rmat", "kind": "batch", "program": "ppr", "graph": "rmat",
         "vertices": 524288, "edge_factor": 16, "symmetric": True, "queries": 100, "delta": 0},
        # a graph used once: build from the host edge list, run, fetch
        {"name": "build_sssp_rmat", "kind": "build", "program": "sssp", "graph": "rmat",
         "vertices": 1048576, "edge_factor": 16, "symmetric": True, "w_lo": 1, "w_hi": 255},
        # a burst of mixed queries at a server with five resident graphs
        {"name": "serve_mix", "kind": "serve", "graph": "mix", "scales": "12,14,16,18",
         "side": 256, "queries": 192},
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "steps", "batch", "batch", "build", "serve"])
    if kind == "serve":
        scales = sorted(rng.sample(range(12, 19), rng.randint(2, 4)))
        return {"kind": "serve", "graph": "mix", "scales": ",".join(map(str, scales)),
                "side": _between(rng, 48, 256), "queries": _between(rng, 24, 192)}
    lattice = rng.random() < 0.35
    program = rng.choice({"batch": ["bfs", "sssp", "ppr"], "build": ["bfs", "sssp", "cc"],
                          "steps": ["bfs", "sssp", "cc"]}.get(kind, ["bfs", "sssp", "cc", "pagerank"]))
    case = {"kind": kind, "program": program}
    if lattice and program in ("bfs", "sssp", "cc"):
        most = {"run": 1024, "build": 1024, "batch": 512, "steps": 128}[kind]
        case.update(graph="lattice", rows=_between(rng, 40, most), cols=_between(rng, 40, most),
                    w_lo=1, w_hi=100)
    else:
        most = {"run": 2097152, "build": 1048576, "batch": 262144, "steps": 262144}[kind]
        case.update(graph="rmat", vertices=_between(rng, 4096, most), edge_factor=rng.choice([8, 12, 16]),
                    symmetric=program != "pagerank")
        if program == "sssp":
            case.update(w_lo=1, w_hi=rng.choice([100, 255]))
    if program == "pagerank":
        case["rounds"] = rng.choice([20, 50])
    if kind == "batch":
        most = 64 if case["graph"] == "lattice" else 100 if program == "ppr" else 256
        case["queries"] = _between(rng, 4, most)
        case["delta"] = 512 if case["graph"] == "lattice" and program == "sssp" else 0
    return case


# ------------------------------------------------------------------ graphs

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _weights(s, d, n, seed, lo, hi):
    """Whole numbers in [lo, hi], the same for both directions of an edge."""
    key = torch.minimum(s, d) * n + torch.maximum(s, d) + seed * 1000003
    key = (key * 0x2545F4914F6CDD1D) ^ (key >> 29)
    key = (key * 0x5851F42D4C957F2D) ^ (key >> 32)
    return (lo + ((key >> 17) & 0x7FFFFFFF) % (hi - lo + 1)).to(torch.int32)


def _rmat(vertices, edge_factor, symmetric, seed):
    """(n, srcs, dsts) as int64 device tensors, sorted by (src, dst)."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    scale = max(1, (vertices - 1).bit_length())
    m = edge_factor * vertices
    s = torch.zeros(m, dtype=torch.int64, device=dev)
    d = torch.zeros(m, dtype=torch.int64, device=dev)
    for _ in range(scale):
        r = torch.rand(m, generator=gen, device=dev)
        s = s * 2 + (r >= 0.76)
        d = d * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    keep = (s != d) & (s < vertices) & (d < vertices)
    s, d = s[keep], d[keep]
    key = s * vertices + d
    if symmetric:
        key = torch.cat([key, d * vertices + s])
    key = torch.unique(key)
    return vertices, key // vertices, key % vertices


def _lattice(rows, cols, seed):
    """A 4-neighbour lattice without 15 % of its edges."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    n = rows * cols
    ids = torch.arange(n, device=dev).reshape(rows, cols)
    u = torch.cat([ids[:, :-1].reshape(-1), ids[:-1].reshape(-1)])
    v = torch.cat([ids[:, 1:].reshape(-1), ids[1:].reshape(-1)])
    keep = torch.rand(u.numel(), generator=gen, device=dev) >= 0.15
    u, v = u[keep], v[keep]
    key, _ = torch.sort(torch.cat([u * n + v, v * n + u]))
    return n, key // n, key % n


def _live(graph, n, s, d):
    """The vertices a query may start at: those with out-edges of an R-MAT
    graph, the largest component of a lattice."""
    if graph != "lattice":
        return torch.unique(s).cpu().numpy()
    label = torch.arange(n, device=s.device)
    while True:  # hook to the smaller label, then halve the paths
        new = label.scatter_reduce(0, label[d], label[s], "amin")
        new = new[new]
        if torch.equal(new, label):
            break
        label = new
    return torch.nonzero(label == torch.bincount(label, minlength=n).argmax()).reshape(-1).cpu().numpy()


def _graph(case, seed):
    if case["graph"] == "lattice":
        n, s, d = _lattice(case["rows"], case["cols"], seed)
    else:
        n, s, d = _rmat(case["vertices"], case["edge_factor"], case["symmetric"], seed)
    w = _weights(s, d, n, seed, case["w_lo"], case["w_hi"]) if "w_lo" in case else None
    return n, s, d, w


def _host(t):
    return None if t is None else t.to(torch.int32).cpu().numpy()


def _pinned(shape, dtype):
    count = int(np.prod(shape)) * np.dtype(dtype).itemsize
    return torch.empty(count, dtype=torch.uint8, pin_memory=torch.cuda.is_available()).numpy() \
        .view(dtype).reshape(shape)


def _initial(program, n, s, source):
    """The state the reference's drivers start from, page-locked."""
    if program == "pagerank":
        vd = _pinned(n, PR_DTYPE)
        vd["rank"] = np.float32(0.15)
        vd["numOutEdges"] = torch.bincount(s, minlength=n).to(torch.int32).cpu().numpy()
        return vd
    vd = _pinned(n, np.int32)
    if program == "cc":
        vd[:] = np.arange(n, dtype=np.int32)
    else:
        vd[:] = -1 if program == "bfs" else UNREACHED
        if program == "sssp":
            vd[source] = 0
    return vd


def _sources(graph, n, s, d, seed, count):
    """Any vertex of _live as likely as another."""
    return np.random.default_rng(seed).choice(_live(graph, n, s, d), count).astype(np.int32)


# ---------------------------------------------------------------- the calls

class _Batch:
    """A batch handle of the C ABI with the result buffer its program keeps."""

    def __init__(self, n, s, d, w, delta):
        self.lib = load()
        self.h = C.c_void_p()
        check(self.lib.gas_batch_create(0, C.c_void_p(0), C.byref(self.h)), "gas_batch_create")
        self.n = n
        ptr = lambda a: None if a is None else a.ctypes.data_as(C.POINTER(C.c_int32))
        check(self.lib.gas_batch_set_graph(self.h, n, len(s), ptr(s), ptr(d), ptr(w)),
              "gas_batch_set_graph")
        check(self.lib.gas_batch_set_delta(self.h, delta), "gas_batch_set_delta")

    def run(self, program, sources, out):
        i32 = C.POINTER(C.c_int32)
        check(self.lib.gas_batch_run(self.h, program, len(sources), sources.ctypes.data_as(i32),
                                     out.ctypes.data_as(i32), None), "gas_batch_run")

    def __del__(self):
        if self.h:
            self.lib.gas_batch_destroy(self.h)
            self.h = None


def _mix(case, seed):
    """The server's graphs and its queries: (graph, program, source)."""
    gs = [_rmat(1 << int(x), 16, True, seed + k) for k, x in enumerate(case["scales"].split(","))]
    ws = [_weights(s, d, n, seed, 1, 255) for n, s, d in gs]
    gs.append(_lattice(case["side"], case["side"], seed))
    ws.append(_weights(gs[-1][1], gs[-1][2], gs[-1][0], seed, 1, 100))
    pool = [_sources("lattice" if k == len(gs) - 1 else "rmat", n, s, d, seed + 7 + k, case["queries"])
            for k, (n, s, d) in enumerate(gs)]
    rng = np.random.default_rng(case["queries"])
    queries = []
    for k in range(case["queries"]):  # half traversals, 3 in 10 distances, 2 in 10 ranks
        g = int(rng.integers(len(gs)))
        p = rng.choice(["bfs", "sssp", "ppr"], p=[0.5, 0.3, 0.2])
        queries.append((g, str(p), int(pool[g][k])))
    return gs, ws, queries


def prepare(case, seed):
    if case["kind"] == "serve":
        gs, ws, queries = _mix(case, seed)
        server = GASServer()
        ids = [server.add_graph(n, _host(s), _host(d), _host(w)) for (n, s, d), w in zip(gs, ws)]
        out, rows, at = {}, [], {}
        for g, p, _ in queries:
            at[g, p] = at.get((g, p), 0) + 1
        for (g, p), count in at.items():
            out["%s_%d" % (p, g)] = _pinned((count, gs[g][0]), np.float32 if p == "ppr" else np.int32)
        used = {}
        for g, p, _ in queries:
            rows.append(out["%s_%d" % (p, g)][used.get((g, p), 0)])
            used[g, p] = used.get((g, p), 0) + 1
        plan = [(ids[g], PROGRAMS[p], x) for g, p, x in queries]
        return {"kind": "serve", "server": server, "plan": plan, "rows": rows, "out": out}
    n, s, d, w = _graph(case, seed)
    hs, hd, hw = _host(s), _host(d), _host(w)
    program = case["program"]
    state = {"kind": case["kind"], "program": program, "n": n}
    if case["kind"] == "batch":
        state["sources"] = _sources(case["graph"], n, s, d, seed, case["queries"])
        state["batch"] = _Batch(n, hs, hd, hw, case["delta"])
        state["out"] = _pinned((case["queries"], n), np.float32 if program == "ppr" else np.int32)
        return state
    # traversals start at a vertex of the largest component: the one of
    # highest degree on a power-law graph, any of a lattice
    source = int(_sources("lattice", n, s, d, seed, 1)[0]) if case["graph"] == "lattice" \
        else int(torch.bincount(s, minlength=n).argmax())
    state["init"] = _initial(program, n, s, source)
    state["vd"] = _pinned(n, state["init"].dtype)
    state["range"] = (source, source + 1) if program == "bfs" else (0, n)
    state["rounds"] = case.get("rounds", 0)
    state["engine"] = GASEngine(PROGRAMS[program])
    if case["kind"] == "build":
        state["edges"] = (hs, hd, hw)
    else:
        state["vd"][:] = state["init"]
        state["engine"].set_graph(n, state["vd"], hs, hd, hw)
    return state


def run(state):
    kind = state["kind"]
    if kind == "serve":
        server = state["server"]
        tickets = [server.submit(g, p, x) for g, p, x in state["plan"]]
        for t, row in zip(tickets, state["rows"]):
            server.wait(t, out=row)
        return state["out"]
    if kind == "batch":
        state["batch"].run(PROGRAMS[state["program"]], state["sources"], state["out"])
        return state["out"]
    e = state["engine"]
    if kind == "build":
        state["vd"][:] = state["init"]
        hs, hd, hw = state["edges"]
        e.set_graph(state["n"], state["vd"], hs, hd, hw)
    else:
        e.set_vertex_data(state["init"])
    e.set_active(*state["range"])
    if kind == "steps":
        rounds = 0
        gather = state["program"] != "bfs"
        e.set_iteration(0)
        while e.count_active():
            e.gather_apply(gather)
            e.scatter_activate(gather)
            e.next_iter()
            rounds += 1
            e.set_iteration(rounds)
    else:
        rounds = e.run(state["rounds"])
    e.get_results()
    vd = state["vd"]
    return {"rounds": rounds, "values": vd["rank"] if vd.dtype == PR_DTYPE else vd}


# ------------------------------------------------------- what a pass needs

def _edges_of(case):
    """Edges after duplicates and self-loops are gone (measured on seed 1 to
    a few per cent; the count differs a little with the seed)."""
    if case["graph"] == "lattice":
        return int(0.85 * 2 * (2 * case["rows"] * case["cols"] - case["rows"] - case["cols"]))
    return int(case["vertices"] * case["edge_factor"] * 0.9 * (2 if case["symmetric"] else 1))


def work(case):
    if case["kind"] == "serve":
        parts = [(1 << int(x), int((1 << int(x)) * 16 * 1.7)) for x in case["scales"].split(",")]
        parts.append((case["side"] ** 2, int(3.4 * case["side"] ** 2)))
        mean_v = sum(v for v, _ in parts) / len(parts)
        mean_e = sum(e for _, e in parts) / len(parts)
        graph = sum(8 * v + 12 * e for v, e in parts)
        return {"bytes": graph + 4 * case["queries"] * mean_v,
                "flops": case["queries"] * mean_e * (0.8 + 0.2 * 2 * PPR_ROUNDS)}
    e = _edges_of(case)
    v = case["vertices"] if case["graph"] == "rmat" else case["rows"] * case["cols"]
    q = case.get("queries", 1)
    rounds = {"pagerank": case.get("rounds", 50), "ppr": PPR_ROUNDS}.get(case["program"], 1)
    vd = 8 if case["program"] == "pagerank" else 4
    weight = 4 if "w_lo" in case and case["program"] == "sssp" else 0
    # the adjacency (and weights) once, the initial state in, the results out
    moved = 4 * (v + 1) + e * (4 + weight) + v * vd * (1 + q)
    if case["kind"] == "build":
        moved += e * (8 + weight)  # the edge list it is made from
    return {"bytes": moved, "flops": 2 * e * q * rounds}


# ------------------------------------------------------------ in 64 bits

def _by_dst(n, s, d):
    """In-edges as a CSR matrix of ones, 64 bits."""
    order = torch.argsort(d, stable=True)
    at = torch.zeros(n + 1, dtype=torch.int64, device=s.device)
    at[1:] = torch.cumsum(torch.bincount(d, minlength=n), 0)
    return torch.sparse_csr_tensor(at, s[order], torch.ones(s.numel(), dtype=torch.float64, device=s.device),
                                   size=(n, n))


def _pagerank64(n, s, d, rounds):
    a = _by_dst(n, s, d)
    base, tol = float(np.float32(0.15)), float(np.float32(0.01))
    damp = float(np.float32(1.0) - np.float32(0.15))
    deg = torch.bincount(s, minlength=n).to(torch.float64).clamp(min=1)
    rank = torch.full((n,), base, dtype=torch.float64, device=s.device)
    active = torch.ones(n, dtype=torch.bool, device=s.device)
    for _ in range(rounds):
        if not bool(active.any()):
            break
        new = base + damp * torch.mv(a, rank / deg)
        moved = active & ((new - rank).abs() >= tol)
        rank = torch.where(active, new, rank)
        active = torch.mv(a, moved.to(torch.float64)) > 0
    return rank


def _ppr64(n, s, d, sources):
    a = _by_dst(n, s, d)
    alpha = np.float32(0.15)
    damp = float(np.float32(1.0) - alpha)
    deg = torch.bincount(s, minlength=n).to(torch.float64).clamp(min=1).unsqueeze(1)
    src = torch.as_tensor(np.asarray(sources, dtype=np.int64), device=s.device)
    parts = []
    for x in src.split(32):
        q = torch.arange(x.numel(), device=s.device)
        rank = torch.zeros(n, x.numel(), dtype=torch.float64, device=s.device)
        rank[x, q] = 1.0
        tele = torch.zeros_like(rank)
        tele[x, q] = float(alpha)
        for _ in range(PPR_ROUNDS):
            rank = tele + damp * (a @ (rank / deg))
        parts.append(rank.t().contiguous())
    return torch.cat(parts)


def exact(case, seed):
    """Ranks in 64 bits; depths, distances and labels are whole numbers."""
    if case["kind"] == "serve":
        gs, _, queries = _mix(case, seed)
        out = {"%s_%d" % (p, g): None for g, p, _ in queries}
        for key in out:
            p, g = key.split("_")
            if p == "ppr":
                n, s, d = gs[int(g)]
                out[key] = _ppr64(n, s, d, [x for h, q, x in queries if q == p and h == int(g)])
        return out
    if case["program"] == "pagerank":
        n, s, d, _ = _graph(case, seed)
        return {"rounds": None, "values": _pagerank64(n, s, d, case["rounds"])}
    if case["program"] == "ppr":
        n, s, d, _ = _graph(case, seed)
        return _ppr64(n, s, d, _sources(case["graph"], n, s, d, seed, case["queries"]))
    return None
