"""Timed cases: one call of the engine on a graph that is resident on the GPU.

A case names an algorithm ("alg"), a seeded synthetic graph and the call's
options.  Graphs: "rmat" (2^scale vertices, edge_factor * 2^scale draws, the
benchmark's a/b/c), "grid" (rows x cols, 4 neighbours, the road-like shape)
and "chunglu" (power law; vertices and draws of any size).  The call writes its result to
a buffer on the GPU that the caller owns; a run's result is complete when the
call returns.
"""
import random

import torch

import cggraph_b200 as cg

BFS, SSSP, CC, PR = (int(cg.Algorithm_type.BFS), int(cg.Algorithm_type.SSSP), int(cg.Algorithm_type.CC),
                     int(cg.Algorithm_type.PR))
FLAG_CC_WEAK = 0x8  # CGB_FLAG_CC_WEAK


def _rmat(name, alg, scale, **more):
    return {"name": name, "alg": alg, "graph": "rmat", "scale": scale, "edge_factor": 16, "wmax": 64, **more}


def listed():
    return [
        # a small graph: the call's latency and its launches
        _rmat("bfs_rmat12", "bfs", 12),
        # the benchmark's graph: 16.8 M vertices, 263 M directed edges
        _rmat("bfs_rmat24", "bfs", 24),
        # a road-like graph: thousands of levels with frontiers of about a thousand vertices
        {"name": "bfs_grid1200x1250", "alg": "bfs", "graph": "grid", "rows": 1200, "cols": 1250, "wmax": 1000},
        # weighted distances: an ordinary graph, the benchmark's, and a road-like one
        _rmat("sssp_rmat18", "sssp", 18),
        _rmat("sssp_rmat24", "sssp", 24),
        {"name": "sssp_grid700x901", "alg": "sssp", "graph": "grid", "rows": 700, "cols": 901, "wmax": 1000},
        # weak components of the benchmark's directed graph
        _rmat("cc_weak_rmat24", "cc", 24, weak=True),
        # PageRank in FP64: a small graph, the benchmark's, and a power-law graph whose
        # size is no power of two (a tenth of the benchmark's large skewed shape)
        _rmat("pr_rmat16", "pr", 16, iters=20),
        _rmat("pr_rmat24", "pr", 24, iters=20),
        {"name": "pr_chunglu4m", "alg": "pr", "graph": "chunglu", "vertices": 4_160_000, "draws": 160_000_000,
         "wmax": 64, "iters": 20},
        # many roots in one call
        _rmat("bfs64_rmat22", "bfs", 22, roots=64),
        _rmat("sssp64_rmat20", "sssp", 20, roots=64),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    alg = rng.choice(["bfs", "bfs", "sssp", "sssp", "cc", "pr", "pr", "bfs", "sssp"])
    roots = 0
    if alg in ("bfs", "sssp") and rng.random() < 0.25:
        roots = rng.randint(2, 64)
    # (a grid's components and PageRank are the same for every seed)
    kind = rng.choice(["rmat", "rmat", "grid", "chunglu"] if alg in ("bfs", "sssp") else ["rmat", "rmat", "chunglu"])
    if kind == "grid":
        # long and short sides, no multiples of the warp size; many-root runs on smaller ones
        area = _log_int(rng, 1_000, (60_000 if roots else 1_500_000) if alg == "bfs" else (40_000 if roots else 600_000))
        rows = _log_int(rng, max(2, int(area ** 0.3)), max(3, int(area ** 0.6)))
        case = {"alg": alg, "graph": "grid", "rows": rows, "cols": max(2, area // rows),
                "wmax": rng.choice([1, 64, 1000, 1000])}
    elif kind == "rmat":
        top = 24 if not roots else (21 if alg == "bfs" else 19)
        scale, ef = rng.randint(10, top), rng.choice([4, 8, 16, 16, 32])
        while ef > 4 and (ef << scale) > (16 << top):
            ef //= 2
        case = {"alg": alg, "graph": "rmat", "scale": scale, "edge_factor": ef, "wmax": 64}
    else:
        top = 4_160_000 if not roots else (1_000_000 if alg == "bfs" else 300_000)
        vertices = _log_int(rng, 2_000, top)
        case = {"alg": alg, "graph": "chunglu", "vertices": vertices, "draws": vertices * rng.randint(4, 38),
                "wmax": 64}
    if roots:
        case["roots"] = roots
    if alg == "sssp" and rng.random() < 0.2:
        case["wmax"] = 0  # no weights: unit lengths
    if alg == "cc":
        # weak components of a directed graph, or components of a symmetric one
        if rng.random() < 0.4:
            case["sym"] = True
            if kind == "rmat":
                case["scale"] = min(case["scale"], 23)
            else:
                case["draws"] = max(1, case["draws"] // 2)
        else:
            case["weak"] = True
    if alg == "pr":
        case["iters"] = rng.randint(1, 20)
    return case


def _size(case):
    """(vertices, edges): the edges as drawn, before duplicates are dropped."""
    if case["graph"] == "rmat":
        v = 1 << case["scale"]
        e = case["edge_factor"] * v
    elif case["graph"] == "grid":
        r, c = case["rows"], case["cols"]
        return r * c, 2 * (r * (c - 1) + c * (r - 1))
    else:
        v, e = case["vertices"], case["draws"]
    return v, e * (2 if case.get("sym") else 1)


def _graph(case, seed):
    sym = bool(case.get("sym"))
    if case["graph"] == "rmat":
        return cg.Graph.rmat(case["scale"], case["edge_factor"], seed=seed, symmetrise=sym, wmax=case["wmax"])
    if case["graph"] == "grid":
        return cg.Graph.grid(case["rows"], case["cols"], seed=seed, wmax=case["wmax"])
    v, draws = case["vertices"], case["draws"]
    # the top vertex has about 7 % of the vertices as neighbours, as in the benchmark's shape
    offset = cg.chunglu_weight_offset(v, draws, max(1, int(v * 0.072)))
    return cg.Graph.chunglu(v, draws, offset, seed=seed, symmetrise=sym, wmax=case["wmax"])


class _DeviceWords:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 3}


def _csr(g):
    """The resident CSR's offsets and destinations (views of the engine's memory)."""
    off, dst, _ = g.device_csr()
    return (torch.as_tensor(_DeviceWords(off, g.vertexNum + 1), device="cuda"),
            torch.as_tensor(_DeviceWords(dst, g.edgeNum), device="cuda"))


def _roots(g, n, seed):
    """n seeded roots: each the vertex with the most out-edges of 64 random ones."""
    rng = random.Random(seed * 7919 + 17)
    off = _csr(g)[0].to(torch.int64)
    pick = torch.tensor([[rng.randrange(g.vertexNum) for _ in range(64)] for _ in range(n)], device="cuda")
    deg = off[pick + 1] - off[pick]
    return pick.gather(1, deg.argmax(1, keepdim=True))[:, 0].tolist()


def prepare(case, seed):
    alg = {"bfs": BFS, "sssp": SSSP, "cc": CC, "pr": PR}[case["alg"]]
    g = _graph(case, seed)
    n = case.get("roots", 0)
    s = {"graph": g, "alg": alg, "options": None, "roots": None, "arg": 0}
    if n:
        s["roots"] = _roots(g, n, seed)
        s["out"] = torch.empty((n, g.vertexNum), dtype=torch.int32, device="cuda")
        return s
    s["out"] = torch.empty(g.vertexNum, dtype=torch.float64 if alg == PR else torch.int32, device="cuda")
    if alg in (BFS, SSSP):
        s["arg"] = _roots(g, 1, seed)[0]
    elif alg == PR:
        s["arg"] = case["iters"]
    elif case.get("weak"):
        s["options"] = cg.make_options(flags=FLAG_CC_WEAK)
    return s


def run(s):
    if s["roots"] is not None:
        return s["graph"].run_batch(s["alg"], s["roots"], out=s["out"])[0]
    return s["graph"].run(s["alg"], s["arg"], s["options"], out=s["out"])[0]


def work(case):
    v, e = _size(case)
    if case["alg"] == "pr":
        # each iteration: offsets and sources of the in-edges, the old values, the new values
        return {"bytes": case["iters"] * (4 * e + 20 * v), "flops": case["iters"] * (e + 3 * v)}
    results = 4 * v * case.get("roots", 1)
    edges = (8 if case["alg"] == "sssp" and case["wmax"] else 4) * e
    return {"bytes": 4 * v + edges + results, "flops": 0}


def exact(case, seed):
    if case["alg"] != "pr":
        return None  # whole numbers
    with _graph(case, seed) as g:
        off, dst = _csr(g)
        deg = (off[1:] - off[:-1]).to(torch.int64)
        v = g.vertexNum
        src = torch.repeat_interleave(torch.arange(v, dtype=torch.int32, device="cuda"), deg)
        inv = torch.where(deg > 0, 1.0 / deg.clamp(min=1).to(torch.float64), torch.zeros((), dtype=torch.float64,
                                                                                       device="cuda"))
        pr = torch.full((v,), 1.0 / v, dtype=torch.float64, device="cuda")
        for _ in range(case["iters"]):
            share = pr * inv
            new = torch.zeros_like(pr)
            step = 1 << 26
            for a in range(0, g.edgeNum, step):
                new.index_add_(0, dst[a:a + step], share[src[a:a + step]])
            pr = 0.15 / v + 0.85 * new
        torch.cuda.synchronize()
        return pr
