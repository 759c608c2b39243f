"""What this engine's performance is measured on: calls that a user's program makes, through the package's public API.

A case names an entry point ("call"), a graph family with its size, and the number of sources. Sizes and families are those of
bench.py's workloads and of the tests: Graph500 R-MAT graphs, the road-like Wilson grids, plain grids, Erdos-Renyi meshes and the
batched mix of the three. The state holds what a service keeps between calls: the engine with its graph uploaded, and the buffer that
the rows are written to. The seed draws both the graph's edges and the sources.
"""
import atexit
import math
import os
import shutil
import tempfile

import numpy as np
import torch

import webgpu_bfs_gb300 as m

UNREACHED = 0xFFFFFFFF
_tuned = {}  # the batched form's autotuner cache file of this process


def listed():
    return [
        # one small query on a small graph: launches and per-level latency are all there is
        dict(name="grid64_s64", call="rows", graph="grid", w=64, h=64, S=64),
        # a lone shortest-path query on a city-sized road network (about 1,000 levels)
        dict(name="road339_s1", call="rows", graph="road", w=339, h=338, extra=5000, S=1),
        # the same network's distance matrix from many sources (centrality, isochrones)
        dict(name="road339_s2048", call="rows", graph="road", w=339, h=338, extra=5000, S=2048),
        # a country-sized road network, beyond one block's shared memory; one request of the served mix
        dict(name="road1448_s64", call="rows", graph="road", w=1448, h=1448, extra=41934, S=64),
        # the headline: a social-network-like graph, a full pass of 512 sources, rows in HBM
        dict(name="rmat22_s512", call="rows", graph="rmat", scale=22, ef=16, directed=False, S=512),
        # a served request: per-source eccentricity / reach / distance sums, no matrix
        dict(name="rmat21_s64_stats", call="stats", graph="rmat", scale=21, ef=16, directed=False, S=64),
        # the smallest served request on a large graph: its latency
        dict(name="rmat20_s1_stats", call="stats", graph="rmat", scale=20, ef=16, directed=False, S=1),
        # a mesh without hubs (the bottom-up path), two passes, the second one ragged
        dict(name="er100k_s700", call="rows", graph="er", n=100000, deg=16, S=700),
        # reachability of a directed graph (web links), an odd number of sources, bitmask to the host
        dict(name="reach_rmat18d_s333", call="reach", graph="rmat", scale=18, ef=8, directed=True, S=333),
        # the drop-in call of the original API: a fresh host array of all distances
        dict(name="host_rmat17_s129", call="host", graph="rmat", scale=17, ef=16, directed=False, S=129),
        # many small graphs of uneven size in one launch, every row back on the host
        dict(name="batch60", call="batch", graph="mix", n_er=36, n_grid=18, n_rmat=6, S=0),
        # a resident graph answering a burst of small requests from its queue
        dict(name="served_rmat20", call="served", graph="rmat", scale=20, ef=16, directed=False, S=0, requests=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["road", "road", "grid", "rmat", "rmat", "stats", "er", "reach", "host", "batch", "served"])
    if kind == "road":
        w, h = _log_int(rng, 40, 1448), _log_int(rng, 40, 1448)
        S = min(_log_int(rng, 1, 2048), (1 << 28) // (w * h))
        return dict(call="rows", graph="road", w=w, h=h, extra=1 + int(w * h * rng.uniform(0.005, 0.08)), S=S)
    if kind == "grid":
        return dict(call="rows", graph="grid", w=_log_int(rng, 16, 400), h=_log_int(rng, 16, 400), S=_log_int(rng, 1, 512))
    if kind == "er":
        return dict(call="rows", graph="er", n=_log_int(rng, 1000, 400000), deg=rng.randint(6, 32), S=_log_int(rng, 1, 1024))
    if kind == "batch":
        return dict(call="batch", graph="mix", n_er=rng.randint(4, 36), n_grid=rng.randint(2, 18), n_rmat=rng.randint(1, 6), S=0)
    scale = rng.randint(10, 21)
    case = dict(call="rows" if kind == "rmat" else kind, graph="rmat", scale=scale, ef=rng.choice([8, 16]), directed=rng.random() < 0.3,
                S=_log_int(rng, 1, 1024))
    if kind == "host":
        case["S"] = min(case["S"], max(1, (1 << 26) >> scale))
    if kind == "served":
        case.update(S=0, requests=rng.randint(4, 48), directed=False)
    return case


def _rmat(scale, ef, directed, seed):
    """Graph500 R-MAT (0.57, 0.19, 0.19, 0.05), symmetrised unless directed, no self-loops or duplicates: CSR arrays."""
    gen = torch.Generator("cuda").manual_seed(seed)
    n = ef << scale
    u = torch.zeros(n, dtype=torch.int64, device="cuda")
    v = torch.zeros(n, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(n, generator=gen, device="cuda")
        u = u * 2 + (r >= 0.76)
        v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    if not directed:
        u, v = torch.cat([u, v]), torch.cat([v, u])
    key = torch.unique(((u << 32) | v)[u != v])
    off = torch.zeros((1 << scale) + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.bincount(key >> 32, minlength=1 << scale).cumsum(0)
    off = off.to(torch.int32).cpu().numpy().view(np.uint32)
    idx = (key & 0xFFFFFFFF).to(torch.int32).cpu().numpy().view(np.uint32)
    return m.CsrGraph(1 << scale, off, idx)


def _graph(case, seed):
    if case["graph"] == "rmat":
        return _rmat(case["scale"], case["ef"], case["directed"], seed)
    if case["graph"] == "road":
        return m.wilson_grid(case["w"], case["h"], case["extra"], seed)
    if case["graph"] == "grid":
        return m.generate_grid2d(case["w"], case["h"])
    return m.generate_erdos_renyi_np(case["n"], case["deg"] / (case["n"] - 1), seed)


def _sources(g, count, rng):
    """Distinct vertices with out-edges, in random order (with repeats where the graph has too few)."""
    ok = np.flatnonzero(np.diff(g.row_offsets.astype(np.int64)) > 0)
    return rng.choice(ok, count, replace=count > ok.size).astype(np.uint32)


def _tuning_cache():
    if "path" not in _tuned:
        d = tempfile.mkdtemp(prefix="batch_tuning_")
        atexit.register(shutil.rmtree, d, True)
        _tuned["path"] = os.path.join(d, "cache.txt")
    return _tuned["path"]


def _quantiles(n, shift):
    """n evenly spread values of (0, 1) in a scattered order: the batch's sizes, the same for every seed."""
    return (np.arange(n) * 0.6180339887 + shift) % 1.0


def _batch_items(case, seed):
    """Graphs of the batched workload's distributions, each with its own sources."""
    rng = np.random.default_rng(seed)
    graphs = []
    for i, x in enumerate(_quantiles(case["n_er"], 0.3)):
        n = int(1000 * 65.536 ** x)
        graphs.append(m.generate_erdos_renyi_np(n, 8.0 / (n - 1), seed + i))
    for i, x in enumerate(_quantiles(case["n_grid"], 0.7)):
        k = int(32 + 225 * x)
        graphs.append(m.wilson_grid(k, k, max(1, round(0.02 * (k * k - 1))), seed + 10000 + i))
    for i in range(case["n_rmat"]):
        graphs.append(m.generate_graph500_rmat(16, 8, seed + 20000 + i))
    counts = [int(257.0 ** x) for x in _quantiles(len(graphs), 0.5)]
    return [(g, rng.integers(0, g.num_vertices, S).astype(np.uint32)) for g, S in zip(graphs, counts)]


def prepare(case, seed):
    call = case["call"]
    st = {"call": call}
    if call == "batch":
        st["batch"] = m.BatchedBfs(_batch_items(case, seed))
        st["batch"].autotune(samples_per_class=1, cache_path=_tuning_cache())
        return st
    rng = np.random.default_rng(seed)
    g = st["g"] = _graph(case, seed)
    if call == "served":
        st["server"] = m.BfsServer(g, slots=2, max_sources_per_launch=512)
        st["requests"] = [_sources(g, (1, 8, 64)[i % 3], rng) for i in range(case["requests"])]
        return st
    st["src"] = _sources(g, case["S"], rng)
    st["eng"] = m.GpuBfsEngine(m.GpuBfsMethod.Auto)
    st["eng"].upload(g)
    if call == "rows":
        st["out"] = torch.empty((case["S"], g.num_vertices), dtype=torch.int32, device="cuda")
    return st


def _fields(rows):
    return {k: rows[k].astype(np.int64) for k in ("distance_sum", "eccentricity", "reached")}


def run(st):
    call = st["call"]
    if call == "rows":
        st["eng"].run_ms_bfs_device(st["g"], st["src"], st["out"].data_ptr())
        return st["out"]
    if call == "stats":
        return _fields(st["eng"].run_ms_bfs_stats(st["g"], st["src"]))
    if call == "reach":
        return st["eng"].run_ms_reachability(st["g"], st["src"]).words.view(np.int32)
    if call == "host":
        return st["eng"].run_ms_bfs(st["g"], st["src"]).view(np.int32)
    if call == "batch":
        st["batch"].run()
        return [st["batch"].result(i).view(np.int32) for i in range(len(st["batch"]))]
    tickets = [st["server"].submit(s) for s in st["requests"]]
    return _fields(np.concatenate([st["server"].wait(t)[0] for t in tickets]))


def _size(case):
    """(vertices, stored edges) of the case's graph, about."""
    if case["graph"] == "rmat":
        return 1 << case["scale"], (case["ef"] << case["scale"]) * (0.95 if case["directed"] else 1.9)
    if case["graph"] == "road":
        return case["w"] * case["h"], 2 * (case["w"] * case["h"] - 1 + case["extra"])
    if case["graph"] == "grid":
        return case["w"] * case["h"], 4 * case["w"] * case["h"] - 2 * (case["w"] + case["h"])
    return case["n"], case["n"] * case["deg"]


def work(case):
    """Bytes that a call cannot do without: the graph read once, and its results written once (no arithmetic to speak of)."""
    if case["call"] == "batch":
        sizes = [(15500, 124000)] * case["n_er"] + [(24600, 50000)] * case["n_grid"] + [(65536, 980000)] * case["n_rmat"]
        return {"bytes": sum(4 * (v + e) + 4 * 46 * v for v, e in sizes), "flops": 0}
    V, E = _size(case)
    S = case["S"]
    if case["call"] == "served":
        S = sum((1, 8, 64)[i % 3] for i in range(case["requests"]))
    out = {"rows": 4 * S * V, "host": 4 * S * V, "reach": 4 * V * ((S + 31) // 32)}.get(case["call"], 16 * S)
    return {"bytes": 4 * (V + 1 + E) + 4 * S + out, "flops": 0}


def exact(case, seed):
    """The distance rows by a plain level-by-level search, where that is quick."""
    if case["call"] != "rows" or case["graph"] == "rmat" or _size(case)[0] * case["S"] > 1 << 21:
        return None
    g = _graph(case, seed)
    src = _sources(g, case["S"], np.random.default_rng(seed)).astype(np.int64)
    off, idx = g.row_offsets.astype(np.int64), g.col_indices.astype(np.int64)
    dist = np.full((src.size, g.num_vertices), UNREACHED, np.uint32)
    for row, s in zip(dist, src):
        row[s], level, front = 0, 0, np.array([s])
        while front.size:
            level += 1
            n = off[front + 1] - off[front]
            at = np.repeat(off[front] - np.cumsum(n) + n, n) + np.arange(n.sum())
            front = np.unique(idx[at])
            front = front[row[front] == UNREACHED]
            row[front] = level
    return dist.view(np.int32)
