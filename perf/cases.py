"""The calls this library's users make, as cases to time: searches, batches of searches, the queue codec, the bitmap OR.

A case is a dict of plain values; `prepare` builds what a program holds before the call (graphs, workspaces, buffers on the
GPU), `run` is one pass through the public entry points, `work` the bytes that pass cannot do without.  Every result is
whole numbers (parents, levels, encoded words, bits), so there is no 64-bit value for `exact` to give.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gpugraph500_gb300 as g5

MODES = {"d4": g5.CODEC_D4, "dm": g5.CODEC_DM}
ID_SPACE = 1 << 24  # queue values: vertex ids of a scale-24 graph


def listed():
    return [
        # one query on a graph small enough that only latency counts
        {"name": "bfs_s10", "kind": "bfs", "scale": 10, "edgefactor": 16, "roots": 1, "levels": False, "host": False,
         "codec": "none", "tuned": False},
        # the reference driver's loop on its CPU configuration: runBFS, then parents and levels on the host
        {"name": "bfs_s16_host", "kind": "bfs", "scale": 16, "edgefactor": 16, "roots": 1, "levels": True, "host": True,
         "codec": "none", "tuned": False},
        # every level's queue through the codec inside the level loop
        {"name": "bfs_s22_codec", "kind": "bfs", "scale": 22, "edgefactor": 16, "roots": 2, "levels": False,
         "host": False, "codec": "d4", "tuned": False},
        # the headline search: scale 26, thresholds as the autotuner picks them, parents stay on the GPU
        {"name": "bfs_s26", "kind": "bfs", "scale": 26, "edgefactor": 16, "roots": 4, "levels": False, "host": False,
         "codec": "none", "tuned": True},
        # a user's own graph (uploaded CSR, odd size, no hubs), many roots in one pipelined call, pinned host parents
        {"name": "many_ragged", "kind": "many", "n": 1000003, "degree": 12, "roots": 8},
        # 64 roots of one graph in one bit-sliced search
        {"name": "batch_s24", "kind": "batch", "scales": "24", "roots": 64},
        # uneven graphs in one batch, 16 roots each
        {"name": "batch_mixed", "kind": "batch", "scales": "14,15,16,17,18,18,19,20", "roots": 16},
        # one large level queue, each direction
        {"name": "encode_5m", "kind": "encode", "n": 5000003, "mode": "d4"},
        {"name": "decode_5m", "kind": "decode", "n": 5000003, "mode": "d4"},
        # the reference's plugin calls on a small host queue, there and back
        {"name": "plugin_3k", "kind": "plugin", "n": 3000, "mode": "dm"},
        # all level queues of several searches in one call each way
        {"name": "codec_batch", "kind": "codec_batch", "searches": 8, "scale": 22, "mode": "d4"},
        # 8 frontier bitmaps of 2^24 bits
        {"name": "or_8x2m", "kind": "or", "words": 1 << 18, "sources": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bfs", "bfs", "bfs", "many", "batch", "batch", "encode", "decode", "plugin", "codec_batch", "or"])
    if kind == "bfs":
        scale = rng.randint(8, 25)
        return {"kind": kind, "scale": scale, "edgefactor": rng.choice([8, 16, 16, 24]), "roots": rng.randint(1, 4),
                "levels": rng.random() < 0.3, "host": scale <= 20 and rng.random() < 0.4,
                "codec": rng.choice(["none", "none", "none", "d4", "dm"]) if scale <= 23 else "none",
                "tuned": rng.random() < 0.5}
    if kind == "many":
        return {"kind": kind, "n": _log(rng, 500, 4_000_000) | 1, "degree": rng.randint(3, 24),
                "roots": rng.randint(2, 16)}
    if kind == "batch":
        top = rng.randint(9, 23)
        scales = [top] + [rng.randint(max(8, top - 6), top) for _ in range(rng.choice([0, 0, 1, 3, 7]))]
        while sum(1 << s for s in scales) > 1 << 24:
            scales.pop()
        return {"kind": kind, "scales": ",".join(map(str, scales)), "roots": rng.randint(1, 64)}
    if kind in ("encode", "decode"):
        return {"kind": kind, "n": _log(rng, 1, 8_000_000), "mode": rng.choice(["d4", "d4", "dm"])}
    if kind == "plugin":
        return {"kind": kind, "n": _log(rng, 20, 200_000), "mode": rng.choice(["dm", "dm", "d4"])}
    if kind == "codec_batch":
        return {"kind": kind, "searches": rng.randint(1, 16), "scale": rng.randint(14, 22),
                "mode": rng.choice(["d4", "dm"])}
    return {"kind": "or", "words": _log(rng, 1000, 1 << 21), "sources": rng.randint(1, 16)}


# ---- inputs ------------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _queue(n, gen, space=ID_SPACE):
    """n sorted distinct vertex ids: a frontier of a graph whose labels are permuted is a uniform random subset."""
    x = torch.unique(torch.randint(space, (min(space, int(1.1 * n + 64 + n * n // space)),), generator=gen, device="cuda"))
    while len(x) < n:
        x = torch.unique(torch.cat([x, torch.randint(space, (n,), generator=gen, device="cuda")]))
    keep = torch.randperm(len(x), generator=gen, device="cuda")[:n]
    return x[keep].sort().values.to(torch.int32)


def _ragged_csr(n, degree, gen):
    """Symmetric CSR of a uniform random graph: rows sorted, no self loops or duplicates (host arrays, as a user uploads)."""
    m = n * degree // 2
    a = torch.randint(n, (m,), generator=gen, device="cuda")
    b = torch.randint(n, (m,), generator=gen, device="cuda")
    keep = a != b
    a, b = a[keep], b[keep]
    key = torch.unique(torch.cat([a * n + b, b * n + a]))
    src, dst = key // n, key % n
    ro = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ro[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    return ro.cpu().numpy(), dst.cpu().numpy().astype(np.uint32)


def _level_queues(case, gen):
    """Every level's queue of some searches of one graph, one after another: a handful of vertices, two levels that hold most
    of the reached half, and a thin end."""
    n = 1 << case["scale"]
    queues = []
    for i in range(case["searches"]):
        wide = 1.0 - 0.05 * (i % 8)
        for q in (1, 24 + i, n // 600 + 7, int(wide * n / 4) + 3, int(n / (5 * wide)) + 1, n // 300 + i, 61, 2):
            queues.append(_queue(q, gen, n))
    return queues


def prepare(case, seed):
    kind = case["kind"]
    if kind == "bfs":
        graph = g5.Graph.kronecker(case["scale"], case["edgefactor"], seed1=seed + 1)
        tuned = {"alpha": 25.0, "beta": 1000.0, "tile_edges": 128, "bu_serial": 16} if case["tuned"] else {}
        search = g5.CudaBFS(graph, codec=MODES.get(case["codec"], g5.CODEC_NONE), want_levels=case["levels"], **tuned)
        roots = [int(r) for r in g5.select_roots(graph, case["roots"])]
        n, k = graph.n, len(roots)
        pred = level = None
        if not case["host"]:
            pred = torch.empty((k, n), dtype=torch.int64, device="cuda")
            level = torch.empty((k, n), dtype=torch.int32, device="cuda") if case["levels"] else None
        return {"case": case, "search": search, "graph": graph, "roots": roots, "pred": pred, "level": level}
    if kind == "many":
        ro, col = _ragged_csr(case["n"], case["degree"], _generator(seed))
        graph = g5.Graph.from_csr(ro, col)
        roots = g5.select_roots(graph, case["roots"])
        pred = [torch.empty(graph.n, dtype=torch.int64, pin_memory=True) for _ in roots]
        return {"case": case, "search": g5.CudaBFS(graph), "graph": graph, "roots": roots, "pred": pred}
    if kind == "batch":
        graphs = [g5.Graph.kronecker(int(s), seed1=seed + 1 + i) for i, s in enumerate(case["scales"].split(","))]
        roots = [g5.select_roots(g, case["roots"]) for g in graphs]
        out = torch.empty(sum(g.n * len(r) for g, r in zip(graphs, roots)), dtype=torch.int32, device="cuda")
        return {"case": case, "batch": g5.Batch(graphs), "graphs": graphs, "roots": np.concatenate(roots),
                "counts": [len(r) for r in roots], "out": out}
    if kind in ("encode", "decode"):
        n, gen = case["n"], _generator(seed)
        codec = g5.Codec(n)
        values = _queue(n, gen)
        stream = torch.zeros(g5.Codec.bound(n) + 4, dtype=torch.int32, device="cuda")
        state = {"case": case, "codec": codec, "values": values, "stream": stream}
        if kind == "decode":
            torch.cuda.synchronize()
            state["words"] = codec.encode(values, n, stream, MODES[case["mode"]])
            state["values"] = torch.zeros(n + 128, dtype=torch.int32, device="cuda")
        return state
    if kind == "plugin":
        plugin = g5.GpuSimd()
        plugin.reconfigure(64, "s4-bp128-" + case["mode"])
        # the stream goes into a send buffer of fixed size, as the reference's exchange holds it
        return {"case": case, "plugin": plugin, "queue": _queue(case["n"], _generator(seed)).cpu().numpy().astype(np.int64),
                "send": np.zeros(g5.Codec.bound(case["n"]), np.uint32)}
    if kind == "codec_batch":
        queues = _level_queues(case, _generator(seed))
        off = np.concatenate([[0], np.cumsum([len(q) for q in queues])]).astype(np.uint64)
        values = torch.cat(queues)
        stream = torch.zeros(g5.Codec.batch_bound(off), dtype=torch.int32, device="cuda")
        return {"case": case, "codec": g5.Codec(len(values)), "values": values, "off": off,
                "n": np.diff(off), "stream": stream, "back": torch.zeros_like(values)}
    words, gen = case["words"], _generator(seed)

    def bitmap(density):  # the reduction's inputs: 1 % to 60 % of the bits set
        bits = torch.rand((words, 8), generator=gen, device="cuda") < density
        byte = torch.randint(256, (words, 8), generator=gen, device="cuda", dtype=torch.int64) * bits
        return (byte << (8 * torch.arange(8, device="cuda"))).sum(1)

    srcs = [bitmap(0.01 + 0.6 * i / case["sources"]) for i in range(case["sources"])]
    return {"case": case, "dst": bitmap(0.01), "srcs": srcs}


# ---- one pass ------------------------------------------------------------------------------


def _ok(code, what):
    if code != g5.G5_OK:
        raise g5.G5Error(code, what)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "bfs":
        search = state["search"]
        if case["host"]:
            out = []
            for root in state["roots"]:
                search.runBFS(root)
                out.append(search.getPredecessor())
                if case["levels"]:
                    out.append(search.getLevels())
            # each search's arrays are the workspace's own: the last one's are what a caller still holds
            return out[-2:] if case["levels"] else out[-1:]
        for i, root in enumerate(state["roots"]):
            _ok(search.run(root, state["pred"][i], state["level"][i] if case["levels"] else None), "run")
        return {"pred": state["pred"], "level": state["level"]}
    if kind == "many":
        state["search"].run_many(state["roots"], state["pred"])
        return state["pred"]
    if kind == "batch":
        state["batch"].run(state["roots"], state["counts"], state["out"])
        return state["out"]
    if kind == "encode":
        words = state["codec"].encode(state["values"], case["n"], state["stream"], MODES[case["mode"]])
        return {"words": words, "stream": state["stream"]}
    if kind == "decode":
        n = state["codec"].decode(state["stream"], state["words"], state["values"], case["n"] + 128, MODES[case["mode"]])
        return {"n": n, "values": state["values"]}
    if kind == "plugin":
        stream, size = state["plugin"].compress(state["queue"])
        state["send"][:size] = stream
        return {"stream": state["send"], "size": size,
                "back": state["plugin"].decompress(state["send"][:size], size, case["n"])}
    if kind == "codec_batch":
        mode = MODES[case["mode"]]
        off, words = state["codec"].encode_batch(state["values"], state["off"], state["stream"], 64, mode)
        back_off, _ = state["codec"].decode_batch(state["stream"], off[:-1], words, state["n"], state["back"], 64, mode)
        return {"off": off.astype(np.int64), "words": words.astype(np.int64), "stream": state["stream"],
                "back_off": back_off.astype(np.int64), "back": state["back"]}
    g5.bitmap_or(state["dst"], state["srcs"], case["words"], torch.cuda.current_stream().cuda_stream)
    return state["dst"]


# ---- the bytes a pass cannot do without ------------------------------------------------------


def _stream_words(n, space=ID_SPACE):
    """About the words of an encoded queue: a miniblock's width holds its largest gap over four values."""
    gap = 4.0 * space / max(n, 1)
    bits = min(32.0, math.ceil(math.log2(1.0 + 3.0 * gap)))
    return 4 + n * bits / 32.0


def work(case):
    kind = case["kind"]
    if kind == "bfs":
        # per vertex its row bounds, one adjacency entry and its parent (and level): a search may skip every other entry
        n = 1 << case["scale"]
        b = case["roots"] * n * (8 + 4 + 8 + (4 if case["levels"] else 0))
        if case["codec"] != "none":
            b += case["roots"] * (4 * n + 4 * _stream_words(n, n)) / 2  # about half the vertices have edges
        return {"bytes": float(b), "flops": 0.0}
    if kind == "many":
        return {"bytes": float(case["roots"] * case["n"] * 20), "flops": 0.0}
    if kind == "batch":
        n = sum(1 << int(s) for s in case["scales"].split(","))
        return {"bytes": float(n * (8 + 4 * 2 * 16 + 4 * case["roots"])), "flops": 0.0}
    if kind in ("encode", "decode"):
        return {"bytes": 4.0 * (case["n"] + _stream_words(case["n"])), "flops": 0.0}
    if kind == "plugin":
        # 8 bytes a value in and out, and the stream both ways
        return {"bytes": 16.0 * case["n"] + 8.0 * _stream_words(case["n"]), "flops": 0.0}
    if kind == "codec_batch":
        n = case["searches"] * (1 << case["scale"]) // 2
        return {"bytes": 8.0 * (n + _stream_words(1 << case["scale"], 2 << case["scale"]) * case["searches"] / 2), "flops": 0.0}
    return {"bytes": 8.0 * case["words"] * (case["sources"] + 2), "flops": 0.0}
