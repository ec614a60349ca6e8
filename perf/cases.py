"""The work whose speed is watched: exact triangle counts through the public
entry points, from the smallest graphs to the largest that one call takes, and
the dispatcher model's forward and backward passes.

A case is a dict: ``kind`` names the entry point (see ``run``), ``family`` the
graph (see ``_graph``), ``order`` / ``dispatch`` the counter's options. The
graphs are the families of the benchmark and the tests (R-MAT with the Graph500
quadrants, Chung-Lu, Erdos-Renyi, planted partition, disjoint cliques, and the
mixed batch), made on the GPU from the seed alone: raw entries in random order
with duplicates and self-loops, as an edge list comes.
"""
import math
import os
import tempfile

import numpy as np
import torch

import tribit_b200 as tb

MODEL = os.path.join(os.path.dirname(os.path.abspath(tb.__file__)), "models", "dispatch_mlp.bin")


def listed():
    return [
        # The smallest call: a graph of a few thousand edges in ordinary numpy
        # memory, one blocking count. Launches and host work are all of it.
        {"name": "er_1k_host", "kind": "host", "family": "er", "n": 1003, "entries": 7919, "order": "degree",
         "dispatch": "plain"},
        # A caller that may not allocate, counting a wiki-Vote-sized graph of
        # its own device memory on its own stream.
        {"name": "chung_lu_7k_noalloc", "kind": "noalloc", "family": "chung_lu", "n": 7115, "entries": 115300},
        # The same graph through a context with the learned dispatcher, as the
        # command line counts a small social network.
        {"name": "chung_lu_7k_device", "kind": "device", "family": "chung_lu", "n": 7115, "entries": 115300,
         "order": "degree", "dispatch": "learned"},
        # `tribit -i graph.mtx`: a Matrix Market file of a million lines read,
        # parsed and counted.
        {"name": "rmat16_mtx", "kind": "mtx", "family": "rmat", "scale": 16, "entries": 1048573, "order": "degree",
         "dispatch": "learned"},
        # The reference's own orientation (by id), which leaves the hubs' long
        # rows in place.
        {"name": "rmat17_id_order", "kind": "device", "family": "rmat", "scale": 17, "entries": 2097143, "order": "id",
         "dispatch": "plain"},
        # An ordinary power-law graph already on the device.
        {"name": "rmat20_device", "kind": "device", "family": "rmat", "scale": 20, "entries": 16777213,
         "order": "degree", "dispatch": "learned"},
        # Communities (the planted partition of the benchmark): similar degrees
        # everywhere, few triangles across.
        {"name": "planted_device", "kind": "device", "family": "planted", "communities": 20000, "size": 100,
         "p_in": 0.3, "inter": 2, "order": "degree", "dispatch": "plain"},
        # Dense blocks: disjoint cliques, which go to the tensor-core tiles.
        {"name": "cliques_device", "kind": "device", "family": "cliques", "count": 512, "min_size": 256,
         "max_size": 512, "order": "degree", "dispatch": "plain"},
        # A graph prepared once and counted again: the counting launch alone,
        # with its result read.
        {"name": "rmat22_launch", "kind": "launch", "family": "rmat", "scale": 22, "entries": 67108859,
         "order": "degree", "dispatch": "learned"},
        # Many small graphs at once from host memory.
        {"name": "batch_512_host", "kind": "batch", "graphs": 512, "min_n": 64, "max_n": 65536, "dispatch": "learned"},
        # The headline graph end to end from pinned host memory: upload,
        # preprocessing, count, result.
        {"name": "rmat24_host", "kind": "host", "family": "rmat", "scale": 24, "entries": 268435456, "pinned": True,
         "order": "degree", "dispatch": "learned"},
        # The dispatcher's model on the row blocks of a two-million-vertex
        # graph: predictions, and one training gradient.
        {"name": "mlp_65k", "kind": "mlp", "rows": 65521},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["device", "device", "device", "host", "launch", "noalloc", "mtx", "batch", "mlp"])
    if kind == "mlp":
        return {"kind": kind, "rows": _log_int(rng, 1000, 200000)}
    dispatch = rng.choice(["plain", "learned"])
    if kind == "batch":
        return {"kind": kind, "graphs": _log_int(rng, 3, 400), "min_n": 64, "max_n": _log_int(rng, 2000, 65536),
                "dispatch": dispatch}
    if kind == "noalloc":
        n = _log_int(rng, 500, 50000)
        family = rng.choice(["er", "chung_lu"])
        return {"kind": kind, "family": family, "n": n, "entries": _log_int(rng, 4 * n, min(32 * n, 600000))}
    case = {"kind": kind, "dispatch": dispatch, "order": rng.choice(["degree", "degree", "degree", "id"])}
    top = {"device": 23, "host": 23, "launch": 23, "mtx": 18}[kind]
    family = rng.choice(["rmat", "rmat", "chung_lu", "er", "planted", "cliques"])
    if kind == "mtx" and family in ("planted", "cliques"):
        family = "er"
    case["family"] = family
    if family == "rmat":
        # By id the hubs keep rows of tens of thousands: their count grows
        # with the square of the graph.
        case["scale"] = rng.randint(10, min(top, 18) if case["order"] == "id" else top)
        case["entries"] = int(rng.uniform(6, 16) * (1 << case["scale"])) | 1
    elif family in ("chung_lu", "er"):
        case["n"] = _log_int(rng, 500, {"mtx": 100000}.get(kind, 3000000))
        if family == "chung_lu" and case["order"] == "id":
            case["n"] = min(case["n"], 200000)
        case["entries"] = int(rng.uniform(4, 16) * case["n"]) | 1
    elif family == "planted":
        case["communities"] = _log_int(rng, 50, 20000)
        case["size"] = rng.randint(30, 120)
        case["p_in"] = round(rng.uniform(0.1, 0.3), 3)
        case["inter"] = rng.randint(1, 4)
    else:
        case["count"] = _log_int(rng, 8, 400)
        case["min_size"] = rng.randint(20, 200)
        case["max_size"] = case["min_size"] + rng.randint(1, 300)
    if kind == "host":
        case["pinned"] = rng.random() < 0.5
    if kind == "launch":
        case["capture"] = rng.random() < 0.5
    return case


# ---- inputs -------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rmat(scale, entries, g):
    """R-MAT entries (a, b, c, d = 0.57, 0.19, 0.19, 0.05), without a permutation of the ids."""
    out = torch.empty(entries, dtype=torch.int64, device="cuda")
    step = 1 << 26
    for at in range(0, entries, step):
        k = min(step, entries - at)
        row = torch.zeros(k, dtype=torch.int32, device="cuda")
        col = torch.zeros(k, dtype=torch.int32, device="cuda")
        for _ in range(scale):
            x = torch.rand(k, generator=g, device="cuda")
            down = x >= 0.76
            right = ((x >= 0.57) & (x < 0.76)) | (x >= 0.95)
            row = row * 2 + down
            col = col * 2 + right
        out[at:at + k] = (row.to(torch.int64) << 32) | col.to(torch.int64)
    return out


def _chung_lu(n, entries, g):
    """Endpoints drawn by weight (i + 1)^(-1), no expected degree above 1,000 or the structural cut-off."""
    w = 1.0 / torch.arange(1, n + 1, dtype=torch.float64, device="cuda")
    most = max(1000.0, math.sqrt(2.0 * entries)) if n < 10000 else math.sqrt(2.0 * entries)
    for _ in range(8):
        w = torch.minimum(w, most * w.sum() / (2.0 * entries))
    cdf = torch.cumsum(w, 0)
    ends = torch.rand((2, entries), generator=g, device="cuda", dtype=torch.float64) * cdf[-1]
    ids = torch.searchsorted(cdf, ends, right=True).clamp_(max=n - 1)
    return (ids[0] << 32) | ids[1]


def _planted(communities, size, p_in, inter, g):
    i, j = torch.triu_indices(size, size, 1, device="cuda")
    n = communities * size
    perm = torch.randperm(n, generator=g, device="cuda")
    parts = []
    step = max(1, (1 << 25) // i.numel())
    for at in range(0, communities, step):
        k = min(step, communities - at)
        hit = (torch.rand((k, i.numel()), generator=g, device="cuda") < p_in).nonzero()
        base = (hit[:, 0] + at) * size
        parts.append((perm[base + i[hit[:, 1]]] << 32) | perm[base + j[hit[:, 1]]])
    away = torch.randint(n, (n * inter,), generator=g, device="cuda")
    here = torch.arange(n, device="cuda").repeat_interleave(inter)
    parts.append((perm[here] << 32) | perm[away])
    return torch.cat(parts)


def _cliques(sizes):
    parts, at = [], 0
    for s in sizes:
        i, j = torch.triu_indices(s, s, 1, device="cuda")
        parts.append(((i + at) << 32) | (j + at))
        at += s
    return torch.cat(parts)


def _graph(case, seed):
    """(entries on the GPU as int64 words (a << 32) | b, number of vertices)."""
    g = _generator(seed)
    family = case["family"]
    if family == "rmat":
        return _rmat(case["scale"], case["entries"], g), 1 << case["scale"]
    if family == "er":
        ids = torch.randint(case["n"], (2, case["entries"]), generator=g, device="cuda")
        return (ids[0] << 32) | ids[1], case["n"]
    if family == "chung_lu":
        return _chung_lu(case["n"], case["entries"], g), case["n"]
    if family == "planted":
        return (_planted(case["communities"], case["size"], case["p_in"], case["inter"], g),
                case["communities"] * case["size"])
    sizes = np.random.RandomState(seed % (1 << 32)).randint(case["min_size"], case["max_size"] + 1, case["count"])
    return _cliques([int(s) for s in sizes]), int(sizes.sum())


def _mlp_inputs(rows, seed):
    """Features and targets in the ranges of real row blocks, and a model's parameters and normalisation."""
    r = np.random.RandomState(seed % (1 << 32))
    mean, std = r.uniform(0, 8, 16), r.uniform(0.5, 3, 16)
    x = (mean + std * r.standard_normal((rows, 16))).astype(np.float32)
    y = (10 + 2 * r.standard_normal((rows, 3)) + 0.3 * x[:, 1:2]).astype(np.float32)
    norm = np.concatenate([x.mean(0), x.std(0) + 1e-3, y.mean(0), y.std(0) + 1e-3]).astype(np.float32)
    lim = np.concatenate([np.full(16 * 64, math.sqrt(6 / 16)), np.zeros(64), np.full(64 * 64, math.sqrt(6 / 64)),
                          np.zeros(64), np.full(64 * 3, math.sqrt(6 / 64)), np.zeros(3)])
    params = (lim * r.uniform(-1, 1, lim.size)).astype(np.float32)
    return x, y, norm, params


def _counter(case):
    c = tb.Counter(order=case.get("order", "degree"), dispatch=case["dispatch"])
    if case["dispatch"] == "learned":
        c.load_model(MODEL)
    return c


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        x, y, norm, params = _mlp_inputs(case["rows"], seed)
        c = tb.Counter()
        c.model_init(norm)
        c.set_model_params(params)
        return {"kind": kind, "counter": c, "x": x, "y": y}
    if kind == "batch":
        e, off, nn = tb.gen_batch(case["graphs"], seed=seed, min_n=case["min_n"], max_n=case["max_n"])
        host = torch.empty(e.size, dtype=torch.int64, pin_memory=True)
        host.numpy()[:] = e.view(np.int64)
        return {"kind": kind, "counter": _counter(case), "keep": host, "entries": host.numpy().view(np.uint64),
                "offsets": off, "nodes": nn}
    d, n = _graph(case, seed)
    state = {"kind": kind, "n": n, "entries": d}
    if kind == "noalloc":
        state["result"] = torch.zeros(4, dtype=torch.int64, device="cuda")
        return state
    state["counter"] = c = _counter(case)
    if kind == "host":
        host = torch.empty(d.numel(), dtype=torch.int64, pin_memory=bool(case.get("pinned")))
        host.copy_(d)
        state["keep"], state["entries"] = host, host.numpy().view(np.uint64)
    elif kind == "mtx":
        state["dir"] = tempfile.TemporaryDirectory()
        state["path"] = os.path.join(state["dir"].name, "graph.mtx")
        tb.write_mtx(state["path"], n, d.cpu().numpy().view(np.uint64))
        state["entries"] = None
    elif kind == "launch":
        torch.cuda.synchronize()
        c.prepare_device(d.data_ptr(), d.numel(), n)
        if case.get("capture"):
            c.capture_count()
        state["entries"] = None  # the prepared graph holds all that the launches read
    torch.cuda.synchronize()  # the counter's own stream reads what torch's wrote
    return state


# ---- a pass ---------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "noalloc":
        e = state["entries"]
        tb.count_edges_noalloc(e.data_ptr(), e.numel(), state["n"], state["result"].data_ptr(),
                               torch.cuda.current_stream().cuda_stream)
        return {"result": state["result"]}
    c = state["counter"]
    if kind == "mlp":
        pred = c.model_predict(state["x"])
        grad, loss = c.model_gradients(state["x"], state["y"])
        return {"pred": pred, "grad": grad, "loss": loss}
    if kind == "batch":
        counts, r = c.count_batch(state["entries"], state["offsets"], state["nodes"])
        return {"triangles": r.triangles, "edges": r.edges, "counts": counts.view(np.int64)}
    if kind == "host":
        r = c.count_edges(state["entries"], state["n"])
    elif kind == "mtx":
        r = c.count_mtx(state["path"])
    elif kind == "launch":
        c.launch_count()
        r = c.read_count()
    else:
        r = c.count_edges_device(state["entries"].data_ptr(), state["entries"].numel(), state["n"])
    return {"triangles": r.triangles, "edges": r.edges}


def _entries(case):
    """Entries of the case's graph, as expected where they are drawn."""
    if case.get("entries"):
        return case["entries"]
    if case["kind"] == "batch":
        span = math.log(case["max_n"] / case["min_n"])
        return case["graphs"] * (case["max_n"] - case["min_n"]) / span * 18
    if case["family"] == "planted":
        s = case["size"]
        return case["communities"] * (case["p_in"] * s * (s - 1) / 2 + s * case["inter"])
    a, b = case["min_size"], case["max_size"]
    return case["count"] * sum(s * (s - 1) / 2 for s in range(a, b + 1)) / (b - a + 1)


def work(case):
    """Every entry read once and the counts written; a prepared graph's oriented
    rows (4 bytes an edge, an offset a vertex) read once."""
    if case["kind"] == "mlp":
        # x and y read, predictions and the gradient written; two products a
        # weight forward (twice, the prediction's and the gradient's) and four back
        rows = case["rows"]
        weights = 16 * 64 + 64 * 64 + 64 * 3
        return {"bytes": 4 * (rows * (16 + 16 + 3 + 3) + 3 * 5443), "flops": 8 * rows * weights}
    e = _entries(case)
    if case["kind"] == "mtx":
        ids = 1 << case["scale"] if case["family"] == "rmat" else case["n"]
        return {"bytes": e * (2 * math.log10(ids) + 1.8) + 16, "flops": 0}
    if case["kind"] == "launch":
        n = {"rmat": lambda: 1 << case["scale"], "er": lambda: case["n"], "chung_lu": lambda: case["n"],
             "planted": lambda: case["communities"] * case["size"],
             "cliques": lambda: case["count"] * (case["min_size"] + case["max_size"]) / 2}[case["family"]]()
        return {"bytes": 4 * (n + 1) + 4 * e + 16, "flops": 0}
    return {"bytes": 8 * e + 16 + 8 * case.get("graphs", 0), "flops": 0}


def tolerance(case):
    # Counts are integers. The model's sums are in 32 bits: predictions sum 64
    # products a unit, a gradient the rows of the batch, the loss by atomics.
    return {"rel": 2e-5, "max": 1e-3} if case["kind"] == "mlp" else "exact"


# ---- the answers, in plain torch and numpy ---------------------------------------

MOST_WEDGES = 2_000_000_000  # above this a plain count takes over a few seconds


def _count(a, b, n, group=None, groups=0):
    """(triangles, edges, triangles per group or None) of the entries (a, b) on n
    vertices; group: of each vertex. None when it would take too long."""
    keep = a != b
    lo, hi = torch.minimum(a, b)[keep], torch.maximum(a, b)[keep]
    key = torch.unique(lo * n + hi)
    lo, hi = key // n, key % n
    deg = torch.bincount(lo, minlength=n) + torch.bincount(hi, minlength=n)
    order = torch.argsort(deg * n + torch.arange(n, device=deg.device))
    rank = torch.empty_like(order)
    rank[order] = torch.arange(n, device=deg.device)
    u, v = torch.minimum(rank[lo], rank[hi]), torch.maximum(rank[lo], rank[hi])
    key = torch.sort(u * n + v).values
    u, v = key // n, key % n
    m = key.numel()
    start = torch.cumsum(torch.bincount(u, minlength=n), 0)
    later = start[u] - torch.arange(m, device=key.device) - 1  # neighbours of u after this one
    total = int(later.sum())
    if total > MOST_WEDGES:
        return None
    per = torch.zeros(groups, dtype=torch.int64, device=key.device) if groups else None
    triangles = 0
    ends = torch.cumsum(later, 0)
    at = 0
    while at < m:
        base = int(ends[at - 1]) if at else 0
        to = max(at + 1, int(torch.searchsorted(ends, base + (1 << 25))))
        to = min(to, m)
        k = later[at:to]
        e = torch.arange(at, to, device=key.device).repeat_interleave(k)
        first = (ends[at:to] - k - base).repeat_interleave(k)
        q = e + 1 + (torch.arange(e.numel(), device=key.device) - first)
        want = v[e] * n + v[q]
        pos = torch.searchsorted(key, want).clamp_(max=m - 1)
        hit = key[pos] == want
        triangles += int(hit.sum())
        if groups:
            per += torch.bincount(group[order[u[e[hit]]]], minlength=groups)
        at = to
    return triangles, m, per


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        return _mlp_exact(case, seed)
    if kind == "batch":
        e, off, nn = tb.gen_batch(case["graphs"], seed=seed, min_n=case["min_n"], max_n=case["max_n"])
        nodes = torch.from_numpy(nn.astype(np.int64)).cuda()
        base = torch.cumsum(nodes, 0) - nodes
        sizes = torch.from_numpy(np.diff(off.astype(np.int64))).cuda()
        shift = base.repeat_interleave(sizes)
        d = torch.from_numpy(e.view(np.int64)).cuda()
        group = torch.arange(nodes.numel(), device="cuda").repeat_interleave(nodes)
        got = _count((d >> 32) + shift, (d & 0xffffffff) + shift, int(nodes.sum()), group, nodes.numel())
        return None if got is None else {"triangles": got[0], "edges": got[1], "counts": got[2].cpu().numpy()}
    if kind == "noalloc" or (case["family"] == "rmat" and case["scale"] > 20):
        return None  # whole words, flags of the call among them; or too long
    d, n = _graph(case, seed)
    got = _count(d >> 32, d & 0xffffffff, n)
    return None if got is None else {"triangles": got[0], "edges": got[1]}


def _mlp_exact(case, seed):
    x, y, norm, params = _mlp_inputs(case["rows"], seed)
    p = torch.from_numpy(params)
    shapes = [(16, 64), (64,), (64, 64), (64,), (64, 3), (3,)]
    parts, at = [], 0
    for s in shapes:
        k = math.prod(s)
        t = p[at:at + k].reshape(s)
        parts.append((t.to(torch.bfloat16) if len(s) == 2 else t).to(torch.float64).cuda().requires_grad_())
        at += k
    w1, b1, w2, b2, w3, b3 = parts
    nm = torch.from_numpy(norm).to(torch.float64).cuda()
    xn = (torch.from_numpy(x).to(torch.float64).cuda() - nm[:16]) / nm[16:32]
    t = (torch.from_numpy(y).to(torch.float64).cuda() - nm[32:35]) / nm[35:38]
    out = torch.relu(torch.relu(xn @ w1 + b1) @ w2 + b2) @ w3 + b3
    loss = ((out - t) ** 2).mean()
    loss.backward()
    grad = torch.cat([q.grad.reshape(-1) for q in parts])
    return {"pred": (out.detach() * nm[35:38] + nm[32:35]).cpu().numpy(), "grad": grad.cpu().numpy(),
            "loss": float(loss)}
