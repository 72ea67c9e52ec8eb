"""Cases that the framework's speed is measured on: what a program that uses it has it do.

The data are the repository's own workloads, seeded: databases of many small
connected graphs (the 1,000-graph and the 20,000-graph shapes of the
benchmark), one large R-MAT graph of the benchmark's skew and labels at sizes
that load quickly, and connected query patterns grown inside the data, so that
every query has at least one embedding.

Kinds of a case, one per public entry point:

  match   geneva_b200.match: one query at a time, what a gpumine user has;
          `rows` copies the embeddings into a host buffer that the program
          keeps (the first rows of it, if there are more), else they are counted
  batch   geneva_b200.batch_count: planned queries, counts and supports (or
          counts per graph) of all of them
  texts   geneva_b200.batch_count_texts: query texts in, counts out
  mine    geneva_b200.mine: frequent patterns by graph support
  mni     geneva_b200.mni_support: minimum image-based support on one graph

Data families (`data`):

  flat    graphs of 10-30 vertices, average degree 3, 4 uniform vertex labels,
          one edge label
  zipf    graphs of 20-60 vertices, average degree 4, 16 vertex labels
          Zipf(1.2), 3 edge labels
  rmat    one R-MAT graph (a=0.57, b=c=0.19) of 2^scale vertices with `degree`
          edges per vertex, 32 vertex labels Zipf(1.0), one edge label
"""
import math

import numpy as np
import torch

import geneva_b200 as gv

# Queries of the match cases: edges over vertices 0..n-1, and the rank of each
# vertex's label among the data's labels (0: the most frequent).
SHAPES = {
    "edge": ([(0, 1)], [0, 1]),
    "wedge": ([(0, 1), (1, 2)], [1, 0, 2]),
    "triangle": ([(0, 1), (1, 2), (0, 2)], [0, 1, 2]),
    "path4": ([(0, 1), (1, 2), (2, 3)], [0, 1, 0, 2]),
    "star4": ([(0, 1), (0, 2), (0, 3)], [0, 1, 1, 2]),
    "square": ([(0, 1), (1, 2), (2, 3), (0, 3)], [0, 0, 1, 1]),
    "tailed": ([(0, 1), (1, 2), (0, 2), (2, 3)], [0, 1, 2, 0]),
    "path6": ([(0, 1), (1, 2), (2, 3), (3, 4), (4, 5)], [0, 0, 1, 0, 0, 1]),
}

FAMILIES = {
    "flat": dict(vmin=10, vmax=30, degree=3.0, labels=4, zipf=0.0, edge_labels=1),
    "zipf": dict(vmin=20, vmax=60, degree=4.0, labels=16, zipf=1.2, edge_labels=3),
    "rmat": dict(labels=32, zipf=1.0, edge_labels=1),
}


def listed():
    return [
        # the smallest call: one three-vertex query over a small database, counted
        dict(name="match_small_count", kind="match", data="flat", graphs=1000, shape="triangle", rows=False),
        # one ordinary query over the benchmark's large database, its embeddings read back
        dict(name="match_graphs_rows", kind="match", data="zipf", graphs=20000, shape="path4", rows=True),
        # one query with a triangle on a skewed graph: long candidate lists, a reduction
        dict(name="match_rmat_count", kind="match", data="rmat", scale=18, degree=16, shape="tailed", rows=False),
        # one query on a skewed graph, millions of embeddings read back
        dict(name="match_rmat_rows", kind="match", data="rmat", scale=16, degree=16, shape="wedge", rows=True),
        # what a server admits between two rounds: a handful of queries of mixed size
        dict(name="batch_few", kind="batch", data="zipf", graphs=20000, queries=16, vmin=3, vmax=10, induced=False,
             per_graph=False),
        # the benchmark's 4,096 induced queries, an int64 count per (query, graph)
        dict(name="batch_per_graph", kind="batch", data="flat", graphs=1000, queries=4096, vmin=3, vmax=8,
             induced=True, per_graph=True),
        # the benchmark's default list: 16,384 patterns over the 20,000-graph database, with supports
        dict(name="batch_list", kind="batch", data="zipf", graphs=20000, queries=16384, vmin=2, vmax=7, induced=False,
             per_graph=False),
        # queries of three and four vertices on a skewed graph: uneven frontiers, hub rows
        dict(name="batch_rmat", kind="batch", data="rmat", scale=14, degree=12, queries=61, vmin=3, vmax=4,
             induced=False, per_graph=False),
        # query texts end to end, an odd number of them over a middling database
        dict(name="texts_middle", kind="texts", data="zipf", graphs=5003, queries=1501, vmin=2, vmax=7, induced=False,
             per_graph=False),
        # a whole mining run: patterns of up to 4 edges in at least 2 % of the graphs
        dict(name="mine_graphs", kind="mine", data="zipf", graphs=4000, max_edges=4, support=0.02),
        # supports of a mining level's candidates on one graph, capped at the minimum support
        dict(name="mni_capped", kind="mni", data="rmat", scale=17, degree=16, queries=1200, vmin=3, vmax=5, cap=1000),
        # exact supports of a few given patterns
        dict(name="mni_exact", kind="mni", data="rmat", scale=16, degree=16, queries=37, vmin=3, vmax=5, cap=0),
    ]


def _log(rng, lo, hi):
    """An integer in [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["match", "match", "batch", "batch", "batch", "texts", "mine", "mni"])
    if kind == "match":
        if rng.random() < 0.5:
            return dict(kind=kind, data=rng.choice(["flat", "zipf"]), graphs=_log(rng, 300, 20000),
                        shape=rng.choice(sorted(SHAPES)), rows=rng.random() < 0.5)
        return dict(kind=kind, data="rmat", scale=rng.randint(13, 17), degree=rng.randint(5, 16),
                    shape=rng.choice(["edge", "wedge", "triangle", "tailed"]), rows=rng.random() < 0.5)
    if kind == "batch" and rng.random() < 0.2:
        return dict(kind=kind, data="rmat", scale=rng.randint(11, 13), degree=rng.randint(5, 12),
                    queries=_log(rng, 1, 64), vmin=3, vmax=4, induced=rng.random() < 0.5, per_graph=False)
    if kind in ("batch", "texts"):
        per_graph = kind == "batch" and rng.random() < 0.3
        vmin = rng.randint(2, 4)
        return dict(kind=kind, data=rng.choice(["flat", "zipf"]), graphs=_log(rng, 300, 1500 if per_graph else 20000),
                    queries=_log(rng, 1, 3000 if per_graph else 16000), vmin=vmin, vmax=vmin + rng.randint(1, 5),
                    induced=rng.random() < 0.5, per_graph=per_graph)
    if kind == "mine":
        return dict(kind=kind, data=rng.choice(["flat", "zipf"]), graphs=_log(rng, 300, 4000),
                    max_edges=rng.randint(2, 4), support=rng.choice([0.02, 0.03, 0.05]))
    cap = rng.choice([0, 100, 1000])
    return dict(kind=kind, data="rmat", scale=rng.randint(13, 16), degree=rng.randint(5, 16),
                queries=_log(rng, 1, 1200 if cap else 150), vmin=3, vmax=rng.randint(4, 5), cap=cap)


PATTERNS = 1 << 16  # most patterns that a mining case finds


def _row_capacity(case):
    """Rows of the host buffer of a match whose embeddings are read back."""
    if case["data"] == "rmat":
        return 24 << case["scale"] if case["shape"] == "edge" else 100 << case["scale"]
    return 64 * case["graphs"]


# ------------------------------------------------------------------- data ---
def _labels(gen, n, k, s):
    """n labels 1..k with weights rank**-s, entry 0 unused."""
    w = torch.arange(1, k + 1, dtype=torch.float64, device="cuda") ** (-s)
    edges = torch.cumsum(w / w.sum(), 0)[:-1].contiguous()
    u = torch.rand(n + 1, dtype=torch.float64, device="cuda", generator=gen)
    lab = torch.searchsorted(edges, u) + 1
    lab[0] = 0
    return lab


def _unique_edges(a, b):
    """Each undirected edge once, as ascending keys; loops dropped."""
    lo, hi = torch.minimum(a, b), torch.maximum(a, b)
    keys = torch.unique(((lo << 32) | hi)[lo != hi])
    return keys


def _graphs(gen, count, vmin, vmax, degree, **_):
    """Connected graphs: a random spanning tree and random further edges up to
    the average degree.  Returns (vertices, edge keys, first vertex per graph)."""
    sizes = torch.randint(vmin, vmax + 1, (count,), device="cuda", generator=gen)
    first = torch.ones(count + 1, dtype=torch.int64, device="cuda")
    first[1:] += torch.cumsum(sizes, 0)
    n = int(first[-1]) - 1
    gid = torch.repeat_interleave(torch.arange(count, device="cuda"), sizes)
    local = torch.arange(1, n + 1, device="cuda") - first[gid]
    parent = first[gid] + (torch.rand(n, device="cuda", generator=gen) * local).long()
    child = local > 0
    extra = (torch.round(sizes * (degree / 2)).long() - (sizes - 1)).clamp(min=0)
    g = torch.repeat_interleave(torch.arange(count, device="cuda"), extra)
    ends = [first[g] + (torch.rand(len(g), device="cuda", generator=gen) * sizes[g]).long() for _ in range(2)]
    a = torch.cat([first[gid][child] + local[child], ends[0]])
    b = torch.cat([parent[child], ends[1]])
    return n, _unique_edges(a, b), first


def _rmat(gen, scale, degree):
    n, m = 1 << scale, (1 << scale) * degree
    a = torch.zeros(m, dtype=torch.int64, device="cuda")
    b = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(m, device="cuda", generator=gen)
        q = (r >= 0.57).long() + (r >= 0.76).long() + (r >= 0.95).long()
        a = (a << 1) | (q >> 1)
        b = (b << 1) | (q & 1)
    return n, _unique_edges(a + 1, b + 1), torch.tensor([1, n + 1], device="cuda")


class _Data:
    def __init__(self, case, seed):
        f = FAMILIES[case["data"]]
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        if case["data"] == "rmat":
            self.n, keys, first = _rmat(gen, case["scale"], case["degree"])
        else:
            self.n, keys, first = _graphs(gen, case["graphs"], **f)
        self.keys = keys
        self.labels = _labels(gen, self.n, f["labels"], f["zipf"])
        self.elabels = torch.randint(1, f["edge_labels"] + 1, (len(keys),), device="cuda", generator=gen)
        self.first, self.gen = first, gen

    def load(self):
        host = [t.to(torch.int64).cpu().numpy().astype(np.uint32)
                for t in (self.labels, self.keys >> 32, self.keys & 0xFFFFFFFF, self.elabels)]
        db = gv.Database.from_edges(*host)
        db.set_graphs(self.first.cpu().numpy())
        return db

    def patterns(self, count, vmin, vmax, induced):
        """Query texts: connected patterns grown edge by edge inside the data,
        every other edge among the chosen vertices kept always (induced) or
        with probability 1/2.  A growth that finds no new vertex stays small."""
        gen = self.gen
        lo, hi = self.keys >> 32, self.keys & 0xFFFFFFFF
        src, dst = torch.cat([lo, hi]), torch.cat([hi, lo])
        src, order = torch.sort(src, stable=True)
        dst = dst[order]
        start = torch.searchsorted(src, torch.arange(self.n + 2, device="cuda"))

        def rand(k):
            return torch.rand(count, device="cuda", generator=gen) * k

        want = vmin + rand(vmax - vmin + 1).long()
        e0 = rand(len(src)).long()
        chosen = torch.zeros(count, vmax, dtype=torch.int64, device="cuda")
        tree = torch.zeros(count, vmax, vmax, dtype=torch.bool, device="cuda")
        at = torch.arange(count, device="cuda")
        chosen[:, 0], chosen[:, 1] = src[e0], dst[e0]
        tree[:, 0, 1] = True
        size = torch.full((count,), 2, dtype=torch.int64, device="cuda")
        for _ in range(6 * (vmax - 2)):
            i = rand(size).long()
            u = chosen[at, i]
            w = dst[start[u] + rand(start[u + 1] - start[u]).long()]
            ok = (size < want) & ~(chosen == w[:, None]).any(1)
            slot = size.clamp(max=vmax - 1)
            chosen[at, slot] = torch.where(ok, w, chosen[at, slot])
            tree[at, i, slot] |= ok
            size += ok
        a, b = torch.triu_indices(vmax, vmax, 1, device="cuda")
        x, y = chosen[:, a], chosen[:, b]
        key = (torch.minimum(x, y) << 32) | torch.maximum(x, y)
        pos = torch.searchsorted(self.keys, key).clamp(max=len(self.keys) - 1)
        edge = (self.keys[pos] == key) & (b[None, :] < size[:, None])
        keep = edge & (tree[:, a, b] | induced | (torch.rand(key.shape, device="cuda", generator=gen) < 0.5))
        lab = self.labels[chosen].cpu().tolist()
        el, keep, size = self.elabels[pos].cpu().tolist(), keep.cpu().tolist(), size.cpu().tolist()
        pairs = [f"e {i} {j} " for i, j in zip(a.cpu().tolist(), b.cpu().tolist())]
        return ["".join([f"v {i} {l[i]}\n" for i in range(k)] + [f"{p}{c}\n" for p, c, ok in zip(pairs, es, ks) if ok])
                for l, es, ks, k in zip(lab, el, keep, size)]


def _shape_text(case):
    edges, ranks = SHAPES[case["shape"]]
    f = FAMILIES[case["data"]]
    lines = [f"v {i} {1 + r % f['labels']}" for i, r in enumerate(ranks)]
    lines += [f"e {a} {b} {1 + i % f['edge_labels']}" for i, (a, b) in enumerate(edges)]
    return "\n".join(lines) + "\n"


def prepare(case, seed):
    data = _Data(case, seed)
    state = dict(case=case, db=data.load())
    if case["kind"] == "match":
        state["plan"] = gv.Plan.from_text(_shape_text(case))
        if case["rows"]:
            state["rows"] = np.zeros((_row_capacity(case), len(SHAPES[case["shape"]][1])), dtype=np.uint32)
    elif case["kind"] != "mine":
        texts = data.patterns(case["queries"], case["vmin"], case["vmax"], case.get("induced", False))
        if case["kind"] == "batch":
            state["plans"] = gv.Plan.batch_from_texts(texts)
        else:
            state["texts"] = texts
    else:
        state["min_support"] = max(2, int(round(case["support"] * case["graphs"])))
        state["found"] = dict(edges=np.zeros(PATTERNS, dtype=np.uint32), supports=np.zeros(PATTERNS, dtype=np.uint32),
                              embeddings=np.zeros(PATTERNS, dtype=np.uint64),
                              text=np.zeros(64 * PATTERNS, dtype=np.uint8))
    return state


def run(state):
    case, db = state["case"], state["db"]
    kind = case["kind"]
    if kind == "match":
        res = gv.match(db, state["plan"], count_only=not case["rows"])
        out = dict(count=res.num_rows, phases=np.array(res.phase_rows, dtype=np.int64))
        if case["rows"]:
            held = min(res.num_rows, len(state["rows"]))
            res.rows(count=held, out=state["rows"][:held])
            out["rows"] = state["rows"]
        return out
    if kind == "batch":
        counts, per_graph, _ = gv.batch_count(db, state["plans"], graph_counts=case["per_graph"], support=True)
        return [counts, per_graph]
    if kind == "texts":
        counts, support, _ = gv.batch_count_texts(db, state["texts"], support=True)
        return [counts, support]
    if kind == "mine":
        pats, _ = gv.mine(db, case["max_edges"], state["min_support"])
        found = state["found"]
        for key in ("edges", "supports", "embeddings"):
            found[key][:len(pats)] = getattr(pats, key)
        text = "".join([pats.text(i) for i in range(len(pats))]).encode()
        found["text"][:len(text)] = np.frombuffer(text, dtype=np.uint8)
        return [np.array([len(pats), len(text)]), found]
    support, _ = gv.mni_support(db, state["texts"], cap=case["cap"])
    return support


def work(case):
    """The data graph read once (4-byte neighbours both ways, labels and list
    starts) and every result written once; the rows of a match are an estimate
    from the data's sizes."""
    f = FAMILIES[case["data"]]
    if case["data"] == "rmat":
        vertices = 1 << case["scale"]
        edges = vertices * case["degree"]
    else:
        vertices = case["graphs"] * (f["vmin"] + f["vmax"]) / 2
        edges = vertices * f["degree"] / 2
    queries = case.get("queries", 1)
    out = queries * 12.0
    if case.get("per_graph"):
        out += 8.0 * queries * case["graphs"]
    if case.get("rows"):
        out += 2.0 * len(SHAPES[case["shape"]][1]) * vertices
    return {"bytes": 8.0 * edges + 8.0 * vertices + out, "flops": 0.0}


def exact(case, seed):
    """Every output is a whole number or text, compared as it is."""
    return None
