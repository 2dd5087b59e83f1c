"""Performance cases: the work that programs on the VEDAS core have it do.

Each case is a plain dict; prepare() makes its inputs on the GPU from a seed
together with what such a program keeps (a context, a resident index, query
texts), run() is one pass through the public Python API of vedas_gb300, and
work() the bytes that one pass cannot do without.  Graphs follow the shapes of
vedas_gb300.workloads (star, chain, hub), drawn here with torch on the device
so that a case is ready in about a second.

The structure of a case's data (which node is tied to which, how often a key
occurs) follows from the case; the seed renames every node, key and value by
random permutations and shuffles the rows.  So each seed gives other inputs and
other outputs, of the same sizes.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import vedas_gb300 as vg
from vedas_gb300 import workloads

GIB = 1 << 30
LITERAL0 = workloads.LITERAL_START_ID
ZIPF_S = {"star": 1.1, "chain": 1.0, "hub": 1.0}
PREDICATES = {"star": 32, "chain": 86, "hub": 86}
# triples per entity: 1M over 50k subjects (star), 100M over 2M entities
# (chain), 500M over 10M (hub), as in the benchmark's graphs
DENSITY = {"star": 20, "chain": 50, "hub": 50}
ENTITY_OBJECTS = {"star": 0.7, "chain": 0.7, "hub": 0.8}   # the others are literals

PARTIAL = ("p_idx_values", "p_idx_offsets", "ps_s_idx_values", "ps_idx_offsets", "po_o_idx_values",
           "po_idx_offsets", "ps_data", "pso_data", "po_data", "pos_data")
FULL = PARTIAL + ("sp_p_idx_values", "sp_idx_offsets", "so_o_idx_values", "so_idx_offsets", "o_idx_values",
                  "o_idx_offsets", "os_data", "op_p_idx_values", "op_idx_offsets", "spo_data", "sop_data",
                  "ops_data", "osp_data")

# the queries of the plain (one at a time) path, by graph shape
QUERIES = {"star": workloads.star_query(3, 7), "chain": workloads.chain_query_open((1, 2, 5, 9)),
           "hub": workloads.snowflake_query(workloads.C3_SNOWFLAKE)}


def listed():
    return [
        # one interactive query: the two-pattern star on the 1M-triple graph
        # (the plain workload's own size); latency and launches count
        {"name": "query_star_1M", "kind": "query", "graph": "star", "n": 1_000_000},
        # one analytical query: seven patterns on the graph with hubs, every
        # relation of millions of rows (a fifth of the 500M-triple workload)
        {"name": "query_snowflake_100M", "kind": "query", "graph": "hub", "n": 100_000_000},
        # a small batch: an application server's few dozen queries at once
        {"name": "batch_64_2M", "kind": "batch", "n": 2_000_000, "queries": 64},
        # the benchmark's workload (20 star, chain and snowflake templates) at
        # its size; results read by the host
        {"name": "batch_4096_100M", "kind": "batch", "n": 100_000_000, "queries": 4096},
        # loading the benchmark's graph: both permutations from device columns
        {"name": "index_100M", "kind": "index", "n": 100_000_000, "full": False, "host": False},
        # a full index (six permutations) from a loader's host columns, ragged
        {"name": "index_full_3M", "kind": "index", "n": 2_999_999, "full": True, "host": True},
        # N-Triples text to ids and dictionaries, literals apart (-ldict)
        {"name": "ingest_1M", "kind": "ingest", "n": 1_000_000, "literals": True},
        # a join of small relations: a selective query's inner step
        {"name": "join_3k", "kind": "join", "left": 3_001, "left_cols": 2, "right": 2_500, "right_cols": 2,
         "keys": 3_000, "hub": False},
        # a join of large relations, left keys with hubs
        {"name": "join_16M", "kind": "join", "left": 16_000_000, "left_cols": 3, "right": 10_000_001,
         "right_cols": 2, "keys": 12_000_000, "hub": True},
        # the join on two shared variables (two patterns over the same pair)
        {"name": "join2_1M", "kind": "join2", "left": 1_000_003, "left_cols": 3, "right": 700_001,
         "right_cols": 3, "keys": 200_000},
        # an index swap of a wide intermediate relation and back
        {"name": "swap_8M", "kind": "swap", "rows": 8_000_000, "cols": 4, "keys": 2_000_000},
        # DISTINCT over whole rows: sort by every column, drop repeated rows
        {"name": "distinct_5M", "kind": "distinct", "rows": 5_000_000, "cols": 3, "keys": 400_000},
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], uniform over its logarithm, odd more often than not."""
    v = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    return min(hi, max(lo, v | (rng.random() < 0.7)))


def draw(rng):
    kind = rng.choice(["query", "batch", "index", "ingest", "join", "join2", "swap", "distinct"])
    if kind == "query":
        graph = rng.choice(["star", "chain", "hub"])
        top = {"star": 4_000_000, "chain": 20_000_000, "hub": 100_000_000}[graph]
        return {"kind": kind, "graph": graph, "n": _log(rng, 200_000, top)}
    if kind == "batch":
        return {"kind": kind, "n": _log(rng, 1_000_000, 100_000_000), "queries": _log(rng, 16, 4096)}
    if kind == "index":
        host = rng.random() < 0.5
        full = rng.random() < 0.5
        return {"kind": kind, "n": _log(rng, 50_000, 5_000_000 if host else 30_000_000 if full else 100_000_000),
                "full": full, "host": host}
    if kind == "ingest":
        return {"kind": kind, "n": _log(rng, 10_000, 1_000_000), "literals": rng.random() < 0.5}
    if kind == "join":
        left, right = _log(rng, 500, 16_000_000), _log(rng, 500, 16_000_000)
        return {"kind": kind, "left": left, "left_cols": rng.randint(1, 4), "right": right,
                "right_cols": rng.randint(1, 4), "keys": int(max(left, right) * rng.uniform(0.7, 2.0)),
                "hub": rng.random() < 0.5}
    if kind == "join2":
        left, right = _log(rng, 1_000, 3_000_000), _log(rng, 1_000, 3_000_000)
        return {"kind": kind, "left": left, "left_cols": rng.randint(2, 4), "right": right,
                "right_cols": rng.randint(2, 4), "keys": int(max(100, max(left, right) * rng.uniform(0.1, 0.4)))}
    rows = _log(rng, 2_000, 8_000_000 if kind == "swap" else 5_000_000)
    return {"kind": kind, "rows": rows, "cols": rng.randint(2, 5 if kind == "swap" else 4),
            "keys": max(10, int(rows * rng.uniform(0.05, 0.5)))}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 1)
    return g


def _structure(case):
    """The generator of the case's structure, the same for every seed."""
    return _gen(sum(v for v in case.values() if isinstance(v, int)) + 77)


class _Names:
    """A random renaming of the ids 1..`count` (and of `literals` literals)."""

    def __init__(self, g, count, literals=0):
        self.e = (torch.randperm(count, generator=g, device="cuda") + 1).to(torch.int32)
        self.l = (torch.randperm(max(1, literals), generator=g, device="cuda") + LITERAL0).to(torch.int32)

    def __call__(self, ids):
        lit = ids >= LITERAL0
        return torch.where(lit, self.l[torch.where(lit, ids - LITERAL0, 0)], self.e[torch.where(lit, 0, ids - 1)])


def _zipf(k, s):
    w = 1.0 / torch.arange(1, k + 1, dtype=torch.float64, device="cuda") ** s
    return w / w.sum()


def _pick(weights, count, g):
    """`count` indices drawn by the weights."""
    c = weights.cumsum(0)
    u = torch.rand(count, generator=g, device="cuda", dtype=torch.float64) * c[-1]
    return torch.searchsorted(c, u, right=True).clamp_(max=weights.shape[0] - 1)


def _ints(lo, hi, count, g):
    return torch.randint(lo, hi, (count,), generator=g, device="cuda", dtype=torch.int32)


def _graph(shape, n, g):
    """s, p, o columns (int32, on the device), the entities and the literals of
    a graph of workloads' shape: subjects uniform, predicates Zipf over their
    ranks, (s, p) pairs with a geometric out-degree of mean 3 (chain, hub),
    objects entities or literals; in the hub graph 30% of the objects are hubs
    with a power law of in-degree.  Repeated triples are left out, as there."""
    entities = max(16, n // DENSITY[shape])
    prob = _zipf(PREDICATES[shape], ZIPF_S[shape])
    m = int(n * (1.3 if shape == "hub" else 1.04)) + 4096
    if shape == "star":
        s = _ints(1, entities + 1, m, g)
        p = (_pick(prob, m, g) + 1).to(torch.int32)
        lits = 4 * entities
    else:
        pairs = int(m / 3 * 1.03) + 4096
        u = torch.rand(pairs, generator=g, device="cuda").clamp_(1e-7, 1 - 1e-7)
        deg = (torch.log(u) / math.log(2.0 / 3.0)).floor_().to(torch.int64) + 1
        s = torch.repeat_interleave(_ints(1, entities + 1, pairs, g), deg)
        p = torch.repeat_interleave((_pick(prob, pairs, g) + 1).to(torch.int32), deg)
        lits = max(1, entities // 10)
    m = s.shape[0]
    o = _ints(1, entities + 1, m, g)
    u = torch.rand(m, generator=g, device="cuda")
    lit = u >= ENTITY_OBJECTS[shape]
    o = torch.where(lit, _ints(LITERAL0, LITERAL0 + lits, m, g), o)
    if shape == "hub":
        nh = max(1, entities // 100)
        hubs = (torch.randperm(entities, generator=g, device="cuda")[:nh] + 1).to(torch.int32)
        w = torch.arange(1, nh + 1, dtype=torch.float64, device="cuda") ** (-1.0 / 1.1)
        o = torch.where(u < 0.3, hubs[_pick(w, m, g)], o)
    # each triple's key, its objects made dense: the first rows of the distinct ones
    key = (p.to(torch.int64) << 52) | (s.to(torch.int64) << 27) | torch.where(o >= LITERAL0, o - LITERAL0 + (1 << 26), o)
    key, at = torch.sort(key, stable=True)
    first = torch.ones(m, dtype=torch.bool, device="cuda")
    first[1:] = key[1:] != key[:-1]
    keep = torch.sort(at[first])[0][:n]
    return s[keep], p[keep], o[keep], entities, lits


def _shuffled(cols, g):
    """The rows of a graph in runs of 3 (a subject's triples mostly lie together
    in a file), the runs in random order."""
    n = cols[0].shape[0]
    runs = torch.randperm((n + 2) // 3, generator=g, device="cuda") * 3
    at = (runs.unsqueeze(1) + torch.arange(3, device="cuda")).flatten()
    at = at[at < n]
    return [c[at].contiguous() for c in cols]


def _queries(s, p, o, count, g, names):
    """`count` queries, round robin over the workload's 20 templates, each with
    the constants of triples along a path that exists in the graph: a triple
    for the first pattern, then out-edges of the nodes bound so far."""
    n_pred = int(p.max())
    usable = torch.zeros(n_pred + 1, dtype=torch.bool, device="cuda")
    usable[1:n_pred] = True                          # never the last predicate
    rare = usable.clone()
    rare[:n_pred // 2 + 1] = False                   # patterns without a constant: the rarer half
    p_sorted, p_pos = torch.sort(p)
    s_sorted, s_pos = torch.sort(s)
    tries = 64
    texts = {}
    for k, (_, template) in enumerate(workloads.TEMPLATES):
        wanted = len(range(k, count, len(workloads.TEMPLATES)))
        if not wanted:
            continue
        q = 16 * wanted + 64                         # walks; some find no way on
        good = torch.ones(q, dtype=torch.bool, device="cuda")
        body = template.split("{", 1)[1].rsplit("}", 1)[0]
        pats = [tuple(t.strip().rstrip(" .").split()) for t in body.split(" . ") if t.strip()]
        subjects = {a for a, _, _ in pats}
        node, used, rows = {}, {}, []
        for i, (a, _, c) in enumerate(pats):
            pool = rare if a.startswith("?") and c.startswith("?") else usable
            u = torch.rand((q, tries), generator=g, device="cuda", dtype=torch.float64)
            if i == 0:
                ids = pool.nonzero().flatten().to(torch.int32)
                pick = ids[torch.randint(0, ids.shape[0], (q, tries), generator=g, device="cuda")]
                lo, hi = (torch.searchsorted(p_sorted, pick, right=r) for r in (False, True))
                pos = p_pos
            else:
                lo, hi = (torch.searchsorted(s_sorted, node[a].unsqueeze(1), right=r) for r in (False, True))
                pos = s_pos
            at = (lo + (u * (hi - lo)).to(torch.int64)).clamp_(max=s.shape[0] - 1)
            t = pos[at]
            score = (pool[p[t].to(torch.int64)] & (hi > lo)).to(torch.int32) * 2
            if c in subjects:                        # a later pattern goes on from this object
                there = torch.searchsorted(s_sorted, o[t]).clamp_(max=s.shape[0] - 1)
                score = score * (s_sorted[there] == o[t])
            for other in used.get(a, ()):            # one predicate per branch where it can be had
                score = score - ((p[t] == other.unsqueeze(1)) & (score > 0)).to(torch.int32)
            best = score.argmax(1, keepdim=True)
            good &= score.gather(1, best).squeeze(1) > 0
            t = t.gather(1, best).squeeze(1)
            used.setdefault(a, []).append(p[t])
            if a.startswith("?"):
                node.setdefault(a, s[t])
            if c.startswith("?"):
                node.setdefault(c, o[t])
            rows.append(torch.stack([names(s[t]), p[t], names(o[t])]))
        took = good.nonzero().flatten()[:wanted]
        rows = [r[:, took].cpu().tolist() for r in rows]
        for j in range(took.shape[0]):
            text = template
            for i in reversed(range(len(pats))):
                num = pats[i][1][1:]
                for letter, value in zip("SPO", rows[i]):
                    text = text.replace(f"{letter}{num} ", f"<{value[j]}> ")
            texts[k + j * len(workloads.TEMPLATES)] = text
    return [texts[i] for i in sorted(texts)]


def _relation_columns(rows, cols, keys, g, values, names, hub=False):
    """A relation sorted by column 0, as joins take it: keys 1..`keys` (with
    hub, 30% of them from a power law over a hundredth) drawn by g, the other
    columns ids drawn by `values`."""
    k = _ints(1, keys + 1, rows, g)
    if hub:
        nh = max(1, keys // 100)
        w = torch.arange(1, nh + 1, dtype=torch.float64, device="cuda") ** (-1.0 / 1.1)
        k = torch.where(torch.rand(rows, generator=g, device="cuda") < 0.3, (_pick(w, rows, g) + 1).to(torch.int32), k)
    return [torch.sort(names(k))[0]] + [_ints(1, LITERAL0, rows, values) for _ in range(cols - 1)]


def _host(t):
    return t.cpu().numpy().view(np.uint32)


class State:
    """What a program keeps between passes; closed with its last reference
    (outputs refer to it, so memory that they view outlives them)."""

    def __init__(self, case, arena_bytes):
        self.case, self.kind = case, case["kind"]
        self.ctx = vg.Context(0, arena_bytes=int(arena_bytes))
        self.index = self.last = None
        self.held = {}

    def drop(self):
        """Releases what the last pass returned."""
        last, self.last = self.last, None
        if last is not None:
            last.free() if hasattr(last, "free") else last.close()

    def __del__(self):
        torch.cuda.synchronize()
        self.drop()
        for x in self.held.values():
            if isinstance(x, vg.Relation):
                x.free()
        if self.index is not None:
            self.index.close()
        self.ctx.close()


class _View:
    """`n` words of device memory as an array; keeps its owner."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": "<i4", "data": (int(ptr), False),
                                         "version": 3, "strides": None}


def _tensor(owner, ptr, n):
    if not n or not ptr:
        return torch.empty(0, dtype=torch.int32, device="cuda")
    return torch.as_tensor(_View(owner, ptr, n), device="cuda")


def _columns(state, rel):
    return [_tensor(state, rel.ir.cols[c], rel.nrows) for c in range(rel.ncols)]


def _device_relation(ctx, cols, state):
    """A relation of the core's from columns that a program has on the device."""
    ir = vg.vg_ir()
    vg.check(vg.lib().vg_ir_alloc(ctx.h, len(cols), cols[0].shape[0], ctypes.byref(ir)))
    rel = vg.Relation(ctx, ir)
    for dst, src in zip(_columns(state, rel), cols):
        dst.copy_(src)
    torch.cuda.current_stream().synchronize()        # the core works on a stream of its own
    return rel


def prepare(case, seed):
    kind = case["kind"]
    gs, g = _structure(case), _gen(seed)             # the structure's, and the seed's
    if kind in ("query", "batch"):
        shape = case.get("graph", "chain")
        n = case["n"]
        s, p, o, entities, lits = _graph(shape, n, gs)
        names = _Names(g, entities, lits)
        texts = [QUERIES[shape]] if kind == "query" else _queries(s, p, o, case["queries"], gs, names)
        s, p, o = _shuffled((names(s), p, names(o)), g)
        torch.cuda.synchronize()
        # room for the index, the relations of the path and their sorts
        st = State(case, 2 * GIB + 160 * n + (6 * GIB + n * case["queries"] // 10 if kind == "batch" else 0))
        st.index = vg.Index(st.ctx, device_ptrs=(s.data_ptr(), p.data_ptr(), o.data_ptr()), n=n)
        # a resident index has answered a query before
        st.index.query(f"SELECT ?x WHERE {{ ?x <1> <{int(o[p == 1][0])}> . }}").close()
        st.held = {"texts": texts}
        if kind == "batch":
            # page-locked memory that any result of such a batch fits
            st.held["pinned"] = torch.zeros(_batch_words(case), dtype=torch.int32, pin_memory=True)
        return st
    if kind == "index":
        s, p, o, entities, lits = _graph("chain", case["n"], gs)
        names = _Names(g, entities, lits)
        cols = _shuffled((names(s), p, names(o)), g)
        torch.cuda.synchronize()
        st = State(case, GIB // 2 + (144 if case["full"] else 96) * case["n"])
        st.held = {"cols": [_host(c) for c in cols] if case["host"] else cols}
        return st
    if kind == "ingest":
        s, p, o, entities, lits = _graph("chain", case["n"], gs)
        names = _Names(g, entities, lits)
        cols = [_host(c) for c in _shuffled((names(s), p, names(o)), g)]
        st = State(case, GIB + 512 * case["n"])
        st.held = {"text": workloads.to_ntriples(workloads.Graph(*cols))}
        return st
    if kind == "join":
        names = _Names(g, case["keys"])
        cols = (_relation_columns(case["left"], case["left_cols"], case["keys"], gs, g, names, case["hub"]),
                _relation_columns(case["right"], case["right_cols"], case["keys"], gs, g, names))
        out = 4 * (case["left_cols"] + case["right_cols"]) * case["left"] * case["right"] / case["keys"]
        st = State(case, GIB // 2 + 40 * (case["left"] + case["right"]) + 2.5 * out)
        st.held = {k: _device_relation(st.ctx, c, st) for k, c in zip("lr", cols)}
        return st
    if kind == "join2":
        second = max(2, case["keys"] // 1000)        # both keys shared by a few rows of each side
        first = max(2, case["keys"] // second)
        n0, n1 = _Names(g, first), _Names(g, second)
        sides = []
        for side in ("left", "right"):
            rows, ncols = case[side], case[side + "_cols"]
            k = torch.randint(0, first * second, (rows,), generator=gs, device="cuda")
            k0, k1 = n0((k // second + 1).to(torch.int32)), n1((k % second + 1).to(torch.int32))
            k = torch.sort(k0.to(torch.int64) << 32 | k1)[0]
            sides.append([(k >> 32).to(torch.int32), (k & 0xFFFFFFFF).to(torch.int32)] +
                         [_ints(1, LITERAL0, rows, g) for _ in range(ncols - 2)])
        out = 32 * case["left"] * case["right"] / (first * second)
        st = State(case, GIB // 2 + 48 * (case["left"] + case["right"]) + 2.5 * out)
        st.held = {k: _device_relation(st.ctx, c, st) for k, c in zip("lr", sides)}
        return st
    rows, ncols = case["rows"], case["cols"]
    if kind == "swap":
        st = State(case, GIB // 2 + 16 * (ncols + 6) * rows)
        names = _Names(g, case["keys"])
        cols = _relation_columns(rows, 1, case["keys"], gs, g, names) + \
            [_ints(1, case["keys"] + 1, rows, g) for _ in range(ncols - 1)]
        st.held = {"rel": _device_relation(st.ctx, cols, st)}
        return st
    if kind == "distinct":
        # a projection's rows: each distinct row a few times over
        k = max(1, case["keys"])
        some = max(1, rows // 3)
        pick = torch.randint(0, some, (rows,), generator=gs, device="cuda")
        pick = pick[torch.randperm(rows, generator=g, device="cuda")]
        st = State(case, GIB // 2 + 16 * (ncols + 6) * rows)
        st.held = {"cols": [_Names(g, k)(_ints(1, k + 1, some, gs))[pick].contiguous() for _ in range(ncols)]}
        return st
    raise ValueError(f"unknown case kind {kind}")


def _batch_words(case):
    """Result words that no batch of the case exceeds (the benchmark's batch
    has 137M for 4096 queries at 100M triples)."""
    return int(4e6 + 1e-3 * case["queries"] * case["n"])


def run(state):
    state.drop()
    ctx, held = state.ctx, state.held
    if state.kind == "query":
        r = state.last = state.index.query(held["texts"][0])
        L = vg.lib()
        return {h: _tensor(state, L.vg_result_column_device(r.h, c), r.nrows) for c, h in enumerate(r.headers)}
    if state.kind == "batch":
        # the batch, then every result column in page-locked memory
        b = state.last = vg.Batch(state.index, held["texts"])
        if b.result_words() > held["pinned"].shape[0]:
            raise RuntimeError(f"{b.result_words()} result words")
        b.download_all(held["pinned"].data_ptr())
        return {"rows": b.rows().astype(np.int64), "words": held["pinned"]}
    if state.kind == "index":
        full, cols = state.case["full"], held["cols"]
        if state.case["host"]:
            ix = vg.Index(ctx, *cols, full=full)
        else:
            ix = vg.Index(ctx, device_ptrs=[c.data_ptr() for c in cols], n=cols[0].shape[0], full=full)
        state.last = ix
        return {name: _tensor(state, *ix.device_array(name)) for name in (FULL if full else PARTIAL)}
    if state.kind == "ingest":
        r = state.last = vg.ingest_ntriples(ctx, held["text"], literal_dict=state.case["literals"])
        out = {k: _tensor(state, ptr, r.n) for k, ptr in zip("spo", r.device_ptrs())}
        return dict(out, terms=[r.dict.size(k) for k in ("so", "p", "l")])
    if state.kind == "join":
        state.last, first_last = vg.join(ctx, held["l"], held["r"])
        return {"cols": _columns(state, state.last), "ends": list(first_last)}
    if state.kind == "join2":
        state.last = vg.join2(ctx, held["l"], held["r"])
        return _columns(state, state.last)
    if state.kind == "swap":
        # by the second variable for one join, back by the first for the next
        vg.swap(ctx, held["rel"], 1)
        vg.swap(ctx, held["rel"], 1)
        return _columns(state, held["rel"])
    rel = state.last = _device_relation(ctx, held["cols"], state)
    vg.sort_rows(ctx, rel)
    vg.unique(ctx, rel)
    return _columns(state, rel)


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------
def _slice_rows(graph, n, pred):
    """Expected triples of the predicate of rank `pred`."""
    k, s = PREDICATES[graph], ZIPF_S[graph]
    return n * pred ** -s / sum(r ** -s for r in range(1, k + 1))


def _query_rows(graph, n):
    """(patterns' input rows, result rows, result columns) expected of QUERIES."""
    e = max(16, n // DENSITY[graph])
    ent = ENTITY_OBJECTS[graph]

    def per(pred):                       # mean triples of one entity under a predicate
        return _slice_rows(graph, n, pred) / e

    if graph == "star":
        preds, rows, cols = (3, 7), e * per(3) * per(7), 3
    elif graph == "chain":
        preds = (1, 2, 5, 9)
        rows, cols = _slice_rows(graph, n, 1) * ent ** 3 * per(2) * per(5) * per(9), 5
    else:
        preds = workloads.C3_SNOWFLAKE
        rows, cols = e * ent, 8
        for p in preds:
            rows *= per(p)
    return sum(_slice_rows(graph, n, p) for p in preds), rows, cols


def work(case):
    """Bytes of one pass: inputs read once, outputs written once."""
    kind = case["kind"]
    flops = 0
    if kind == "query":
        rows_in, rows_out, cols = _query_rows(case["graph"], case["n"])
        data = 8 * rows_in + 4 * cols * rows_out
    elif kind == "batch":
        # two patterns without a constant a query on average, each a slice of
        # one of the rarer predicates (0.32% of the triples), and the results
        # (the benchmark's 550 MB per 4096 queries at 100M triples), written on
        # the device and on the host
        data = case["queries"] * (2 * 8 * 0.0032 * case["n"] + 2 * 1.34e-3 * case["n"])
    elif kind == "index":
        n = case["n"]
        # three columns in; two data columns a permutation out (PSO, POS), six
        # permutations' data and boundaries with the full index
        data = 12 * n + (16 * n if not case["full"] else 16 * n + 4 * 8 * n)
    elif kind == "ingest":
        data = 101 * case["n"] + 12 * case["n"]
    elif kind in ("join", "join2"):
        left, right = case["left"], case["right"]
        rows = left * right / case["keys"]
        nk = 1 if kind == "join" else 2
        data = 4 * (left * case["left_cols"] + right * case["right_cols"]) + \
            4 * rows * (case["left_cols"] + case["right_cols"] - nk)
    elif kind == "swap":
        data = 2 * 2 * 4 * case["cols"] * case["rows"]
    else:
        data = 4 * case["cols"] * case["rows"] * 1.3
    return {"bytes": data, "flops": flops}


def exact(case, seed):
    """Every output is a column of 32-bit ids or a count: nothing is rounded."""
    return None
