"""Workloads that the engine is timed on.

Each case is what a program that uses the engine does over and over: it
keeps one graph (or many) on the device, brings a batch of edges in, and
reads something back.  Graphs are directed R-MAT graphs (a = .57, b = c =
.19) with self loops and duplicates removed, as in the bench, or, for the
skewed stream, half uniform and half R-MAT (.7 / .1 / .1 / .1).

A stream holds about half of its edges at any time.  Its edges are cut into
steps of `batch` inserts and `batch` deletes of stored edges, and go round:
an edge deleted in one step comes back in a later one, so a stream can run
for as long as it likes with the stored set moving all the while.

Kinds
  stream     update calls on one graph, then a read of the result: the
             counts of the step's keys (edge_query), or the whole CSR view
  expiry     a sliding time window: every batch carries the next timestamp
             and the update's threshold expires the oldest ones
  gpma       the same stream on the flat array of GPMA mode, then its view
  many       one batch for each of many graphs in one call, then the CSR
             views of some of them
  reads      neighbour lists, edge queries and a 2-hop BFS on a stored graph
  analytics  PageRank and a full BFS over a stored graph
  build      an empty graph, the bulk load of an edge list, the CSR view
"""
import math

import torch

import lpma_gb300 as L
from lpma_gb300 import rpma

DEV = "cuda"
SRC, DST, TIME = 42, 20, 0xFFFFF


def listed():
    return [
        # an online graph fed edge by edge in small groups: a call is all latency
        dict(name="stream 1K on s21", kind="stream", scale=21, ef=16, batch=1024, calls="two", read="edges"),
        # the small plain stream: scale 16, batches of 16,384, src/dst pairs, the
        # row offsets and columns read after every step
        dict(name="stream 16K on s16, CSR", kind="stream", scale=16, ef=16, batch=16384, calls="two", read="csr",
             pair32=True),
        # a mid-size ingest with stored values and an odd batch size
        dict(name="stream 100K values on s21", kind="stream", scale=21, ef=16, batch=100003, calls="mixed",
             read="edges", values=True),
        # the headline stream: scale 21, 1M-edge batches, then the analytics' view
        dict(name="stream 1M on s21, CSR", kind="stream", scale=21, ef=16, batch=1 << 20, calls="two", read="csr"),
        # hub-heavy mixed batches that rebalance the top of the tree each time
        dict(name="skew 512K+512K on 55M", kind="stream", scale=20, ef=54, batch=1 << 19, calls="mixed",
             read="edges", skew=True),
        # a temporal graph that keeps the last 64 ticks
        dict(name="expiry 64K of 64 ticks", kind="expiry", scale=20, ef=16, batch=65537, ticks=64),
        # batches that arrive in pinned host memory, with values
        dict(name="host 300K on s19", kind="stream", scale=19, ef=16, batch=300001, calls="two", read="edges",
             values=True, host=True),
        # the flat array of GPMA mode
        dict(name="gpma 250K on s20", kind="gpma", scale=20, ef=16, batch=250000),
        # a fleet of graphs of uneven size, one batch of 100..100K edges each per
        # round (a sixteenth of a graph's edges at most)
        dict(name="many 256 graphs", kind="many", graphs=256, lo=100, hi=100000, read=20),
        # what a server answers between updates
        dict(name="reads on s20", kind="reads", scale=20, ef=16, lists=4096, queries=100000, seeds=1024),
        # the analytics step over the stored graph
        dict(name="PageRank 20 and BFS on s20", kind="analytics", scale=20, ef=16, iterations=20),
        # loading an edge list
        dict(name="build s20", kind="build", scale=20, ef=16, values=True),
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["stream"] * 6 + ["skew", "expiry", "gpma", "many", "reads", "analytics", "build"])
    if kind == "stream":
        scale = rng.randint(15, 21)
        # both halves of the edges have to hold many steps
        batch = _log(rng, 200, min(1 << 20, (1 << scale) * 16 // 24))
        return dict(kind="stream", scale=scale, ef=16, batch=batch, calls=rng.choice(["two", "mixed"]),
                    read=rng.choice(["edges", "csr"]) if batch >= 10000 else "edges", values=rng.random() < 0.4,
                    host=rng.random() < 0.15 and scale <= 19, pair32=rng.random() < 0.25)
    if kind == "skew":
        return dict(kind="stream", scale=rng.randint(16, 19), ef=54, batch=_log(rng, 20000, 200000), calls="mixed",
                    read="edges", skew=True)
    if kind == "expiry":
        ticks = rng.randint(16, 100)
        return dict(kind="expiry", scale=rng.randint(16, 20), ef=16, batch=_log(rng, 500, 100000), ticks=ticks)
    if kind == "gpma":
        scale = rng.randint(15, 20)
        return dict(kind="gpma", scale=scale, ef=16, batch=_log(rng, 1000, (1 << scale) * 16 // 20))
    if kind == "many":
        return dict(kind="many", graphs=rng.randint(16, 200), lo=100, hi=_log(rng, 2000, 100000), read=rng.randint(1, 20))
    if kind == "reads":
        return dict(kind="reads", scale=rng.randint(14, 20), ef=rng.randint(8, 24), lists=_log(rng, 1, 20000),
                    queries=_log(rng, 100, 500000), seeds=_log(rng, 1, 4000))
    if kind == "analytics":
        return dict(kind="analytics", scale=rng.randint(14, 20), ef=rng.randint(8, 16), iterations=rng.randint(5, 20))
    return dict(kind="build", scale=rng.randint(14, 20), ef=rng.randint(8, 16), values=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rmat(gen, scale, n, a=0.57, b=0.19, c=0.19):
    """n directed edges as packed keys (src << 42 | dst << 20), loops left out."""
    key = torch.zeros(n, dtype=torch.int64, device=DEV)
    for bit in range(scale):
        r = torch.rand(n, generator=gen, device=DEV)
        key += (r >= a + b).to(torch.int64) << (SRC + scale - 1 - bit)
        key += (((r >= a) & (r < a + b)) | (r >= a + b + c)).to(torch.int64) << (DST + scale - 1 - bit)
    return key[(key >> SRC) != ((key >> DST) & 0x3FFFFF)]


def _shuffled(gen, keys):
    return keys[torch.randperm(keys.numel(), generator=gen, device=DEV)]


def _edges(gen, scale, ef, draw=_rmat):
    """Exactly ef << scale distinct edges in random order."""
    n = ef << scale
    e = torch.unique(draw(gen, scale, n + n // 8))
    while e.numel() < n:
        e = torch.unique(torch.cat([e, draw(gen, scale, n)]))
    return _shuffled(gen, e)[:n]


def _values(gen, n):
    return torch.randint(0, 255, (n,), generator=gen, device=DEV, dtype=torch.uint8)


def _steps(stored, rest, batch):
    """(bulk, steps): steps[i] = `batch` keys to insert, then `batch` stored
    keys to delete.  Both halves are cut to whole batches, so that after all
    steps the stored set is the bulk again."""
    S = stored[:stored.numel() // batch * batch]
    U = rest[:rest.numel() // batch * batch]
    ins, dels = torch.cat([U, S]).view(-1, batch), torch.cat([S, U]).view(-1, batch)
    return S, torch.cat([ins, dels], 1).contiguous()


def _probes(gen, steps):
    """What is asked after each step: is it there?  The step's own keys and
    as many from another step, in random order."""
    perm = torch.randperm(2 * steps.shape[1], generator=gen, device=DEV)
    other = torch.roll(steps, steps.shape[0] // 2 + 1, 0)
    return torch.cat([steps, other], 1).index_select(1, perm)


def _pair32(keys):
    return ((keys >> SRC) << 32) | ((keys >> DST) & 0x3FFFFF)


def _skewed(gen, case):
    """A quarter of the edges stored; 90% of the inserts have a source among
    the top 1% of out-degrees.  The steps run forth and then back."""
    scale, ef, B = case["scale"], case["ef"], case["batch"]
    V = 1 << scale
    e = _edges(gen, scale, ef, lambda g, s, n: torch.cat([_rmat(g, s, n // 2, 0.25, 0.25, 0.25),
                                                         _rmat(g, s, n - n // 2, 0.7, 0.1, 0.1)]))
    hub = torch.zeros(V, dtype=torch.bool, device=DEV)
    hub[torch.topk(torch.bincount(e >> SRC, minlength=V), max(1, V // 100)).indices] = True
    nb = e.numel() // 4
    bulk, rest = e[:nb], e[nb:]
    at_hub = hub[rest >> SRC]
    hubs, cold = rest[at_hub], rest[~at_hub]
    nh = int(B * 0.9)
    n = min(hubs.numel() // nh, cold.numel() // (B - nh), nb // B)
    ins = torch.cat([hubs[:n * nh].view(n, nh), cold[:n * (B - nh)].view(n, B - nh)], 1)
    dels = bulk[:n * B].view(n, B)
    forth, back = torch.cat([ins, dels], 1), torch.cat([dels, ins], 1).flip(0)
    return bulk, torch.cat([forth, back]).contiguous()


def prepare(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    st = {"case": case, "at": 0}
    if kind == "many":
        return _prepare_many(case, seed, st)
    V = 1 << case["scale"]
    if kind == "stream":
        B = case["batch"]
        if case.get("skew"):
            bulk, steps = _skewed(gen, case)
        else:
            e = _edges(gen, case["scale"], case["ef"])
            bulk, steps = _steps(e[:e.numel() // 2], e[e.numel() // 2:], B)
        st["probes"] = _probes(gen, steps)
        fmt = _pair32 if case.get("pair32") else (lambda k: k)
        st["steps"] = fmt(steps) if case.get("pair32") else steps
        st["vals"] = _values(gen, B) if case.get("values") else None
        if case.get("host"):
            st["steps"] = st["steps"].cpu().pin_memory().numpy().view("uint64")
            if st["vals"] is not None:
                st["vals"] = st["vals"].cpu().pin_memory().numpy()
        st["g"] = L.Lpma(V, config=rpma.default_config(key_format=1 if case.get("pair32") else 0))
        st["g"].build(fmt(bulk))
    elif kind == "expiry":
        B, w = case["batch"], case["ticks"]
        e = _edges(gen, case["scale"], case["ef"])
        st["steps"] = e[:e.numel() // B * B].view(-1, B)
        t = torch.arange(w, device=DEV)
        past = st["steps"][-(torch.arange(w) % st["steps"].shape[0]) - 1] + t[:, None]
        st["g"] = L.Lpma(V)
        st["g"].build(past.reshape(-1).contiguous())
        st["now"] = w
        st["probes"] = _probes(gen, st["steps"])
    elif kind == "gpma":
        e = _pair32(_edges(gen, case["scale"], case["ef"]))
        bulk, st["steps"] = _steps(e[:e.numel() // 2], e[e.numel() // 2:], case["batch"])
        st["g"] = L.Lpma(V, config=L.gpma_config())
        st["g"].build(bulk)
    else:
        e = _edges(gen, case["scale"], case["ef"])
        if kind == "build":
            st["edges"], st["vals"] = e, _values(gen, e.numel()) if case["values"] else None
            return st
        st["g"] = L.Lpma(V)
        if kind == "reads":
            e = _prepare_reads(case, gen, e, st)
        st["g"].build(e)
        if kind == "reads":
            st["queries"] = _shuffled(gen, st["queries"])
        else:
            # the source with the most out-edges
            st["source"] = torch.bincount(e >> SRC, minlength=V).argmax().to(torch.int32).view(1)
    return st


def _prepare_reads(case, gen, e, st):
    """The edges get timestamps 0..999.  The lists asked for are those of
    vertices of fixed small degrees, at all times, and of the largest hubs,
    in a time window that holds 8 * ef of a hub's edges."""
    V, n, full = 1 << case["scale"], case["lists"], 8 * case["ef"]
    src = e >> SRC
    deg = torch.bincount(src, minlength=V)
    hubs = torch.topk(deg, 8).indices
    t = torch.randint(0, 1000, (e.numel(),), generator=gen, device=DEV)
    for h in hubs.tolist():
        at = (src == h).nonzero().view(-1)
        t[at] = t[at] % 500 + 500
        t[at[:full]] -= 500
    lists, kinds = [], (16, 0, 1, 2, 4, 8, 32, 3, 6, 12, 24, 0, 1, 2, 5, 10)
    for j, d in enumerate(kinds):
        at = (deg == d).nonzero().view(-1)
        c = (n - 1 - j) // len(kinds) + 1
        lists.append(at[torch.randint(0, at.numel(), (c,), generator=gen, device=DEV)])
    lists = torch.cat(lists)
    windows = torch.full((n,), TIME, dtype=torch.int64, device=DEV)
    k = min(8, n // 100)
    lists[:k], windows[:k] = hubs[:k], 499
    at = torch.randperm(n, generator=gen, device=DEV)
    st["lists"], st["windows"] = lists[at].to(torch.int32), windows[at].contiguous()
    st["seeds"] = torch.randint(0, V, (case["seeds"],), generator=gen, device=DEV, dtype=torch.int32)
    half = case["queries"] // 2
    miss = (torch.randint(0, V, (case["queries"] - half,), generator=gen, device=DEV) << SRC) | \
           (torch.randint(0, V, (case["queries"] - half,), generator=gen, device=DEV) << DST)
    hit = e[torch.randint(0, e.numel(), (half,), generator=gen, device=DEV)]
    st["queries"] = torch.cat([hit, miss]) | TIME  # at any time
    return e | t


def _prepare_many(case, seed, st):
    rng = torch.Generator()
    rng.manual_seed(case["graphs"])  # the sizes go with the case, the edges with the seed
    graphs, steps = [], []
    for i in range(case["graphs"]):
        u = torch.rand(3, generator=rng).tolist()
        scale, ef = 10 + int(u[0] * 9), 8 + int(u[1] * 25)
        gen = _gen(seed * 1000003 + i)
        e = _edges(gen, scale, ef)
        half = e.numel() // 2
        batch = min(int(case["lo"] * (case["hi"] / case["lo"]) ** u[2]), half // 8)
        bulk, s = _steps(e[:half], e[half:], batch)
        g = L.Lpma(1 << scale)
        g.build(bulk)
        graphs.append(g)
        steps.append(s.view(s.shape[0], 2, batch))
    st.update(graphs=graphs, steps=steps, batcher=L.Batcher())
    return st


# ------------------------------------------------------------------ passes
class _Ptr:
    """Device memory of a graph as an array that torch can view (a tensor over
    it keeps the graph alive)."""

    def __init__(self, graph, ptr, n, typestr):
        self.graph = graph
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 2}


def _at(graph, ptr, n, typestr):
    return torch.as_tensor(_Ptr(graph, ptr, n, typestr), device=DEV)


def _csr(g):
    ro, ci, va, nnz = g.csr_view()
    return {"row_offset": _at(g, ro, g.num_vertices + 1, "<i4"), "col_index": _at(g, ci, nnz, "<i4"),
            "values": _at(g, va, nnz, "|u1")}


def _counts(*stats):
    return [[s["n_ins_applied"], s["n_upserts"], s["n_del_applied"], s["n_noop"], s["num_items"], s["height_after"],
             s["levelup"]] for s in stats]


def run(st):
    case = st["case"]
    kind = case["kind"]
    at = st["at"]
    st["at"] += 1
    if kind == "many":
        return _run_many(case, st, at)
    if kind == "stream":
        g, B = st["g"], case["batch"]
        i = at % len(st["steps"])
        step = st["steps"][i]
        if case["calls"] == "two":
            s = [g.update(ins=step[:B], ins_vals=st["vals"]), g.update(dels=step[B:])]
        else:
            s = [g.update(ins=step[:B], ins_vals=st["vals"], dels=step[B:])]
        return {"counts": _counts(*s), "read": _csr(g) if case["read"] == "csr" else g.edge_query(st["probes"][i])}
    if kind == "expiry":
        g, now = st["g"], st["now"]
        st["now"] += 1
        i = at % st["steps"].shape[0]
        s = g.update(ins=st["steps"][i] + now, thres=now - case["ticks"] + 1)
        return {"counts": _counts(s), "read": g.edge_query(st["probes"][i] + now, case["ticks"])}
    if kind == "gpma":
        g, B = st["g"], case["batch"]
        step = st["steps"][at % st["steps"].shape[0]]
        s = [g.update(ins=step[:B]), g.update(dels=step[B:])]
        (ro, k, v), (size, _, _) = g.gpma_view()
        return {"counts": _counts(*s), "row_offset": _at(g, ro, g.num_vertices + 1, "<i4"), "keys": _at(g, k, size, "<i8"),
                "values": _at(g, v, size, "|u1")}
    if kind == "reads":
        g = st["g"]
        offsets, nbrs, vals = g.query_neighbors(st["lists"], st["windows"])
        found = g.edge_query(st["queries"])
        dist, levels, reached = g.bfs(st["seeds"], 2)
        return {"offsets": offsets, "nbrs": nbrs, "values": vals, "found": found, "dist": dist, "levels": levels,
                "reached": reached}
    if kind == "analytics":
        g = st["g"]
        rank = g.pagerank(0.85, case["iterations"])
        dist, levels, reached = g.bfs(st["source"])
        return {"rank": rank, "dist": dist, "levels": levels, "reached": reached}
    if st.get("g") is not None:
        L.destroy_rpma(st["g"])
    st["g"] = g = L.init_csr_rpma(1 << case["scale"])
    s = g.build(st["edges"], st["vals"])
    return {"counts": _counts(s), "read": _csr(g)}


def _run_many(case, st, at):
    # a graph's turns go insert, delete, insert, ...; the odd graphs start one
    # round later, so that inserts and deletes mix in every round
    graphs, batches = st["graphs"], []
    for i, s in enumerate(st["steps"]):
        turn = at - (i & 1)
        if turn < 0:
            batches.append({})
        else:
            key = s[(turn >> 1) % s.shape[0], turn & 1]
            batches.append({"dels": key} if turn & 1 else {"ins": key})
    stats, _ = st["batcher"].update(graphs, batches)
    n = len(graphs)
    picked = [(at * case["read"] + k) % n for k in range(min(case["read"], n))]
    return {"counts": [torch.tensor([[s.n_ins_applied, s.n_del_applied, s.num_items] for s in stats])],
            "views": [_csr(graphs[i]) for i in picked]}


# ------------------------------------------------------------------ what a pass cannot do without
def _update_bytes(items, batch, values=False):
    """The batch read once; every segment of 32 slots that takes one of its
    keys read and written once (8-byte key and 1-byte value a slot).  The
    array's segments hold about 18 items each."""
    nseg = max(1.0, items / 18.0)
    return batch * (9 if values else 8) + nseg * (1 - math.exp(-batch / nseg)) * 2 * 32 * 9


def _stored(case):
    """Keys on the device (edges and one sentinel a vertex), about."""
    edges = case["ef"] << case["scale"]
    return edges // 2 + (1 << case["scale"])


def work(case):
    kind = case["kind"]
    if kind == "stream":
        B = case["batch"]
        if case.get("skew"):
            # half of the array's slots are taken; all are rewritten
            items = (case["ef"] << case["scale"]) / 4 + (1 << case["scale"])
            by = 2 * B * 8 + 2 * items * 18
        else:
            items = _stored(case)
            n = 2 if case["calls"] == "two" else 1
            by = n * _update_bytes(items, 2 * B / n, case.get("values", False))
        by += items * 14 + 4 * (1 << case["scale"]) if case["read"] == "csr" else 4 * B * 12
        return {"bytes": by, "flops": 0}
    if kind == "expiry":
        items = case["batch"] * case["ticks"] + (1 << case["scale"])
        return {"bytes": _update_bytes(items, case["batch"]) + items * 8 + case["batch"] * 24, "flops": 0}
    if kind == "gpma":
        return {"bytes": 2 * _update_bytes(_stored(case), case["batch"]), "flops": 0}
    if kind == "many":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        view = 14 * 20 * 0.5 * ((1 << 19) - (1 << 10)) / 9
        return {"bytes": case["graphs"] * _update_bytes(1e6, mean) + case["read"] * view, "flops": 0}
    V, E = 1 << case["scale"], case["ef"] << case["scale"]
    if kind == "reads":
        deg = case["ef"]
        return {"bytes": case["lists"] * deg * 14 + case["queries"] * 12 + case["seeds"] * deg * 12 + 4 * V, "flops": 0}
    if kind == "analytics":
        return {"bytes": case["iterations"] * (E * 8 + V * 16) + E * 8 + V * 4, "flops": case["iterations"] * E}
    return {"bytes": E * 9 + 2 * (E + V) * 9 + (E + V) * 14 + 4 * V, "flops": 0}


def exact(case, seed):
    """PageRank as float64 tensors give it; the other kinds return whole
    numbers only."""
    if case["kind"] != "analytics":
        return None
    gen = _gen(seed)
    V = 1 << case["scale"]
    e = _edges(gen, case["scale"], case["ef"])
    src, dst = e >> SRC, (e >> DST) & 0x3FFFFF
    deg = torch.bincount(src, minlength=V).to(torch.float64)
    rank = torch.full((V,), 1.0 / V, dtype=torch.float64, device=DEV)
    for _ in range(case["iterations"]):
        contrib = torch.where(deg > 0, rank / deg.clamp(min=1), torch.zeros_like(rank))
        acc = torch.zeros(V, dtype=torch.float64, device=DEV).index_add_(0, dst, contrib[src])
        rank = (1 - 0.85) / V + 0.85 * (acc + rank[deg == 0].sum() / V)
    return {"rank": rank, "dist": None, "levels": None, "reached": None}
