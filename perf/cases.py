"""The work a user has the engine do, as measurable cases.

Each case names one use of the engine by its path, its workload law and its
sizes; `prepare` makes what a user's program holds before the call (host
arrays, a resident graph, a server), `run` is one pass through the public
entry points. The laws are the package's own named workloads at other sizes:

  small   sizes k^-2.5 on [2, 25], Zipf-Mandelbrot(1.2, q = 1000), two
          hyperedges per node: the graphs of the served workload
  hub     sizes k^-2.5 on [2, 25], plain Zipf(1.2): the node-popularity law
          of the CPU-sized static workload, a few hub nodes in most hyperedges
  wide    sizes k^-2.2 on [2, 100], Zipf-Mandelbrot(1.1) with q in proportion
          to the size: the laws of the 2M-hyperedge static workload
"""
import math

import numpy as np

from ipdps26_b200 import engine, gen, workloads

_CTX = []


def _context():
    """One context for the resident graphs, as one program holds it."""
    if not _CTX:
        _CTX.append(engine.Context(0))
    return _CTX[0]


def _law(law, edges, seed):
    if law == "small":
        return gen.params(seed, max(edges // 2, 2), edges, 2, 25, 2.5, 1.2, gen.C5_Q)
    if law == "hub":
        return gen.config1(seed=seed, n_nodes=max(edges // 2, 30), n_edges=edges)
    return gen.from_laws(workloads.config2_laws(edges, max(edges // 2, 110)).scaled(seed=seed))


def _events(edges, seed):
    """The bursty event stream with the full workload's events per time unit."""
    B = workloads.CONFIG4_BURSTS
    p = gen.config4(seed=seed, n_nodes=max(edges * 2 // 5, 30), n_edges=edges)
    return gen.temporal(p, B.burst_rate, B.events_per_burst, B.gap_mean, 200 * edges)


def listed():
    return [
        # A full 26-motif count of one resident graph: the smallest and a
        # large one of those a server keeps.
        {"name": "static-small-1k", "path": "static", "law": "small", "edges": 1_000},
        {"name": "static-small-100k", "path": "static", "law": "small", "edges": 100_003},
        # The same where a few hubs sit in most hyperedges.
        {"name": "static-hub-8k", "path": "static", "law": "hub", "edges": 8_000},
        # The 2M-hyperedge workload's laws at a size counted in a fraction of
        # a second.
        {"name": "static-wide-60k", "path": "static", "law": "wide", "edges": 60_000},
        # Host arrays in, counts out: a graph counted once.
        {"name": "build-count-small-20k", "path": "build", "law": "small", "edges": 20_000},
        # Update batches with their exact delta: a few hundred edits on a
        # served graph, and a large batch on a wide one. Each pass applies a
        # batch (80 % insertions) and the one that undoes it.
        {"name": "update-small-20k-300", "path": "update", "law": "small", "edges": 20_000, "edits": 300},
        {"name": "update-wide-50k-4k", "path": "update", "law": "wide", "edges": 50_021, "edits": 4_000},
        # 96 temporal motifs: a short stream, a long one under a narrow
        # window, one under a wide window.
        {"name": "temporal-2k-1e4", "path": "temporal", "edges": 2_000, "delta": 10_000},
        {"name": "temporal-200k-1e3", "path": "temporal", "edges": 200_000, "delta": 1_000},
        {"name": "temporal-30k-1e5", "path": "temporal", "edges": 30_000, "delta": 100_000},
        # A round of mixed requests to the server: an update of every graph,
        # full counts of some, the updates undone.
        {"name": "serve-24", "path": "serve", "law": "small", "graphs": 24, "edges": 2_000, "edits": 200},
        # A sliding three-layer window: rotate, new newest layer, count.
        {"name": "window-5k", "path": "window", "law": "small", "edges": 5_000},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["static", "static", "static", "build", "update", "update", "temporal", "temporal", "temporal",
                       "serve", "window"])
    if path == "temporal":
        delta = _spread(rng, 1_000, 100_000)
        return {"path": path, "edges": _spread(rng, 2_000, min(200_000, 3_000_000_000 // delta)), "delta": delta}
    if path == "serve":
        return {"path": path, "law": "small", "graphs": rng.randint(4, 24), "edges": _spread(rng, 1_000, 2_000),
                "edits": _spread(rng, 100, 200)}
    if path == "window":
        return {"path": path, "law": "small", "edges": _spread(rng, 300, 5_000)}
    law = rng.choice(["small", "small", "hub", "wide"])
    most = {"small": 100_000, "hub": 8_000, "wide": 60_000 if path == "static" else 50_000}[law]
    c = {"path": path, "law": law, "edges": _spread(rng, 1_000, most)}
    if path == "update":
        c["edits"] = _spread(rng, 100, min(4_000, c["edges"] // 3))
    return c


def _batches(p, n_edges, edits, seed):
    """A batch (80 % insertions) and the members of its deletions, as one
    graph takes them."""
    host = gen.static(p)
    dels, ins = gen.batch(p, seed, np.arange(n_edges, dtype=np.uint32), edits)
    rows = [host.edge(int(d)) for d in dels]
    off = np.cumsum([0] + [len(r) for r in rows]).astype(np.uint64)
    mem = np.concatenate(rows) if rows else np.zeros(0, np.uint32)
    return host, dels, ins, off, mem


def prepare(case, seed):
    path, n = case["path"], case["edges"]
    s = {"path": path}
    if path == "temporal":
        s["graph"] = engine.Graph.from_hypergraph(_context(), _events(n, seed))
        s["delta"] = case["delta"]
        return s
    if path == "serve":
        ctx = engine.Context(0)
        s["ctx"], s["server"] = ctx, engine.Server(ctx)
        s["work"] = []
        for k in range(case["graphs"]):
            m = n + 97 * k  # graphs of uneven size
            host, dels, ins, off, mem = _batches(_law("small", m, 1000 * seed + k), m, case["edits"] + 11 * k, seed + k)
            gid = s["server"].add_graph(host.offsets, host.members, host.n_nodes)
            new = [int(d) for d in dels]  # the freed ids first, then new ones
            new += list(range(m, m + ins.n_edges - len(dels)))
            s["work"].append((gid, dels, ins, np.array(new, np.uint32), off, mem, k % 3 == 0))
        s["server"].start()
        return s
    p = _law(case["law"], n, seed)
    if path == "window":
        s["window"] = engine.Window(_context(), p.n_nodes)
        s["layers"] = [gen.static(_law(case["law"], n + 13 * k, 10 * seed + k)) for k in range(4)]
        for layer in (engine.OLDER, engine.MIDDLE, engine.NEWEST):
            h = s["layers"][layer]
            s["window"].set_layer(layer, h.offsets, h.members % p.n_nodes)
        s["layers"] = [(h.offsets, h.members % p.n_nodes) for h in s["layers"]]
        s["next"] = 3
        return s
    if path == "update":
        host, dels, ins, off, mem = _batches(p, n, case["edits"], seed)
        s["graph"] = engine.Graph.from_hypergraph(_context(), host)
        s["batch"], s["undo"] = (dels, ins.offsets, ins.members), (off, mem)
        return s
    s["host"] = gen.static(p)
    if path == "static":
        s["graph"] = engine.Graph.from_hypergraph(_context(), s["host"])
    return s


def run(s):
    path = s["path"]
    if path == "static":
        return s["graph"].count_static30()
    if path == "temporal":
        return s["graph"].count_temporal(s["delta"])
    if path == "build":
        h = s["host"]
        with engine.Graph(_context(), h.offsets, h.members, h.n_nodes) as g:
            return {"counts": g.count_static30(), "adjacent": g.info().n_adjacent}
    if path == "update":
        ids, delta = s["graph"].apply_batch(*s["batch"])
        ids_back, delta_back = s["graph"].apply_batch(ids, *s["undo"])
        return {"ids": ids, "delta": delta, "ids_back": ids_back, "delta_back": delta_back}
    if path == "window":
        w, k = s["window"], s["next"]
        w.rotate()
        w.set_layer(engine.NEWEST, *s["layers"][k])
        s["next"] = (k + 1) % len(s["layers"])
        return w.count30()
    server, tickets = s["server"], []
    for gid, dels, ins, new, off, mem, count in s["work"]:
        tickets.append(server.submit_update(gid, dels, ins.offsets, ins.members))
        if count:
            tickets.append(server.submit_count(gid))
    for gid, dels, ins, new, off, mem, count in s["work"]:
        tickets.append(server.submit_update(gid, new, off, mem))
    counts, deltas = [], []
    for t in tickets:
        r, _ = server.wait(t, 1 << 14)
        (counts if r.kind == engine.REQ_COUNT else deltas).append(list(r.counts30 if r.kind else r.delta30))
    return {"counts": np.array(counts, np.int64), "deltas": np.array(deltas, np.int64)}


_WORK = {}


def work(case):
    """Bytes of the inputs read once: the adjacency a count walks (neighbour
    and overlap, 5 bytes an entry, bounded by the wedges of the nodes) and the
    member lists; the time-ordered member lists for a temporal count."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _WORK:
        path, n = case["path"], case["edges"]
        if path == "temporal":
            h = _events(n, 1)
            # every event's window, walked once
            per_window = min(case["delta"] / 200.0, n)
            b = 4.0 * len(h.members) + 8.0 * n + 4.0 * len(h.members) * (1.0 + per_window / 8.0)
        else:
            h = gen.static(_law(case["law"], n, 1))
            deg = np.bincount(h.members, minlength=h.n_nodes).astype(np.float64)
            store = 5.0 * float((deg * (deg - 1)).sum()) + 4.0 * len(h.members)
            if path == "update":
                b = 2.0 * store * case["edits"] / n + 8.0 * len(h.members)
            elif path == "serve":
                b = case["graphs"] * (store / 3 + 2.0 * store * case["edits"] / n)
            else:
                b = store * (3 if path == "window" else 1)
        _WORK[key] = {"bytes": b, "flops": 0.0}
    return dict(_WORK[key])


def exact(case, seed):
    """The 30 static classes of a small graph by their definition, from dense
    0/1 incidence in plain numpy; None for the paths whose outputs are updates
    of state, and for graphs too large for it."""
    if case["path"] != "static" or case["edges"] > 1_200:
        return None
    h = gen.static(_law(case["law"], case["edges"], seed))
    n = h.n_edges
    M = np.zeros((n, h.n_nodes), np.float32)
    M[np.repeat(np.arange(n), np.diff(h.offsets).astype(np.int64)), h.members] = 1
    O = (M @ M.T).astype(np.int32)
    size = np.diag(O).copy()
    out = np.zeros(30, np.int64)
    for a in range(n):
        nb = np.flatnonzero(O[a])
        nb = nb[nb != a]
        if len(nb) < 2:
            continue
        own = h.edge(a)
        G = (M[np.ix_(nb, own)] @ M[np.ix_(nb, own)].T).astype(np.int32)
        i, j = np.triu_indices(len(nb), 1)
        b, c = nb[i], nb[j]
        # closed triples at their smallest hyperedge, open ones at their centre
        take = (O[b, c] == 0) | (a < b)
        b, c, g = b[take], c[take], G[i, j][take]
        ab, bc, ca = O[a, b], O[b, c], O[c, a]
        ex = [(x > 0).astype(np.int64) for x in (size[a] - ab - ca + g, size[b] - ab - bc + g, size[c] - bc - ca + g)]
        pr = [(x - g > 0).astype(np.int64) for x in (ab, bc, ca)]
        p, nex = pr[0] + pr[1] + pr[2], ex[0] + ex[1] + ex[2]
        hub = np.where((pr[2] & pr[0]) > 0, ex[0], np.where((pr[0] & pr[1]) > 0, ex[1], ex[2]))
        loner = np.where(pr[0] > 0, ex[2], np.where(pr[1] > 0, ex[0], ex[1]))
        pair = nex - loner
        one = 4 + np.where(loner > 0, np.where(pair == 0, 2, 3 + pair), np.where(pair == 2, 3, pair))
        two = hub + 2 * (nex - hub)
        k = np.where(p == 3, np.where(g > 0, 16, 26) + nex,
                     np.where(p == 2, np.where(g > 0, 10, 20) + two, np.where(p == 1, one, nex)))
        out += np.bincount(k, minlength=30)
    return out.astype(np.uint64)
