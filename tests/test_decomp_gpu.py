"""The static count by decomposition (light pairs in closed form, triangles with
two or three heavy pairs enumerated) at the sizes where its kernels change:
position masks of 32 and 64 members, centres above 64, tables indexed by rank
and hashed, short and long heavy rows, spread owners, and graphs it leaves to
the enumeration of all triangles. Exact integers, so equality."""
import numpy as np
import pytest

from oracle import oracle
from tests.helpers import csr

pytestmark = pytest.mark.gpu


def _rows(rng, n, n_nodes, sizes, hubs=0, n_hubs=6):
    """n hyperedges with the given sizes; `hubs` of each one's members come
    from n_hubs shared nodes (overlaps of two or more)."""
    out = []
    for _ in range(n):
        k = int(rng.choice(sizes))
        h = min(k, hubs)
        r = set(rng.choice(n_hubs, size=min(h, n_hubs), replace=False).tolist())
        while len(r) < k:
            r.add(int(rng.integers(0, n_nodes)))
        out.append(sorted(r))
    return out


CASES = {
    # sizes, hub members per hyperedge, hubs, hyperedges, nodes
    "sizes-1-to-4": ([1, 2, 3, 4], 1, 40, 900, 300),
    "masks-31-32-33": ([2, 3, 31, 32, 33], 2, 12, 260, 220),
    "masks-63-64-65": ([2, 4, 63, 64, 65], 2, 20, 220, 400),
    "centres-above-64": ([66, 90, 130, 255], 3, 30, 120, 900),
    "overlaps-past-3": ([6, 7, 8, 9, 10], 5, 9, 300, 60),
    "rows-of-95-96-97": ([3, 4], 2, 8, 420, 4000),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("seed", range(3))
def test_decomposition_matches_oracle(ctx, name, seed):
    from ipdps26_b200 import engine

    sizes, hubs, n_hubs, n, n_nodes = CASES[name]
    rng = np.random.default_rng(1000 + seed)
    rows = _rows(rng, n, n_nodes, sizes, hubs, n_hubs) + [[0], [0, 1], [1, 2], [0, 1, 2]]
    off, mem = csr(rows)
    want = oracle.static30(off, mem, n_nodes)
    with engine.Graph(ctx, off, mem, n_nodes) as g:
        assert g.count_static30().tolist() == want.tolist()
        g.set_static_groups(False)
        assert g.count_static30().tolist() == want.tolist()
        g.set_static_groups(True)
        assert g.count_static30().tolist() == want.tolist()


@pytest.mark.parametrize("n,law", [(12_287, "small"), (12_288, "small"), (12_289, "small"), (20_000, "wide"),
                                   (12_000, "wide")])
def test_decomposition_equals_enumeration(ctx, n, law):
    """Graphs on both sides of the rank-indexed table's limit, one of them with
    owners that spread their pairs over a node vector; and after an update."""
    from ipdps26_b200 import engine, gen

    p = (gen.params(n, n // 2, n, 2, 25, 2.5, 1.2, 60.0) if law == "small"
         else gen.config2(seed=n, n_nodes=n // 2, n_edges=n, q=10.0))
    h = gen.static(p)
    with engine.Graph.from_hypergraph(ctx, h) as g:
        for _ in range(2):
            got = g.count_static30()
            g.set_static_groups(False)
            assert got.tolist() == g.count_static30().tolist()
            g.set_static_groups(True)
            dels, ins = gen.batch(p, 5, g.live_ids(), 200)
            _, delta = g.apply_batch(dels, ins.offsets, ins.members)
            after = g.count_static30()
            assert (got.astype(np.int64) + delta).tolist() == after.astype(np.int64).tolist()


def test_all_pairs_heavy_is_enumerated(ctx):
    """Every pair shares two nodes: the decomposition would enumerate more than
    the enumeration does, and is not taken."""
    from ipdps26_b200 import engine

    rng = np.random.default_rng(3)
    rows = [[0, 1] + sorted(rng.choice(np.arange(2, 200), size=int(rng.integers(0, 4)), replace=False).tolist())
            for _ in range(400)]
    off, mem = csr(rows)
    with engine.Graph(ctx, off, mem, 200) as g:
        assert g.count_static30().tolist() == oracle.static30(off, mem, 200).tolist()


def _touch_law(name, seed):
    from ipdps26_b200 import gen

    if name == "hub":
        return gen.config1(seed=seed, n_nodes=1500, n_edges=3000), 3000
    if name == "wide":
        return gen.config2(seed=seed, n_nodes=3000, n_edges=6000, q=3.0), 6000
    return gen.params(seed, 600, 3000, 20, 110, 1.1, 1.1, 40.0), 3000  # "large": most centres above 32 members


@pytest.mark.parametrize("law", ["hub", "wide", "large"])
@pytest.mark.parametrize("marked", [400, 1500])
def test_touched_triples_by_decomposition(ctx, law, marked):
    """Batches whose touched-triple counts are large enough to go by the
    decomposition: the count of a marked set equals the walk of id-ordered rows
    (other kernels), marking everything gives the full count, and an update's
    delta equals the difference of two full counts."""
    from ipdps26_b200 import engine, gen

    p, n = _touch_law(law, 7 + marked)
    h = gen.static(p)
    rng = np.random.default_rng(marked)
    ids = np.sort(rng.choice(n, size=marked, replace=False)).astype(np.uint32)
    with engine.Graph.from_hypergraph(ctx, h) as g:
        got = g.count_touching30(ids)
        g.set_touch_orientation(True)
        assert got.tolist() == g.count_touching30(ids).tolist()
        g.set_touch_orientation(False)
        full = g.count_static30()
        assert g.count_touching30(np.arange(n, dtype=np.uint32)).tolist() == full.tolist()
        dels, ins = gen.batch(p, 3, g.live_ids(), marked)
        _, delta = g.apply_batch(dels, ins.offsets, ins.members)
        assert (full.astype(np.int64) + delta).tolist() == g.count_static30().astype(np.int64).tolist()


def _cliques(rng, sizes, n_free):
    """Hyperedges in groups that share two nodes of their own (all pairs of a
    group heavy), each with one of n_free common nodes (light pairs, and closed
    triangles of all kinds)."""
    rows, node = [], n_free
    for k in sizes:
        rows += [sorted([int(rng.integers(0, n_free)), node, node + 1]) for _ in range(k)]
        node += 2
    return rows, node


# Searched pair by pair up to 2^13 heavy entries and a sum of squared heavy
# degrees of 2^18, by centre beyond.
@pytest.mark.parametrize("sizes", [[], [2], [9] * 113 + [2] * 28, [9] * 113 + [2] * 29,
                                   [64] + [9] * 14 + [2] * 32, [64] + [9] * 14 + [2] * 33],
                         ids=["none", "one-pair", "entries-2^13", "entries-past", "tests-2^18", "tests-past"])
def test_few_heavy_pairs_searched_by_entry(ctx, sizes):
    from ipdps26_b200 import engine

    rng = np.random.default_rng(len(sizes))
    rows, n_nodes = _cliques(rng, sizes + [1] * 200, 10)
    off, mem = csr(rows)
    with engine.Graph(ctx, off, mem, n_nodes) as g:
        want = oracle.static30(off, mem, n_nodes).tolist()
        assert g.count_static30().tolist() == want
        assert g.count_static30().tolist() == want  # replayed


@pytest.mark.parametrize("groups", [20, 200])
@pytest.mark.parametrize("marked", [1, 400, 1500])
def test_touched_triples_of_few_heavy_pairs(ctx, groups, marked):
    """Marked sets in graphs searched by entry, with several warps on a pair
    (two hubs hold everything, so 400 marks or more go by the decomposition)."""
    from ipdps26_b200 import engine

    rng = np.random.default_rng(groups + marked)
    rows, n_nodes = _cliques(rng, [4] * groups + [1] * (3000 - 4 * groups), 2)
    off, mem = csr(rows)
    ids = np.sort(rng.choice(3000, size=marked, replace=False)).astype(np.uint32)
    rest_off, rest_mem = csr([r for k, r in enumerate(rows) if k not in set(ids.tolist())])
    with engine.Graph(ctx, off, mem, n_nodes) as g, engine.Graph(ctx, rest_off, rest_mem, n_nodes) as rest:
        got = g.count_touching30(ids)
        assert got.tolist() == (g.count_static30() - rest.count_static30()).tolist()
        g.set_touch_orientation(True)
        assert got.tolist() == g.count_touching30(ids).tolist()


def _core(rng, n, n_nodes, sizes, hubs, n_hubs, light, pad):
    """A heavy core (n hyperedges, each with `hubs` members out of n_hubs shared
    nodes) in a graph whose pairs are mostly light: `light` hyperedges meet in
    one node, which a third of the core holds too, so that the core goes by the
    decomposition; `pad` hyperedges apart from all others take slots only."""
    hub, rows = n_nodes, []
    for k in range(n):
        s = int(rng.choice(sizes))
        r = set(rng.choice(n_hubs, size=min(hubs, s, n_hubs), replace=False).tolist())
        if k % 3 == 0 and len(r) < s:
            r.add(hub)
        while len(r) < s:
            r.add(int(rng.integers(0, n_nodes)))
        rows.append(sorted(r))
    rows += [[hub, hub + 1 + i] for i in range(light)]
    free = hub + 1 + light
    rows += [[free + 2 * i, free + 2 * i + 1] for i in range(pad)]
    return rows, free + 2 * pad


# name: sizes, hub members, hubs, core hyperedges, nodes, light hyperedges, launch shapes that have to run
CORES = {
    "masks-31-32-33": ([2, 3, 31, 32, 33], 2, 12, 260, 220, 500, (1, 2)),
    "masks-63-64-65": ([2, 4, 63, 64, 65], 2, 20, 220, 400, 500, (1, 2, 3)),
    "centres-above-64": ([4, 40, 66, 90, 130, 255], 3, 30, 160, 900, 500, (1, 2, 3)),
    "overlaps-past-3": ([6, 7, 8, 9, 10], 5, 9, 300, 60, 700, (1,)),
    "rows-around-96": ([3, 4], 2, 8, 800, 4000, 900, (0, 1)),
}


@pytest.mark.parametrize("name", sorted(CORES))
@pytest.mark.parametrize("pad", [0, 12_300], ids=["by-rank", "hashed"])
@pytest.mark.parametrize("seed", range(2))
def test_heavy_core_runs_its_kernels(ctx, name, pad, seed):
    """The edges of the table kernels: the launch shapes named above are the ones
    that ran."""
    from ipdps26_b200 import engine

    *law, shapes = CORES[name]
    sizes, hubs, n_hubs, n, n_nodes, light = law
    rows, n_all = _core(np.random.default_rng(50 + seed), n, n_nodes, sizes, hubs, n_hubs, light, pad)
    off, mem = csr(rows)
    with engine.Graph(ctx, off, mem, n_all) as g:
        g.set_static_groups(2)  # whatever its node graph costs
        got = g.count_static30()
        r = g.routes()
        assert r.static_decomposed and not r.static_by_entry
        assert all(r.static_centres[k] for k in shapes), list(r.static_centres)
        assert r.static_spread or name != "centres-above-64"
        assert got.tolist() == oracle.static30(off, mem, n_all).tolist()
        g.set_static_groups(False)
        assert got.tolist() == g.count_static30().tolist()
        assert not g.routes().static_decomposed


@pytest.mark.parametrize("seed", range(2))
def test_large_centres_searched_by_entry(ctx, seed):
    """Few heavy pairs, most of centres above 64 members: the triple overlap of
    each by merging the three lists."""
    from ipdps26_b200 import engine

    rows, n_all = _core(np.random.default_rng(70 + seed), 40, 900, [65, 66, 101, 180, 255], 3, 20, 300, 0)
    off, mem = csr(rows)
    with engine.Graph(ctx, off, mem, n_all) as g:
        g.set_static_groups(2)
        got = g.count_static30()
        assert g.routes().static_decomposed and g.routes().static_by_entry
        assert got.tolist() == oracle.static30(off, mem, n_all).tolist()


@pytest.mark.parametrize("name", sorted(CORES))
@pytest.mark.parametrize("pad", [0, 12_300], ids=["by-rank", "hashed"])
def test_touched_triples_of_a_heavy_core(ctx, name, pad):
    """The same kernels with marks: half of the core and most light hyperedges
    are marked, and the count is the full one minus that of the rest."""
    from ipdps26_b200 import engine

    sizes, hubs, n_hubs, n, n_nodes, _, shapes = CORES[name]
    rng = np.random.default_rng(90)
    rows, n_all = _core(rng, n, n_nodes, sizes, hubs, n_hubs, 700, pad)
    ids = np.sort(np.concatenate([rng.choice(n, size=n // 2, replace=False), np.arange(n, n + 650)])).astype(np.uint32)
    off, mem = csr(rows)
    rest_off, rest_mem = csr([r for k, r in enumerate(rows) if k not in set(ids.tolist())])
    with engine.Graph(ctx, off, mem, n_all) as g:
        g.set_static_groups(2)
        got = g.count_touching30(ids)
        r = g.routes()
        assert r.touch_decomposed and not r.touch_by_entry
        assert all(r.touch_centres[k] for k in shapes if k), list(r.touch_centres)
        want = oracle.static30(off, mem, n_all) - oracle.static30(rest_off, rest_mem, n_all)
        assert got.tolist() == want.tolist()
        g.set_touch_orientation(True)
        assert got.tolist() == g.count_touching30(ids).tolist()
        assert not g.routes().touch_decomposed


def test_rows_past_the_largest_table(ctx):
    """Hub rows of more than 12,288 higher-ranked neighbours (searched), of more
    than 3,072 (large tables), and shorter ones, against the enumeration."""
    from ipdps26_b200 import engine, gen

    n = 16_000
    with engine.Graph.from_hypergraph(ctx, gen.static(gen.config1(seed=4, n_nodes=n // 2, n_edges=n))) as g:
        got = g.count_static30()
        r = g.routes()
        assert r.static_decomposed and r.static_centres[0] and r.static_centres[1] and r.static_centres[3]
        g.set_static_groups(False)
        assert got.tolist() == g.count_static30().tolist()


def _uniform(n, lo, hi, n_nodes):
    rng = np.random.default_rng(n + hi)
    z = rng.integers(lo, hi + 1, n)
    off = np.concatenate([[0], np.cumsum(z)]).astype(np.uint64)
    return off, rng.integers(0, n_nodes, int(off[-1])).astype(np.uint32), n_nodes


@pytest.mark.parametrize("law,static,touched", [
    ((20_000, 60, 100, 2_000_000), False, False),  # large hyperedges, seldom adjacent: refused before the table
    ((20_000, 20, 40, 20_000), False, False),      # refused by the node graph's own size
    ((3_000, 30, 60, 3_000), False, False),
    ((20_000, 8, 16, 10_000), True, True),
    ((30_000, 3, 6, 3_000), True, True),
    ((20_000, 2, 4, 1_000_000), False, False),
    ("hub", True, True),
    ("large", False, False),                       # a hyperedge of 120 members, alone on a warp for most of the count
], ids=str)
def test_closed_forms_where_their_node_graph_is_worth_it(ctx, law, static, touched):
    """The dispatch weighs the node graph's walk against the enumeration, and for
    touched triples against the walk of the marked rows (half of the graph
    marked); both ways give the same counts."""
    from ipdps26_b200 import engine, gen

    if law == "hub":
        h = gen.static(gen.config1(seed=2, n_nodes=2_000, n_edges=4_000))
        off, mem, n_nodes = h.offsets, h.members, h.n_nodes
    elif law == "large":
        h = gen.static(gen.params(50_140, 6_214, 3_458, 1, 200, 2.543, 0.988, 50.0, dedupe=True))
        off, mem, n_nodes = h.offsets, h.members, h.n_nodes
    else:
        off, mem, n_nodes = _uniform(*law)
    n = len(off) - 1
    ids = np.arange(0, n, 2, dtype=np.uint32)
    with engine.Graph(ctx, off, mem, n_nodes) as g:
        got = g.count_static30(), g.count_touching30(ids)
        r = g.routes()
        assert (bool(r.static_decomposed), bool(r.touch_decomposed)) == (static, touched)
        g.set_static_groups(0 if static else 2)
        if static or law == "large" or law[1] < 40:  # the closed forms of the largest take tens of milliseconds and 3 GB
            assert g.count_static30().tolist() == got[0].tolist()
        g.set_static_groups(2)
        g.set_touch_orientation(touched)
        if touched or law == "large" or law[1] < 40:
            assert g.count_touching30(ids).tolist() == got[1].tolist()
            assert bool(g.routes().touch_decomposed) != touched


def test_refused_for_room_is_looked_at_again():
    """A count without room for the closed forms (7 MB of tables, which may take
    half of the room) enumerates, and takes them once the context has the room; a
    batch or a rebuild is not needed."""
    from ipdps26_b200 import engine, gen

    h, other = (gen.static(gen.params(s, 4_000, 8_000, 2, 25, 2.5, 1.2, 1000.0)) for s in (6, 7))
    with engine.Context(0) as c:
        with engine.Graph.from_hypergraph(c, h), engine.Graph.from_hypergraph(c, other):
            used = c.memory()[0]
    with engine.Context(0, mem_budget_bytes=used + (11 << 20)) as c:
        b = engine.Graph.from_hypergraph(c, other)
        with engine.Graph.from_hypergraph(c, h) as g:
            want = g.count_static30().tolist()
            assert not g.routes().static_decomposed
            assert g.count_static30().tolist() == want
            assert not g.routes().static_decomposed
            b.close()
            assert g.count_static30().tolist() == want
            assert g.routes().static_decomposed


def test_closed_forms_take_the_grouped_rows_place(ctx):
    """After tuning (which walks the grouped rows) a full count by closed forms
    gives the grouped rows' memory back."""
    from ipdps26_b200 import engine, gen

    h = gen.static(gen.config1(seed=8, n_nodes=2_000, n_edges=4_000))
    used = lambda: ctx.memory()[0]
    with engine.Graph.from_hypergraph(ctx, h) as g:
        base = used()
        g.count_static30()
        closed = used() - base
    with engine.Graph.from_hypergraph(ctx, h) as g:
        base = used()
        g.autotune()
        tuned = used() - base
        g.count_static30()
        assert g.routes().static_decomposed
        both = used() - base
        oriented = 7 * g.info().n_oriented  # bytes of the grouped rows per oriented entry
        assert both <= tuned + closed - oriented
        g.count_static30_shard(0, 2)  # walks them again, and keeps the closed forms
        assert used() - base >= both + oriented
        g.count_static30()
        assert used() - base >= both + oriented


def test_sharded_counts_have_the_room_they_had():
    """Budgets that hold a store and its oriented rows: sharded counts succeed
    after a full count wherever they do before one."""
    from ipdps26_b200 import engine, gen
    from ipdps26_b200._lib import HM_ERR_NOMEM, HmError

    h = gen.static(gen.config1(seed=9, n_nodes=3_000, n_edges=6_000))

    def run(budget, full):
        with engine.Context(0, mem_budget_bytes=budget) as c:
            try:
                with engine.Graph.from_hypergraph(c, h) as g:
                    if full:
                        g.count_static30()
                    return (g.count_static30_shard(0, 2) + g.count_static30_shard(1, 2)).tolist()
            except HmError as e:
                assert e.status == HM_ERR_NOMEM, str(e)
                return None

    with engine.Context(0) as c:
        with engine.Graph.from_hypergraph(c, h) as g:
            store, want = c.memory()[0], g.count_static30().tolist()
    seen = 0
    for mb in range(0, 400, 10):
        first, after = run(store + (mb << 20), False), run(store + (mb << 20), True)
        assert first in (None, want) and after in (None, want)
        assert first is None or after is not None, mb
        seen += first is not None
    assert seen
