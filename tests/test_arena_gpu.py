"""The H2H arena grows in place (virtual memory mapped at its end) and gives
its free tail back under memory pressure. Growth-heavy batch sequences are
checked against the CPU oracle after every batch, with and without a tight
device-memory budget on the context."""
import numpy as np
import pytest

from tests.helpers import csr
from tests.test_dynamic_gpu import Mirror, random_rows

pytestmark = pytest.mark.gpu


def grow_sequence(g, mirror, rng, n_nodes, batches, n_ins, n_del, kmax):
    """Applies the batches; returns how many succeeded before an error (and
    the error, or None). Every successful batch is checked in full."""
    from ipdps26_b200._lib import HmError

    try:
        total = g.count_static30().astype(np.int64)
    except HmError as e:
        return 0, e
    assert total.tolist() == mirror.counts(n_nodes).astype(np.int64).tolist()
    for step in range(batches):
        live = np.array(sorted(mirror.rows), dtype=np.uint32)
        dels = sorted(rng.choice(live, size=min(n_del, len(live)), replace=False).tolist())
        ins_rows = random_rows(rng, n_ins, n_nodes, kmax)
        io, im = csr(ins_rows)
        try:
            ids, delta = g.apply_batch(dels, io, im)
            full = g.count_static30().astype(np.int64)
        except HmError as e:
            return step, e
        want_ids = mirror.apply(dels, ins_rows)
        assert ids.tolist() == want_ids
        want = mirror.counts(n_nodes).astype(np.int64)
        assert full.tolist() == want.tolist(), f"batch {step}"
        assert (total + delta).tolist() == full.tolist(), f"batch {step}: delta"
        total = full
    return batches, None


def test_arena_grows_in_place(ctx):
    from ipdps26_b200 import engine

    rng = np.random.default_rng(11)
    n_nodes = 1000
    rows = random_rows(rng, 6000, n_nodes, 6)
    mirror = Mirror(rows)
    off, mem = csr(rows)
    with engine.Graph(ctx, off, mem, n_nodes) as g:
        a0 = g.info().n_adjacent
        done, err = grow_sequence(g, mirror, rng, n_nodes, batches=6, n_ins=1500, n_del=200, kmax=6)
        assert err is None and done == 6
        assert g.info().n_adjacent > 2 * a0  # the arena had to grow several times


@pytest.mark.parametrize("factor", [1.5, 2.5, 4.0, 16.0])
def test_tight_budget_trims_or_fails_cleanly(factor):
    """Contexts whose budget leaves little room over the built store: the
    arena grows lean, the oriented copy is built after giving back the
    arena's free tail, and a batch that cannot fit fails with HM_ERR_NOMEM
    instead of faulting. Every batch that succeeds is exact, and with room
    enough every batch succeeds."""
    from ipdps26_b200 import engine
    from ipdps26_b200._lib import HM_ERR_NOMEM

    rng = np.random.default_rng(12)
    n_nodes = 800
    rows = random_rows(rng, 5000, n_nodes, 6)
    off, mem = csr(rows)
    with engine.Context(0) as probe:
        with engine.Graph(probe, off, mem, n_nodes) as g:
            g.count_static30()
            used = probe.memory()[0]
    with engine.Context(0, mem_budget_bytes=int(used * factor)) as tight:
        mirror = Mirror(rows)
        try:
            g = engine.Graph(tight, off, mem, n_nodes)
        except Exception as e:  # the store itself may not fit the smallest budgets
            assert getattr(e, "status", None) == HM_ERR_NOMEM, str(e)
            return
        with g:
            done, err = grow_sequence(g, mirror, rng, n_nodes, batches=6, n_ins=1500, n_del=100, kmax=6)
        if err is not None:
            assert err.status == HM_ERR_NOMEM, str(err)
        if factor >= 16.0:
            assert done == 6, str(err)


def test_pooled_arena_moves_to_chunks_under_every_budget():
    """A small store's arena starts in the context's pool and moves to mapped
    chunks when it grows: in one piece while the budget holds both copies,
    through host memory while it does not. Over budgets from the built store's
    own bytes upwards a batch either fails with HM_ERR_NOMEM or leaves exactly
    the store of an unlimited budget, and it succeeds from some budget on."""
    from ipdps26_b200 import engine
    from ipdps26_b200._lib import HM_ERR_NOMEM, HmError

    rng = np.random.default_rng(13)
    n_nodes = 64
    off, mem = csr([sorted(rng.choice(n_nodes, size=4, replace=False).tolist()) for _ in range(2500)])
    io, im = csr([sorted(rng.choice(n_nodes, size=4, replace=False).tolist()) for _ in range(2500)])

    def run(c):
        with engine.Graph(c, off, mem, n_nodes) as g:
            used = c.memory()[0]
            _, delta = g.apply_batch([], io, im)
            return used, g.info().n_adjacent, g.count_static30().tolist(), delta.tolist()

    with engine.Context(0) as free:
        used, *want = run(free)
    passed = []
    for mb in range(0, 513, 16):
        with engine.Context(0, mem_budget_bytes=int(used + (mb << 20))) as tight:
            try:
                passed.append(list(run(tight)[1:]) == want)
            except HmError as e:
                assert e.status == HM_ERR_NOMEM, str(e)
                assert mb < 512, str(e)
    assert passed and all(passed)


def test_rows_by_bitmaps_or_sorted(ctx):
    """The two ways adjacency rows are built: on both sides of the slot limit the
    same store, and a store of many short rows sorted, short batches into it by
    bitmaps, against the oracle."""
    from ipdps26_b200 import engine, gen
    from oracle import oracle

    n = 113 << 10
    h = gen.static(gen.params(3, n // 2, n, 2, 25, 2.5, 1.2, 1000.0))
    with engine.Graph(ctx, h.offsets, h.members, h.n_nodes + 1) as g:
        assert g.routes().rows_bitmap
        want = g.info().n_adjacent, g.count_static30().tolist()
    off, mem = np.append(h.offsets, h.offsets[-1] + 1).astype(np.uint64), np.append(h.members, h.n_nodes).astype(np.uint32)
    with engine.Graph(ctx, off, mem, h.n_nodes + 1) as g:  # one more hyperedge, apart from the others
        assert not g.routes().rows_bitmap
        assert (g.info().n_adjacent, g.count_static30().tolist()) == want

    rng = np.random.default_rng(15)
    rows = [sorted(6 * (k // 5) + rng.choice(6, size=3, replace=False)) for k in range(40_000)]
    n_nodes = 6 * 8_000
    off, mem = csr(rows)
    with engine.Graph(ctx, off, mem, n_nodes) as g:
        assert not g.routes().rows_bitmap
        before = g.count_static30()
        assert before.tolist() == oracle.static30(off, mem, n_nodes).tolist()
        new = rows[100:400]
        io, im = csr(new)
        _, delta = g.apply_batch(list(range(50)), io, im)
        assert g.routes().rows_bitmap
        off, mem = csr(rows[50:] + new)
        want = oracle.static30(off, mem, n_nodes)
        assert g.count_static30().tolist() == want.tolist()
        assert (before.astype(np.int64) + delta).tolist() == want.astype(np.int64).tolist()


def test_growth_of_a_pooled_arena_fails_whole():
    """Every allocation of a batch that grows a pooled arena fails in turn. The
    batch then ends in HM_ERR_NOMEM or, where the growth was optional, in the
    store of an undisturbed one; the budget's account returns to nothing when
    the graph goes, and the context's next graph is whole."""
    from ipdps26_b200 import engine
    from ipdps26_b200._lib import HM_ERR_NOMEM, HmError, lib

    rng = np.random.default_rng(14)
    n_nodes = 64
    off, mem = csr([sorted(rng.choice(n_nodes, size=4, replace=False).tolist()) for _ in range(2000)])
    io, im = csr([sorted(rng.choice(n_nodes, size=4, replace=False).tolist()) for _ in range(1500)])
    dels = list(range(0, 400, 2))
    with engine.Context(0) as c:

        def run(n):
            with engine.Graph(c, off, mem, n_nodes) as g:
                lib.hm_debug_fail_allocations_after(n)
                try:
                    ids, delta = g.apply_batch(dels, io, im)
                finally:
                    lib.hm_debug_fail_allocations_after(-1)
                return ids.tolist(), delta.tolist(), g.info().n_adjacent, g.count_static30().tolist()

        want = run(-1)
        failed, step = 0, 0
        while step < 2000:
            try:
                got = run(step)
                assert got == want, step
                break  # no allocation left to fail
            except HmError as e:
                assert e.status == HM_ERR_NOMEM, f"{step}: {e}"
                failed += 1
            assert c.memory()[0] == 0, step
            step += 1
        assert failed > 20 and got == want
        assert run(-1) == want


@pytest.mark.parametrize("members", [3, 12])
def test_built_rows_leave_no_holes(ctx, members):
    """Bitmap rows lie one after another, so what the wedge bound reserves past
    them is free for a first batch (of rows taken by warps, and by blocks)."""
    from ipdps26_b200 import engine

    rng = np.random.default_rng(16)
    n, n_nodes = 1200, 40  # most pairs share members: far more wedges than entries
    off, mem = csr([sorted(rng.choice(n_nodes, size=members, replace=False).tolist()) for _ in range(n)])
    with engine.Graph(ctx, off, mem, n_nodes) as g:
        r = g.routes()
        assert r.rows_bitmap and r.arena_tail == r.arena_entries == g.info().n_adjacent
        assert r.arena_capacity > r.arena_tail


def test_small_arenas_stay_lean_in_a_full_context():
    """A small store's arena keeps several times its rows free while the context
    has plenty of room, and half of them once it does not, so that a context
    holds as many updated stores as fit by their rows."""
    from ipdps26_b200 import engine

    rng = np.random.default_rng(17)
    n_nodes = 64
    off, mem = csr([sorted(rng.choice(n_nodes, size=4, replace=False).tolist()) for _ in range(1500)])
    io, im = csr([sorted(rng.choice(n_nodes, size=4, replace=False).tolist()) for _ in range(500)])
    granules = 3 * (2 << 20) / 13  # of the three arrays
    graphs, free = [], []
    with engine.Context(0, mem_budget_bytes=800 << 20) as c:
        for _ in range(14):
            g = engine.Graph(c, off, mem, n_nodes)
            g.apply_batch([], io, im)
            graphs.append(g)
            r = g.routes()
            free.append((r.arena_capacity - 1.5 * r.arena_entries, c.memory()[0] > 150 << 20))
        assert free[0][0] > r.arena_entries and not free[0][1]
        lean = [f for f, full in free if full]
        assert len(lean) > 4 and max(lean) <= granules, free
        for g in graphs:
            g.close()
