"""Contexts on threads of their own: the engine's kernels and their attributes
are shared by every context of the device, the contexts are not."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def _run(jobs):
    """Runs each job on a thread of its own; the first exception is raised."""
    errors = []

    def guarded(f):
        try:
            f()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(f,)) for f in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def _graph(n, seed):
    from ipdps26_b200 import gen

    p = gen.params(seed, max(n // 2, 30), n, 2, 6, 2.5, 1.2, 1000.0)
    return p, gen.static(p)


def test_contexts_build_stores_of_different_sizes_at_once():
    """The row builder's shared memory grows with a store's slots: small and
    large stores built at once by one context per thread."""
    from ipdps26_b200 import engine

    def builds(n, rounds):
        def job():
            _, h = _graph(n, 5)
            with engine.Context(0) as c:
                with engine.Graph.from_hypergraph(c, h) as g:
                    want = g.info().n_adjacent
                for _ in range(rounds):
                    with engine.Graph.from_hypergraph(c, h) as g:
                        assert g.info().n_adjacent == want

        return job

    _run([builds(1_000, 600) for _ in range(6)] + [builds(80_000, 150) for _ in range(3)])


def test_contexts_count_and_update_at_once():
    """Counts capture their launches while other contexts grow, release and
    destroy stores; each context's results are those of a lone one."""
    import numpy as np

    from ipdps26_b200 import engine, gen

    def rounds(n, seed, k, out):
        def job():
            p, h = _graph(n, seed)
            dels, ins = gen.batch(p, 9, np.arange(n, dtype=np.uint32), 60)
            with engine.Context(0) as c:
                for _ in range(k):
                    with engine.Graph.from_hypergraph(c, h) as g:
                        full = g.count_static30().astype(np.int64)
                        _, delta = g.apply_batch(dels, ins.offsets, ins.members)
                        after = g.count_static30().astype(np.int64)
                        assert (full + delta).tolist() == after.tolist()
                        out.append((full.tolist(), after.tolist()))

        return job

    sizes = [(1_000, 150), (80_000, 60), (30_000, 100)]
    got = [[] for _ in sizes]
    _run([rounds(n, 20 + k, r, got[k]) for k, (n, r) in enumerate(sizes)])
    for k, (n, r) in enumerate(sizes):
        alone = []
        rounds(n, 20 + k, 1, alone)()
        assert len(got[k]) == r and all(x == alone[0] for x in got[k])


def test_counts_while_the_program_waits_for_the_device():
    """A first count makes its graphs without capturing a stream, so a wait for
    the whole device on another thread neither fails nor disturbs it."""
    import torch

    from ipdps26_b200 import engine

    done = threading.Event()

    def waits():
        while not done.is_set():
            torch.cuda.synchronize()

    def counts():
        try:
            _, h = _graph(3_000, 31)
            with engine.Context(0) as c:
                want = None
                for _ in range(60):
                    with engine.Graph.from_hypergraph(c, h) as g:
                        for on in (True, False):  # either method
                            g.set_static_groups(on)
                            got = [g.count_static30().tolist() for _ in range(2)]
                            want = want or got[0]
                            assert got == [want, want]
        finally:
            done.set()

    _run([counts, waits])
