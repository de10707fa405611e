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
