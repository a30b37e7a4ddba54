"""Serving rounds inside one launch (needs a B200)."""
import time

import numpy as np
import pytest

import oracle
import xted
from xted import gen

pytestmark = pytest.mark.gpu

SHAPES = ("random", "wide", "deep", "caterpillar")


def _trees(n, seed, lo, hi):
    rng = np.random.default_rng(seed)
    return [gen.tree(SHAPES[i % 4], int(rng.integers(lo, hi + 1)), seed * 1000 + i, "zipf", 12) for i in range(n)]


def _check(ids, ds, q, corpus, k):
    d = oracle.distance_batch([(q, t) for t in corpus], nthreads=8)
    order = sorted(range(len(corpus)), key=lambda i: (d[i], i))[:k]
    assert ids.tolist() == order and ds.tolist() == [int(d[i]) for i in order]


@pytest.mark.timeout(300)
def test_second_round_joins_the_running_launch():
    """Queries one after another, each with a second round: the tables are
    cleared by the launch itself, so a round need not wait for its end (it did,
    and every query took two launches)."""
    corpus, queries = _trees(300, 5, 20, 90), _trees(24, 6, 20, 90)
    with xted.Context() as ctx:
        ctx.corpus_load(corpus)
        for q in queries[:4]:
            ctx.query_wait(ctx.query_submit(q, 5), timeout_s=60)
        before = ctx.serve_stats()
        for q in queries[4:]:
            t = ctx.query_submit(q, 5)
            ids, ds, _, _ = ctx.query_wait(t, timeout_s=60)
            _check(ids, ds, q, corpus, 5)
            time.sleep(0.01)  # (the launch goes idle and ends)
        after = ctx.serve_stats()
        rounds = len(queries) - 4 + after["second_rounds"] - before["second_rounds"]
        assert rounds >= 30
        assert after["launches"] - before["launches"] <= 25  # 20 queries; a slow host may miss the launch now and then


@pytest.mark.timeout(300)
def test_queries_that_arrive_while_others_run():
    """Tables of a new query are cleared while other queries' items run: sizes
    around one piece of the clearing, without and with pruning."""
    corpus, queries = _trees(40, 7, 1, 140), _trees(20, 8, 1, 140)
    with xted.Context() as ctx:
        ctx.corpus_load(corpus)
        for prune in (0, 2):
            ctx.serve_options(prune)
            tickets = []
            for q in queries:
                tickets.append(ctx.query_submit(q, len(corpus)))
                time.sleep(0.001)
            for q, t in zip(queries, tickets):
                ids, ds, _, _ = ctx.query_wait(t, timeout_s=60)
                _check(ids, ds, q, corpus, len(corpus))
        ctx.serve_drain()


@pytest.mark.timeout(300)
def test_lists_larger_than_the_pool():
    """A query whose hand-off words exceed the session's pool (spines with a leg
    per node on a random side) runs in parts, beside small queries, with and
    without a second round."""
    from test_gpu_flow_memory import _zigzag
    corpus = [_zigzag(400 + 3 * k, k) for k in range(6)] + _trees(40, 9, 5, 60)
    queries = [_zigzag(410, 50), gen.tree("random", 33, 3, "zipf", 12), _zigzag(395, 51)]
    with xted.Context(mem_limit=256 << 20) as ctx:
        ctx.corpus_load(corpus)
        for prune in (0, 2):
            ctx.serve_options(prune)
            tickets = [ctx.query_submit(q, 8) for q in queries]
            for q, t in zip(queries, tickets):
                ids, ds, _, _ = ctx.query_wait(t, timeout_s=100)
                _check(ids, ds, q, corpus, 8)
        ctx.serve_drain()


@pytest.mark.timeout(300)
def test_a_failed_query_leaves_its_slot_to_the_next():
    """A query whose work is lost fails and its slot's list is emptied, in the
    stream's order, before the next query's is posted there: more queries than
    slots wait behind it, several times."""
    corpus, queries = _trees(20, 10, 5, 60), _trees(20, 11, 5, 60)
    with xted.Context() as ctx:
        ctx.corpus_load(corpus)
        ctx.serve_options(prune=0)
        for _ in range(4):
            ctx.test_fault(xted.XTED_FAULT_HOLD_PAIR)
            tickets = [ctx.query_submit(q, 3) for q in queries]
            failed = 0
            for q, t in zip(queries, tickets):
                try:
                    ids, ds, _, _ = ctx.query_wait(t, timeout_s=60)
                except xted.XtedError as e:
                    assert e.code == xted.XTED_ETIMEOUT
                    failed += 1
                else:
                    _check(ids, ds, q, corpus, 3)
            assert failed == 1


@pytest.mark.timeout(300)
def test_calls_while_lists_are_posted():
    """Polls and submissions from other threads while the worker plans and posts."""
    import threading
    corpus, queries = _trees(120, 12, 100, 400), _trees(30, 13, 100, 400)
    with xted.Context() as ctx:
        ctx.corpus_load(corpus)
        ctx.serve_options(prune=0)
        want = [ctx.query_wait(ctx.query_submit(q, 4), timeout_s=60)[:2] for q in queries]
        got = [None] * len(queries)

        def client(lo):
            for i in range(lo, len(queries), 3):
                got[i] = ctx.query_wait(ctx.query_submit(queries[i], 4), poll_s=0.0, timeout_s=60)[:2]

        threads = [threading.Thread(target=client, args=(k,)) for k in range(3)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for (a, b), (c, d) in zip(want, got):
            assert np.array_equal(a, c) and np.array_equal(b, d)
        ctx.serve_drain()


@pytest.mark.timeout(300)
def test_closing_with_queries_in_every_state():
    """A context closed while the worker plans, posts and runs."""
    corpus, queries = _trees(120, 12, 100, 400), _trees(30, 13, 100, 400)
    for pause in (0.0, 0.0005, 0.001, 0.002, 0.003, 0.005, 0.01, 0.05):
        with xted.Context() as ctx:
            ctx.corpus_load(corpus)
            ctx.serve_options(2 if pause == 0.05 else 0)
            for q in queries:
                ctx.query_submit(q, 4)
            time.sleep(pause)
