"""One pair planned by one block (needs a B200): sizes around the block's
1,024 threads and the limit of the one-block plan, against the batch's planner
(which a prepared batch uses) and the oracle; plans that do not fit its lists;
and the arena entry point's own checks of its trees."""
import ctypes

import numpy as np
import pytest

import oracle
import xted
from xted import _lib, gen, trees

pytestmark = pytest.mark.gpu


def _noalloc(a, b):
    keep = []
    ta, tb = _lib.ctree(a, keep), _lib.ctree(b, keep)
    out = ctypes.c_int32(-1)
    return _lib.lib().xted_distance_noalloc(ctypes.byref(ta), ctypes.byref(tb), 0, ctypes.byref(out)), out.value


@pytest.mark.timeout(300)
@pytest.mark.parametrize("m,n", [(1, 1), (1, 300), (32, 33), (257, 256), (1023, 260), (1024, 1025), (2048, 2048), (2049, 2048)])
def test_sizes(m, n):
    for k, (sa, sb) in enumerate((("random", "random"), ("wide", "deep"), ("caterpillar", "random"))):
        a, b = gen.tree(sa, m, 3 * m + k, "uniform", 5), gen.tree(sb, n, 7 * n + k, "uniform", 5)
        want = int(oracle.distance_batch([(a, b)], nthreads=8)[0])
        with xted.Context() as ctx:
            assert ctx.distance(a, b) == want
            cells = ctx.stats()["cells"]
            ctx.prepare_batch([(a, b)])
            assert int(ctx.run_prepared()[0]) == want
            assert ctx.stats()["cells"] == cells
        rc, d = _noalloc(a, b)
        assert (rc, d) == (xted.XTED_ETOOBIG, -1) if m > 1500 else (0, want)


def _nested(n):
    adj = [[c for c in (v + 1, v + 2) if c < n] if v % 2 == 0 and v + 1 < n else [] for v in range(n)]
    return trees.from_adjacency([v % 3 for v in range(n)], adj)


@pytest.mark.timeout(300)
def test_plans_that_do_not_fit():
    a = _nested(801)  # keyroot depth 400: more levels than the one-block plan lists
    b = gen.tree("random", 90, 5, "uniform", 3)
    for x, y in ((a, b), (b, a), (a, a)):
        want = int(oracle.distance_batch([(x, y)], nthreads=8)[0])
        with xted.Context(orientation=xted.ORIENT_RIGHT) as ctx:
            assert ctx.distance(x, y) == want
        assert _noalloc(x, y) == (0, want)
    wide, small = gen.tree("wide", 60000, 9, "uniform", 3), gen.tree("random", 3, 1, "uniform", 3)
    want = int(oracle.distance_batch([(wide, small)], nthreads=8)[0])
    assert _noalloc(wide, small) == (0, want)  # its plan is larger than the arena
    assert _noalloc(small, small)[0] == 0


@pytest.mark.timeout(300)
def test_arena_checks_trees_like_the_host():
    rng = np.random.default_rng(3)
    bad = 0
    for k in range(120):
        t = gen.tree(("random", "wide", "deep")[k % 3], int(rng.integers(2, 70)), k, "uniform", 4)
        labels, off, idx = (np.array(x, dtype=np.int32) for x in (t.labels, t.off, t.idx))
        for _ in range(int(rng.integers(1, 3))):
            arr = off if rng.integers(2) else idx
            arr[int(rng.integers(len(arr)))] += int(rng.integers(-2, 3)) if k % 4 else int(rng.choice([-2**30, 2**30]))
        c = trees.Tree(labels, off, idx)
        keep = []
        want = _lib.lib().xted_validate(ctypes.byref(_lib.ctree(c, keep)))
        assert _noalloc(c, t)[0] == want and _noalloc(t, c)[0] == want
        bad += want != 0
    assert 30 < bad < 120


@pytest.mark.timeout(300)
@pytest.mark.parametrize("m,n", [(1, 1), (40, 57), (300, 251)])
def test_a_pair_runs_again(m, n):
    """A call leaves its plan prepared: run again it starts from cleared
    counters, also from the graph that the second run captures."""
    a, b = gen.tree("random", m, 5, "uniform", 5), gen.tree("deep", n, 6, "uniform", 5)
    out = ctypes.c_int32(-1)
    with xted.Context() as ctx:
        want = ctx.distance(a, b)
        assert want == oracle.distance(a, b)
        for _ in range(4):
            out.value = -1
            assert _lib.lib().xted_run_prepared(ctx.handle, ctypes.byref(out)) == 0
            assert out.value == want


@pytest.mark.timeout(300)
@pytest.mark.parametrize("n", [1, 2, 13, 14, 15, 16, 63, 64, 65, 66])
def test_arena_smallest_pairs(n):
    """Around the sizes up to which the arena's own kernel runs a pair (14 nodes
    a side, paths of 64), valid and malformed."""
    path = trees.from_adjacency([v % 3 for v in range(n)], [[v + 1] if v + 1 < n else [] for v in range(n)])
    for other in (gen.tree("random", n, 3, "uniform", 3), gen.tree("wide", max(n - 1, 1), 4, "uniform", 3), path,
                  trees.from_adjacency([v % 2 for v in range(64)], [[v + 1] if v < 63 else [] for v in range(64)])):
        for a, b in ((path, other), (other, path), (other, other)):
            assert _noalloc(a, b) == (0, oracle.distance(a, b))
    if n > 2:
        bad = trees.Tree(np.array(path.labels, np.int32), np.array(path.off, np.int32), np.array(path.idx, np.int32))
        bad.idx[n // 2] += 1
        assert _noalloc(bad, path)[0] == _noalloc(path, bad)[0] == xted.XTED_EINVAL


@pytest.mark.timeout(300)
def test_no_room_for_the_one_block_plan():
    """With a few MB of device memory left a pair is planned by the batch's
    kernels, whose buffers the context holds already."""
    import torch
    a, b = gen.tree("random", 300, 1, "uniform", 4), gen.tree("deep", 280, 2, "uniform", 4)
    want = oracle.distance(a, b)
    with xted.Context() as ctx:
        ctx.prepare_batch([(a, b)])
        assert ctx.run_prepared()[0] == want
        torch.zeros(1, device="cuda")
        hold = []
        while (free := torch.cuda.mem_get_info()[0]) > 24 << 20:
            size = max(free - (16 << 20), 1 << 20) if free < 64 << 30 else 32 << 30
            try:
                hold.append(torch.cuda.caching_allocator_alloc(size))
            except torch.cuda.OutOfMemoryError:
                break
        try:
            assert torch.cuda.mem_get_info()[0] < 32 << 20
            assert ctx.distance(a, b) == want
        finally:
            for p in hold:
                torch.cuda.caching_allocator_delete(p)
            torch.cuda.empty_cache()
        assert ctx.distance(a, b) == want
