"""Hand-off words larger than their buffer (needs a B200): a list then runs in
parts, launches that share the buffer. Trees whose tables are costly in both
decompositions have the most words (a spine with a leg per node on a random
side: 1,000 nodes a side 11.6 GB). Exact against the oracle."""
import numpy as np
import pytest

import oracle
import xted
from xted import gen, trees

pytestmark = pytest.mark.gpu


def _zigzag(n, seed):
    rng = np.random.default_rng(seed)
    spine = (n + 1) // 2
    adj, ids, later, at = [[] for _ in range(n)], [], [], 0
    for k in range(spine):
        ids.append(at)
        at += 1
        if k < n - spine:
            if k < spine - 1 and rng.integers(2):
                adj[ids[k]].append(at)
                at += 1
            else:
                later.append(k)
        if k > 0:
            adj[ids[k - 1]].append(ids[k])
    for k in reversed(later):
        adj[ids[k]].append(at)
        at += 1
    return trees.from_adjacency([int(x) for x in rng.integers(0, 4, n)], adj)


def _held():
    import torch
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.mark.timeout(300)
def test_words_stay_bounded():
    """One pair and a batch whose words would be 11.6 and 47 GB: as a call, then
    prepared and run again from a graph; both keep the buffer at its floor."""
    pairs = [(_zigzag(1000 + k, 2 * k), _zigzag(1001 - k, 2 * k + 1)) for k in range(4)]
    want = [804, 810, 790, 811]  # oracle.distance_batch: a minute a pair on one core
    before = _held()
    with xted.Context() as ctx:
        assert ctx.distance(*pairs[0]) == want[0]
        assert ctx.distance_batch(pairs).tolist() == want
        ctx.prepare_batch(pairs)
        for _ in range(3):
            assert ctx.run_prepared().tolist() == want
        assert _held() - before < 10 << 30


@pytest.mark.timeout(300)
@pytest.mark.parametrize("limit_mb", [400, 160, 96, 64])
def test_under_a_limit(limit_mb):
    """Less room than one launch's words: parts, down to a few units each; a
    context whose buffers hold the limit still takes other work."""
    wide = [(_zigzag(500, k), _zigzag(499, 50 + k)) for k in range(2)]  # 1 GB of words
    many = [(gen.tree("random", 60, k, "uniform", 4), gen.tree("deep", 70, k, "uniform", 4)) for k in range(600)]
    with xted.Context(mem_limit=limit_mb << 20) as ctx:
        for pairs in (wide, many, wide):
            assert np.array_equal(ctx.distance_batch(pairs), oracle.distance_batch(pairs, nthreads=8))


@pytest.mark.timeout(300)
def test_room_of_many_trees():
    """Planning 4,000 trees of 800,000 nodes together: 238 MB suffice."""
    pairs = [(gen.tree("random", 400, k, "uniform", 4), gen.tree("random", 1, k, "uniform", 4)) for k in range(2000)]
    with xted.Context(mem_limit=238 << 20) as ctx:
        assert np.array_equal(ctx.distance_batch(pairs), oracle.distance_batch(pairs, nthreads=8))
