"""The DP launch at the sizes where its item kinds change (needs a B200):
chunks of up to 256 columns on one warp, column stripes of 256 beyond
that (a boundary may fall on any node), row runs around the 32 rows that
a warp looks ahead, stacks deeper than the shared-memory window, and long
lists of path columns, exports and far columns across a stripe
boundary. Exact against the oracle: distances are whole numbers."""
import numpy as np
import pytest

import oracle
import xted
from xted import gen, trees

pytestmark = pytest.mark.gpu


def _comb(n, seed, leaf_first):
    """A spine on which every node carries one leaf, before or after the next
    spine node: right-path keyroots nested to depth n / 2, or one long path."""
    adj = []
    for v in range(n):
        if v % 2 or v + 1 >= n:
            adj.append([])
        elif leaf_first:
            adj.append([c for c in (v + 1, v + 2) if c < n])
        else:
            adj.append([])
    if not leaf_first:  # spine 0 .. d-1, then the leaves from the innermost out
        d = n // 2 + 1
        adj = [[] for _ in range(n)]
        for v in range(d - 1):
            adj[v].append(v + 1)
        for k in range(n - d):
            adj[d - 2 - k].append(d + k)
    labels = np.random.default_rng(seed).integers(0, 4, n)
    return trees.from_adjacency([int(x) for x in labels], adj)


@pytest.mark.timeout(300)
@pytest.mark.parametrize("n", [253, 256, 257, 260, 508, 511, 512, 513, 516, 1023, 1025, 1537])
def test_chunk_widths(n):
    """Column trees around every width limit, both decompositions."""
    pairs = []
    for k, shape in enumerate(("random", "wide", "deep", "caterpillar")):
        pairs.append((gen.tree(shape, 31 + 2 * k, n + k, "uniform", 5), gen.tree("random", n, 7 * n + k, "uniform", 5)))
        pairs.append((gen.tree("random", 64 + k, n + k, "uniform", 5), gen.tree(shape, n, 3 * n + k, "uniform", 5)))
    want = oracle.distance_batch(pairs, nthreads=8)
    for orient in (xted.ORIENT_RIGHT, xted.ORIENT_LEFT):
        with xted.Context(orientation=orient) as ctx:
            assert np.array_equal(ctx.distance_batch(pairs), want)


@pytest.mark.timeout(300)
@pytest.mark.parametrize("m,n", [(1, 700), (2, 513), (32, 600), (33, 257), (35, 1030), (97, 129)])
def test_long_lists_and_deep_stacks(m, n):
    """Combs: every second column of the root chunk on its right path, or one
    export per nested keyroot (lists longer than 64), and row stacks as deep as
    half the tree; also under general costs."""
    pairs = [(_comb(m, 1, a), _comb(n, 2, b)) for a in (True, False) for b in (True, False)]
    pairs += [(_comb(n, 3, a), _comb(m, 4, True)) for a in (True, False)]
    for orient in (xted.ORIENT_AUTO, xted.ORIENT_RIGHT, xted.ORIENT_LEFT):
        with xted.Context(orientation=orient) as ctx:
            assert np.array_equal(ctx.distance_batch(pairs), oracle.distance_batch(pairs, nthreads=8))
    with xted.Context(costs=(2, 3, 7)) as ctx:  # a rename dearer than delete + insert
        assert ctx.distance_batch(pairs).tolist() == [oracle.distance(a, b, costs=(2, 3, 7)) for a, b in pairs]


@pytest.mark.timeout(300)
@pytest.mark.parametrize("narrow,run_rows", [(256, 1), (64, 7), (0, 33), (256, 200)])
def test_many_segments(narrow, run_rows):
    """Chunks of many small segments (caterpillars, wide trees) and runs of many
    small tables, at several granularities."""
    rng = np.random.default_rng(narrow + run_rows)
    pairs = []
    for k in range(24):
        m, n = int(rng.integers(1, 400)), int(rng.integers(1, 400))
        pairs.append((gen.tree(("caterpillar", "wide", "random")[k % 3], m, k, "uniform", 3),
                      gen.tree(("wide", "caterpillar", "deep")[k // 3 % 3], n, 50 + k, "uniform", 3)))
    with xted.Context(narrow_width=narrow, run_rows=run_rows) as ctx:
        assert np.array_equal(ctx.distance_batch(pairs), oracle.distance_batch(pairs, nthreads=8))


@pytest.mark.timeout(300)
@pytest.mark.parametrize("n", [301, 601])
def test_more_far_values_than_places(n):
    """Forced right-path tables of a comb whose nested keyroots cross every
    stripe boundary with a far column each: more than have a place in shared
    memory (64)."""
    a, b = _comb(9, 5, False), _comb(n, 6, False)
    with xted.Context(orientation=xted.ORIENT_RIGHT) as ctx:
        assert ctx.distance(a, b) == oracle.distance(a, b)


@pytest.mark.timeout(300)
@pytest.mark.parametrize("npairs", [1023, 1024])
def test_launch_of_many_pairs(npairs):
    """From 1,024 pairs on the launch takes five blocks an SM: every chunk kind,
    first as a batch, then prepared and run again from a graph."""
    small = [(gen.tree("random", 1 + k % 37, k, "uniform", 4), gen.tree("deep", 1 + k % 61, 2 * k, "uniform", 4)) for k in range(npairs - 6)]
    pairs = small + [(_comb(130, 1, a), _comb(n, 2, a)) for a in (True, False) for n in (255, 600, 1100)]
    want = oracle.distance_batch(pairs, nthreads=8)
    with xted.Context() as ctx:
        assert np.array_equal(ctx.distance_batch(pairs), want)
        ctx.prepare_batch(pairs)
        for _ in range(3):
            assert np.array_equal(ctx.run_prepared(), want)


@pytest.mark.timeout(300)
@pytest.mark.parametrize("n", [303, 304, 305, 340, 513])
def test_far_values_of_other_stripes(n):
    """The same combs with 47, 48 (the places beside the usual stack rows), 49,
    84 and 255 far values of other stripes in a stripe, against rows that pop the
    stack one by one and rows that leave and refill its window; in a batch wide
    enough that stripes wait for each other."""
    rows = [_comb(9, 5, False), _comb(61, 7, False), _comb(40, 8, True), gen.tree("deep", 90, 9, "uniform", 4),
            gen.tree("random", 120, 10, "uniform", 4)]
    pairs = [(a, _comb(n, s, False)) for a in rows for s in (6, 11)]
    want = oracle.distance_batch(pairs, nthreads=8)
    with xted.Context(orientation=xted.ORIENT_RIGHT) as ctx:
        assert np.array_equal(ctx.distance_batch(pairs), want)
        assert [ctx.distance(a, b) for a, b in pairs[:3]] == want[:3].tolist()
        assert np.array_equal(ctx.distance_batch(pairs * 40), np.tile(want, 40))


def _path(n, seed):
    labels = np.random.default_rng(seed).integers(0, 3, n)
    return trees.from_adjacency([int(x) for x in labels], [[v + 1] if v + 1 < n else [] for v in range(n)])


def _star(n, seed):
    labels = np.random.default_rng(seed).integers(0, 3, n)
    return trees.from_adjacency([int(x) for x in labels], [list(range(1, n))] + [[] for _ in range(n - 1)])


@pytest.mark.timeout(300)
@pytest.mark.parametrize("m", [31, 63, 64, 65, 97, 300])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 66, 129, 255, 257, 513])
def test_many_path_columns(m, n):
    """Items whose rows and columns lie on their paths, all of them (paths;
    runs and chunks of single nodes) or most (combs, whose chunks also hold
    longer segments), around 64 columns, 64 rows and the stripes' edges; words of
    later items are waited for (a batch), costs other than one."""
    rows = [_path(m, 1), _star(m, 2), _comb(m, 3, False), _comb(m, 4, True)]
    cols = [_path(n, 5), _star(n, 6), _comb(n, 7, False), gen.tree("caterpillar", n, 8, "uniform", 3)]
    pairs = [(a, b) for a in rows for b in cols]
    want = oracle.distance_batch(pairs, nthreads=8)
    for orient in (xted.ORIENT_RIGHT, xted.ORIENT_LEFT):
        with xted.Context(orientation=orient) as ctx:
            assert np.array_equal(ctx.distance_batch(pairs), want)
    with xted.Context(run_rows=256) as ctx:  # (runs of many small tables)
        assert np.array_equal(ctx.distance_batch(pairs * 3), np.tile(want, 3))
    with xted.Context(costs=(2, 3, 4)) as ctx:
        assert ctx.distance_batch(pairs).tolist() == [oracle.distance(a, b, costs=(2, 3, 4)) for a, b in pairs]
