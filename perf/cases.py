"""The work that a user of this library has it do, as cases that can be timed.

Every case goes through the public entry points of the ``xted`` package on
seeded synthetic trees (``xted.gen``), the shapes, sizes and label
distributions of the benchmark: random recursive, wide-shallow, deep-narrow
and caterpillar trees, from tens of nodes to 20,000.

A case's ``kind`` names the call:

  ted       ``standard_ted``: string labels and adjacency lists, one distance
  pair      ``Context.distance``: one pair of trees in CSR form
  noalloc   ``distance_noalloc``: one pair in the library's fixed arena
  batch     ``Context.distance_batch``: many pairs, planned on every call
  prepared  ``Context.run_prepared``: a batch planned once and run again
  matrix    ``Context.distance_matrix``: all pairs of a list of trees
  serve     ``Context.query_submit`` / ``query_wait``: exact top-k queries,
            sent together, against a resident corpus
"""
import math
import os
import random
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "x-ted_b200"))

import xted  # noqa: E402
from xted import gen  # noqa: E402

SHAPES = ("random", "wide", "deep", "caterpillar")


def listed():
    return [
        # a document diff through the reference's own entry point: two small trees with string labels
        {"name": "ted strings 40x57", "kind": "ted", "shape_a": "random", "shape_b": "wide", "m": 40, "n": 57,
         "labels": "uniform", "alphabet": 26},
        # the plain single pair: two 100-node random recursive trees, 26 labels; latency and launches
        {"name": "pair 100x100", "kind": "pair", "shape_a": "random", "shape_b": "random", "m": 100, "n": 100,
         "labels": "uniform", "alphabet": 26, "costs": ""},
        # the 1,000-node pair of mixed shapes: every keyroot level, tables from one warp to a block
        {"name": "pair 1000x1000 wide deep", "kind": "pair", "shape_a": "wide", "shape_b": "deep", "m": 1000,
         "n": 1000, "labels": "zipf", "alphabet": 10000, "costs": ""},
        # the largest pair: 20,000-node random recursive trees (1.6 GB of distances)
        {"name": "pair 20000x20000 random", "kind": "pair", "shape_a": "random", "shape_b": "random", "m": 20000,
         "n": 20000, "labels": "uniform", "alphabet": 64, "costs": ""},
        # two long caterpillars of unequal, odd sizes: few levels, one very large table
        {"name": "pair 19999x13571 caterpillar", "kind": "pair", "shape_a": "caterpillar", "shape_b": "caterpillar",
         "m": 19999, "n": 13571, "labels": "uniform", "alphabet": 64, "costs": ""},
        # a caller that must not allocate device memory: one pair in the fixed arena
        {"name": "noalloc 300x251", "kind": "noalloc", "shape_a": "random", "shape_b": "deep", "m": 300, "n": 251,
         "labels": "zipf", "alphabet": 1000},
        # all distances of a small collection of records (clustering, deduplication)
        {"name": "matrix 96 trees", "kind": "matrix", "trees": 96, "lo": 20, "hi": 250, "alphabet": 64, "costs": ""},
        # the headline batch, end to end: 4,096 pairs of 50-2,000 nodes planned and run in one call
        {"name": "batch 4096 mixed", "kind": "batch", "pairs": 4096, "lo": 50, "hi": 2000, "alphabet": 1000,
         "costs": ""},
        # a mid-sized batch planned once and evaluated again from resident inputs
        {"name": "prepared 1024 mixed", "kind": "prepared", "pairs": 1024, "lo": 50, "hi": 2000, "alphabet": 1000,
         "costs": ""},
        # a small batch under general edit costs (delete 2, insert 3, rename 4)
        {"name": "batch 500 costs", "kind": "batch", "pairs": 500, "lo": 50, "hi": 1000, "alphabet": 1000,
         "costs": "2,3,4"},
        # serving: exact top-10 of queries that arrive together, over 1,000 resident trees
        {"name": "serve 1000 trees", "kind": "serve", "trees": 1000, "queries": 4, "lo": 100, "hi": 1000, "k": 10,
         "alphabet": 1000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("ted", "pair", "pair", "pair", "noalloc", "batch", "batch", "prepared", "matrix", "serve"))
    alphabet = _log_int(rng, 4, 10000)
    labels = rng.choice(("uniform", "zipf"))
    costs = rng.choice(("", "", "", "1,1,2", "2,3,4"))
    if kind in ("ted", "pair", "noalloc"):
        hi = {"ted": 250, "pair": 20000, "noalloc": 600}[kind]
        m, n = _log_int(rng, 20, hi), _log_int(rng, 20, hi)
        # trees of many thousands of nodes come in the two shapes whose tables stay affordable
        shapes = SHAPES if max(m, n) <= 2000 else ("random", "caterpillar")
        sa = rng.choice(shapes)
        # a caterpillar against a tree of another kind has no cheap decomposition once both are large
        sb = sa if max(m, n) > 2000 else rng.choice(shapes)
        c = {"kind": kind, "shape_a": sa, "shape_b": sb, "m": m, "n": n, "labels": labels, "alphabet": alphabet}
        # costs of up to 4 keep a pair of 20,000-node trees within the library's bound only at unit cost
        return dict(c, costs=costs if max(m, n) <= 10000 else "") if kind == "pair" else c
    if kind == "matrix":
        return {"kind": kind, "trees": _log_int(rng, 8, 160), "lo": rng.randint(5, 60), "hi": rng.randint(80, 300),
                "alphabet": alphabet, "costs": costs}
    if kind == "serve":
        return {"kind": kind, "trees": _log_int(rng, 100, 1000), "queries": rng.randint(1, 6),
                "lo": rng.randint(20, 200), "hi": rng.randint(300, 1000), "k": rng.randint(1, 12),
                "alphabet": alphabet}
    return {"kind": kind, "pairs": _log_int(rng, 64, 3000), "lo": rng.randint(20, 100), "hi": rng.randint(300, 2000),
            "alphabet": alphabet, "costs": costs}


def _two_trees(case, seed):
    return (gen.tree(case["shape_a"], case["m"], 2 * seed + 1, case["labels"], case["alphabet"]),
            gen.tree(case["shape_b"], case["n"], 2 * seed + 2, case["labels"], case["alphabet"]))


def _tree_list(count, lo, hi, alphabet, seed):
    """Trees of every shape with sizes uniform in [lo, hi]."""
    rng = random.Random(seed)
    return [gen.tree(rng.choice(SHAPES), rng.randint(lo, hi), rng.getrandbits(48), "zipf", alphabet)
            for _ in range(count)]


def _pair_list(case, seed):
    """Pairs with log-uniform sizes, every tree drawn by itself."""
    return gen.mixed_batch(case["pairs"], seed, case["lo"], case["hi"], case["alphabet"])


def _strings(tree):
    return ["n%d" % x for x in tree.labels.tolist()], tree.adjacency()


def _context(case):
    costs = tuple(int(x) for x in case["costs"].split(",")) if case.get("costs") else None
    return xted.Context(costs=costs)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ted":
        a, b = _two_trees(case, seed)
        return kind, _context(case), (*_strings(a), *_strings(b))
    if kind == "pair":
        return kind, _context(case), _two_trees(case, seed)
    if kind == "noalloc":
        return kind, None, _two_trees(case, seed)
    if kind == "matrix":
        return kind, _context(case), _tree_list(case["trees"], case["lo"], case["hi"], case["alphabet"], seed)
    if kind == "serve":
        ctx = _context(case)
        ctx.corpus_load(_tree_list(case["trees"], case["lo"], case["hi"], case["alphabet"], seed))
        queries = _tree_list(case["queries"], case["lo"], case["hi"], case["alphabet"], seed + 1000003)
        return kind, ctx, (queries, case["k"])
    ctx = _context(case)
    pairs = _pair_list(case, seed)
    if kind == "prepared":
        ctx.prepare_batch(pairs)
    return kind, ctx, pairs


def run(state):
    kind, ctx, data = state
    if kind == "ted":
        return xted.standard_ted(*data, ctx=ctx)
    if kind == "pair":
        return ctx.distance(*data)
    if kind == "noalloc":
        return xted.distance_noalloc(*data)
    if kind == "batch":
        return ctx.distance_batch(data)
    if kind == "prepared":
        return ctx.run_prepared()
    if kind == "matrix":
        return ctx.distance_matrix(data)
    queries, k = data
    tickets = [ctx.query_submit(q, k) for q in queries]
    return [ctx.query_wait(t)[:2] for t in tickets]


def _keyroot_sums(tree):
    """Sum of subtree sizes over the keyroots (root and non-last, or non-first, children): right, left path."""
    n, off, idx = tree.n, tree.off, tree.idx
    parent = np.full(n, -1)
    parent[idx] = np.repeat(np.arange(n), np.diff(off))
    size = np.ones(n, np.int64)
    for v in range(n - 1, 0, -1):
        size[parent[v]] += size[v]
    has = np.diff(off) > 0
    last, first = idx[off[1:][has] - 1], idx[off[:-1][has]]
    total = int(size.sum())
    return total - int(size[last].sum()), total - int(size[first].sum())


def work(case):
    """Every input array read once and every distance written once; three
    integer operations (add, add-min, add-min) per cell of the forest tables
    of the cheaper decomposition."""
    kind = case["kind"]

    def tree_bytes(t):
        return 4 * (3 * t.n + 1)

    if kind in ("ted", "pair", "noalloc"):
        trees, pairs = list(_two_trees(case, 0)), [(0, 1)]
    elif kind == "matrix":
        trees = _tree_list(case["trees"], case["lo"], case["hi"], case["alphabet"], 0)
        pairs = [(i, j) for i in range(len(trees)) for j in range(i)]
    elif kind == "serve":
        trees = _tree_list(case["trees"] + case["queries"], case["lo"], case["hi"], case["alphabet"], 0)
        # exact top-k needs at least k distances of each query
        pairs = [(len(trees) - 1 - q, t) for q in range(case["queries"]) for t in range(case["k"])]
    else:  # a sample of the batch stands for all of it
        few = min(case["pairs"], 128)
        trees = [t for p in _pair_list(dict(case, pairs=few), 0) for t in p]
        pairs = [(2 * i, 2 * i + 1) for i in range(few)]
    sums = [_keyroot_sums(t) for t in trees]
    cells = sum(min(sums[a][0] * sums[b][0], sums[a][1] * sums[b][1]) for a, b in pairs)
    moved = sum(tree_bytes(t) for t in trees) + 4 * len(pairs)
    scale = case["pairs"] / few if kind in ("batch", "prepared") else 1.0
    return {"bytes": moved * scale, "flops": 3.0 * cells * scale}


def _distance(a, b, dele, ins, ren):
    """Tree edit distance by keyroot tables in 64-bit numpy: the row keyroots
    innermost first, against all column keyroots of one nesting depth at once."""
    def facts(t):
        n = t.n
        parent = np.full(n, -1)
        parent[t.idx] = np.repeat(np.arange(n), np.diff(t.off))
        size = np.ones(n, np.int64)
        for v in range(n - 1, 0, -1):
            size[parent[v]] += size[v]
        key = np.ones(n, bool)
        has = np.diff(t.off) > 0
        key[t.idx[t.off[1:][has] - 1]] = False
        return n, np.arange(n) + size, np.flatnonzero(key)  # end = one past the subtree

    m, end_a, keys_a = facts(a)
    n, end_b, keys_b = facts(b)
    depth = {}
    for k in reversed(keys_b.tolist()):
        inner = [depth[q] for q in keys_b[(keys_b > k) & (keys_b < end_b[k])].tolist()]
        depth[k] = 1 + max(inner) if inner else 0
    dist = np.zeros((m, n), np.int64)
    big = 1 << 40
    groups = []
    for d in range(max(depth.values()) + 1):
        # columns of all depth-d tables side by side, one border column after each
        node, seg_end, seg = [], [], 0
        for k in keys_b.tolist():
            if depth[k] == d:
                node += list(range(k, end_b[k])) + [-1]
                seg_end += [(len(node) - 1, seg)] * (end_b[k] - k + 1)
                seg += 1
        node = np.array(node)
        last = np.array([e for e, _ in seg_end])
        which = np.array([s for _, s in seg_end])
        groups.append((node, last, which))
    for i0 in reversed(keys_a.tolist()):
        imax = int(end_a[i0])
        for node, last, which in groups:
            at = np.arange(node.size)
            border = node < 0
            col = np.where(border, 0, node)
            far_col = np.minimum(at + np.where(border, 0, end_b[col] - col), node.size - 1)
            on_path = ~border & (far_col == last)
            ramp = at * ins + which * big
            table = np.zeros((imax - i0 + 1, node.size), np.int64)
            table[-1] = (last - at) * ins
            for i in range(imax - 1, i0 - 1, -1):
                r, below = i - i0, table[i - i0 + 1]
                best = dist[i, col] + table[end_a[i] - i0, far_col]
                if end_a[i] == imax:
                    match = np.append(below[1:], 0) + np.where(a.labels[i] == b.labels[col], 0, ren)
                    best = np.where(on_path, match, best)
                best = np.where(border, (imax - i) * dele, np.minimum(best, below + dele))
                row = np.minimum.accumulate((best + ramp)[::-1])[::-1] - ramp
                table[r] = row
                if end_a[i] == imax:
                    dist[i, col[on_path]] = row[on_path]
    return int(dist[0, 0])


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("ted", "pair", "noalloc") or case["m"] * case["n"] > 250000:
        return None
    costs = [int(x) for x in case["costs"].split(",")] if case.get("costs") else [1, 1, 1]
    return _distance(*_two_trees(case, seed), *costs)
