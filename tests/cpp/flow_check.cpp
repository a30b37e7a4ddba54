// flow_check.cpp -- TEST INFRASTRUCTURE: the DP launch's item list on the CPU.
//
// Plans pairs with the host planner of the list (serve_plan.h: serve_plan_items;
// flow_plan.h lays out the same list on the device) and runs its items one
// after another in list order, cell by cell in the savings form of flow.cu.
// Checked: every word an item reads (tables, first columns, exported columns)
// was written by an item before it, which is what lets a launch wait for words
// without a deadlock; every word is written once, so no two units share
// hand-off words; every index lies in its pool; the distance is the oracle's.
// The list is run whole and in parts (flow_cut) that share one buffer: parts
// consist of whole units, hold at most their limit or one unit, and cover the list.
// Then as serving divides and places it (serve_cut, serve_fixup_items).
//   usage: flow_check <rounds> <max_nodes> <seed>
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../../include/xted.h"
#include "../../x-ted_b200/csrc/serve_plan.h"

extern "C" int xo_distance(int m, const int32_t *la, const int32_t *aoff, const int32_t *aidx, int n,
                           const int32_t *lb, const int32_t *boff, const int32_t *bidx);
using namespace xted;

#define FAIL(...)                     \
    do {                              \
        std::printf(__VA_ARGS__);     \
        std::printf("\n");            \
        std::exit(1);                 \
    } while (0)

struct HTree {
    std::vector<int32_t> lab, off, idx;
    int n = 0;
};

static HTree from_children(const std::vector<std::vector<int>> &ch, std::mt19937_64 &g, int alpha) {
    HTree t;
    t.n = (int)ch.size();
    std::vector<int> order, st{0};
    while (!st.empty()) {
        const int v = st.back();
        st.pop_back();
        order.push_back(v);
        for (int k = (int)ch[(size_t)v].size() - 1; k >= 0; k--) st.push_back(ch[(size_t)v][(size_t)k]);
    }
    std::vector<int> id((size_t)t.n);
    for (int k = 0; k < t.n; k++) id[(size_t)order[(size_t)k]] = k;
    t.off.assign(1, 0);
    for (int k = 0; k < t.n; k++) {
        t.lab.push_back((int32_t)(g() % (uint64_t)alpha));
        for (int c : ch[(size_t)order[(size_t)k]]) t.idx.push_back(id[(size_t)c]);
        t.off.push_back((int32_t)t.idx.size());
    }
    return t;
}

// Shapes: random, wide, a spine with a leg per node after it, before it or on
// a random side (then neither decomposition is cheap), a path.
static HTree gen(int n, std::mt19937_64 &g, int shape) {
    std::vector<std::vector<int>> ch((size_t)n);
    int spine = 0;
    for (int i = 1; i < n; i++) {
        int p = i - 1;
        if (shape == 0) p = (int)(g() % (uint64_t)i);
        else if (shape == 1) p = (int)(g() % (uint64_t)std::min(i, 1 + n / 20));
        else if (shape < 5) p = spine;
        const bool before = shape == 3 || (shape == 4 && g() % 2);
        if (shape >= 2 && shape < 5 && i % 2 == 0) {  // the next spine node
            ch[(size_t)p].push_back(i);
            spine = i;
            if (ch[(size_t)p].size() == 2 && !before) std::swap(ch[(size_t)p][0], ch[(size_t)p][1]);
        } else {
            ch[(size_t)p].push_back(i);
        }
    }
    return from_children(ch, g, 1 + (int)(g() % 5));
}

struct Plan {
    ServePools H;
    QPlan q;
};

// Runs items [from, to) of a plan; word w0 of the list is the buffer's first.
static void run_items(const Plan &p, int from, int to, int64_t w0, std::vector<int32_t> &dt, std::vector<int32_t> &buf,
                      const std::vector<int32_t> &smap) {
    const ServePools &H = p.H;
    const XPair &pr = p.q.pairs[0];
    const int2 *rows = H.node.data() + pr.row_base, *nodes = H.node.data() + pr.col_base;
    auto far_of = [](const int2 *t, int v) { return (t[v].y & XTED_ROW_ORL_MASK) + 1; };
    for (int g = from; g < to; g++) {
        const XItem &it = p.q.items[(size_t)g];
        const XRun &run = H.runs[(size_t)it.run];
        const XChunk &ch = H.chunks[(size_t)it.chunk];
        const XChunkX &cx = H.chunkx[(size_t)it.chunk];
        // the item's columns: node, end of its segment
        std::vector<int> node, seg_end;
        int j0 = 0, je = 0, lead = 0;
        if (ch.nseg > 1) {
            if (it.stripe != 0 || cx.K != 1) FAIL("stripes of several segments");
            for (int q = ch.k_lo; q < ch.k_lo + ch.nseg; q++)
                for (int j = H.krd[(size_t)q], e = far_of(nodes, j); j < e; j++) {
                    node.push_back(j);
                    seg_end.push_back(e);
                }
        } else {
            j0 = H.krd[(size_t)ch.k_lo];
            je = far_of(nodes, j0);
            lead = j0 & (XTED_PITCH - 1);
            if (cx.K != chunk_stripes(ch, H.krd.data()) || it.stripe < 0 || it.stripe >= cx.K) FAIL("stripe %d of %d", it.stripe, cx.K);
            const int base = j0 - lead + it.stripe * XTED_SW;
            for (int j = std::max(base, j0); j < std::min(base + XTED_SW, je); j++) {
                node.push_back(j);
                seg_end.push_back(je);
            }
        }
        const int w = (int)node.size(), first = w ? node[0] : 0;
        if (w == 0 || (ch.nseg > 1 && w != ch.width)) FAIL("an item of %d columns", w);
        const int64_t R = run.rows, K = cx.K, X = cx.X;
        auto word = [&](int64_t at, int64_t i) -> int32_t & {
            const int64_t k = it.buf - w0 + at + i;
            if (k < 0 || k >= (int64_t)buf.size()) FAIL("hand-off word %lld of %zu", (long long)k, buf.size());
            return buf[(size_t)k];
        };
        auto place = [&](int f) {  // column of node f in this item, or -1: in a stripe to the right
            if (ch.nseg == 1) return f - first < w ? f - first : -1;
            return (int)(std::lower_bound(node.begin(), node.end(), f) - node.begin());
        };
        int64_t t = 0;  // row of the run
        for (int kq = run.kr_lo; kq < run.kr_hi; kq++) {
            const int i0 = H.krd[(size_t)kq], ie = far_of(rows, i0);
            std::vector<std::vector<int32_t>> S((size_t)(ie - i0 + 1), std::vector<int32_t>((size_t)w + 1, 0));
            std::vector<int64_t> at((size_t)(ie - i0 + 1), -1);
            for (int i = ie - 1; i >= i0; i--, t++) {
                at[(size_t)(i - i0)] = t;
                std::vector<int32_t> &row = S[(size_t)(i - i0)], &below = S[(size_t)(i - i0 + 1)];
                const int fi = far_of(rows, i);
                int32_t right = 0;
                if (it.stripe + 1 < K) {
                    right = word((int64_t)it.stripe * R, t);
                    if (right < 0) FAIL("a first column is not there yet");
                }
                row[(size_t)w] = right;
                for (int c = w - 1; c >= 0; c--) {
                    const int j = node[(size_t)c], fj = far_of(nodes, j), e = seg_end[(size_t)c];
                    int32_t term;
                    if (fi == ie && fj == e) {
                        const bool edge = j + 1 == e || i + 1 == ie;
                        term = (edge ? 0 : below[(size_t)c + 1]) + (rows[i].x == nodes[j].x ? 2 : 1);
                    } else {
                        const int32_t tree = dt[(size_t)(pr.dt_off + (int64_t)i * pr.pitch + j)];
                        if (tree < 0) FAIL("table word %d %d is not there yet", i, j);
                        int32_t far = 0;
                        if (fi < ie && fj < e) {
                            const int fc = place(fj);
                            if (fc >= 0) {
                                far = S[(size_t)(fi - i0)][(size_t)fc];
                            } else {
                                if (K == 1) FAIL("a far column outside its chunk");
                                const int32_t x = smap[(size_t)(cx.map + fj - j0)];
                                if (x < 0 || x >= X) FAIL("export %d of %lld", x, (long long)X);
                                far = word((K - 1) * R + at[(size_t)(fi - i0)] * X, x);
                                if (far < 0) FAIL("an exported column is not there yet");
                            }
                        }
                        term = tree + far;
                    }
                    const int32_t after = j + 1 == e ? 0 : row[(size_t)c + 1];
                    row[(size_t)c] = std::max(term, std::max(below[(size_t)c], after));
                    if (fi == ie && fj == e) {
                        int32_t &o = dt[(size_t)(pr.dt_off + (int64_t)i * pr.pitch + j)];
                        if (o >= 0) FAIL("table word %d %d is written twice", i, j);
                        o = row[(size_t)c];
                    }
                    if (K > 1) {
                        const int32_t x = smap[(size_t)(cx.map + j - j0)];
                        const bool pushed = i > i0 && far_of(rows, i - 1) == i;  // a row read as a far row
                        if (x >= 0 && pushed) {
                            int32_t &o = word((K - 1) * R + t * X, x);
                            if (o >= 0) FAIL("an export is written twice");
                            o = row[(size_t)c];
                        }
                    }
                }
                if (it.stripe > 0) {
                    int32_t &o = word((int64_t)(it.stripe - 1) * R, t);
                    if (o >= 0) FAIL("a first column is written twice");
                    o = row[0];
                }
            }
        }
        if (t != R) FAIL("a run of %lld rows has %lld", (long long)R, (long long)t);
    }
}

int main(int argc, char **argv) {
    const int rounds = argc > 1 ? std::atoi(argv[1]) : 10, maxn = argc > 2 ? std::atoi(argv[2]) : 400;
    std::mt19937_64 g(argc > 3 ? (uint64_t)std::atoll(argv[3]) : 7);
    long long items = 0, words = 0, parts = 0, striped = 0;
    for (int r = 0; r < rounds; r++) {
        const HTree a = gen(1 + (int)(g() % (uint64_t)maxn), g, (int)(g() % 6));
        const HTree b = gen(1 + (int)(g() % (uint64_t)maxn), g, r % 6);
        const xted_tree ta{a.lab.data(), a.off.data(), a.idx.data(), a.n};
        Plan p;
        static const int narrow[4] = {0, 256, 17, 100}, rr[4] = {16, 1, 256, 50};
        serve_pools_build(p.H, &ta, 1, 1, maxn, rr[g() % 4], narrow[g() % 4], XTED_HALF_DEFAULT);
        serve_plan_items(p.H, 0, b.lab.data(), b.off.data(), b.idx.data(), b.n, r % 3, p.q);
        size_t maps = 0;  // of the column tree's decomposition that the pair uses, and no other
        const DOTree &O = p.H.otrees[(size_t)(p.q.pairs[0].col_base == p.H.otrees[3].node_base ? 3 : 2)];
        for (int d = 0; d <= O.D; d++) {
            const DDepth &dd = p.H.depths[(size_t)(O.depth_base + d)];
            for (int c = dd.chunk_lo; c < dd.chunk_lo + dd.nnarrow + dd.nhalf + dd.nwide; c++)
                if (chunk_stripes(p.H.chunks[(size_t)c], p.H.krd.data()) > 1) maps += (size_t)p.H.chunks[(size_t)c].width;
        }
        if (p.q.smap.size() != maps) FAIL("%zu words of export maps, %zu of the columns in use", p.q.smap.size(), maps);
        const int n = (int)p.q.items.size();
        items += n;
        words += p.q.words;
        for (int k = 1; k < n; k++)
            if (p.q.items[(size_t)k].buf < p.q.items[(size_t)k - 1].buf) FAIL("hand-off words fall along the list");
        const int want = a.n + b.n - xo_distance(a.n, a.lab.data(), a.off.data(), a.idx.data(), b.n, b.lab.data(), b.off.data(), b.idx.data());
        // whole, then in parts of at most: one word (a unit each), a tenth of the words, all but one
        for (int64_t cap : {p.q.words, (int64_t)1, p.q.words / 10 + 1, std::max<int64_t>(p.q.words - 1, 1)}) {
            std::vector<int32_t> dt((size_t)p.q.dt_elems, -1);
            int np = 0;
            for (int from = 0, to; from < n; from = to, np++) {
                to = flow_cut(p.q.items.data(), n, p.q.words, from, cap);
                if (to <= from || to > n) FAIL("a part [%d, %d) of %d items", from, to, n);
                const int64_t w0 = p.q.items[(size_t)from].buf, w1 = to < n ? p.q.items[(size_t)to].buf : p.q.words;
                auto unit = [&](int k) { return std::make_pair(p.q.items[(size_t)k].run, p.q.items[(size_t)k].chunk); };
                if (to < n && unit(to) == unit(to - 1)) FAIL("a unit lies in two parts");
                if (w1 - w0 > cap)  // one unit with words, and no other
                    for (int k = from; k < to; k++)
                        if (p.q.items[(size_t)k].buf != w0) FAIL("a part of several units has %lld words", (long long)(w1 - w0));
                std::vector<int32_t> buf((size_t)(w1 - w0), -1);
                run_items(p, from, to, w0, dt, buf, p.q.smap);
            }
            if (cap >= p.q.words && np != 1) FAIL("%d parts", np);
            parts += np;
            if (dt[(size_t)p.q.pairs[0].dt_off] != want) FAIL("distance: saving %d, want %d", dt[(size_t)p.q.pairs[0].dt_off], want);
        }
        striped += p.q.words > 0;
        // as serving posts it: parts bounded in words and items, at an offset of
        // a pool that holds tables, the part's words and export maps side by side
        const int64_t item_cap = 1 + (int64_t)(g() % (uint64_t)(n + 1));
        serve_cut(p.q, p.q.words / 4 + 1, item_cap);
        const int64_t off = 4 * (int64_t)(g() % 100), at = off + p.q.dt_elems;
        serve_fixup_items(p.H, p.q, 0, off);
        std::vector<int32_t> pool((size_t)at, -1);
        pool.resize((size_t)(at + p.q.max_words), 7);
        pool.insert(pool.end(), p.q.smap.begin(), p.q.smap.end());
        if (p.q.cuts.front() != 0 || p.q.cuts.back() != n) FAIL("parts do not cover the list");
        for (size_t k = 0; k + 1 < p.q.cuts.size(); k++) {
            const int from = p.q.cuts[k], to = p.q.cuts[k + 1];
            if (to - from > p.q.max_items || p.q.part_words[k] > p.q.max_words) FAIL("a part beyond the largest");
            std::fill(pool.begin() + (long)at, pool.begin() + (long)(at + p.q.part_words[k]), -1);
            run_items(p, from, to, 0, pool, pool, pool);
        }
        if (pool[(size_t)p.q.pairs[0].dt_off] != want) FAIL("distance in parts of a pool");
        for (size_t k = 0; k < p.q.smap.size(); k++)
            if (pool[(size_t)(at + p.q.max_words) + k] != p.q.smap[k]) FAIL("an export map was overwritten");
    }
    if (striped == 0 && maxn > 600) FAIL("no striped units");
    std::printf("ok: %lld items, %lld words, %lld parts, %lld striped pairs\n", items, words, parts, striped);
    return 0;
}
