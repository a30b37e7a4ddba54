// flow_plan.h -- the item list of the DP launch (flow.cu), as functions of
// one chunk, one level or one item, so that the planning kernels (prep.cu)
// and the host planner of serving queries (serve_plan.h) lay out the same
// list.
//
// A level of a pair is the set of tables whose keyroot depths add up to it.
// Its units are (row run of depth a) x (column chunk of depth d - a); a chunk
// of one segment too wide for a warp gives every unit K stripes, each an item
// of its own, rightmost first. The items of a level are laid out by row depth
// from the deepest down, so the longest runs start first.
#pragma once

#include "plan_core.h"

namespace xted {

// Stripes of a chunk: stripe s covers the nodes [base + s SW, base + (s+1) SW)
// of the column tree, base = the segment's first node rounded down to
// XTED_PITCH (16-byte copies of a table row start there).
XT_HD inline int32_t chunk_stripes(const XChunk &c, const int32_t *krd) {
    if (c.nseg != 1) return 1;
    const int32_t lead = krd[c.k_lo] & (XTED_PITCH - 1);
    return (lead + c.width + XTED_SW - 1) / XTED_SW;
}

// Column c of a striped segment is in stripe (lead + c) / SW. Its far column
// f = c + foff is read across a stripe boundary if it lies in another stripe
// (and inside the segment): column f is then exported.
XT_HD inline bool far_crosses(int32_t c, int32_t foff, int32_t width, int32_t lead) {
    const int32_t f = c + foff;
    return f < width && (lead + f) / XTED_SW != (lead + c) / XTED_SW;
}

XT_HD inline int32_t table_pitch(int32_t n) { return (n + XTED_PITCH - 1) & ~(XTED_PITCH - 1); }

struct FlowCtx {
    const DOTree *ot;
    const DDepth *depths;
    const XRun *runs;
    const XChunk *chunks;
    const XChunkX *chunkx;
    const int32_t *cumw;
};

// Items and hand-off words of level d of a pair (row tree A, column tree B),
// and an estimate of its time (only its order of magnitude matters: it ranks
// pairs by the work left behind their slowest tables).
XT_HD inline void flow_level_count(const FlowCtx &C, const DOTree &A, const DOTree &B, int d, int64_t *items,
                                   int64_t *words, int64_t *est) {
    const DDepth *da = C.depths + A.depth_base, *db = C.depths + B.depth_base;
    const int lo = d - B.D > 0 ? d - B.D : 0, hi = A.D < d ? A.D : d;
    int64_t n = 0, w = 0, e = 0;
    for (int a = lo; a <= hi; a++) {
        const DDepth &ra = da[a], &cb = db[d - a];
        n += (int64_t)(ra.run_hi - ra.run_lo) * cb.nitems;
        w += (int64_t)ra.rows * cb.wsum;
        if (ra.maxrows > e) e = ra.maxrows;
    }
    *items = n;
    *words = w;
    *est = e + 1;
}

// Item `at` of the items of row depth a at level d; buf is the level's (and
// depth's) first hand-off word.
XT_HD inline XItem flow_item(const FlowCtx &C, const DDepth &ra, const DDepth &cb, int32_t pair, int64_t at,
                             int64_t buf) {
    const int32_t KS = cb.nitems, nch = cb.nnarrow + cb.nhalf + cb.nwide;
    const int32_t r = ra.run_lo + (int32_t)(at / KS), k = (int32_t)(at % KS);
    XItem it;
    it.run = r;
    it.pair = pair;
    it.gen = it.pad = 0;
    int32_t c = cb.chunk_lo + k;
    it.stripe = 0;
    it.buf = buf;
    if (KS != nch) {  // some chunk of this depth is striped: the last one whose kpre <= k
        int32_t lo = cb.chunk_lo, hi = cb.chunk_lo + nch - 1;
        while (lo < hi) {
            const int32_t mid = (lo + hi + 1) >> 1;
            if (C.chunkx[mid].kpre <= k) lo = mid;
            else hi = mid - 1;
        }
        c = lo;
        const XChunkX &x = C.chunkx[c];
        it.stripe = x.K - 1 - (k - x.kpre);
        // hand-off words: the depth's runs in order, in a run its chunks in order
        it.buf = buf + (int64_t)C.cumw[C.runs[r].kr_lo] * cb.wsum + (int64_t)C.runs[r].rows * x.wpre;
    }
    it.chunk = c;
    return it;
}

// A list whose hand-off words exceed the buffer runs in parts, launches one
// after another that each use the buffer from its start: an item needs items
// before it, whose part has ended. `buf` never falls along the list, and a unit's
// words end where the next unit's begin. Returns the end of the part that
// starts at item g: whole units of at most cap words together, or one unit alone.
XT_HD inline int32_t flow_cut(const XItem *items, int32_t n, int64_t words, int32_t g, int64_t cap) {
    const int64_t top = items[g].buf + cap;
    if (words <= top) return n;
    int32_t lo = g, hi = n - 1;  // the last item whose words start at or below top ...
    while (lo < hi) {
        const int32_t mid = lo + (hi - lo + 1) / 2;
        if (items[mid].buf <= top) lo = mid;
        else hi = mid - 1;
    }
    const int32_t last = lo;
    lo = g, hi = last;  // ... and the first of those with the same start: its unit may end above top
    while (lo < hi) {
        const int32_t mid = lo + (hi - lo) / 2;
        if (items[mid].buf < items[last].buf) lo = mid + 1;
        else hi = mid;
    }
    return lo > g ? lo : last + 1;
}

// Hand-off words per row of a chunk: the first column of every stripe but the
// leftmost, and the exported columns.
XT_HD inline int32_t chunk_words(int32_t K, int32_t X) { return K > 1 ? K - 1 + X : 0; }

// Export map of a striped chunk (sequentially; k_chunk_maps in prep.cu does
// the same with a block); nodes are the column tree's records. Returns X.
XT_HD inline int32_t chunk_export_map(const XChunk &c, const int32_t *krd, const int2 *nodes, int32_t *map) {
    const int32_t j0 = krd[c.k_lo], lead = j0 & (XTED_PITCH - 1);
    for (int32_t k = 0; k < c.width; k++) map[k] = -1;
    for (int32_t k = 0; k < c.width; k++) {
        const int32_t foff = (nodes[j0 + k].y & XTED_ROW_ORL_MASK) + 1 - (j0 + k);
        if (far_crosses(k, foff, c.width, lead)) map[k + foff] = 0;
    }
    int32_t X = 0;
    for (int32_t k = 0; k < c.width; k++)
        if (map[k] == 0) map[k] = X++;
    return X;
}

// The item totals of one depth of one oriented tree, from its chunks' K and X
// (sequentially; prep.cu does the same with a warp).
XT_HD inline void flow_depth_totals(DDepth &dd, const XRun *runs, const int32_t *cumw, XChunkX *chunkx) {
    int32_t k = 0, w = 0;
    for (int32_t c = dd.chunk_lo; c < dd.chunk_lo + dd.nnarrow + dd.nhalf + dd.nwide; c++) {
        chunkx[c].kpre = k;
        chunkx[c].wpre = w;
        k += chunkx[c].K;
        w += chunk_words(chunkx[c].K, chunkx[c].X);
    }
    dd.nitems = k;
    dd.wsum = w;
    dd.rows = dd.run_hi > dd.run_lo ? cumw[runs[dd.run_hi - 1].kr_lo] + runs[dd.run_hi - 1].rows : 0;
}

}  // namespace xted
