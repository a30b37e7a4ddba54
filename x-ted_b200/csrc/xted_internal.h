// xted_internal.h -- data layout shared by the host planner and the kernels.
//
// Terminology (reference names in brackets):
//   row tree A (m nodes) and column tree B (n nodes) of one pair;
//   orl(v)      rightmost leaf of v's subtree = v + size(v) - 1
//               [outermost_right_leaves, X-TED_CPU/TED.cpp:21-42];
//   keyroot     root or a node that is not the last child of its parent
//               [key_roots, X-TED_CPU/TED.cpp:46-77];
//   kdepth(k)   keyroot level: 1 + max kdepth of keyroots strictly inside
//               sub(k), 0 if none [X-TED_CPU/parallel_computing.cpp:93-119];
//   table (i0,j0) the forest-distance table of one keyroot pair, whose level
//               is kdepth(i0) + kdepth(j0) [parallel_computing.cpp:121-123].
//
// Work decomposition. All keyroots of B with the same kdepth have disjoint
// subtrees ("segments"); their columns are concatenated per depth into one
// column list. A *chunk* is a run of whole segments of one depth. A *row run*
// is a run of whole keyroots of A of one depth. A *unit* = (row run, chunk):
// every table (i0, j0) with i0 in the run and j0 in the chunk, computed row by
// row (rows descending, a suffix maximum across the chunk's columns). An *item*
// is what one warp claims: a unit, or one column stripe of a unit whose chunk
// is a segment wider than a warp holds.
#pragma once

#include <stdint.h>
#include <vector_types.h>  // int2, int4 (CUDA toolkit header, host-includable)

#define XTED_CTA_THREADS 256
#define XTED_WARPS (XTED_CTA_THREADS / 32)
#define XTED_NARROW_MAX 256       // widest chunk of several segments (8 columns per lane)
#define XTED_KEY_BIG (1 << 17)    // key step between segments of one chunk
#define XTED_INF 0x3fffffff

// rowinfo.y bit layout: orl in the low 20 bits.
#define XTED_ROW_ORL_MASK 0x000fffff
#define XTED_ROW_ISKR (1u << 29)     // node is a keyroot
#define XTED_ROW_PREVLEAF (1u << 30) // node i-1 is a leaf

// Node record (both trees use the same pool): x = label, y = orl | flags.

// Granularity of one tree-size bucket: trees with fewer than max_n nodes use
// this row-run length and this widest chunk of several segments (half_width: no effect on the launch).
#define XTED_TUNE_ROWS 8
struct XTuneRow {
    int32_t max_n, run_rows, narrow_width, half_width;
};

struct XRun {      // a run of keyroots of one depth of a row tree
    int32_t kr_lo; // index into the keyroot pool (global)
    int32_t kr_hi;
    int32_t rows;  // total rows = sum of subtree sizes
    int32_t depth;
};

struct XChunk {     // a run of whole segments of one depth of a column tree
    int32_t k_lo;   // keyroot-pool index of its first segment
    int32_t width;
    int32_t depth;
    int32_t nseg;
};

struct XPair {
    int64_t dt_off;   // element offset of this pair's m x n distance table
    int32_t m, n;     // rows (A) and columns (B)
    int32_t row_base; // index of A's node 0 in the node-record pool
    int32_t col_base; // index of B's node 0 in the node-record pool
    int32_t pitch;    // row pitch of the table: n rounded up to XTED_PITCH columns
    int32_t pad;
};

// From here to XEntry: the level schedule of plan_core.h, blocks that run units
// level by level. The launch has only items; the schedule is what
// tests/cpp/plan_emu.cpp and serve_emu.cpp run over the same trees, runs and chunks.
struct XUnit {
    int32_t run;   // global run index (row tree)
    int32_t chunk; // global chunk index (column tree)
};

#define XTED_WIDE_REG_MAX 2048      // widest chunk of a whole-block unit, wider ones in column stripes
#define XTED_HALF_MAX 1024          // ... of a half-block unit
#define XTED_HALF_DEFAULT 512
#define XTED_TASK_WIDE 0x80000000u  // one unit run by a whole block
#define XTED_TASK_HALF 0x40000000u  // units run by a block's two halves
#define XTED_TASK_STRIPED 0x20000000u  // (with WIDE) one column stripe of a striped unit, rightmost first:
                                    // kind_n = WIDE | STRIPED | (stripe << XTED_STRIPE_SHIFT) | 1
#define XTED_STRIPE_SHIFT 16
#define XTED_STRIPE_MASK 0xfffu
#define XTED_STRIPE 2048        // widest stripe (8 columns per thread)
#define XTED_STRIPE_MIN_W 2     // narrowest stripe: 2 columns per thread (512 columns)
#define XTED_STRIPES_MAX 128    // stripes of one unit: a wider segment takes wider stripes

struct XStripe {       // a striped unit
    int32_t unit;      // its unit
    int32_t K;         // stripes
    int32_t sww;       // columns per thread: a stripe is 256 * sww columns
    int32_t X;         // far columns read across a stripe boundary
    int32_t w, R;      // width (one segment) and rows
    int32_t pair, pad;
    int64_t map_off;   // its export map (w ints): column -> export index, or -1
    int64_t buf_off;   // its hand-off words
};

#ifndef XTED_TASK_UNITS
#define XTED_TASK_UNITS 32   // narrow units per task
#endif

struct XTask {
    int32_t pair;
    int32_t entry;    // its (pair, level) entry
    uint32_t kind_n;  // XTED_TASK_* | number of units
    int32_t unit_lo;  // first unit
};

#define XTED_BUCKETS 16
struct XEntry {
    int32_t task_off;  // first task
    int32_t ntasks;
    int32_t bucket;    // priority: larger = longer remaining critical path of the pair
    int32_t next;      // entry of the pair's next level, -1 after the last level
    int32_t nnarrow;   // tasks [task_off, task_off + nnarrow) are narrow, the rest group tasks
    int32_t pad;
};

// ---- the DP launch (flow.cu) ----
//
// Every warp of the launch claims *items* from one list and runs each to its
// end. An item is a unit (row run x chunk) or, for a single segment wider
// than a warp holds, one column stripe of a unit. The list is sorted so that
// an item only needs values of items before it: a unit of keyroot depths
// (a, b) reads tables of depths (a', b') with a' <= a, b' <= b, and the
// stripes of a unit go rightmost first. A warp that needs a value which is not
// there yet waits for it: every word that one item writes for another starts
// at -1 and is written once, with a value >= 0.
#define XTED_PITCH 4          // rows of a table start on 16 bytes
#define XTED_SW 256           // columns of a stripe: the widest slice one warp holds (8 per lane)
#define XTED_FLOW_WARPS 4     // warps per block, each with its own shared memory

struct XItem {
    int32_t run, chunk, pair;
    int32_t stripe;           // stripe of the unit's chunk (0 for a chunk one warp holds)
    int64_t buf;              // striped unit: its hand-off words in XKernelParams::buf
    int32_t gen;              // serving: the generation of its list
    int32_t pad;
};

// What a column chunk adds to the plan (same index as its XChunk).
struct XChunkX {
    int32_t K;     // stripes (1: one warp holds the chunk)
    int32_t kpre;  // stripes of the chunks before it at its depth
    int32_t X;     // columns that a stripe further left reads as far columns
    int32_t wpre;  // hand-off words per row of the chunks before it at its depth
    int64_t map;   // striped: its export map in XKernelParams::smap (width ints: export index or -1)
};

// A plan made without reading anything back (k_plan_pair): what the launch
// needs of it, in device memory.
struct XPlanOut {
    int32_t items, stack_rows, levels;
    int32_t status;  // nonzero: no plan, nothing to run
    int64_t cells, cells_right;
    int64_t words, scratch;  // hand-off words; ints left for the warps' stacks
};

// What a serving list's warps set to -1 before they run its items: n words of
// the table pool from off on (16-byte aligned), in pieces of XTED_CLEAR_INTS.
#define XTED_CLEAR_INTS 16384
struct XServeClear {
    int64_t off, n;
    int32_t pieces, claimed, done, pad;
};

struct XKernelParams {
    const int2 *rowinfo;  // node records of every oriented tree
    const int32_t *krd;   // keyroots grouped by depth (node ids within their tree)
    const int32_t *cumw;  // position of each keyroot's segment in its depth's column list
    const XRun *runs;
    const XChunk *chunks;
    const XChunkX *chunkx;
    const XPair *pairs;
    const XItem *items;
    int32_t *dt;          // every pair's tree-distance savings, -1 = not computed yet
    int32_t *buf;         // hand-off words of striped units, -1 = not written yet
    const int32_t *smap;  // export maps of striped chunks
    int32_t *scratch;     // per-warp far-row stacks: rows that left the shared window
    int64_t scratch_per_warp;  // int32 elements
    int32_t stack_rows;   // stack capacity in rows
    int32_t nitems, npairs;
    const XPlanOut *plan;  // if set: in place of nitems and stack_rows; the stacks lie below scratch, and
                           // warps whose stack does not fit leave at once
    int32_t *next;        // items claimed (batch launch)
    int32_t *progress;    // items finished
    int32_t *error;       // 0 = ok; else an XTED error code
    int32_t *error_info;  // [4] diagnostics of the first error
    uint64_t timeout_ns;  // bound on every wait, without progress of any item
    unsigned long long *trace; // optional, 4 words per item: claim ns, start ns, end ns, info
    // ---- serving session (serve = 1); a batch launch leaves these zero ----
    int32_t serve;
    uint64_t idle_exit_ns;  // the launch ends once every warp has had no work for this long
    unsigned long long *lists;  // [XTED_SERVE_SLOTS] (end << 32) | next item of the slot's list
    XServeClear *clears;    // [XTED_SERVE_SLOTS]
    const int32_t *ages;    // [XTED_SERVE_SLOTS] arrival number of the slot's query
    int32_t *ctl;           // XTED_CTL_* words
    int32_t *slot_done;     // [XTED_SERVE_SLOTS] items finished in the slot's current round
    const int32_t *slot_need, *slot_gen;  // items to finish, generation to report
    int32_t *results;       // [slots * serve_pairs] distances, mapped host memory
    int32_t *flags;         // [XTED_SERVE_SLOTS] generation of the last finished round, mapped host memory
    // ---- test hook (xted_test_fault): level 0 of this pair is never computed; -1: none ----
    int32_t hold_pair;
    // ---- edit costs: delete a row-tree node, insert a column-tree node, change a label ----
    int32_t c_del, c_ins, c_ren;
};

#define XTED_SERVE_SLOTS 16
#define XTED_CTL_IDLE 0     // warps currently without work
#define XTED_CTL_CLOSED 1   // nonzero: the launch is ending, warps claim nothing more
#define XTED_CTL_STOP 2     // nonzero: warps leave when idle (host)
#define XTED_CTL_PROGRESS 3 // items finished
#define XTED_CTL_INTS 8
