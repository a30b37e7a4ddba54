// tune_table.h -- granularity per tree-size bucket, read and rewritten by
// x-ted_b200/xted/autotune.py, which measures candidates bucket by bucket and
// keeps a changed row only if whole mixed batches gain. The present rows were set
// from the measurements below, all buckets alike.
//
// Row k applies to trees with fewer than max_n nodes (the last row to all
// larger ones): the row-run length of the tree as a row tree, and the widest
// chunks of several segments of the tree as a column tree (the last column has no effect).
// batch of 4,096 pairs of 50-1,000 nodes, DP ms: 160.1 with narrow 128 and runs of 32-128 rows by size;
// narrow 256: runs of 64 rows 145.9, 128 144.5, 192 144.2, 256 144.1, 512 143.9
// 1,024 pairs: 42.5 before; narrow 256 with 64 / 128 / 256 rows 38.3 / 38.2 / 38.4
// 20,000 x 20,000 random: 56.6 before; narrow 256 with 64 / 128 / 256 / 512 rows 50.2 / 48.9 / 47.6 / 47.1
// (a launch of few cells takes shorter runs than these: ctx_granularity)
#pragma once

#include "xted_internal.h"

static const XTuneRow kTuneTable[] = {
    {128, 256, 256, -1},
    {256, 256, 256, -1},
    {512, 256, 256, -1},
    {1024, 256, 256, -1},
    {2048, 256, 256, -1},
    {1 << 30, 256, 256, -1},
};
static const int kTuneRows = (int)(sizeof(kTuneTable) / sizeof(kTuneTable[0]));
