// pair_plan.h -- one pair planned and run without reading anything back
// (prep.cu: k_plan_pair). The memory is one range of fixed size: the context's
// buffer for a single small pair, or the arena of xted_distance_noalloc.
#pragma once

#include <cuda_runtime.h>

#include "plan_core.h"

namespace xted {

struct PairLayout {
    int32_t m, n;
    int32_t *raw;   // both trees (labels, offsets, children; the second from 3 m + 1 on); hdr follows
    int32_t *hdr;   // PAIR_* words, zero before the plan and between runs (the first 16); the tables follow
    int64_t upload_ints;  // raw .. the end of hdr
    int32_t *dt;
    int64_t dt_ints;
    int32_t *room;  // items | hand-off words | ... the warps' stacks from the end down
    int64_t room_ints;
    PlanPools P;
    DTree *trees;
    XChunkX *chunkx;
    int32_t *smap, *list;
    void *levels;
    int32_t cap_map, cap_list, cap_levels;
};

#define PAIR_NEXT 0       // items claimed
#define PAIR_PROGRESS 1   // items finished
#define PAIR_ERROR 2      // error code, then 4 words about it
#define PAIR_CTL_INTS 16
#define PAIR_OUT 16       // XPlanOut
#define PAIR_PAIR 32      // XPair
#define PAIR_HDR_INTS 64
#define PLAN_OVERFLOW (-100)  // XPlanOut::status: a list did not fit

// Lays a pair (m, n >= 1) out in `bytes` bytes at base (256-byte aligned; may be null to measure).
// Returns the bytes before the room, or 0 if none is left for it. Uses no heap.
size_t pair_layout(void *base, size_t bytes, int32_t m, int32_t n, PairLayout *L);
// The plan; with check, the trees are validated first (status XTED_EINVAL).
cudaError_t launch_plan_pair(const PairLayout &L, int32_t orientation, bool check, cudaStream_t s);
// Every table and hand-off word of the plan to -1 (not written).
cudaError_t launch_pair_clear(const PairLayout &L, int32_t blocks, cudaStream_t s);
void pair_params(const PairLayout &L, XKernelParams &K);
cudaError_t pair_kernels_load();  // loads the kernels above onto the current device
// Blocks of the DP launch: `grid`, or fewer for a small pair. A 100-node pair has 40 items; every
// 1,024 products of two nodes are given a block's four warps, so that no pair waits for one.
inline int32_t pair_grid(int32_t grid, int32_t m, int32_t n) {
    const int64_t want = 16 + (int64_t)m * n / 1024;
    return want < grid ? (int32_t)want : grid;
}

}  // namespace xted
