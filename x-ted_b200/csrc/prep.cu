// prep.cu -- device-side preprocessing and work decomposition of a batch.
//
// The reference computes orl, keyroots and keyroot depths on the host, then
// for every depth level fetches, sizes, sorts and bins tables with host
// round trips (X-TED_CPU/TED.cpp:163-166, X-TED_GPU/parallel_X_TED.cu:184-224,
// 304-387). Here the raw trees go up once and everything else is built on the
// device, a warp or a block per tree / oriented tree, one thread per pair / (pair, level):
//
//   k_tree_basic   sizes, depths, parents, keyroot-size sums (both decompositions)
//   k_orient       per orientation: node records, kdepth, keyroots by depth,
//                  column-list positions, row runs, column chunks (the records
//                  plan_core.h's orient_tree builds for the host planners)
//   k_pair_setup   decomposition choice, level count
//   k_map_reserve, k_chunk_maps   export maps of column chunks too wide for a warp
//   k_depth_totals items and hand-off words per keyroot depth (flow_plan.h)
//   k_level_*      item counts per (pair, level), the levels in the order of
//                  the launch's list, then the items themselves
//
// The list holds the levels of all pairs by the time estimated to be left of
// their pair behind them, longest first (a pair's levels in order), so the
// pairs with the longest chains of tables start first and the launch ends
// with short ones. Two small device-to-host reads size the buffers.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "ctx.h"
#include "flow_plan.h"
#include "pair_plan.h"
#include "plan_core.h"

namespace xted {

namespace {

__device__ __forceinline__ int warp_incl_sum(int v, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += o;
    }
    return v;
}

// The threads that plan one tree together: a warp for trees of up to
// PLAN_WARP_NODES nodes (four trees to a block), a block of 1,024 threads
// beyond. A batch's thousands of small trees fill the GPU with warps; one
// large tree leaves it idle: the two 20,000-node caterpillars took 2.2 ms in
// k_tree_basic and 13.1 ms in k_orient with a warp each.
#define PLAN_WARP_NODES 1024
#define PLAN_BLOCK_TREES 296  // more trees than this (two blocks an SM) fill the GPU with a warp each
template <int NT>
struct Team {
    static constexpr int WARPS = NT / 32;
    int tid;
    int *part;  // shared, [WARPS + 1] (blocks)
    __device__ void sync() const {
        if (NT == 32) __syncwarp();
        else __syncthreads();
    }
    // inclusive sum over the team's threads, and its total
    __device__ int incl_sum(int v, int *total) const {
        const int lane = tid & 31, w = tid >> 5;
        int x = warp_incl_sum(v, lane);
        if (NT == 32) {
            *total = __shfl_sync(0xffffffffu, x, 31);
            return x;
        }
        if (lane == 31) part[w] = x;
        __syncthreads();
        if (w == 0) {
            const int y = warp_incl_sum(lane < WARPS ? part[lane] : 0, lane);
            if (lane < WARPS) part[lane] = y;
        }
        __syncthreads();
        if (w > 0) x += part[w - 1];
        *total = part[WARPS - 1];
        __syncthreads();
        return x;
    }
    __device__ bool any(bool p) const {
        if (NT == 32) return __any_sync(0xffffffffu, p);
        return __syncthreads_or(p) != 0;
    }
};

// The outputs of tree_basic (plan_core.h: sizes, depths and parents of every
// node, the keyroot-size sums of both decompositions), with the work spread
// over the team: parents straight from the child lists; each node's orl
// (rightmost leaf) by pointer jumping along last children, its size orl - v +
// 1; depths as a prefix sum of +1 at every node and -1 just past its subtree (u
// is an ancestor of v exactly when u <= v <= orl(u)); the sums as thread sums.
template <int NT>
__device__ void tree_basic_team(const Team<NT> &team, const PlanPools &P, int t, DTree *trees_out, int64_t (*acc)[32]) {
    DTree T = P.trees[t];
    const int n = T.n, tid = team.tid;
    const int32_t *off = P.raw + T.raw + n, *idx = P.raw + T.raw + 2 * n + 1;
    int32_t *size = P.size + T.nbase, *depth = P.depth + T.nbase, *par = P.parent + T.nbase;
    int32_t *jump = P.opar + 2 * (int64_t)T.nbase;  // scratch: this tree's orientation pool, unused until k_orient
    if (n > 0) {
        for (int v = tid; v < n; v += NT) {
            const int32_t lo = off[v], hi = off[v + 1];
            for (int32_t e = lo; e < hi; e++) par[idx[e]] = v;
            size[v] = hi > lo ? idx[hi - 1] : v;  // last child, or the node itself for a leaf
            depth[v] = 0;
        }
        if (tid == 0) par[0] = -1;
        team.sync();
        int32_t *cur = size, *nxt = jump;
        for (int round = 0; round < 32; round++) {
            bool changed = false;
            for (int v = tid; v < n; v += NT) {
                const int32_t a = cur[v], b = cur[a];
                nxt[v] = b;
                changed |= b != a;
            }
            team.sync();
            int32_t *tmp = cur;
            cur = nxt;
            nxt = tmp;
            if (!team.any(changed)) break;
        }
        // cur[v] = orl(v). Depth: +1 at every u, -1 at orl(u) + 1, then an inclusive prefix sum
        for (int u = tid; u < n; u += NT) {
            atomicAdd(&depth[u], 1);
            const int32_t o1 = cur[u] + 1;
            if (o1 < n) atomicSub(&depth[o1], 1);
        }
        team.sync();
        int carry = 0;
        for (int base = 0; base < n; base += NT) {
            const int v = base + tid;
            int total;
            const int x = team.incl_sum(v < n ? __ldcg(&depth[v]) : 0, &total);
            if (v < n) depth[v] = carry + x - 1;
            carry += total;
        }
        for (int v = tid; v < n; v += NT) size[v] = cur[v] - v + 1;
        team.sync();
        // keyroot-size sums, right path and left path: all subtree sizes less
        // those of last (first) children
        int64_t sr = 0, sl = 0;
        for (int v = tid; v < n; v += NT) {
            const int32_t lo = off[v], hi = off[v + 1];
            const int64_t z = size[v];
            sr += z;
            sl += z;
            if (hi > lo) {
                sr -= size[idx[hi - 1]];
                sl -= size[idx[lo]];
            }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            sr += __shfl_down_sync(0xffffffffu, sr, d);
            sl += __shfl_down_sync(0xffffffffu, sl, d);
        }
        if (NT == 32) {
            T.S[0] = sr;
            T.S[1] = sl;
        } else {
            if ((tid & 31) == 0) {
                acc[0][tid >> 5] = sr;
                acc[1][tid >> 5] = sl;
            }
            __syncthreads();
            T.S[0] = T.S[1] = 0;
            for (int w = 0; w < Team<NT>::WARPS; w++) {
                T.S[0] += acc[0][w];
                T.S[1] += acc[1][w];
            }
        }
    } else {
        T.S[0] = T.S[1] = 0;
    }
    if (tid == 0) trees_out[t] = T;
    team.sync();
}

template <int NT>
__global__ void k_tree_basic(PlanPools P, DTree *trees_out) {
    __shared__ int part[33];
    __shared__ int64_t acc[2][32];
    const Team<NT> team{NT == 32 ? (int)(threadIdx.x & 31) : (int)threadIdx.x, part};
    const int t = NT == 32 ? (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) : (int)blockIdx.x;
    if (t < P.ntrees) tree_basic_team<NT>(team, P, t, trees_out, acc);  // whole teams
}

// The decomposition of every pair (as pair_setup chooses it), so that k_orient
// builds each tree in the orientations that some pair needs only: the left
// path of a caterpillar has a keyroot depth per spine node and took nearly all
// of its planning, for nothing.
__global__ void k_pair_orient(const DTree *trees, const int32_t *pair_trees, int orientation, int npairs,
                              int32_t *need) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npairs) return;
    const int ta = pair_trees[2 * p], tb = pair_trees[2 * p + 1];
    const DTree &A = trees[ta], &B = trees[tb];
    if (A.n == 0 || B.n == 0) return;
    const int o = pair_orientation(A, B, orientation);
    need[2 * ta + o] = 1;
    need[2 * tb + o] = 1;
}

// One team per oriented tree: the records of orient_tree (plan_core.h, which
// the host planners run), with its passes spread over the threads:
//   * node records and the previous-node-is-leaf flags: one node per thread;
//   * A(x), the keyroots on x's root path (x included): a prefix sum over
//     preorder of +1 at each keyroot and -1 just past its subtree;
//   * keyroot depth kd(u) = (max of A over u's subtree) - A(u), the height of u
//     among the keyroots nested in it: each thread scans the subtrees of its
//     keyroots, over the maxima of 32 nodes at a time where they fit;
//   * keyroots grouped by depth in preorder: a counting sort by one warp, 32
//     nodes at a time, lanes of one depth ranked by lane;
//   * row runs and column chunks per depth, a depth per warp: sizes and column
//     positions loaded and summed 32 keyroots at a time, the greedy packing
//     then decided by the whole warp from shuffled sizes (every lane holds the
//     same packing state). A depth's runs and chunks start at its first keyroot's
//     place in the pools, so the depths do not wait for each other. The launch
//     takes chunks of every width alike: all count as narrow.
template <int NT>
__device__ void orient_team(const Team<NT> &team, const PlanPools &P, int ot, bool needed, int *s_max) {
    const unsigned FULL = 0xffffffffu;
    const int tid = team.tid, lane = tid & 31, warp = tid >> 5;
    const int t = ot >> 1, o = ot & 1;
    const DTree T = P.trees[t];
    const int n = T.n;
    DOTree O;
    O.n = n;
    O.node_base = 2 * T.nbase + o * n;
    O.depth_base = 2 * (T.nbase + t) + o * (n + 1);
    O.D = -1;
    O.maxka = 0;
    O.maxw_wide = 0;
    O.S = T.S[o];
    if (n == 0 || !needed) {
        if (tid == 0) P.otrees[ot] = O;
        return;
    }
    const int32_t *lab = P.raw + T.raw;
    const int32_t *off = P.raw + T.raw + n;
    const int32_t *idx = P.raw + T.raw + 2 * n + 1;
    const int32_t *size = P.size + T.nbase, *depth = P.depth + T.nbase, *par = P.parent + T.nbase;
    int2 *node = P.node + O.node_base;
    int32_t *okd = P.okd + O.node_base, *oka = P.oka + O.node_base, *bmax = P.opar + O.node_base;
    // node records in this orientation
    for (int v = tid; v < n; v += NT) {
        const int32_t u = o ? mirror_id(v, n, size, depth) : v;
        bool kr = true;
        if (v > 0) {
            const int32_t p = par[v];
            kr = o ? idx[off[p]] != v : idx[off[p + 1] - 1] != v;
        }
        node[u].x = lab[v];
        node[u].y = (int32_t)((uint32_t)(u + size[v] - 1) | (kr ? XTED_ROW_ISKR : 0u));
        oka[u] = 0;
    }
    team.sync();
    for (int u = 1 + tid; u < n; u += NT) {
        const int32_t prev_orl = node[u - 1].y & XTED_ROW_ORL_MASK;  // (its flag bits may change meanwhile)
        if (prev_orl == u - 1) node[u].y = (int32_t)((uint32_t)node[u].y | XTED_ROW_PREVLEAF);
    }
    // A(x): +1 at a keyroot, -1 just past its subtree, summed over preorder
    for (int u = tid; u < n; u += NT) {
        const int32_t y = node[u].y;
        if (y & XTED_ROW_ISKR) {
            atomicAdd(&oka[u], 1);
            const int e = (y & XTED_ROW_ORL_MASK) + 1;
            if (e < n) atomicSub(&oka[e], 1);
        }
    }
    if (tid == 0) *s_max = 1;
    team.sync();
    int carry = 0, maxa = 1;
    for (int base = 0; base < n; base += NT) {
        const int x = base + tid;
        int total;
        const int a = carry + team.incl_sum(x < n ? __ldcg(&oka[x]) : 0, &total);
        if (x < n) {
            oka[x] = a;
            maxa = max(maxa, a);
        }
        const int wm = __reduce_max_sync(FULL, x < n ? a : 0);
        if (lane == 0 && x < n) bmax[x >> 5] = wm;  // the maximum of 32 nodes
        carry += total;
    }
    maxa = __reduce_max_sync(FULL, maxa);
    if (NT == 32) {
        O.maxka = maxa;
        __syncwarp();
    } else {
        if (lane == 0) atomicMax(s_max, maxa);
        __syncthreads();
        O.maxka = *s_max;
    }
    // keyroot depths
    DDepth *dep = P.depths + O.depth_base;
    for (int u = tid; u < n; u += NT) {
        const int32_t y = node[u].y;
        int kd = -1;
        if (y & XTED_ROW_ISKR) {
            const int e = (y & XTED_ROW_ORL_MASK) + 1, au = oka[u];
            int m = au, x = u + 1;
            for (; x < e && (x & 31); x++) m = max(m, oka[x]);
            for (; x + 32 <= e; x += 32) m = max(m, bmax[x >> 5]);
            for (; x < e; x++) m = max(m, oka[x]);
            kd = m - au;
        }
        okd[u] = kd;
    }
    team.sync();
    const int D = okd[0];  // the root is a keyroot
    O.D = D;
    // keyroots grouped by depth (counting sort, preorder inside a depth)
    for (int d = tid; d <= D; d += NT) {
        dep[d].krd_lo = 0;
        dep[d].krd_hi = 0;
    }
    team.sync();
    for (int u = tid; u < n; u += NT)
        if (okd[u] >= 0) atomicAdd(&dep[okd[u]].krd_hi, 1);
    team.sync();
    carry = O.node_base;
    for (int base = 0; base <= D; base += NT) {
        const int d = base + tid;
        const int c = d <= D ? __ldcg(&dep[d].krd_hi) : 0;
        int total;
        const int incl = team.incl_sum(c, &total);
        if (d <= D) {
            dep[d].krd_lo = carry + incl - c;
            dep[d].krd_hi = carry + incl - c;  // fill cursor
        }
        carry += total;
    }
    team.sync();
    if (NT == 32 || warp == 0) {
        const unsigned below = (1u << lane) - 1u;
        for (int base = 0; base < n; base += 32) {
            const int u = base + lane;
            const int kd = u < n ? okd[u] : -1;
            const unsigned same = __match_any_sync(FULL, kd);  // lanes holding keyroots of this depth
            if (kd >= 0) {
                const int leader = __ffs(same) - 1;
                int at = 0;
                if (lane == leader) {
                    at = dep[kd].krd_hi;
                    dep[kd].krd_hi = at + __popc(same);
                }
                at = __shfl_sync(same, at, leader);
                P.krd[at + __popc(same & below)] = u;
            }
            __syncwarp();
        }
    }
    team.sync();
    // column-list positions, row runs and chunks per depth
    int run_rows, nw, hw;
    tree_granularity(P, n, &run_rows, &nw, &hw);
    const int group_w = nw > 0 ? nw : XTED_NARROW_MAX;
    for (int d = warp; d <= D; d += Team<NT>::WARPS) {
        DDepth dd = dep[d];  // krd_lo, krd_hi
        const int klo = dd.krd_lo, khi = dd.krd_hi;
        int run_cur = klo, chunk_cur = klo;
        dd.run_lo = dd.chunk_lo = klo;
        dd.maxrows = 0;
        int pos = 0, r_lo = klo, r_rows = 0, c_lo = klo, c_w = 0;
        for (int kb = klo; kb < khi; kb += 32) {
            const int k = kb + lane;
            int sz = 0;
            if (k < khi) {
                const int32_t u = P.krd[k];
                sz = (node[u].y & XTED_ROW_ORL_MASK) - u + 1;
            }
            const int incl = warp_incl_sum(sz, lane);
            if (k < khi) P.cumw[k] = pos + incl - sz;
            pos += __shfl_sync(FULL, incl, 31);
            const int cnt = min(32, khi - kb);
            for (int j = 0; j < cnt; j++) {
                const int szj = __shfl_sync(FULL, sz, j), kk = kb + j;
                if (r_rows > 0 && r_rows + szj > run_rows) {
                    dd.maxrows = max(dd.maxrows, r_rows);
                    if (lane == 0) P.runs[run_cur] = XRun{r_lo, kk, r_rows, d};
                    run_cur++;
                    r_lo = kk;
                    r_rows = 0;
                }
                r_rows += szj;
                if (c_w > 0 && c_w + szj > group_w) {
                    if (lane == 0) P.chunks[chunk_cur] = XChunk{c_lo, c_w, d, kk - c_lo};
                    chunk_cur++;
                    c_lo = kk;
                    c_w = 0;
                }
                c_w += szj;
            }
        }
        dd.maxrows = max(dd.maxrows, r_rows);
        if (lane == 0) {
            P.runs[run_cur] = XRun{r_lo, khi, r_rows, d};
            P.chunks[chunk_cur] = XChunk{c_lo, c_w, d, khi - c_lo};
        }
        dd.run_hi = run_cur + 1;
        dd.nnarrow = chunk_cur + 1 - klo;
        dd.nhalf = dd.nwide = 0;
        if (lane == 0) dep[d] = dd;
        __syncwarp();
    }
    if (tid == 0) P.otrees[ot] = O;
    team.sync();
}

template <int NT>
__global__ void k_orient(PlanPools P, const int32_t *need) {
    __shared__ int part[33];
    __shared__ int s_max;
    const Team<NT> team{NT == 32 ? (int)(threadIdx.x & 31) : (int)threadIdx.x, part};
    const int ot = NT == 32 ? (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) : (int)blockIdx.x;
    if (ot < 2 * P.ntrees) orient_team<NT>(team, P, ot, need[ot] != 0, &s_max);  // whole teams
}

__global__ void k_pair_setup(const DTree *trees, const DOTree *ot, const int32_t *pair_trees, int orientation,
                             int npairs, DPair *pairs, int64_t *L, int64_t *cells, int32_t *used) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npairs) return;
    pair_setup(trees, ot, pair_trees, orientation, p, pairs);
    const DPair q = pairs[p];
    L[p] = q.L;
    cells[p] = q.trivial >= 0 ? 0 : (int64_t)trees[q.ta].n * table_pitch(trees[q.tb].n);
    if (q.trivial < 0) used[2 * q.tb + q.o] = 1;  // a column tree
}

// Exclusive scan of n int64 values in one block; out[n] = total.
__global__ void k_scan64(const int64_t *v, int n, int64_t *out) {
    __shared__ int64_t part[1024];
    const int tid = threadIdx.x, nt = blockDim.x;
    const int per = (n + nt - 1) / nt;
    const int lo = min(tid * per, n), hi = min(lo + per, n);
    int64_t s = 0;
    for (int i = lo; i < hi; i++) s += v[i];
    part[tid] = s;
    __syncthreads();
    for (int d = 1; d < nt; d <<= 1) {
        int64_t x = tid >= d ? part[tid - d] : 0;
        __syncthreads();
        part[tid] += x;
        __syncthreads();
    }
    int64_t run = part[tid] - s;
    for (int i = lo; i < hi; i++) {
        out[i] = run;
        run += v[i];
    }
    if (tid == nt - 1) out[n] = part[nt - 1];
}

#define PLAN_PAIR_THREADS 1024
#define ITEM_INTS ((int64_t)(sizeof(XItem) / sizeof(int32_t)))

struct Summary {
    int64_t entries, dt_elems;
    int64_t items, words;        // items of the launch, hand-off words of striped units
    int64_t map_ints;            // export maps of striped chunks
    int32_t nmaps, stack_rows;
    int64_t cells, cells_right;
    int32_t levels_max, pad;
    int64_t chain_max;
};

__global__ void k_pair_offsets(DPair *pairs, const DTree *trees, const DOTree *ot, int npairs, const int64_t *Lscan,
                               const int64_t *dtscan, Summary *sum) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) {
        sum->entries = Lscan[npairs];
        sum->dt_elems = dtscan[npairs];
    }
    if (p >= npairs) return;
    DPair &q = pairs[p];
    q.lvl_base = (int32_t)Lscan[p];
    q.dt_off = dtscan[p];
    if (q.trivial < 0) {
        const DOTree &A = ot[2 * q.ta + q.o];
        atomicMax(&sum->stack_rows, A.maxka + 1);
        atomicMax(&sum->levels_max, q.L);
        atomicAdd((unsigned long long *)&sum->cells, (unsigned long long)q.cells);
        atomicAdd((unsigned long long *)&sum->cells_right,
                  (unsigned long long)(trees[q.ta].S[0] * trees[q.tb].S[0]));
    }
}

// A warp per oriented tree: reserves export-map space for the striped chunks
// of the trees that some pair uses as its column tree, and lists them.
__global__ void k_map_reserve(PlanPools P, const int32_t *used, XChunkX *chunkx, int32_t *list, Summary *sum) {
    const int lane = threadIdx.x & 31;
    const int ot = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (ot >= 2 * P.ntrees || !used[ot]) return;
    const DOTree O = P.otrees[ot];
    for (int d = 0; d <= O.D; d++) {
        const DDepth &dd = P.depths[O.depth_base + d];
        const int hi = dd.chunk_lo + dd.nnarrow + dd.nhalf + dd.nwide;
        for (int c = dd.chunk_lo + lane; c < hi; c += 32)
            if (chunk_stripes(P.chunks[c], P.krd) > 1) {
                chunkx[c].map = (int64_t)atomicAdd((unsigned long long *)&sum->map_ints,
                                                   (unsigned long long)P.chunks[c].width);
                list[atomicAdd(&sum->nmaps, 1)] = c;
            }
    }
}

// The export map of a striped chunk, by a block: the far columns that a stripe
// reads from a stripe to its right, numbered in column order (-1 elsewhere).
// nodes are the column tree's records. Returns the number of exports.
template <int NT>
__device__ int chunk_map_team(const Team<NT> &team, const XChunk &ch, const int32_t *krd, const int2 *nodes, int32_t *map) {
    const int w = ch.width, j0 = krd[ch.k_lo], lead = j0 & (XTED_PITCH - 1), tid = team.tid;
    for (int c = tid; c < w; c += NT) map[c] = 0;
    team.sync();
    for (int c = tid; c < w; c += NT) {
        const int foff = (nodes[j0 + c].y & XTED_ROW_ORL_MASK) + 1 - (j0 + c);
        if (far_crosses(c, foff, w, lead)) map[c + foff] = 1;
    }
    team.sync();
    int before = 0;
    for (int base = 0; base < w; base += NT) {
        const int c = base + tid, m = c < w ? map[c] : 0;
        int total;
        const int incl = team.incl_sum(m, &total);
        if (c < w) map[c] = m ? before + incl - 1 : -1;
        before += total;
    }
    return before;
}

// One block per striped chunk. The tree whose node records it needs is found
// from the chunk's keyroot pool index, which lies in the tree's range of the
// node pool.
__global__ void k_chunk_maps(PlanPools P, const int32_t *list, XChunkX *chunkx, int32_t *smap) {
    __shared__ int part[33];
    __shared__ int s_base;
    const Team<XTED_CTA_THREADS> team{(int)threadIdx.x, part};
    const int c0 = list[blockIdx.x];
    const XChunk ch = P.chunks[c0];
    if (team.tid == 0) {  // the oriented tree whose pool range holds the chunk
        int lo = 0, hi = 2 * P.ntrees - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (P.otrees[mid].node_base <= ch.k_lo) lo = mid;
            else hi = mid - 1;
        }
        s_base = P.otrees[lo].node_base;
    }
    __syncthreads();
    const int X = chunk_map_team(team, ch, P.krd, P.node + s_base, smap + chunkx[c0].map);
    if (team.tid == 0) chunkx[c0].X = X;
}

// Stripes and hand-off words of one depth's chunks summed by a warp
// (flow_depth_totals, flow_plan.h, with the lanes over the chunks).
__device__ void depth_totals_warp(const PlanPools &P, XChunkX *chunkx, DDepth &dd, int lane) {
    const unsigned FULL = 0xffffffffu;
    const int lo = dd.chunk_lo, hi = lo + dd.nnarrow + dd.nhalf + dd.nwide;
    int k = 0, w = 0;
    for (int cb = lo; cb < hi; cb += 32) {
        const int c = cb + lane;
        int K = 0, words = 0;
        if (c < hi) {
            K = chunk_stripes(P.chunks[c], P.krd);
            if (K == 1) chunkx[c].X = 0;
            words = chunk_words(K, chunkx[c].X);
        }
        const int ki = warp_incl_sum(K, lane), wi = warp_incl_sum(words, lane);
        if (c < hi) {
            chunkx[c].K = K;
            chunkx[c].kpre = k + ki - K;
            chunkx[c].wpre = w + wi - words;
        }
        k += __shfl_sync(FULL, ki, 31);
        w += __shfl_sync(FULL, wi, 31);
    }
    if (lane == 0) {
        dd.nitems = k;
        dd.wsum = w;
        const int last = dd.run_hi - 1;
        dd.rows = P.cumw[P.runs[last].kr_lo] + P.runs[last].rows;  // every depth up to D has a keyroot
    }
}

// A warp per oriented tree: the totals of its depths.
__global__ void k_depth_totals(PlanPools P, XChunkX *chunkx) {
    const int lane = threadIdx.x & 31;
    const int ot = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (ot >= 2 * P.ntrees) return;
    const DOTree O = P.otrees[ot];
    for (int d = 0; d <= O.D; d++) depth_totals_warp(P, chunkx, P.depths[O.depth_base + d], lane);
}

// One (pair, level) of the batch.
struct Level {
    int32_t pair, level;
    int64_t items, words;
    int64_t rem;              // estimate, then the time left of the pair from this level on
    int64_t item_off, buf_off;
};

// Where k_plan_pair writes, and how much fits.
struct PairPlan {
    int32_t n[2];  // the trees' sizes (raw: the first's arrays, then the second's)
    int32_t orientation, check;
    XPair *pair;
    XChunkX *chunkx;
    int32_t *smap, *list;
    Level *levels;
    int32_t *room;  // items, then hand-off words; stacks from the end down
    XPlanOut *out;
    int32_t cap_map, cap_list, cap_levels;
    int64_t room_ints;
};

// A pair's levels (a warp): their counts, and the time left of the pair from
// each on. Returns the whole pair's time.
__device__ int64_t level_count_warp(const FlowCtx &C, const DOTree &A, const DOTree &B, int p, int L, Level *lv, int lane) {
    int64_t rem = 0;
    for (int hi = L; hi > 0; hi -= 32) {  // from the last level down, 32 at a time
        const int d = hi - 1 - lane;
        int64_t items = 0, words = 0, est = 0;
        if (d >= 0) flow_level_count(C, A, B, d, &items, &words, &est);
        int64_t incl = est;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (d >= 0) {
            Level &E = lv[d];
            E.pair = p;
            E.level = d;
            E.items = items;
            E.words = words;
            E.rem = rem + incl;
        }
        rem += __shfl_sync(0xffffffffu, incl, 31);
    }
    return rem;
}

__global__ void k_level_count(FlowCtx C, const DPair *pairs, int npairs, Level *lv, Summary *sum) {
    const int lane = threadIdx.x & 31;
    const int p = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (p >= npairs) return;
    const DPair q = pairs[p];
    if (q.L == 0) return;
    const int64_t rem = level_count_warp(C, C.ot[2 * q.ta + q.o], C.ot[2 * q.tb + q.o], p, q.L, lv + q.lvl_base, lane);
    if (lane == 0) atomicMax((unsigned long long *)&sum->chain_max, (unsigned long long)rem);
}

// The order of the levels in the launch's list and their offsets, in one
// block: a stable radix sort (four passes of four bits) of the levels by the
// time left of their pair, longest first (stable: a pair's levels stay in
// order), then the scans of items and hand-off words in that order.
#define ORDER_THREADS 512
__global__ void __launch_bounds__(ORDER_THREADS) k_level_order(Level *lv, int n, bool sort, int32_t *ord0, int32_t *ord1,
                                                               Summary *sum) {
    __shared__ int32_t cnt[16 * ORDER_THREADS];
    __shared__ int64_t part[2][ORDER_THREADS];
    const int tid = threadIdx.x;
    const int per = (n + ORDER_THREADS - 1) / ORDER_THREADS, lo = min(tid * per, n), hi = min(lo + per, n);
    int32_t *src = ord0, *dst = ord1;
    for (int i = lo; i < hi; i++) src[i] = i;
    if (sort) {
        const double scale = 65535.0 / (double)max(sum->chain_max, (int64_t)1);
        for (int shift = 0; shift < 16; shift += 4) {
            auto digit = [&](int e) { return ((65535 - (int)((double)lv[e].rem * scale)) >> shift) & 15; };
            for (int b = 0; b < 16; b++) cnt[b * ORDER_THREADS + tid] = 0;
            for (int i = lo; i < hi; i++) cnt[digit(src[i]) * ORDER_THREADS + tid]++;
            __syncthreads();
            int s = 0;
            for (int b = 0; b < 16; b++) s += cnt[16 * tid + b];
            part[0][tid] = s;
            __syncthreads();
            for (int d = 1; d < ORDER_THREADS; d <<= 1) {
                const int64_t x = tid >= d ? part[0][tid - d] : 0;
                __syncthreads();
                part[0][tid] += x;
                __syncthreads();
            }
            int run = (int)part[0][tid] - s;
            for (int b = 0; b < 16; b++) {
                const int c = cnt[16 * tid + b];
                cnt[16 * tid + b] = run;
                run += c;
            }
            __syncthreads();
            for (int i = lo; i < hi; i++) {
                const int e = src[i];
                dst[cnt[digit(e) * ORDER_THREADS + tid]++] = e;
            }
            __syncthreads();
            int32_t *x = src;
            src = dst;
            dst = x;
        }
    }
    int64_t a = 0, b = 0;
    for (int i = lo; i < hi; i++) {
        a += lv[src[i]].items;
        b += lv[src[i]].words;
    }
    part[0][tid] = a;
    part[1][tid] = b;
    __syncthreads();
    for (int d = 1; d < ORDER_THREADS; d <<= 1) {
        const int64_t x = tid >= d ? part[0][tid - d] : 0, y = tid >= d ? part[1][tid - d] : 0;
        __syncthreads();
        part[0][tid] += x;
        part[1][tid] += y;
        __syncthreads();
    }
    int64_t ia = part[0][tid] - a, ib = part[1][tid] - b;
    for (int i = lo; i < hi; i++) {
        Level &E = lv[src[i]];
        E.item_off = ia;
        E.buf_off = ib;
        ia += E.items;
        ib += E.words;
    }
    if (tid == ORDER_THREADS - 1) {
        sum->items = part[0][tid];
        sum->words = part[1][tid];
    }
}

// The items of one level, by a block: by row depth from the deepest down (the
// longest runs first), then by run, then by chunk.
__device__ void level_fill_block(const FlowCtx &C, const DOTree &A, const DOTree &B, const Level &E, XItem *items) {
    const int lo = max(E.level - B.D, 0), hi = min(A.D, E.level);
    int64_t at = E.item_off, buf = E.buf_off;
    for (int a = hi; a >= lo; a--) {
        const DDepth ra = C.depths[A.depth_base + a], cb = C.depths[B.depth_base + E.level - a];
        const int64_t n = (int64_t)(ra.run_hi - ra.run_lo) * cb.nitems;
        for (int64_t k = threadIdx.x; k < n; k += blockDim.x) items[at + k] = flow_item(C, ra, cb, E.pair, k, buf);
        at += n;
        buf += (int64_t)ra.rows * cb.wsum;
    }
}

__global__ void k_level_fill(FlowCtx C, const DPair *pairs, const Level *lv, int64_t nent, XItem *items) {
    for (int64_t e = blockIdx.x; e < nent; e += gridDim.x) {
        const Level E = lv[e];
        const DPair q = pairs[E.pair];
        level_fill_block(C, C.ot[2 * q.ta + q.o], C.ot[2 * q.tb + q.o], E, items);
    }
}

// A preorder CSR tree is well formed (validate_tree, plan.cpp, by a block, every
// index checked before it is used): offsets rise from 0 to n - 1, every node but
// the root is one node's child, and the children of v start at v + 1 and follow
// each other's last nodes (cur: 2 n ints of scratch).
template <int NT>
__device__ bool valid_team(const Team<NT> &team, int n, const int32_t *off, const int32_t *idx, int32_t *cur) {
    const int tid = team.tid;
    int32_t *nxt = cur + n;
    bool bad = off[0] != 0 || off[n] != n - 1;
    for (int v = tid; v < n; v += NT) {
        bad |= off[v + 1] < off[v] || off[v] < 0 || off[v + 1] > n - 1;
        nxt[v] = 0;
    }
    if (team.any(bad)) return false;
    for (int v = tid; v < n; v += NT) {
        const int32_t lo = off[v], hi = off[v + 1];
        int32_t last = v;
        for (int32_t e = lo; e < hi; e++) {
            const int32_t c = idx[e];
            if (c <= last || c >= n || (e == lo && c != v + 1)) {
                bad = true;
                break;
            }
            atomicAdd(&nxt[c], 1);
            last = c;
        }
        cur[v] = last;
    }
    if (team.any(bad)) return false;
    for (int v = 1 + tid; v < n; v += NT) bad |= __ldcg(&nxt[v]) != 1;
    if (team.any(bad)) return false;
    for (int round = 0; round < 32; round++) {  // each node's last descendant (links rise: they end)
        bool changed = false;
        for (int v = tid; v < n; v += NT) {
            const int32_t x = cur[v], y = cur[x];
            nxt[v] = y;
            changed |= y != x;
        }
        team.sync();
        int32_t *tmp = cur;
        cur = nxt;
        nxt = tmp;
        if (!team.any(changed)) break;
    }
    bad = cur[0] != n - 1;
    for (int v = tid; v < n; v += NT)
        for (int32_t e = off[v] + 1; e < off[v + 1]; e++) bad |= idx[e] != cur[idx[e - 1]] + 1;
    return !team.any(bad);
}

// The whole plan of one pair in one block, in memory of fixed size: nothing
// is read back, so a call on two small trees makes one launch for its plan and
// none of its waits (a pair of 100 nodes spent 118 us on eleven planning kernels
// and two reads; the trees of one pair never fill more than a block or two
// anyway). out->status: 0, XTED_EINVAL (check: the trees are validated here),
// or PLAN_OVERFLOW when a list does not fit (the launch then runs nothing).
__global__ void __launch_bounds__(PLAN_PAIR_THREADS) k_plan_pair(PlanPools P, DTree *trees, PairPlan B) {
    constexpr int NT = PLAN_PAIR_THREADS;
    __shared__ int part[33];
    __shared__ int64_t acc[2][32];
    __shared__ int s_max, s_maps, s_nmaps;
    const Team<NT> team{(int)threadIdx.x, part};
    const int tid = team.tid, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_maps = s_nmaps = 0;
        B.out->status = PLAN_OVERFLOW;  // until all is in place
        B.out->items = 0;
        B.out->stack_rows = 1;
        B.out->words = 0;
        B.out->scratch = 0;
        for (int t = 0; t < P.ntrees; t++) {
            DTree T;
            T.n = B.n[t];
            T.raw = t == 0 ? 0 : 3 * B.n[0] + 1;
            T.nbase = t == 0 ? 0 : B.n[0];
            T.t = t;
            T.S[0] = T.S[1] = 0;
            trees[t] = T;
        }
    }
    __syncthreads();
    if (B.check)
        for (int t = 0; t < P.ntrees; t++) {
            const DTree T = trees[t];
            const int32_t *off = P.raw + T.raw + T.n;
            if (!valid_team(team, T.n, off, off + T.n + 1, P.opar + 2 * (int64_t)T.nbase)) {
                if (tid == 0) B.out->status = XTED_EINVAL;
                return;
            }
        }
    for (int t = 0; t < P.ntrees; t++) tree_basic_team(team, P, t, trees, acc);
    const int tb = P.ntrees - 1;  // (one tree: against itself)
    const int o = pair_orientation(trees[0], trees[tb], B.orientation);
    for (int t = 0; t < P.ntrees; t++) orient_team(team, P, 2 * t + o, true, &s_max);
    const DOTree A = P.otrees[o], Bt = P.otrees[2 * tb + o];
    // striped chunks of the column tree: export maps, then the depths' totals
    for (int d = warp; d <= Bt.D; d += NT / 32) {
        const DDepth &dd = P.depths[Bt.depth_base + d];
        for (int c = dd.chunk_lo + lane; c < dd.chunk_lo + dd.nnarrow; c += 32)
            if (chunk_stripes(P.chunks[c], P.krd) > 1) {
                B.chunkx[c].map = atomicAdd(&s_maps, P.chunks[c].width);
                const int i = atomicAdd(&s_nmaps, 1);
                if (i < B.cap_list) B.list[i] = c;
            }
    }
    __syncthreads();
    if (s_maps > B.cap_map || s_nmaps > B.cap_list) return;
    for (int i = 0; i < s_nmaps; i++) {
        const int c = B.list[i];
        const int X = chunk_map_team(team, P.chunks[c], P.krd, P.node + Bt.node_base, B.smap + B.chunkx[c].map);
        if (tid == 0) B.chunkx[c].X = X;
    }
    __syncthreads();
    for (int t = 0; t < P.ntrees; t++) {
        const DOTree &O = t == 0 ? A : Bt;
        for (int d = warp; d <= O.D; d += NT / 32) depth_totals_warp(P, B.chunkx, P.depths[O.depth_base + d], lane);
    }
    __syncthreads();
    FlowCtx C;
    C.ot = P.otrees;
    C.depths = P.depths;
    C.runs = P.runs;
    C.chunks = P.chunks;
    C.chunkx = B.chunkx;
    C.cumw = P.cumw;
    const int L = A.D + Bt.D + 1;
    if (L > B.cap_levels) return;
    if (warp == 0) {
        level_count_warp(C, A, Bt, 0, L, B.levels, lane);
        __syncwarp();
        if (lane == 0) {  // one pair: its levels in order
            int64_t items = 0, words = 0;
            for (int d = 0; d < L; d++) items += B.levels[d].items;
            const int64_t total = items;
            items = 0;
            for (int d = 0; d < L; d++) {
                Level &E = B.levels[d];
                E.item_off = items;
                E.buf_off = ITEM_INTS * total + words;
                items += E.items;
                words += E.words;
            }
            acc[0][0] = items;
            acc[0][1] = words;
        }
    }
    __syncthreads();
    const int64_t items = acc[0][0], words = acc[0][1];
    const int64_t left = B.room_ints - ITEM_INTS * items - ((words + 3) & ~(int64_t)3);
    if (left < (A.maxka + 1) * (int64_t)XTED_SW) return;  // at least one warp's stack
    for (int d = 0; d < L; d++) level_fill_block(C, A, Bt, B.levels[d], (XItem *)B.room);
    if (tid == 0) {
        XPair x;
        x.dt_off = 0;
        x.m = trees[0].n;
        x.n = trees[tb].n;
        x.row_base = A.node_base;
        x.col_base = Bt.node_base;
        x.pitch = table_pitch(x.n);
        x.pad = 0;
        *B.pair = x;
        XPlanOut out;
        out.items = (int32_t)items;
        out.stack_rows = A.maxka + 1;
        out.levels = L;
        out.status = 0;
        out.cells = A.S * Bt.S;
        out.cells_right = trees[0].S[0] * trees[tb].S[0];
        out.words = words;
        out.scratch = left;
        *B.out = out;
    }
}

// A planned pair's tables and hand-off words to -1, 16 bytes a store.
__global__ void k_pair_clear(const XPlanOut *out, int4 *dt, int64_t dt4, int32_t *room) {
    if (out->status != 0) return;
    const int64_t w4 = (out->words + 3) / 4, step = (int64_t)gridDim.x * blockDim.x;
    int4 *w = (int4 *)(room + ITEM_INTS * (int64_t)out->items);
    const int4 none = make_int4(-1, -1, -1, -1);
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < dt4 + w4; k += step)
        *(k < dt4 ? dt + k : w + (k - dt4)) = none;
}

__global__ void k_pair_finalize(const DPair *pairs, const DTree *trees, const DOTree *ot, int npairs, XPair *xp,
                                int32_t *trivial) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npairs) return;
    const DPair q = pairs[p];
    XPair x;
    x.dt_off = q.dt_off;
    x.m = trees[q.ta].n;
    x.n = trees[q.tb].n;
    x.row_base = ot[2 * q.ta + q.o].node_base;
    x.col_base = ot[2 * q.tb + q.o].node_base;
    x.pitch = table_pitch(x.n);
    x.pad = 0;
    xp[p] = x;
    trivial[p] = q.trivial;
}

// The parts of a list (flow_cut): where each starts, at most max of them, and
// their count (one thread: some fifty loads a part, on lists that need more than one).
__global__ void k_parts(const XItem *items, int n, int64_t words, int64_t cap, XPart *parts, int max, int32_t *count) {
    int k = 0;
    for (int g = 0; g < n && k < max; g = flow_cut(items, n, words, g, cap)) parts[k++] = XPart{items[g].buf, g, 0};
    *count = k;
}

inline unsigned blocks_for(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

}  // namespace

// Carves a device buffer into aligned sections.
struct Carver {
    char *base;
    size_t off = 0;
    template <class T>
    T *take(size_t count) {
        off = (off + 255) & ~(size_t)255;
        T *p = (T *)(base + off);
        off += sizeof(T) * (count > 0 ? count : 1);
        return p;
    }
};

size_t pair_layout(void *base, size_t bytes, int32_t m, int32_t n, PairLayout *L) {
    const size_t N = (size_t)m + n, N2 = 2 * N;
    Carver cv{(char *)base};
    L->m = m;
    L->n = n;
    const size_t raw_ints = (3 * N + 2 + 63) & ~(size_t)63;
    L->dt_ints = (int64_t)m * table_pitch(n);
    L->upload_ints = (int64_t)raw_ints + PAIR_HDR_INTS;
    L->raw = cv.take<int32_t>(raw_ints + PAIR_HDR_INTS + (size_t)L->dt_ints);
    L->hdr = L->raw + raw_ints;
    L->dt = L->hdr + PAIR_HDR_INTS;
    PlanPools &P = L->P;
    P.raw = L->raw;
    L->trees = cv.take<DTree>(2);
    P.trees = L->trees;
    P.ntrees = 2;
    P.size = cv.take<int32_t>(N);
    P.depth = cv.take<int32_t>(N);
    P.parent = cv.take<int32_t>(N);
    P.node = cv.take<int2>(N2);
    P.krd = cv.take<int32_t>(N2);
    P.cumw = cv.take<int32_t>(N2);
    P.runs = cv.take<XRun>(N2);
    P.chunks = cv.take<XChunk>(N2);
    P.opar = cv.take<int32_t>(N2);
    P.okd = cv.take<int32_t>(N2);
    P.oka = cv.take<int32_t>(N2);
    P.depths = cv.take<DDepth>(N2 + 4);
    P.otrees = cv.take<DOTree>(4);
    L->chunkx = cv.take<XChunkX>(N2);
    L->list = cv.take<int32_t>((size_t)n);
    L->cap_list = n;
    L->cap_map = 32 * n;  // (each column of 32 tables wider than a warp holds)
    L->smap = cv.take<int32_t>((size_t)L->cap_map);
    // keyroot depths of most trees grow with the logarithm of their nodes (a spine with a leg per node on the wrong side
    // has half of them: its plan overflows and goes to the batch's kernels)
    L->cap_levels = 64;
    L->levels = cv.take<Level>((size_t)L->cap_levels);
    L->room = cv.take<int32_t>(0);
    const size_t used = (size_t)((char *)L->room - (char *)base);
    if (bytes <= used) return 0;
    L->room_ints = (int64_t)(bytes - used) / 4;
    return used;
}

cudaError_t launch_plan_pair(const PairLayout &L, int32_t orientation, bool check, cudaStream_t s) {
    PairPlan B;
    B.n[0] = L.m;
    B.n[1] = L.n;
    B.orientation = orientation;
    B.check = check;
    B.pair = (XPair *)(L.hdr + PAIR_PAIR);
    B.chunkx = L.chunkx;
    B.smap = L.smap;
    B.list = L.list;
    B.levels = (Level *)L.levels;
    B.room = L.room;
    B.out = (XPlanOut *)(L.hdr + PAIR_OUT);
    B.cap_map = L.cap_map;
    B.cap_list = L.cap_list;
    B.cap_levels = L.cap_levels;
    B.room_ints = L.room_ints;
    k_plan_pair<<<1, PLAN_PAIR_THREADS, 0, s>>>(L.P, L.trees, B);
    return cudaGetLastError();
}

cudaError_t launch_pair_clear(const PairLayout &L, int32_t blocks, cudaStream_t s) {
    k_pair_clear<<<(unsigned)blocks, 256, 0, s>>>((const XPlanOut *)(L.hdr + PAIR_OUT), (int4 *)L.dt, L.dt_ints / 4, L.room);
    return cudaGetLastError();
}

cudaError_t pair_kernels_load() {
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, k_plan_pair);
    return e != cudaSuccess ? e : cudaFuncGetAttributes(&a, k_pair_clear);
}

void pair_params(const PairLayout &L, XKernelParams &K) {
    K.rowinfo = L.P.node;
    K.krd = L.P.krd;
    K.cumw = L.P.cumw;
    K.runs = L.P.runs;
    K.chunks = L.P.chunks;
    K.chunkx = L.chunkx;
    K.pairs = (const XPair *)(L.hdr + PAIR_PAIR);
    K.items = (const XItem *)L.room;
    K.dt = L.dt;
    K.buf = L.room;
    K.smap = L.smap;
    K.scratch = L.room + L.room_ints;
    K.plan = (const XPlanOut *)(L.hdr + PAIR_OUT);
    K.npairs = 1;
    K.next = L.hdr + PAIR_NEXT;
    K.progress = L.hdr + PAIR_PROGRESS;
    K.error = L.hdr + PAIR_ERROR;
    K.error_info = L.hdr + PAIR_ERROR + 1;
    K.hold_pair = -1;
}

int dev_parts(xted_ctx *c, int64_t cap, int64_t *need) {
    std::vector<XPart> &parts = c->parts;
    const int64_t words = c->plan_words;
    const int n = c->kp.nitems;
    parts.assign(1, XPart{0, 0, 0});
    if (words > cap) {
        // two neighbouring parts have more than cap words together
        const int64_t max = std::min<int64_t>(2 * (words / std::max<int64_t>(cap, 1)) + 2, n);
        int rc = ctx_dev_reserve(c, c->levels, sizeof(XPart) * (size_t)max + 256);  // (the levels have been used)
        if (rc) return rc;
        int32_t *d_count = (int32_t *)c->levels.p, count = 0;
        XPart *d_parts = (XPart *)((char *)c->levels.p + 256);
        k_parts<<<1, 1, 0, c->stream>>>(c->kp.items, n, words, cap, d_parts, (int)max, d_count);
        if (cudaMemcpyAsync(&count, d_count, 4, cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
            cudaStreamSynchronize(c->stream) != cudaSuccess) {
            cudaGetLastError();
            return XTED_ECUDA;
        }
        parts.resize((size_t)count);
        if (cudaMemcpy(parts.data(), d_parts, sizeof(XPart) * (size_t)count, cudaMemcpyDeviceToHost) != cudaSuccess) {
            cudaGetLastError();
            return XTED_ECUDA;
        }
    }
    parts.push_back(XPart{words, n, 0});
    *need = 0;
    for (size_t k = 0; k + 1 < parts.size(); k++) *need = std::max(*need, parts[k + 1].word - parts[k].word);
    return XTED_OK;
}

int dev_plan(xted_ctx *c, const xted_tree *a, const xted_tree *b, int32_t npairs, XKernelParams &K) {
    cudaStream_t s = c->stream;
    // ---- host: unique trees, flat raw input, pair list ----
    c->tree_ids.clear();
    c->uniq.clear();
    std::vector<int32_t> &pt = c->pair_trees;
    pt.resize(2 * (size_t)npairs);
    int64_t N = 0, R = 0, products = 0;
    int32_t maxn = 0;
    for (int p = 0; p < npairs; p++) {
        products += (int64_t)std::max(a[p].n, 0) * std::max(b[p].n, 0);
        for (int side = 0; side < 2; side++) {
            const xted_tree &t = side ? b[p] : a[p];
            TreeKey key{t.labels, t.child_off, t.child_idx, t.n};
            auto it = c->tree_ids.find(key);
            int id;
            if (it == c->tree_ids.end()) {
                id = (int)c->uniq.size();
                c->tree_ids.emplace(key, id);
                if (t.n < 0 || t.n > XTED_MAX_NODES) return XTED_EINVAL;
                c->uniq.push_back(TreeView{t.n, t.labels, t.child_off, t.child_idx});
                N += t.n;
                R += 3 * (int64_t)t.n + 1;
                maxn = std::max(maxn, t.n);
            } else {
                id = it->second;
            }
            pt[2 * (size_t)p + side] = id;
        }
    }
    const int T = (int)c->uniq.size();
    if (N > (int64_t)1 << 30) return XTED_ENOMEM;
    {   // every unique tree is checked before anything reads it (host threads for big batches)
        std::vector<int> bad((size_t)std::max(T, 1), 0);
        parallel_for(T, 512, [&](int64_t lo, int64_t hi) {
            for (int64_t t = lo; t < hi; t++) bad[(size_t)t] = validate_tree(c->uniq[(size_t)t]);
        });
        for (int t = 0; t < T; t++)
            if (bad[(size_t)t]) return bad[(size_t)t];
    }
    std::vector<DTree> &ht = c->htrees;
    ht.resize((size_t)T);
    // staging: raw trees | DTree[T] | pair_trees
    const size_t raw_bytes = (size_t)R * 4, tr_bytes = sizeof(DTree) * (size_t)T,
                 pt_bytes = 8 * (size_t)npairs;
    const size_t stage_bytes = raw_bytes + tr_bytes + pt_bytes + 1024;
    int rc = ctx_host_reserve(c->stage, stage_bytes);
    if (rc) return rc;
    char *h = (char *)c->stage.p;
    int32_t *hraw = (int32_t *)h;
    {
        int64_t rpos = 0, nb = 0;
        for (int t = 0; t < T; t++) {
            const TreeView &tv = c->uniq[(size_t)t];
            DTree &d = ht[(size_t)t];
            d.n = tv.n;
            d.raw = (int32_t)rpos;
            d.nbase = (int32_t)nb;
            d.t = t;
            d.S[0] = d.S[1] = 0;
            rpos += 3 * (int64_t)tv.n + 1;
            nb += tv.n;
        }
        parallel_for(T, 512, [&](int64_t lo, int64_t hi) {
            for (int64_t t = lo; t < hi; t++) {
                const TreeView &tv = c->uniq[(size_t)t];
                int32_t *dst = hraw + ht[(size_t)t].raw;
                const int n = tv.n;
                if (n > 0) {
                    std::memcpy(dst, tv.labels, 4 * (size_t)n);
                    std::memcpy(dst + n, tv.off, 4 * ((size_t)n + 1));
                    if (n > 1) std::memcpy(dst + 2 * n + 1, tv.idx, 4 * ((size_t)n - 1));
                } else {
                    dst[0] = 0;  // child_off[0]
                }
            }
        });
    }
    size_t hoff = (raw_bytes + 255) & ~(size_t)255;
    std::memcpy(h + hoff, ht.data(), tr_bytes);
    const size_t hoff_pt = (hoff + tr_bytes + 255) & ~(size_t)255;
    std::memcpy(h + hoff_pt, pt.data(), pt_bytes);
    const size_t upload = hoff_pt + pt_bytes;

    // ---- device buffer A: input + per-tree pools (sizes known from N, T, npairs) ----
    const size_t N2 = 2 * (size_t)std::max<int64_t>(N, 1);
    size_t need = upload + 4096;
    need += 3 * sizeof(int32_t) * (size_t)std::max<int64_t>(N, 1);  // size, depth, parent
    need += N2 * (sizeof(int2) + 2 * sizeof(int32_t) + sizeof(XRun) + sizeof(XChunk) + sizeof(XChunkX) + sizeof(int32_t));
    need += sizeof(DDepth) * (N2 + 2 * (size_t)T) + sizeof(DOTree) * 2 * (size_t)T + sizeof(DTree) * (size_t)T +
            4 * sizeof(int32_t) * (size_t)T;
    need += (size_t)npairs * (sizeof(DPair) + sizeof(XPair) + 4 + 4 * 8) + 24 * 256 + sizeof(Summary);
    rc = ctx_dev_reserve(c, c->meta, need);
    if (rc) return rc;
    Carver cv{(char *)c->meta.p};
    char *d_in = cv.take<char>(upload);
    if (cudaMemcpyAsync(d_in, h, upload, cudaMemcpyHostToDevice, s) != cudaSuccess) return XTED_ECUDA;
    c->h2d_bytes = (int64_t)upload;
    PlanPools P;
    P.raw = (const int32_t *)d_in;
    DTree *d_trees = (DTree *)(d_in + hoff);
    P.trees = d_trees;
    const int32_t *d_pt = (const int32_t *)(d_in + hoff_pt);
    P.ntrees = T;
    P.size = cv.take<int32_t>((size_t)N);
    P.depth = cv.take<int32_t>((size_t)N);
    P.parent = cv.take<int32_t>((size_t)N);
    P.node = cv.take<int2>(N2);
    P.krd = cv.take<int32_t>(N2);
    P.cumw = cv.take<int32_t>(N2);
    P.runs = cv.take<XRun>(N2);
    P.chunks = cv.take<XChunk>(N2);
    // k_orient's scratch, and where it was, from k_map_reserve on, what the chunks add to the plan
    char *chunk_room = cv.take<char>(N2 * (sizeof(XChunkX) + sizeof(int32_t)));
    P.opar = (int32_t *)chunk_room;
    P.okd = P.opar + N2;
    P.oka = P.okd + N2;
    static_assert(sizeof(XChunkX) + sizeof(int32_t) >= 3 * sizeof(int32_t), "room for both");
    XChunkX *d_chunkx = (XChunkX *)chunk_room;
    int32_t *d_list = (int32_t *)(d_chunkx + N2);
    P.depths = cv.take<DDepth>(N2 + 2 * (size_t)T);
    P.otrees = cv.take<DOTree>(2 * (size_t)T);
    ctx_granularity(c, products, P);
    DPair *d_pairs = cv.take<DPair>((size_t)npairs);
    XPair *d_xpairs = cv.take<XPair>((size_t)npairs);
    int32_t *d_trivial = cv.take<int32_t>((size_t)npairs);
    int64_t *d_L = cv.take<int64_t>((size_t)npairs + 1);
    int64_t *d_cells = cv.take<int64_t>((size_t)npairs + 1);
    int64_t *d_Ls = cv.take<int64_t>((size_t)npairs + 1);
    int64_t *d_dts = cv.take<int64_t>((size_t)npairs + 1);
    int32_t *d_used = cv.take<int32_t>(2 * (size_t)T), *d_need = cv.take<int32_t>(2 * (size_t)T);
    Summary *d_sum = cv.take<Summary>(1);
    if (cv.off > c->meta.cap) return XTED_ENOMEM;
    const bool stripes = maxn + XTED_PITCH > XTED_SW;  // some chunk may be wider than a warp holds

    const int BS = 128;
    cudaMemsetAsync(d_used, 0, (size_t)((char *)(d_sum + 1) - (char *)d_used), s);
    const bool big = maxn > PLAN_WARP_NODES && T <= PLAN_BLOCK_TREES;
    if (big) k_tree_basic<1024><<<(unsigned)T, 1024, 0, s>>>(P, d_trees);
    else k_tree_basic<32><<<blocks_for(32 * (int64_t)T, BS), BS, 0, s>>>(P, d_trees);
    k_pair_orient<<<blocks_for(std::max(npairs, 1), BS), BS, 0, s>>>(d_trees, d_pt, c->opts.orientation, npairs, d_need);
    if (big) k_orient<1024><<<2 * (unsigned)T, 1024, 0, s>>>(P, d_need);
    else k_orient<32><<<blocks_for(64 * (int64_t)T, BS), BS, 0, s>>>(P, d_need);
    k_pair_setup<<<blocks_for(std::max(npairs, 1), BS), BS, 0, s>>>(d_trees, P.otrees, d_pt, c->opts.orientation, npairs,
                                                                    d_pairs, d_L, d_cells, d_used);
    k_scan64<<<1, 1024, 0, s>>>(d_L, npairs, d_Ls);
    k_scan64<<<1, 1024, 0, s>>>(d_cells, npairs, d_dts);
    k_pair_offsets<<<blocks_for(std::max(npairs, 1), BS), BS, 0, s>>>(d_pairs, d_trees, P.otrees, npairs, d_Ls,
                                                                      d_dts, d_sum);
    if (stripes) k_map_reserve<<<blocks_for(64 * (int64_t)T, BS), BS, 0, s>>>(P, d_used, d_chunkx, d_list, d_sum);
    rc = ctx_host_reserve(c->summary, sizeof(Summary));
    if (rc) return rc;
    Summary *hs = (Summary *)c->summary.p;
    cudaMemcpyAsync(hs, d_sum, sizeof(Summary), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) {
        cudaGetLastError();
        return XTED_ECUDA;
    }
    const int64_t nent = hs->entries;
    if (nent > INT32_MAX / 2) return XTED_ENOMEM;
    if (hs->nmaps > 0) {
        rc = ctx_dev_reserve(c, c->smap, (size_t)hs->map_ints * sizeof(int32_t));
        if (rc) return rc;
        k_chunk_maps<<<(unsigned)hs->nmaps, XTED_CTA_THREADS, 0, s>>>(P, d_list, d_chunkx, (int32_t *)c->smap.p);
    }
    // ---- buffer B: the levels ----
    const size_t E1 = (size_t)nent + 1;
    rc = ctx_dev_reserve(c, c->levels, sizeof(Level) * E1 + 2 * sizeof(int32_t) * E1 + 4 * 256);
    if (rc) return rc;
    Carver cb{(char *)c->levels.p};
    Level *d_lv = cb.take<Level>(E1);
    int32_t *d_ord0 = cb.take<int32_t>(E1), *d_ord1 = cb.take<int32_t>(E1);
    FlowCtx C;
    C.ot = P.otrees;
    C.depths = P.depths;
    C.runs = P.runs;
    C.chunks = P.chunks;
    C.chunkx = d_chunkx;
    C.cumw = P.cumw;
    k_pair_finalize<<<blocks_for(std::max(npairs, 1), BS), BS, 0, s>>>(d_pairs, d_trees, P.otrees, npairs, d_xpairs,
                                                                       d_trivial);
    if (nent > 0) {
        k_depth_totals<<<blocks_for(64 * (int64_t)T, BS), BS, 0, s>>>(P, d_chunkx);
        k_level_count<<<blocks_for(32 * (int64_t)npairs, BS), BS, 0, s>>>(C, d_pairs, npairs, d_lv, d_sum);
        k_level_order<<<1, ORDER_THREADS, 0, s>>>(d_lv, (int)nent, npairs > 1, d_ord0, d_ord1, d_sum);
    }
    cudaMemcpyAsync(hs, d_sum, sizeof(Summary), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) {
        cudaGetLastError();
        return XTED_ECUDA;
    }
    const int64_t nitems = hs->items;
    if (nitems > INT32_MAX / 2) return XTED_ENOMEM;
    // ---- buffer C: the items and the launch's counters ----
    rc = ctx_dev_reserve(c, c->work, sizeof(XItem) * (size_t)(nitems + 1) + 2 * 256 + 64);
    if (rc) return rc;
    Carver cw{(char *)c->work.p};
    XItem *d_items = cw.take<XItem>((size_t)nitems);
    int32_t *d_ctl = cw.take<int32_t>(2);  // items claimed, items finished
    if (nent > 0)
        k_level_fill<<<(unsigned)std::min<int64_t>(nent, 1 << 16), 128, 0, s>>>(C, d_pairs, d_lv, nent, d_items);
    if (cudaGetLastError() != cudaSuccess) return XTED_ECUDA;

    std::memset(&K, 0, sizeof(K));
    K.rowinfo = P.node;
    K.krd = P.krd;
    K.cumw = P.cumw;
    K.runs = P.runs;
    K.chunks = P.chunks;
    K.pairs = d_xpairs;
    K.chunkx = d_chunkx;
    K.items = d_items;
    K.nitems = (int32_t)nitems;
    K.npairs = npairs;
    K.next = d_ctl;
    K.progress = d_ctl + 1;
    K.smap = (const int32_t *)c->smap.p;
    K.hold_pair = -1;
    c->d_trivial = d_trivial;
    c->plan_dt_elems = hs->dt_elems;
    c->plan_stack_rows = std::max(hs->stack_rows, 1);
    c->plan_words = hs->words;
    c->plan_cells = hs->cells;
    c->plan_cells_right = hs->cells_right;
    c->plan_levels_max = hs->levels_max;
    return XTED_OK;
}

}  // namespace xted
