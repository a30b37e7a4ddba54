// api.cpp -- the C ABI (include/xted.h): context, device memory, launches.
//
// xted_distance / xted_distance_batch replace the reference's
// standard_ted (X-TED_CPU/TED.cpp:177-190; X-TED_GPU/TED.cu:116-128): the
// planner (prep.cu) lays out every keyroot table of every pair as a list of
// items, one launch of the persistent DP kernel (flow.cu) runs
// them, and a gather kernel reads Dtree[0][0] of each pair
// (X-TED_CPU/TED.cpp:188). Errors are returned, never printed or exited on
// (the reference prints CUDA errors and continues, X-TED_GPU/utils/cuda_utils.h:35-41,
// or exits, X-TED_GPU/help.h:6-14).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/xted.h"
#include "ctx.h"
#include "plan.h"
#include "tune_table.h"

namespace xted {
int dp_occupancy(int *blocks_per_sm, bool full);
cudaError_t launch_dp(const XKernelParams &P, int grid, bool full, cudaStream_t s);
cudaError_t launch_gather(const XPair *pairs, const int32_t *trivial, const int32_t *dt, int npairs,
                          int32_t *out, int c_del, int c_ins, int32_t *error, cudaStream_t s);
}  // namespace xted

using namespace xted;

namespace {

inline double now_ms() {
    using namespace std::chrono;
    return duration<double, std::milli>(steady_clock::now().time_since_epoch()).count();
}

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace

namespace xted {

bool costs_fit(const xted_opts &o, int64_t m, int64_t n) {
    return (int64_t)o.cost_del * m + (int64_t)o.cost_ins * n < XTED_COST_BOUND;
}

static void dev_release(xted_ctx *c, DevBuf &b) {
    if (b.p) cudaFree(b.p);
    c->held -= (int64_t)b.cap;
    b = DevBuf{};
}

int ctx_dev_reserve(xted_ctx *c, DevBuf &b, size_t bytes) {
    if (b.cap >= bytes) return XTED_OK;
    size_t want = align_up(std::max(bytes, b.cap + b.cap / 2), (size_t)2 << 20);
    dev_release(c, b);
    void *p = nullptr;
    for (;;) {
        const int64_t room = c->opts.mem_limit > 0 ? c->opts.mem_limit - c->held : INT64_MAX;
        if ((int64_t)want > room) want = align_up(bytes, 256);
        if ((int64_t)want <= room) {
            if (cudaMalloc(&p, want) == cudaSuccess) break;
            cudaGetLastError();
        }
        // the stacks and hand-off words of an earlier plan may have taken all there is: they come in any size
        if (&b == &c->scratch || &b == &c->sbuf || (!c->scratch.p && !c->sbuf.p)) return XTED_ENOMEM;
        dev_release(c, c->scratch);
        dev_release(c, c->sbuf);
    }
    b.p = p;
    b.cap = want;
    c->held += (int64_t)want;
    return XTED_OK;
}

int ctx_host_reserve(HostBuf &b, size_t bytes) {
    if (b.cap >= bytes) return XTED_OK;
    size_t want = align_up(std::max(bytes, b.cap + b.cap / 2), (size_t)1 << 20);
    if (b.p) cudaFreeHost(b.p);
    b.p = nullptr;
    b.cap = 0;
    if (cudaHostAlloc(&b.p, want, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        b.p = nullptr;
        return XTED_ENOMEM;
    }
    b.cap = want;
    return XTED_OK;
}

// From this many pairs on a launch takes five blocks an SM. It is a line on
// mixed pairs of 50-2,000 nodes (ms with four / five): 128 pairs 5.35 / 5.50, 512
// 20.5 / 20.2, 768 26.4 / 26.1, 1,023 36.7 / 35.5, 1,500 57.1 / 54.8. A count does
// not see the shapes: pairs of deep trees gain from 20 pairs on (20 of 2,000 nodes
// 59.4 / 56.5), random trees lose at any number (1,600 of 300 5.18 / 5.47, 16,000
// of 100 8.84 / 9.23), and so do many small pairs beside a large one.
#define XTED_FULL_PAIRS 1024

// One pair is planned by one block up to this many nodes together, by the
// batch's kernels beyond. A call on two trees of 40 nodes takes 165 us this way
// and 239 the other, of 1,000 nodes each 1,531 and 1,730, of 2,048 each 2,701
// and 2,720; of 2,500 each the batch's kernels are level.
#define XTED_PAIR_NODES 4096
// Its items, hand-off words and stacks: what does not fit is planned by the batch's kernels.
#define XTED_PAIR_ROOM ((size_t)32 << 20)

// Lays one pair out and enqueues its plan; nothing is read back (ctx_run finds
// out whether the plan fitted).
static int pair_prepare(xted_ctx *c, const xted_tree &a, const xted_tree &b) {
    const xted_tree *t[2] = {&a, &b};
    for (int k = 0; k < 2; k++) {
        const int rc = validate_tree(TreeView{t[k]->n, t[k]->labels, t[k]->child_off, t[k]->child_idx});
        if (rc) return rc;
    }
    PairLayout &L = c->pair;
    pair_layout(nullptr, 0, a.n, b.n, &L);
    const size_t fixed = (size_t)((char *)L.room - (char *)nullptr);
    int rc = ctx_dev_reserve(c, c->meta, fixed + XTED_PAIR_ROOM);
    if (!rc) rc = ctx_host_reserve(c->stage, (size_t)L.upload_ints * 4);
    if (!rc) rc = ctx_host_reserve(c->result, (PAIR_HDR_INTS + 1) * sizeof(int32_t));
    if (rc) return rc;
    pair_layout(c->meta.p, fixed + XTED_PAIR_ROOM, a.n, b.n, &L);
    ctx_granularity(c, (int64_t)a.n * b.n, L.P);
    int32_t *h = (int32_t *)c->stage.p;
    std::memset(h + L.upload_ints - PAIR_HDR_INTS, 0, PAIR_HDR_INTS * sizeof(int32_t));
    for (int k = 0; k < 2; k++) {
        const size_t n = (size_t)t[k]->n;
        std::memcpy(h, t[k]->labels, 4 * n);
        std::memcpy(h + n, t[k]->child_off, 4 * (n + 1));
        if (n > 1) std::memcpy(h + 2 * n + 1, t[k]->child_idx, 4 * (n - 1));
        h += 3 * n + 1;
    }
    c->h2d_bytes = L.upload_ints * 4;
    if (cudaMemcpyAsync(L.raw, c->stage.p, (size_t)c->h2d_bytes, cudaMemcpyHostToDevice, c->stream) != cudaSuccess ||
        launch_plan_pair(L, c->opts.orientation, false, c->stream) != cudaSuccess) {
        cudaGetLastError();
        return XTED_ECUDA;
    }
    XKernelParams &K = c->kp;
    std::memset(&K, 0, sizeof(K));
    pair_params(L, K);
    K.c_del = c->opts.cost_del;
    K.c_ins = c->opts.cost_ins;
    K.c_ren = c->opts.cost_ren;
    K.timeout_ns = (uint64_t)(c->opts.wait_timeout_s * 1e9);
    c->npairs = 1;
    c->prepared = true;
    return XTED_OK;
}

// A launch holds as many bytes of hand-off words as of tables, and this many at least; a list with more runs in
// parts. The words of a pair that is costly in both decompositions grow with the fourth power of its nodes (zigzags of
// 1,000 nodes 11.6 GB beside 4 MB of tables, of 2,000 nodes 212 GB), those of most others stay below their tables or
// this floor (4,096 mixed pairs 4.0 GB beside 4.7). Every part but the last ends with the GPU running empty: the deep
// pair of 20,000 nodes takes 407 ms whole, with 10 GB, and 471 in parts of 2 GB.
#define XTED_WORDS_MIN ((int64_t)8 << 30)

// Reserves the launch's stacks and hand-off words and divides the list into
// parts. Both come in any size: the stacks down to one block's, the words down
// to the largest unit's. Where not all fits, the stacks take at most half.
static int reserve_launch(xted_ctx *c) {
    XKernelParams &K = c->kp;
    const int64_t block = (int64_t)c->plan_stack_rows * XTED_SW * XTED_FLOW_WARPS * (int64_t)sizeof(int32_t);
    const int64_t bytes = c->plan_words * (int64_t)sizeof(int32_t);
    int64_t cap = std::max(XTED_WORDS_MIN, c->plan_dt_elems * (int64_t)sizeof(int32_t));
    if (c->opts.mem_limit > 0 && bytes > 0) {
        const int64_t left = c->opts.mem_limit - c->held + (int64_t)c->scratch.cap + (int64_t)c->sbuf.cap;
        if (block * c->run_grid + std::min(bytes, cap) > left) {
            dev_release(c, c->scratch);
            dev_release(c, c->sbuf);
            c->run_grid = (int32_t)std::max<int64_t>(std::min<int64_t>(c->run_grid, left / 2 / block), 1);
            cap = std::min(cap, left - block * c->run_grid);
        }
    }
    for (bool old = c->sbuf.p != nullptr;; old = false) {
        int rc = ctx_dev_reserve(c, c->scratch, (size_t)(block * c->run_grid));
        for (int64_t most = cap, before = INT64_MAX; !rc && bytes > 0;) {
            int64_t need = 0;
            rc = dev_parts(c, std::max<int64_t>(most / (int64_t)sizeof(int32_t), 1), &need);
            if (!rc) rc = ctx_dev_reserve(c, c->sbuf, (size_t)need * sizeof(int32_t));
            if (rc != XTED_ENOMEM || need >= before) break;
            rc = XTED_OK;
            before = need;
            most = need * (int64_t)sizeof(int32_t) / 2;
        }
        if (!rc) rc = ctx_dev_reserve(c, c->scratch, (size_t)(block * c->run_grid));  // (given up for the list of parts?)
        if (rc != XTED_ENOMEM || (c->run_grid == 1 && !old)) {
            K.scratch = (int32_t *)c->scratch.p;
            return rc;
        }
        dev_release(c, c->scratch);
        dev_release(c, c->sbuf);
        if (!old) c->run_grid = (c->run_grid + 1) / 2;  // (first without what an earlier plan left)
    }
}

// Plans a batch on the device (prep.cu) and sizes every buffer the DP launch
// needs; the kernel parameters stay in the context so the batch can be run
// repeatedly from device-resident inputs. With one_block, one small pair is
// planned by a block instead (not under a memory limit, whose lists are sized
// by reading their lengths back, nor for a trace of the items).
int ctx_prepare(xted_ctx *c, const xted_tree *a, const xted_tree *b, int32_t npairs, bool one_block) {
    c->prepared = false;
    ctx_drop_graph(c);  // the graph holds the previous plan's buffers and sizes
    for (int32_t p = 0; p < npairs; p++)
        if (!costs_fit(c->opts, a[p].n, b[p].n)) return XTED_EINVAL;
    XKernelParams &K = c->kp;
    const char *tr = std::getenv("XTED_TRACE");
    if (one_block && npairs == 1 && a->n > 0 && b->n > 0 && (int64_t)a->n + b->n <= XTED_PAIR_NODES &&
        c->opts.mem_limit == 0 && !(tr && *tr)) {
        const int rc = pair_prepare(c, *a, *b);
        if (rc != XTED_ENOMEM) return rc;  // (the batch's kernels size their lists and need less room)
    }
    int rc = dev_plan(c, a, b, npairs, K);
    if (rc) return rc;
    K.c_del = c->opts.cost_del;
    K.c_ins = c->opts.cost_ins;
    K.c_ren = c->opts.cost_ren;
    rc = ctx_dev_reserve(c, c->dt, (size_t)std::max<int64_t>(c->plan_dt_elems, 1) * sizeof(int32_t));
    if (rc) return rc;
    // per-warp scratch: the far-row stack's rows outside the shared window
    const int64_t stack_rows = c->plan_stack_rows;
    const int64_t per = stack_rows * XTED_SW;
    c->full = npairs >= XTED_FULL_PAIRS && c->grid_full > 0;
    c->run_grid = c->full ? c->grid_full : c->grid;
    // counters: [1] error, [2..5] error info, then out[npairs]
    rc = ctx_dev_reserve(c, c->counters, (8 + 2 * (size_t)npairs) * sizeof(int32_t));
    if (rc) return rc;
    rc = ctx_host_reserve(c->result, ((size_t)npairs + 8) * sizeof(int32_t));
    if (rc) return rc;
    int32_t *cnt = (int32_t *)c->counters.p;
    K.dt = (int32_t *)c->dt.p;
    K.scratch_per_warp = per;
    K.stack_rows = (int32_t)stack_rows;
    K.error = cnt + 1;
    K.error_info = cnt + 2;
    K.timeout_ns = (uint64_t)(c->opts.wait_timeout_s * 1e9);
    // Optional per-item trace (XTED_TRACE=<file>): timestamps of every item,
    // written as raw uint64 quadruples after each run.
    K.trace = nullptr;
    if (tr && *tr && K.nitems > 0) {
        rc = ctx_dev_reserve(c, c->trace, (size_t)K.nitems * 4 * sizeof(unsigned long long));
        if (rc) return rc;
        K.trace = (unsigned long long *)c->trace.p;
    }
    c->parts.assign({XPart{0, 0, 0}, XPart{0, K.nitems, 0}});
    rc = reserve_launch(c);
    if (rc) return rc;
    c->npairs = npairs;
    c->prepared = true;
    return XTED_OK;
}

// Runs the prepared plan: counter reset, the persistent DP launch, the
// gather, and the copy of results + error word to pinned memory. Synchronous.
// One step of the prepared plan, enqueued on the context's stream: counter
// resets, the persistent DP launch, the gather, and the copy of results + error word to pinned memory.
// first: nothing has run since the plan was uploaded.
static int enqueue_step(xted_ctx *c, bool events, bool first) {
    const XKernelParams &K = c->kp;
    const int npairs = c->npairs;
    int32_t *cnt = (int32_t *)c->counters.p;
    int32_t *d_out = cnt + 8 + npairs;
    int32_t *hres = (int32_t *)c->result.p;
    const size_t res_bytes = (size_t)npairs * sizeof(int32_t);
    if (events && cudaEventRecord(c->ev0, c->stream) != cudaSuccess) return XTED_ECUDA;
    if (K.plan) {
        const PairLayout &L = c->pair;
        const int grid = pair_grid(c->grid, L.m, L.n);
        if ((!first &&  // (the first run finds the words zero, as uploaded)
             cudaMemsetAsync(L.hdr, 0, PAIR_CTL_INTS * sizeof(int32_t), c->stream) != cudaSuccess) ||
            launch_pair_clear(L, grid, c->stream) != cudaSuccess ||
            (events && cudaEventRecord(c->evk0, c->stream) != cudaSuccess) ||
            launch_dp(K, grid, false, c->stream) != cudaSuccess ||
            (events && cudaEventRecord(c->evk1, c->stream) != cudaSuccess) ||
            (events && cudaEventRecord(c->ev1, c->stream) != cudaSuccess) ||
            cudaMemcpyAsync(hres, L.hdr, (PAIR_HDR_INTS + 1) * sizeof(int32_t), cudaMemcpyDeviceToHost, c->stream) !=
                cudaSuccess)
            return XTED_ECUDA;
        return XTED_OK;
    }
    // per-run reset: the error words; every table to -1 (not written), and of each part the claim counter and the
    // hand-off words
    if (cudaMemsetAsync(cnt, 0, 8 * sizeof(int32_t), c->stream) != cudaSuccess ||
        (K.nitems > 0 &&
         cudaMemsetAsync(K.dt, 0xff, (size_t)c->plan_dt_elems * sizeof(int32_t), c->stream) != cudaSuccess))
        return XTED_ECUDA;
    for (size_t k = 0; k + 1 < c->parts.size() && K.nitems > 0; k++) {
        const XPart &p = c->parts[k], &q = c->parts[k + 1];
        XKernelParams part = K;
        part.items = K.items + p.item;
        part.nitems = q.item - p.item;
        part.buf = (int32_t *)((uintptr_t)c->sbuf.p - (uintptr_t)p.word * sizeof(int32_t));
        if (K.trace) part.trace = K.trace + 4 * (int64_t)p.item;
        if (cudaMemsetAsync(K.next, 0, 2 * sizeof(int32_t), c->stream) != cudaSuccess ||
            (q.word > p.word &&
             cudaMemsetAsync(c->sbuf.p, 0xff, (size_t)(q.word - p.word) * sizeof(int32_t), c->stream) != cudaSuccess) ||
            (events && k == 0 && cudaEventRecord(c->evk0, c->stream) != cudaSuccess) ||
            launch_dp(part, c->run_grid, c->full, c->stream) != cudaSuccess)
            return XTED_ECUDA;
    }
    if (events && K.nitems == 0 && cudaEventRecord(c->evk0, c->stream) != cudaSuccess) return XTED_ECUDA;
    if (events && cudaEventRecord(c->evk1, c->stream) != cudaSuccess) return XTED_ECUDA;
    if (launch_gather(K.pairs, c->d_trivial, K.dt, npairs, d_out, K.c_del, K.c_ins, K.error, c->stream) != cudaSuccess)
        return XTED_ECUDA;
    if ((events && cudaEventRecord(c->ev1, c->stream) != cudaSuccess) ||
        cudaMemcpyAsync(hres, cnt, 8 * sizeof(int32_t), cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
        (npairs && cudaMemcpyAsync(hres + 8, d_out, res_bytes, cudaMemcpyDeviceToHost, c->stream) != cudaSuccess))
        return XTED_ECUDA;
    return XTED_OK;
}

void ctx_drop_graph(xted_ctx *c) {
    if (c->step_graph) cudaGraphExecDestroy(c->step_graph);
    c->step_graph = nullptr;
    c->runs_prepared = 0;
}

// Captures the step into a graph; false (and no graph is tried again for this
// context) if the runtime refuses any part of it.
static bool capture_step(xted_ctx *c) {
    cudaGraph_t g = nullptr;
    if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const int rc = enqueue_step(c, false, false);  // events recorded inside a graph cannot be timed
    const cudaError_t e = cudaStreamEndCapture(c->stream, &g);
    bool ok = rc == XTED_OK && e == cudaSuccess && g != nullptr &&
              cudaGraphInstantiate(&c->step_graph, g, 0) == cudaSuccess;
    if (g) cudaGraphDestroy(g);
    if (!ok) {
        cudaGetLastError();
        c->step_graph = nullptr;
    }
    return ok;
}

// Runs the prepared plan. Synchronous. With allow_graph, the second and later
// runs of one prepared plan replay a CUDA graph of the step (one launch of
// the whole sequence instead of eleven enqueues).
int ctx_run(xted_ctx *c, int32_t *out, bool allow_graph) {
    if (!c->prepared) return XTED_EINVAL;
    const XKernelParams &K = c->kp;
    const int npairs = c->npairs;
    int32_t *hres = (int32_t *)c->result.p;
    const size_t res_bytes = (size_t)npairs * sizeof(int32_t);
    bool replay = false;
    if (allow_graph && !K.trace && !c->graph_failed && c->runs_prepared >= 1) {
        if (!c->step_graph && !capture_step(c)) c->graph_failed = true;
        replay = c->step_graph != nullptr;
    }
    const bool first = c->runs_prepared == 0;
    c->runs_prepared++;
    if (replay) {
        // timed from outside: the DP time of a replay includes the step's
        // clearing of the tables and its gather
        if (cudaEventRecord(c->ev0, c->stream) != cudaSuccess || cudaEventRecord(c->evk0, c->stream) != cudaSuccess ||
            cudaGraphLaunch(c->step_graph, c->stream) != cudaSuccess ||
            cudaEventRecord(c->evk1, c->stream) != cudaSuccess || cudaEventRecord(c->ev1, c->stream) != cudaSuccess) {
            cudaGetLastError();
            return XTED_ECUDA;
        }
    } else {
        const int rc = enqueue_step(c, true, first);
        if (rc) {
            cudaGetLastError();
            return rc;
        }
    }
    c->stats.graph = replay ? 1 : 0;
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) {
        cudaGetLastError();
        return XTED_ECUDA;
    }
    float ms = 0.f, kms = 0.f;
    cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    cudaEventElapsedTime(&kms, c->evk0, c->evk1);
    cudaGetLastError();  // a failed timing read must not surface in a later call
    c->stats.device_ms = ms;
    c->stats.dp_ms = kms;
    c->stats.h2d_bytes = c->h2d_bytes;
    if (K.plan) {
        const XPlanOut plan = *(const XPlanOut *)(hres + PAIR_OUT);
        c->stats.d2h_bytes = (PAIR_HDR_INTS + 1) * sizeof(int32_t);
        c->stats.grid = pair_grid(c->grid, c->pair.m, c->pair.n);
        if (plan.status != 0) return plan.status;
        c->kp.nitems = plan.items;  // (for the statistics: the launch reads the plan's)
        c->plan_cells = plan.cells;
        c->plan_cells_right = plan.cells_right;
        c->plan_levels_max = plan.levels;
        std::memcpy(c->err_info, hres + PAIR_ERROR + 1, sizeof(c->err_info));
        if (hres[PAIR_ERROR] != 0) return hres[PAIR_ERROR];
        const int32_t v = hres[PAIR_HDR_INTS];  // the root table's saving
        if (v < 0) return XTED_ETIMEOUT;
        out[0] = c->pair.m * K.c_del + c->pair.n * K.c_ins - v;
        return XTED_OK;
    }
    c->stats.d2h_bytes = (int64_t)(res_bytes + 8 * sizeof(int32_t));
    c->stats.grid = c->run_grid;
    std::memcpy(c->err_info, hres + 2, sizeof(c->err_info));
    if (K.trace) {
        std::vector<unsigned long long> tr((size_t)K.nitems * 4);
        if (cudaMemcpy(tr.data(), K.trace, tr.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost) ==
            cudaSuccess) {
            if (FILE *f = std::fopen(std::getenv("XTED_TRACE"), "wb")) {
                std::fwrite(tr.data(), sizeof(unsigned long long), tr.size(), f);
                std::fclose(f);
            }
            // the plan beside it: the items in list order
            std::vector<XItem> it((size_t)K.nitems);
            const std::string base = std::getenv("XTED_TRACE");
            if (cudaMemcpy(it.data(), K.items, it.size() * sizeof(XItem), cudaMemcpyDeviceToHost) == cudaSuccess)
                if (FILE *f = std::fopen((base + ".items").c_str(), "wb")) {
                    std::fwrite(it.data(), sizeof(XItem), it.size(), f);
                    std::fclose(f);
                }
        }
    }
    if (hres[1] != 0) return hres[1];
    if (npairs) std::memcpy(out, hres + 8, res_bytes);
    return XTED_OK;
}

const XTuneRow *ctx_tune_table(const xted_ctx *c, int *nrows) {
    if (c->ntune > 0) {
        *nrows = c->ntune;
        return c->tune;
    }
    *nrows = kTuneRows;
    return kTuneTable;
}

// The granularity a launch is planned with. A run of rows ends the wait of the
// tables that need it, so short runs shorten the chain of a launch that does
// not fill the GPU; a full one pays for every run's start (its copies are not
// yet in flight). The lines lie where the node products of the launch's pairs
// together pass 2, 20 and 100 million. Device ms at runs of 16 / 32 / 128 / 256 rows:
//   one pair of 60 0.095 / 0.113 / 0.125 / 0.126, of 1,000 1.22 / 1.25 / 1.57 / 2.00;
//   64 pairs of 400 (10 M) 0.908 / 0.890 / 0.967 / 1.03, 16 of 1,000 (16 M) 1.93 / 1.91 / 2.00 / 2.25;
//   256 of 400 (41 M) 2.09 / 1.97 / 1.89 / 1.94, 64 of 1,000 (64 M) 4.25 / 4.15 / 4.17 / 4.16;
//   1,024 of 400 (164 M) 6.38 / 5.89 / 5.47 / 5.38, 256 of 1,000 11.8 / 11.1 / 10.5 / 10.4.
// A table set by xted_set_tune_table, or the options of an untuned context, is taken as it is.
void ctx_granularity(const xted_ctx *c, int64_t products, PlanPools &P) {
    P.run_rows = c->opts.run_rows;
    P.narrow_width = c->opts.narrow_width;
    P.half_width = c->opts.half_width == 0 ? XTED_HALF_DEFAULT : c->opts.half_width;
    P.ntune = 0;
    if (!c->opts.tuned) return;
    const int32_t cap = products < 2000000 ? 16 : products < 20000000 ? 32 : products < 100000000 ? 128 : INT32_MAX;
    int nt = 0;
    const XTuneRow *tt = ctx_tune_table(c, &nt);
    for (int k = 0; k < nt && k < XTED_TUNE_ROWS; k++) {
        P.tune[k] = tt[k];
        if (c->ntune <= 0) P.tune[k].run_rows = std::min(tt[k].run_rows, cap);
        P.ntune++;
    }
}

void fill_stats(xted_ctx *c, double plan_ms) {
    c->stats.pairs = c->npairs;
    c->stats.cells = c->plan_cells;
    c->stats.cells_right = c->plan_cells_right;
    c->stats.tasks = c->kp.nitems;
    c->stats.units = c->kp.nitems;
    c->stats.levels_max = c->plan_levels_max;
    c->stats.host_plan_ms = plan_ms;
}

}  // namespace xted

extern "C" {

void xted_opts_default(xted_opts *o) {
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->device = 0;
    o->orientation = XTED_ORIENT_AUTO;
    o->narrow_width = XTED_NARROW_MAX;
    o->run_rows = 64;
    o->ctas_per_sm = 0;
    o->wide_rows = 0;
    o->half_width = 0;
    o->tuned = 1;
    o->wait_timeout_s = 20.0;
    o->mem_limit = 0;
    o->stripe_min_cells = 0;
    o->cost_del = o->cost_ins = o->cost_ren = 1;
}

const char *xted_strerror(int code) {
    switch (code) {
        case XTED_OK: return "ok";
        case XTED_EINVAL: return "invalid argument or malformed tree";
        case XTED_ENOMEM: return "out of memory (device, host or the context's limit)";
        case XTED_ETIMEOUT: return "a bounded device wait timed out";
        case XTED_ECUDA: return "CUDA runtime error";
        case XTED_ENODEV: return "no usable sm_100 CUDA device";
        case XTED_ENOTFOUND: return "unknown ticket";
        case XTED_EAGAIN: return "serving queue full";
        case XTED_ETOOBIG: return "pair does not fit the fixed arena of xted_distance_noalloc";
        default: return "unknown error";
    }
}

int xted_create(xted_ctx **out, const xted_opts *opts) {
    if (!out) return XTED_EINVAL;
    *out = nullptr;
    xted_opts o;
    if (opts) o = *opts;
    else xted_opts_default(&o);
    if (o.narrow_width < 0 || o.narrow_width > XTED_NARROW_MAX || o.run_rows < 1 ||
        o.orientation < 0 || o.orientation > 2 || o.wait_timeout_s <= 0 || o.ctas_per_sm < 0 ||
        o.cost_del < 0 || o.cost_ins < 0 || o.cost_ren < 0 || o.cost_del >= XTED_COST_BOUND ||
        o.cost_ins >= XTED_COST_BOUND || o.cost_ren >= XTED_COST_BOUND)
        return XTED_EINVAL;
    if (o.cost_del == 0 && o.cost_ins == 0 && o.cost_ren == 0) o.cost_del = o.cost_ins = o.cost_ren = 1;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || o.device < 0 || o.device >= ndev) {
        cudaGetLastError();
        return XTED_ENODEV;
    }
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, o.device) != cudaSuccess || prop.major != 10) return XTED_ENODEV;
    if (cudaSetDevice(o.device) != cudaSuccess) return XTED_ECUDA;
    xted_ctx *c = new (std::nothrow) xted_ctx();
    if (!c) return XTED_ENOMEM;
    c->opts = o;
    c->sms = prop.multiProcessorCount;
    int occ = 0;
    int occ_full = 0;
    if (dp_occupancy(&occ, false) != 0 || occ < 1 || dp_occupancy(&occ_full, true) != 0) {
        delete c;
        return XTED_ECUDA;
    }
    // (under a limit on blocks or on memory, whose stacks would be a quarter more, only the smaller launch)
    if (occ_full > occ && o.ctas_per_sm == 0 && o.mem_limit == 0) c->grid_full = occ_full * c->sms;
    if (o.ctas_per_sm > 0) occ = std::min(occ, o.ctas_per_sm);
    c->grid = occ * c->sms;
    if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&c->ev0) != cudaSuccess || cudaEventCreate(&c->ev1) != cudaSuccess ||
        cudaEventCreate(&c->evk0) != cudaSuccess || cudaEventCreate(&c->evk1) != cudaSuccess) {
        delete c;
        return XTED_ECUDA;
    }
    *out = c;
    return XTED_OK;
}

int xted_destroy(xted_ctx *c) {
    if (!c) return XTED_OK;
    cudaSetDevice(c->opts.device);
    xted::serve_shutdown(c);
    cudaStreamSynchronize(c->stream);
    ctx_drop_graph(c);
    for (DevBuf *b : {&c->meta, &c->levels, &c->work, &c->dt, &c->scratch, &c->counters, &c->trace, &c->smap, &c->sbuf})
        if (b->p) cudaFree(b->p);
    for (HostBuf *b : {&c->stage, &c->result, &c->summary})
        if (b->p) cudaFreeHost(b->p);
    for (cudaEvent_t e : {c->ev0, c->ev1, c->evk0, c->evk1})
        if (e) cudaEventDestroy(e);
    cudaStreamDestroy(c->stream);
    delete c;
    return XTED_OK;
}

int xted_distance_batch(xted_ctx *c, const xted_tree *a, const xted_tree *b, int32_t npairs,
                        int32_t *out) {
    if (!c || npairs < 0 || (npairs > 0 && (!a || !b || !out))) return XTED_EINVAL;
    const double t0 = now_ms();
    if (cudaSetDevice(c->opts.device) != cudaSuccess) return XTED_ECUDA;
    int rc = ctx_prepare(c, a, b, npairs, true);
    double t1 = now_ms();
    std::memset(&c->stats, 0, sizeof(c->stats));
    if (rc) return rc;
    const bool hold = c->fault == XTED_FAULT_HOLD_PAIR && npairs > 0;
    if (hold) {  // test hook: pair 0's level 0 is never published
        c->fault = 0;
        c->kp.hold_pair = 0;
    }
    rc = ctx_run(c, out, false);
    if (rc == PLAN_OVERFLOW) {  // one pair, planned by one block: a list did not fit
        rc = ctx_prepare(c, a, b, npairs, false);
        t1 = now_ms();
        if (rc) return rc;
        if (hold) c->kp.hold_pair = 0;
        rc = ctx_run(c, out, false);
    }
    c->kp.hold_pair = -1;
    fill_stats(c, t1 - t0);
    c->stats.total_ms = now_ms() - t0;
    return rc;
}

int xted_prepare_batch(xted_ctx *c, const xted_tree *a, const xted_tree *b, int32_t npairs) {
    if (!c || npairs < 0 || (npairs > 0 && (!a || !b))) return XTED_EINVAL;
    if (cudaSetDevice(c->opts.device) != cudaSuccess) return XTED_ECUDA;
    const double t0 = now_ms();
    int rc = ctx_prepare(c, a, b, npairs, false);
    std::memset(&c->stats, 0, sizeof(c->stats));
    if (rc) return rc;
    c->prep_ms = now_ms() - t0;
    c->stats.host_plan_ms = c->prep_ms;
    return cudaStreamSynchronize(c->stream) == cudaSuccess ? XTED_OK : XTED_ECUDA;
}

int xted_run_prepared(xted_ctx *c, int32_t *out) {
    if (!c || !out) return XTED_EINVAL;
    if (cudaSetDevice(c->opts.device) != cudaSuccess) return XTED_ECUDA;
    const int rc = ctx_run(c, out, true);
    fill_stats(c, c->prep_ms);
    return rc;
}

int xted_distance(xted_ctx *c, const xted_tree *a, const xted_tree *b, int32_t *out) {
    return xted_distance_batch(c, a, b, 1, out);
}

int xted_distance_matrix(xted_ctx *c, const xted_tree *trees, int32_t ntrees, int64_t pair_budget, int32_t *out) {
    if (!c || ntrees < 0 || (ntrees > 0 && (!trees || !out)) || pair_budget < 0) return XTED_EINVAL;
    int64_t budget = pair_budget > 0 ? pair_budget
                                     : (c->opts.mem_limit > 0 ? c->opts.mem_limit / 16 : (int64_t)1 << 30);
    const int64_t max_pairs = (int64_t)1 << 20;
    // TED is symmetric when deleting and inserting cost the same: each
    // unordered pair once, mirrored; else both orders
    const bool sym = c->opts.cost_del == c->opts.cost_ins;
    std::vector<xted_tree> A, B;
    std::vector<int64_t> at;  // i * ntrees + j of each pair in the chunk
    std::vector<int32_t> res;
    auto flush = [&]() -> int {
        if (A.empty()) return XTED_OK;
        res.resize(A.size());
        const int rc = xted_distance_batch(c, A.data(), B.data(), (int32_t)A.size(), res.data());
        if (rc) return rc;
        for (size_t k = 0; k < A.size(); k++) {
            const int64_t i = at[k] / ntrees, j = at[k] % ntrees;
            out[i * ntrees + j] = res[k];
            if (sym) out[j * ntrees + i] = res[k];
        }
        A.clear();
        B.clear();
        at.clear();
        return XTED_OK;
    };
    int64_t cells = 0;
    for (int32_t i = 0; i < ntrees; i++) {
        out[(int64_t)i * ntrees + i] = 0;
        for (int32_t j = sym ? i + 1 : 0; j < ntrees; j++) {
            if (j == i) continue;
            const int64_t c2 = (int64_t)std::max(trees[i].n, 1) * std::max(trees[j].n, 1);
            if (!A.empty() && (cells + c2 > budget || (int64_t)A.size() >= max_pairs)) {
                const int rc = flush();
                if (rc) return rc;
                cells = 0;
            }
            A.push_back(trees[i]);
            B.push_back(trees[j]);
            at.push_back((int64_t)i * ntrees + j);
            cells += c2;
        }
    }
    return flush();
}

int xted_test_fault(xted_ctx *c, int32_t kind) {
    if (!c || kind < 0 || kind > XTED_FAULT_HOLD_PAIR) return XTED_EINVAL;
    if (c->serve) {
        std::lock_guard<std::mutex> g(serve_mutex(c));
        c->fault = kind;
    } else {
        c->fault = kind;
    }
    return XTED_OK;
}

int xted_last_stats(const xted_ctx *c, xted_stats *out) {
    if (!c || !out) return XTED_EINVAL;
    *out = c->stats;
    return XTED_OK;
}

int xted_set_tune_table(xted_ctx *c, const int32_t *rows, int32_t nrows) {
    if (!c || nrows < 0 || nrows > XTED_TUNE_ROWS || (nrows > 0 && !rows)) return XTED_EINVAL;
    for (int k = 0; k < nrows; k++) {
        const int32_t *r = rows + 4 * k;
        if (r[0] <= 0 || (k > 0 && r[0] <= rows[4 * (k - 1)]) || r[1] < 1 || r[2] < 0 || r[2] > XTED_NARROW_MAX ||
            r[3] < -1 || r[3] > XTED_HALF_MAX)
            return XTED_EINVAL;
    }
    for (int k = 0; k < nrows; k++) c->tune[k] = XTuneRow{rows[4 * k], rows[4 * k + 1], rows[4 * k + 2], rows[4 * k + 3]};
    c->ntune = nrows > 0 ? nrows : -1;
    return XTED_OK;
}

int xted_pair_cells(const xted_tree *a, const xted_tree *b, int32_t orientation, int64_t *out3) {
    if (!a || !b || !out3 || orientation < 0 || orientation > 2) return XTED_EINVAL;
    TreeView A{a->n, a->labels, a->child_off, a->child_idx};
    TreeView B{b->n, b->labels, b->child_off, b->child_idx};
    int rc = validate_tree(A);
    if (!rc) rc = validate_tree(B);
    if (rc) return rc;
    int64_t sa[2], sb[2];
    keyroot_sums(A, sa);
    keyroot_sums(B, sb);
    out3[0] = sa[0] * sb[0];
    out3[1] = sa[1] * sb[1];
    out3[2] = orientation == XTED_ORIENT_RIGHT ? out3[0]
              : orientation == XTED_ORIENT_LEFT ? out3[1]
                                                : std::min(out3[0], out3[1]);
    return XTED_OK;
}

int xted_validate(const xted_tree *t) {
    if (!t) return XTED_EINVAL;
    return validate_tree(TreeView{t->n, t->labels, t->child_off, t->child_idx});
}

}  // extern "C"
