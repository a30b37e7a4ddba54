// serve.cpp -- a resident corpus and exact top-k TED queries, with continuous
// batching into one running persistent DP launch.
//
// Nothing in the reference serves queries (its only caller computes one pair,
// X-TED_CPU/TED_test.cpp:26-47); the per-pair work is the same keyroot-table
// DP as the batch path (X-TED_CPU/parallel_computing.cpp:4-182).
//
// Layout. The corpus trees are planned once (both orientations) on the host
// with the batch planner's own functions (plan_core.h) and stay resident on
// the device. A query is one more tree planned into one of XTED_SERVE_SLOTS
// slots: its node pools, its pairs (query x every corpus tree, the corpus
// tree as the row tree so the far-row stack depth is a corpus property),
// their items. Tables, hand-off words and export maps come from a pool of
// device memory; a query is admitted when a slot is free and these and its
// items fit ("DP scratch bytes"), in arrival order.
//
// Continuous batching. An admitted query's plan is copied to the device on a
// copy stream, its slot's list word written last; the launch sets its tables to
// "not written" before it runs the list's items. The warps of the DP kernel, launched once
// and kept running while there is work, claim items from the lists of all
// slots, the oldest query's first, so earlier queries finish first while later
// ones fill idle warps. The item that ends a pair writes its distance into
// pinned host memory; the last item of a query raises the slot's flag. Warps
// leave the launch after an idle spell; a worker thread relaunches when new
// work arrives.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <climits>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <thread>
#include <unordered_map>
#include <vector>

#include "../../include/xted.h"
#include "ctx.h"
#include "plan.h"
#include "plan_core.h"
#include "serve_plan.h"

namespace xted {
int serve_occupancy(int *blocks_per_sm);
cudaError_t launch_dp(const XKernelParams &P, int grid, bool full, cudaStream_t s);
}

static_assert(XTED_SERVE_SLOTS == XTED_SERVE_SLOTS_MAX, "slot count of the ABI and the kernels");

namespace xted {

namespace {

double now_ms() {
    using namespace std::chrono;
    return duration<double, std::milli>(steady_clock::now().time_since_epoch()).count();
}

// First-fit allocator over [0, cap) (elements).
class Extents {
public:
    void reset(int64_t cap) {
        free_.clear();
        if (cap > 0) free_[0] = cap;
        cap_ = cap;
    }
    int64_t cap() const { return cap_; }
    bool alloc(int64_t n, int64_t *off) {
        n = std::max<int64_t>(n, 1);
        for (auto it = free_.begin(); it != free_.end(); ++it)
            if (it->second >= n) {
                const int64_t lo = it->first, len = it->second;
                free_.erase(it);
                if (len > n) free_[lo + n] = len - n;
                *off = lo;
                return true;
            }
        return false;
    }
    // n = 0: nothing is held (a slot whose extents were already released)
    void release(int64_t off, int64_t n) {
        if (n <= 0) return;
        auto it = free_.emplace(off, n).first;
        auto nx = std::next(it);
        if (nx != free_.end() && it->first + it->second == nx->first) {
            it->second += nx->second;
            free_.erase(nx);
        }
        if (it != free_.begin()) {
            auto pv = std::prev(it);
            if (pv->first + pv->second == it->first) {
                pv->second += it->second;
                free_.erase(it);
            }
        }
    }

private:
    std::map<int64_t, int64_t> free_;
    int64_t cap_ = 0;
};

struct Query {
    std::vector<int32_t> lab, off, idx;
    int32_t n = 0, k = 0;
    std::vector<int32_t> lb, dist;  // per corpus tree: label lower bound; distance once known (-1 before)
    int state = 0;  // 0 queued, 1 admitted, 2 done, < 0 error code
    std::vector<int32_t> ids, dists;
    double t_submit = 0, t_admit = 0, t_done = 0;
};

struct Slot {
    bool busy = false;
    int round = 1;               // 1: the most promising corpus trees; 2: what may still beat them
    bool need_post = false;      // a planned next round waits for device room
    std::vector<uint8_t> inc;    // corpus trees computed in this round
    uint64_t ticket = 0;
    int64_t seq = 0;
    int32_t gen = 0;
    int part = 0;                // of the plan's list
    int64_t dt_off = 0, dt_n = 0, i_off = 0, i_n = 0;  // table pool and item pool ranges
    QPlan plan;
};

}  // namespace

struct ServeState {
    xted_ctx *c = nullptr;
    int T = 0, S = XTED_SERVE_SLOTS, Qmax = XTED_SERVE_MAX_QUERY;  // XTED_SERVE_SLOTS == XTED_SERVE_SLOTS_MAX
    int32_t max_tree = 0;  // largest corpus tree
    int grid = 0;          // blocks of the launch
    int64_t Nc_nonempty = 0;
    ServePools pools;  // host planning pools: the corpus, then one region per slot
    // device
    std::vector<void *> dev_allocs;
    int2 *d_node = nullptr;
    int32_t *d_krd = nullptr, *d_cumw = nullptr, *d_ctl = nullptr, *d_slot = nullptr, *d_err = nullptr,
            *d_scratch = nullptr, *d_dt = nullptr;
    XRun *d_runs = nullptr;
    XChunk *d_chunks = nullptr;
    XPair *d_pairs = nullptr;
    XChunkX *d_chunkx = nullptr;
    XItem *d_items = nullptr;
    unsigned long long *d_lists = nullptr;
    XServeClear *d_clears = nullptr;
    int32_t *h_results = nullptr, *h_flags = nullptr;  // mapped pinned host memory
    Extents dt_ext, i_ext;
    int64_t dt_cap = 0;  // distances of a query's tables, at most
    XKernelParams K{};
    cudaStream_t ks = nullptr, cs = nullptr;
    cudaEvent_t kev = nullptr;
    bool running = false;
    // requests
    std::mutex mu;
    std::condition_variable cv_work, cv_done;
    std::deque<uint64_t> pending;
    std::unordered_map<uint64_t, Query> queries;
    uint64_t next_ticket = 1;
    int64_t next_seq = 0;
    int32_t next_gen = 1;
    Slot slots[XTED_SERVE_SLOTS];
    int error = 0;
    bool stop = false;
    std::thread worker;
    // counters
    int64_t launches = 0, served = 0, pairs_served = 0, cells_served = 0, pairs_pruned = 0, second_rounds = 0;
    int64_t bound_us = 0, plan_us = 0;  // host time spent on bounds and on planning
    // exact top-k pruning by lower bounds: 0 off, 1 label multisets, 2 preorder sequences
    int prune = 2;
    int first_round = 32;                            // at least this many trees, and 4k, in round 1
    std::vector<std::vector<int32_t>> sorted_labels;  // per corpus tree
    std::unordered_map<int32_t, int32_t> dense;       // corpus label -> dense symbol
    std::vector<std::vector<int32_t>> dense_seq;      // per corpus tree: preorder dense symbols
};

namespace {

constexpr int kMaxPending = 1 << 16;
constexpr int64_t kItemCap = 12 << 20;
constexpr int64_t kItemPart = kItemCap / 2;  // a longer list is posted in parts, beside which others fit
constexpr int64_t kDtCapMax = (int64_t)4 << 30;  // int32 elements (16 GiB)

template <class T>
int dev_alloc(ServeState *s, T **p, size_t count) {
    void *q = nullptr;
    if (cudaMalloc(&q, sizeof(T) * std::max<size_t>(count, 1)) != cudaSuccess) {
        cudaGetLastError();
        return XTED_ENOMEM;
    }
    s->dev_allocs.push_back(q);
    *p = (T *)q;
    return XTED_OK;
}

int upload(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    if (bytes == 0) return XTED_OK;
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st) == cudaSuccess ? XTED_OK : XTED_ECUDA;
}

void free_all(ServeState *s) {
    for (void *p : s->dev_allocs) cudaFree(p);
    s->dev_allocs.clear();
    if (s->h_results) cudaFreeHost(s->h_results);
    if (s->h_flags) cudaFreeHost(s->h_flags);
    s->h_results = s->h_flags = nullptr;
    if (s->kev) cudaEventDestroy(s->kev);
    if (s->ks) cudaStreamDestroy(s->ks);
    if (s->cs) cudaStreamDestroy(s->cs);
    s->kev = nullptr;
    s->ks = s->cs = nullptr;
}

// Table-pool elements of a planned query: tables, hand-off words of a part,
// export maps (whole 16-byte pieces, so every query's tables start on one).
int64_t pool_elems(const QPlan &p) {
    const int64_t n = std::max<int64_t>(p.dt_elems + p.max_words + (int64_t)p.smap.size(), 1);
    return (n + XTED_PITCH - 1) / XTED_PITCH * XTED_PITCH;
}

// Divides a planned query's list: hand-off words of at most a quarter of the
// table pool, or what its tables leave of it, at a time.
void divide(ServeState *s, QPlan &p) {
    const int64_t left = s->dt_ext.cap() - p.dt_elems - (int64_t)p.smap.size() - XTED_PITCH;
    serve_cut(p, std::max<int64_t>(std::min(left, s->dt_ext.cap() / 4), 1), kItemPart);
}

// Reserves device room for a planned query; false if it does not fit now.
bool reserve(ServeState *s, Slot &sl) {
    const QPlan &p = sl.plan;
    sl.dt_n = pool_elems(p);
    sl.i_n = std::max<int64_t>(p.max_items, 1);
    if (!s->dt_ext.alloc(sl.dt_n, &sl.dt_off)) return false;
    if (!s->i_ext.alloc(sl.i_n, &sl.i_off)) {
        s->dt_ext.release(sl.dt_off, sl.dt_n);
        return false;
    }
    return true;
}

bool never_fits(ServeState *s, const QPlan &p) {
    return p.distances > s->dt_cap || pool_elems(p) > s->dt_ext.cap() || p.max_items > s->i_ext.cap();
}

bool take_hold(ServeState *s) {
    const bool hold = s->c->fault == XTED_FAULT_HOLD_PAIR;
    if (hold) s->c->fault = 0;
    return hold;
}

int32_t next_gen(ServeState *s) {
    const int32_t g = s->next_gen++;
    if (s->next_gen <= 0) s->next_gen = 1;
    return g;
}

void release_extents(ServeState *s, Slot &sl) {
    s->dt_ext.release(sl.dt_off, sl.dt_n);
    s->i_ext.release(sl.i_off, sl.i_n);
    sl.dt_n = sl.i_n = 0;
}

void release(ServeState *s, Slot &sl) {
    release_extents(s, sl);
    sl = Slot{};
}

// Copies part sl.part of the plan's list, its slot words and last its list
// word to the device, in that order, on the copy stream. Called without the
// lock (a list may be 200 MB, and a poll would wait for its copy): the slot is
// the worker's own. hold: the test hook, one computed pair is never computed.
int post_part(ServeState *s, int slot, Slot &sl, bool hold) {
    QPlan &p = sl.plan;
    cudaStream_t st = s->cs;
    XItem *items = p.items.data() + p.cuts[(size_t)sl.part];
    int64_t n = p.cuts[(size_t)sl.part + 1] - p.cuts[(size_t)sl.part];
    const int32_t words[2] = {(int32_t)n, sl.gen};
    for (int64_t k = 0; k < n; k++) items[k].gen = sl.gen;
    if (hold) {
        const int32_t held = items[0].pair;
        n = std::remove_if(items, items + n, [&](const XItem &i) { return i.pair == held; }) - items;
    }
    const int64_t done = sl.part > 0 ? p.dt_elems : 0;  // the tables stay between parts
    const int64_t clear = p.dt_elems - done + p.part_words[(size_t)sl.part];
    const XServeClear cl{sl.dt_off + done, clear, (int32_t)((clear + XTED_CLEAR_INTS - 1) / XTED_CLEAR_INTS), 0, 0, 0};
    const unsigned long long list = ((unsigned long long)(sl.i_off + n) << 32) | (unsigned long long)sl.i_off;
    const int32_t age = (int32_t)sl.seq;
    int rc = XTED_OK;
    rc |= upload(s->d_items + sl.i_off, items, (size_t)n * sizeof(XItem), st);
    rc |= upload(s->d_slot + XTED_SERVE_SLOTS + slot, &words[0], 4, st);      // slot_need
    rc |= upload(s->d_slot + 2 * XTED_SERVE_SLOTS + slot, &words[1], 4, st);  // slot_gen
    rc |= upload(s->d_slot + 3 * XTED_SERVE_SLOTS + slot, &age, 4, st);
    rc |= upload(s->d_clears + slot, &cl, sizeof(cl), st);
    rc |= upload(s->d_lists + slot, &list, sizeof(list), st);
    return rc ? XTED_ECUDA : XTED_OK;
}

// Fixes the plan up to its device offsets and copies it to the device, with the
// first part of its list.
int post(ServeState *s, int slot, Slot &sl, bool hold) {
    QPlan &p = sl.plan;
    const int T = s->T;
    const int64_t pair_base = (int64_t)slot * T;
    serve_fixup_items(s->pools, p, slot, sl.dt_off);
    const ServePools &H = s->pools;
    const DTree &Q = H.trees[(size_t)(T + slot)];
    const size_t nb = 2 * (size_t)Q.nbase, n2 = 2 * (size_t)Q.n;
    cudaStream_t st = s->cs;
    int rc = XTED_OK;
    rc |= upload(s->d_dt + sl.dt_off + p.dt_elems + p.max_words, p.smap.data(), p.smap.size() * 4, st);
    rc |= upload(s->d_node + nb, H.node.data() + nb, n2 * sizeof(int2), st);
    rc |= upload(s->d_krd + nb, H.krd.data() + nb, n2 * 4, st);
    rc |= upload(s->d_cumw + nb, H.cumw.data() + nb, n2 * 4, st);
    rc |= upload(s->d_runs + nb, H.runs.data() + nb, n2 * sizeof(XRun), st);
    rc |= upload(s->d_chunks + nb, H.chunks.data() + nb, n2 * sizeof(XChunk), st);
    rc |= upload(s->d_chunkx + nb, H.chunkx.data() + nb, n2 * sizeof(XChunkX), st);
    rc |= upload(s->d_pairs + pair_base, p.pairs.data(), p.pairs.size() * sizeof(XPair), st);
    sl.part = 0;
    return rc ? XTED_ECUDA : post_part(s, slot, sl, hold);
}

// Empties a slot's list, so that no launch claims the rest of it (on the copy
// stream: what is posted to the slot next comes after it).
void close_list(ServeState *s, int slot) {
    const unsigned long long none = 0;
    if (upload(s->d_lists + slot, &none, sizeof(none), s->cs) || upload(s->d_slot + slot, &none, 4, s->cs))
        cudaGetLastError();
}

// Finishes a query from its known distances: every corpus tree not computed
// has a bound that cannot beat the k-th of them (prune_round2 saw to it).
void finish_query(ServeState *s, Query &q) {
    q.ids.assign((size_t)q.k, -1);
    q.dists.assign((size_t)q.k, -1);
    topk_known(q.dist, q.k, q.ids.data(), q.dists.data());
    for (int32_t d : q.dist) s->pairs_pruned += d < 0;
    q.state = 2;
    q.t_done = now_ms();
}

// Round 1 of a query: the bound of every corpus tree (host threads), the
// distances of empty-tree pairs, and the trees computed first.
void first_round(ServeState *s, const Query &q, std::vector<int32_t> &lb, std::vector<int32_t> &dist,
                 std::vector<uint8_t> &inc) {
    const int T = s->T, level = s->prune;
    // distances are TED(query, corpus tree): deleting a query node costs
    // cost_del, inserting a corpus node cost_ins
    const xted_opts &o = s->c->opts;
    const bool unit = o.cost_del == 1 && o.cost_ins == 1 && o.cost_ren == 1;
    lb.assign((size_t)T, 0);
    dist.assign((size_t)T, -1);
    for (int t = 0; t < T; t++) {
        const int32_t ct = (int32_t)s->sorted_labels[(size_t)t].size();
        if (q.n == 0) dist[(size_t)t] = ct * o.cost_ins;  // X-TED_CPU/TED.cpp:181-186, with costs
        else if (ct == 0) dist[(size_t)t] = q.n * o.cost_del;
    }
    if (!unit && level > 0) {
        // weighted bounds: the label bound under the costs, and the unit
        // Levenshtein bound times the cheapest operation (an alignment of
        // distance L makes at least L operations)
        std::vector<int32_t> ql(q.lab);
        std::sort(ql.begin(), ql.end());
        std::vector<int32_t> qd;
        SeqBits P;
        if (level >= 2 && q.n > 0) {
            qd.resize((size_t)q.n);
            for (int v = 0; v < q.n; v++) {
                auto it = s->dense.find(q.lab[(size_t)v]);
                qd[(size_t)v] = it == s->dense.end() ? -1 : it->second;
            }
            P.build(qd.data(), q.n, (int)s->dense.size());
        }
        const int cmin = std::min(o.cost_del, std::min(o.cost_ins, o.cost_ren));
        parallel_for(T, 16, [&](int64_t lo, int64_t hi) {
            std::vector<uint64_t> work;
            for (int64_t t = lo; t < hi; t++) {
                if (dist[(size_t)t] >= 0) continue;
                const std::vector<int32_t> &tl = s->sorted_labels[(size_t)t];
                int32_t b = label_lower_bound_cost(label_common(ql.data(), q.n, tl.data(), (int)tl.size()), q.n,
                                                   (int)tl.size(), o.cost_del, o.cost_ins, o.cost_ren);
                if (level >= 2) {
                    const std::vector<int32_t> &sq = s->dense_seq[(size_t)t];
                    b = std::max<int32_t>(b, cmin * P.distance(sq.data(), (int)sq.size(), work));
                }
                lb[(size_t)t] = b;
            }
        });
    } else if (level == 1) {
        std::vector<int32_t> ql(q.lab);
        std::sort(ql.begin(), ql.end());
        parallel_for(T, 64, [&](int64_t lo, int64_t hi) {
            for (int64_t t = lo; t < hi; t++) {
                const std::vector<int32_t> &tl = s->sorted_labels[(size_t)t];
                lb[(size_t)t] = label_lower_bound(ql.data(), q.n, tl.data(), (int)tl.size());
            }
        });
    } else if (level >= 2 && q.n > 0) {
        std::vector<int32_t> qd((size_t)q.n);
        for (int v = 0; v < q.n; v++) {
            auto it = s->dense.find(q.lab[(size_t)v]);
            qd[(size_t)v] = it == s->dense.end() ? -1 : it->second;
        }
        SeqBits P;
        P.build(qd.data(), q.n, (int)s->dense.size());
        parallel_for(T, 16, [&](int64_t lo, int64_t hi) {
            std::vector<uint64_t> work;
            for (int64_t t = lo; t < hi; t++) {
                const std::vector<int32_t> &sq = s->dense_seq[(size_t)t];
                if (dist[(size_t)t] < 0) lb[(size_t)t] = P.distance(sq.data(), (int)sq.size(), work);
            }
        });
    }
    prune_round1(lb, dist, std::max<size_t>((size_t)s->first_round, 4 * (size_t)q.k), level > 0, inc);
}

void fail_inflight(ServeState *s, int code) {
    for (int i = 0; i < s->S; i++) {
        Slot &sl = s->slots[i];
        if (!sl.busy) continue;
        auto it = s->queries.find(sl.ticket);
        if (it != s->queries.end()) it->second.state = code;
        release(s, sl);
    }
}

// One pass of the serving loop (called with the lock held; drops it while planning).
bool step(ServeState *s, std::unique_lock<std::mutex> &lk) {
    bool progress = false;
    const int T = s->T;
    // 1. completions
    for (int i = 0; i < s->S; i++) {
        Slot &sl = s->slots[i];
        if (!sl.busy || sl.gen == 0) continue;
        if (((volatile int32_t *)s->h_flags)[i] != sl.gen) continue;
        std::atomic_thread_fence(std::memory_order_acquire);
        progress = true;
        auto it = s->queries.find(sl.ticket);
        if ((size_t)sl.part + 2 < sl.plan.cuts.size() && it != s->queries.end()) {  // the next part of its list
            Query &q = it->second;  // (stays where it is until it is done or has failed)
            sl.part++;
            sl.gen = next_gen(s);
            const bool hold = take_hold(s);
            lk.unlock();
            const int rc = post_part(s, i, sl, hold);
            lk.lock();
            if (rc != XTED_OK) {
                q.state = XTED_ECUDA;
                release(s, sl);
            }
            continue;
        }
        s->pairs_served += sl.plan.need;
        s->cells_served += sl.plan.cells;
        if (it == s->queries.end()) {
            release(s, sl);
            continue;
        }
        Query &q = it->second;
        const int32_t *res = s->h_results + (size_t)i * T;
        for (int t = 0; t < T; t++)
            if (sl.plan.trivial[(size_t)t] < 0 && sl.inc[(size_t)t]) q.dist[(size_t)t] = res[t];
        if (sl.round == 1 && s->prune > 0) {
            std::vector<uint8_t> inc2;
            if (prune_round2(q.lb, q.dist, q.k, inc2)) {  // plan round 2 in the same slot
                release_extents(s, sl);
                sl.gen = 0;
                sl.round = 2;
                Query qcopy = q;
                lk.unlock();
                const double t1 = now_ms();
                QPlan plan;
                serve_plan_items(s->pools, i, qcopy.lab.data(), qcopy.off.data(), qcopy.idx.data(), qcopy.n,
                                 s->c->opts.orientation, plan, inc2.data());
                divide(s, plan);
                const double t2 = now_ms();
                lk.lock();
                if (s->stop) {  // shutting down: no further round
                    sl = Slot{};
                    continue;
                }
                sl.plan = std::move(plan);
                sl.inc = std::move(inc2);
                s->plan_us += (int64_t)((t2 - t1) * 1e3);
                s->second_rounds++;
                if (never_fits(s, sl.plan)) {  // round 2 covers more trees than round 1 did
                    q.state = XTED_ENOMEM;
                    release(s, sl);
                    continue;
                }
                sl.need_post = true;
                continue;
            }
        }
        finish_query(s, q);
        s->served++;
        release(s, sl);
    }
    // next rounds waiting for device room
    for (int i = 0; i < s->S; i++) {
        Slot &sl = s->slots[i];
        if (!sl.busy || !sl.need_post || !reserve(s, sl)) continue;
        sl.need_post = false;
        sl.gen = next_gen(s);
        const bool hold = take_hold(s);
        lk.unlock();
        const int rc = post(s, i, sl, hold);
        lk.lock();
        auto it = s->queries.find(sl.ticket);
        if (rc != XTED_OK) {
            if (it != s->queries.end()) it->second.state = XTED_ECUDA;
            release(s, sl);
        }
        progress = true;
    }
    if (progress) s->cv_done.notify_all();
    // 2. the launch: notice its end (and any error), relaunch for work in flight.
    // One query: the launch may end between two of them.
    const cudaError_t kq = s->running ? cudaEventQuery(s->kev) : cudaErrorNotReady;
    if (s->running && kq == cudaSuccess) {
        s->running = false;
        int32_t err = 0;
        if (cudaMemcpy(&err, s->d_err, 4, cudaMemcpyDeviceToHost) != cudaSuccess) err = XTED_ECUDA;
        cudaStreamSynchronize(s->cs);  // every list posted so far is in place
        if (err != 0) {
            s->error = err;
            fail_inflight(s, err);
            cudaMemsetAsync(s->d_err, 0, 8 * sizeof(int32_t), s->cs);  // (a launch waits for this stream)
            for (int i = 0; i < s->S; i++) close_list(s, i);  // what is left of them is void
            s->cv_done.notify_all();
            progress = true;
        } else {
            // A launch leaves only when every warp is idle, so a query whose
            // items were all claimed has finished. One that has not (its work
            // was lost) fails instead of waiting forever; one with items left
            // goes on in the next launch.
            unsigned long long lists[XTED_SERVE_SLOTS] = {};
            if (cudaMemcpy(lists, s->d_lists, sizeof(lists), cudaMemcpyDeviceToHost) != cudaSuccess) cudaGetLastError();
            for (int i = 0; i < s->S; i++) {
                Slot &sl = s->slots[i];
                if (!sl.busy || sl.gen == 0) continue;
                if (((volatile int32_t *)s->h_flags)[i] == sl.gen) continue;  // done: step 1 takes it
                if ((uint32_t)lists[i] < (uint32_t)(lists[i] >> 32)) continue;
                if (std::getenv("XTED_SERVE_DEBUG")) {
                    int32_t done = -1;
                    cudaMemcpy(&done, s->d_slot + i, 4, cudaMemcpyDeviceToHost);
                    std::fprintf(stderr,
                                 "xted serve: launch %lld ended with slot %d unfinished: round %d gen %d items %zu "
                                 "done %d flag %d\n",
                                 (long long)s->launches, i, sl.round, sl.gen, sl.plan.items.size(), done,
                                 ((volatile int32_t *)s->h_flags)[i]);
                }
                auto it = s->queries.find(sl.ticket);
                if (it != s->queries.end()) it->second.state = XTED_ETIMEOUT;
                s->error = XTED_ETIMEOUT;
                close_list(s, i);  // the slot's finished-item count restarts for its next query
                release(s, sl);
                s->cv_done.notify_all();
                progress = true;
            }
        }
    } else if (s->running && kq != cudaErrorNotReady) {
        cudaGetLastError();
        s->running = false;
        s->error = XTED_ECUDA;
        fail_inflight(s, XTED_ECUDA);
        s->cv_done.notify_all();
    }
    // 3. admission, in arrival order
    while (!s->pending.empty()) {
        const uint64_t ticket = s->pending.front();
        auto it = s->queries.find(ticket);
        if (it == s->queries.end()) {
            s->pending.pop_front();
            continue;
        }
        Query &q = it->second;
        int slot = -1;
        for (int i = 0; i < s->S; i++)
            if (s->slots[i].busy && s->slots[i].ticket == ticket) slot = i;
        if (slot < 0) {
            const int64_t seq = s->next_seq;
            for (int i = 0; i < s->S && slot < 0; i++)
                if (!s->slots[i].busy) slot = i;
            if (slot < 0) break;
            Slot &sl = s->slots[slot];
            sl.busy = true;
            sl.ticket = ticket;
            sl.seq = seq;
            s->next_seq++;
            Query qcopy = q;  // plan outside the lock
            lk.unlock();
            const double t0 = now_ms();
            std::vector<int32_t> lb, dist;
            std::vector<uint8_t> inc;
            first_round(s, qcopy, lb, dist, inc);
            const double t1 = now_ms();
            QPlan plan;  // (a shutdown empties the slots meanwhile)
            serve_plan_items(s->pools, slot, qcopy.lab.data(), qcopy.off.data(), qcopy.idx.data(), qcopy.n,
                             s->c->opts.orientation, plan, inc.data());
            divide(s, plan);
            const double t2 = now_ms();
            lk.lock();
            s->bound_us += (int64_t)((t1 - t0) * 1e3);
            s->plan_us += (int64_t)((t2 - t1) * 1e3);
            if (s->stop || !sl.busy || sl.ticket != ticket) break;  // shut down meanwhile
            q.lb = std::move(lb);
            q.dist = std::move(dist);
            sl.plan = std::move(plan);
            sl.inc = std::move(inc);
            sl.round = 1;
            progress = true;
        }
        Slot &sl = s->slots[slot];
        if (never_fits(s, sl.plan)) {
            q.state = XTED_ENOMEM;
            sl = Slot{};
            s->pending.pop_front();
            s->cv_done.notify_all();
            continue;
        }
        if (sl.plan.need == 0) {  // empty query or empty corpus trees only
            finish_query(s, q);
            sl = Slot{};
            s->pending.pop_front();
            s->cv_done.notify_all();
            progress = true;
            continue;
        }
        if (!reserve(s, sl)) break;  // wait for memory to free up
        sl.gen = next_gen(s);
        s->pending.pop_front();
        q.state = 1;
        const bool hold = take_hold(s);
        lk.unlock();
        const int rc = post(s, slot, sl, hold);
        lk.lock();
        if (rc) {
            q.state = rc;
            release(s, sl);
            s->cv_done.notify_all();
            continue;
        }
        q.t_admit = now_ms();
        progress = true;
    }
    // 4. keep a launch running while queries are in flight
    bool inflight = false;
    for (const Slot &sl : s->slots) inflight |= sl.busy && sl.gen != 0;
    if (inflight && !s->running && s->stop) {
        // shutting down: a query that its launch has not finished is not started again
        for (int i = 0; i < s->S; i++) {
            Slot &sl = s->slots[i];
            if (!sl.busy || sl.gen == 0) continue;
            if (((volatile int32_t *)s->h_flags)[i] == sl.gen) continue;  // done: step 1 takes it
            auto it = s->queries.find(sl.ticket);
            if (it != s->queries.end()) it->second.state = XTED_ETIMEOUT;
            release(s, sl);
        }
        s->cv_done.notify_all();
        return true;
    }
    if (inflight && !s->running) {
        cudaStreamSynchronize(s->cs);
        bool ok = cudaMemsetAsync(s->d_ctl, 0, XTED_CTL_INTS * 4, s->ks) == cudaSuccess &&
                  launch_dp(s->K, s->grid, false, s->ks) == cudaSuccess &&
                  cudaEventRecord(s->kev, s->ks) == cudaSuccess;
        if (!ok) {
            cudaGetLastError();
            s->error = XTED_ECUDA;
            fail_inflight(s, XTED_ECUDA);
            s->cv_done.notify_all();
        } else {
            s->running = true;
            s->launches++;
        }
        progress = true;
    }
    return progress;
}

void worker_main(ServeState *s) {
    cudaSetDevice(s->c->opts.device);
    std::unique_lock<std::mutex> lk(s->mu);
    for (;;) {
        const bool progress = step(s, lk);
        bool inflight = false;
        for (const Slot &sl : s->slots) inflight |= sl.busy;
        if (s->stop && !inflight && s->pending.empty() && !s->running) break;
        if (!progress) s->cv_work.wait_for(lk, std::chrono::microseconds(inflight || s->running ? 50 : 2000));
    }
}

void stop_worker(ServeState *s) {
    {
        std::lock_guard<std::mutex> g(s->mu);
        s->stop = true;
        for (uint64_t t : s->pending) {
            auto it = s->queries.find(t);
            if (it != s->queries.end() && it->second.state == 0) it->second.state = XTED_EINVAL;
        }
        s->pending.clear();
        for (Slot &sl : s->slots)
            if (sl.busy && sl.gen == 0) sl = Slot{};  // planned but never posted
        const int32_t one = 1;
        if (s->cs) cudaMemcpyAsync(s->d_ctl + XTED_CTL_STOP, &one, 4, cudaMemcpyHostToDevice, s->cs);
    }
    s->cv_work.notify_all();
    if (s->worker.joinable()) s->worker.join();
}

int load(xted_ctx *c, ServeState *s, const xted_tree *tr, int32_t ntrees) {
    s->c = c;
    s->T = ntrees;
    const int T = ntrees, S = s->S, Qm = s->Qmax;
    int64_t N = 0, R = 0, nonempty = 0;
    for (int t = 0; t < T; t++) {
        TreeView tv{tr[t].n, tr[t].labels, tr[t].child_off, tr[t].child_idx};
        const int rc = validate_tree(tv);
        if (rc) return rc;
        N += tr[t].n;
        s->max_tree = std::max(s->max_tree, tr[t].n);
        R += 3 * (int64_t)tr[t].n + 1;
        nonempty += tr[t].n;
    }
    const int64_t Nall = N + (int64_t)S * Qm;
    if (2 * Nall + 2 * (int64_t)(T + S) >= INT32_MAX / 2 || (int64_t)S * T >= INT32_MAX / 2) return XTED_ENOMEM;
    s->Nc_nonempty = nonempty;
    s->sorted_labels.resize((size_t)T);
    s->dense_seq.resize((size_t)T);
    for (int t = 0; t < T; t++) {
        std::vector<int32_t> &v = s->sorted_labels[(size_t)t];
        v.assign(tr[t].labels, tr[t].labels + tr[t].n);
        std::sort(v.begin(), v.end());
        std::vector<int32_t> &d = s->dense_seq[(size_t)t];
        d.resize((size_t)tr[t].n);
        for (int v2 = 0; v2 < tr[t].n; v2++)
            d[(size_t)v2] = s->dense.emplace(tr[t].labels[v2], (int32_t)s->dense.size()).first->second;
    }
    int ntune = 0;
    const XTuneRow *tune = ctx_tune_table(c, &ntune);
    serve_pools_build(s->pools, tr, T, S, Qm, c->opts.run_rows, c->opts.narrow_width,
                      c->opts.half_width == 0 ? XTED_HALF_DEFAULT : c->opts.half_width,
                      c->opts.tuned ? tune : nullptr, c->opts.tuned ? ntune : 0);
    const ServePools &H = s->pools;
    const size_t n2 = H.node.size();
    int occ = 0;  // (a launch ends once all its warps are idle: no more blocks than are resident)
    if (serve_occupancy(&occ) != 0 || occ < 1) return XTED_ECUDA;
    s->grid = std::min(c->grid, occ * c->sms);
    // device memory
    int64_t dt_cap = std::min<int64_t>(kDtCapMax, (int64_t)S * Qm * std::max<int64_t>(nonempty, 1));
    if (c->opts.mem_limit > 0) dt_cap = std::min<int64_t>(dt_cap, c->opts.mem_limit / 8);  // half of the limit
    dt_cap = std::max<int64_t>(dt_cap, 1);
    s->dt_cap = dt_cap;
    dt_cap += std::max<int64_t>(dt_cap / 32, 1 << 20);  // hand-off words and export maps beside the largest tables
    int rc = XTED_OK;
    rc |= dev_alloc(s, &s->d_node, n2);
    rc |= dev_alloc(s, &s->d_krd, n2);
    rc |= dev_alloc(s, &s->d_cumw, n2);
    rc |= dev_alloc(s, &s->d_runs, n2);
    rc |= dev_alloc(s, &s->d_chunks, n2);
    rc |= dev_alloc(s, &s->d_pairs, (size_t)S * T);
    rc |= dev_alloc(s, &s->d_chunkx, n2);
    rc |= dev_alloc(s, &s->d_items, (size_t)kItemCap);
    rc |= dev_alloc(s, &s->d_lists, XTED_SERVE_SLOTS);
    rc |= dev_alloc(s, &s->d_ctl, XTED_CTL_INTS);
    rc |= dev_alloc(s, &s->d_clears, XTED_SERVE_SLOTS);
    rc |= dev_alloc(s, &s->d_slot, 4 * XTED_SERVE_SLOTS);
    rc |= dev_alloc(s, &s->d_err, 8);
    rc |= dev_alloc(s, &s->d_dt, (size_t)dt_cap);
    // per-warp scratch: the far-row stack's rows outside the shared window
    const int64_t per = (int64_t)H.stack_rows * XTED_SW;
    rc |= dev_alloc(s, &s->d_scratch, (size_t)per * (size_t)s->grid * XTED_FLOW_WARPS);
    if (rc) return XTED_ENOMEM;
    if (cudaHostAlloc((void **)&s->h_results, sizeof(int32_t) * std::max<size_t>((size_t)S * T, 1),
                      cudaHostAllocMapped) != cudaSuccess ||
        cudaHostAlloc((void **)&s->h_flags, sizeof(int32_t) * XTED_SERVE_SLOTS, cudaHostAllocMapped) != cudaSuccess) {
        cudaGetLastError();
        return XTED_ENOMEM;
    }
    std::memset(s->h_flags, 0, sizeof(int32_t) * XTED_SERVE_SLOTS);
    int32_t *d_results = nullptr, *d_flags = nullptr;
    if (cudaHostGetDevicePointer((void **)&d_results, s->h_results, 0) != cudaSuccess ||
        cudaHostGetDevicePointer((void **)&d_flags, s->h_flags, 0) != cudaSuccess ||
        cudaStreamCreateWithFlags(&s->ks, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&s->cs, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&s->kev, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        return XTED_ECUDA;
    }
    const size_t ncorp = 2 * (size_t)N;
    if (upload(s->d_node, H.node.data(), ncorp * sizeof(int2), s->cs) ||
        upload(s->d_krd, H.krd.data(), ncorp * 4, s->cs) || upload(s->d_cumw, H.cumw.data(), ncorp * 4, s->cs) ||
        upload(s->d_runs, H.runs.data(), ncorp * sizeof(XRun), s->cs) ||
        upload(s->d_chunks, H.chunks.data(), ncorp * sizeof(XChunk), s->cs) ||
        cudaMemsetAsync(s->d_lists, 0, XTED_SERVE_SLOTS * 8, s->cs) != cudaSuccess ||
        cudaMemsetAsync(s->d_slot, 0, 4 * XTED_SERVE_SLOTS * 4, s->cs) != cudaSuccess ||
        cudaMemsetAsync(s->d_ctl, 0, XTED_CTL_INTS * 4, s->cs) != cudaSuccess ||
        cudaMemsetAsync(s->d_err, 0, 8 * 4, s->cs) != cudaSuccess || cudaStreamSynchronize(s->cs) != cudaSuccess) {
        cudaGetLastError();
        return XTED_ECUDA;
    }
    s->dt_ext.reset(dt_cap);
    s->i_ext.reset(kItemCap);
    XKernelParams &K = s->K;
    std::memset(&K, 0, sizeof(K));
    K.rowinfo = s->d_node;
    K.krd = s->d_krd;
    K.cumw = s->d_cumw;
    K.runs = s->d_runs;
    K.chunks = s->d_chunks;
    K.pairs = s->d_pairs;
    K.chunkx = s->d_chunkx;
    K.items = s->d_items;
    K.dt = K.buf = s->d_dt;
    K.smap = s->d_dt;
    K.scratch = s->d_scratch;
    K.scratch_per_warp = per;
    K.stack_rows = H.stack_rows;
    K.npairs = S * T;
    K.progress = s->d_ctl + XTED_CTL_PROGRESS;
    K.error = s->d_err;
    K.error_info = s->d_err + 1;
    K.timeout_ns = (uint64_t)(c->opts.wait_timeout_s * 1e9);
    K.trace = nullptr;
    K.serve = 1;
    K.idle_exit_ns = 2000000;  // 2 ms
    K.lists = s->d_lists;
    K.clears = s->d_clears;
    K.ages = s->d_slot + 3 * XTED_SERVE_SLOTS;
    K.ctl = s->d_ctl;
    K.slot_done = s->d_slot;
    K.slot_need = s->d_slot + XTED_SERVE_SLOTS;
    K.slot_gen = s->d_slot + 2 * XTED_SERVE_SLOTS;
    K.results = d_results;
    K.flags = d_flags;
    K.hold_pair = -1;
    // the kernel's row tree is the corpus tree and its column tree the query:
    // TED(query, corpus tree) deletes query nodes and inserts corpus nodes,
    // so the kernel's row deletions cost cost_ins and its column insertions cost_del
    K.c_del = c->opts.cost_ins;
    K.c_ins = c->opts.cost_del;
    K.c_ren = c->opts.cost_ren;
    s->worker = std::thread(worker_main, s);
    return XTED_OK;
}

}  // namespace

std::mutex &serve_mutex(xted_ctx *c) { return c->serve->mu; }

void serve_shutdown(xted_ctx *c) {
    ServeState *s = c->serve;
    if (!s) return;
    stop_worker(s);
    if (s->ks) cudaStreamSynchronize(s->ks);
    if (s->cs) cudaStreamSynchronize(s->cs);
    free_all(s);
    delete s;
    c->serve = nullptr;
}

}  // namespace xted

using namespace xted;

extern "C" {

int xted_corpus_load(xted_ctx *c, const xted_tree *trees, int32_t ntrees) {
    if (!c || ntrees < 1 || !trees) return XTED_EINVAL;
    if (cudaSetDevice(c->opts.device) != cudaSuccess) return XTED_ECUDA;
    serve_shutdown(c);
    ServeState *s = new (std::nothrow) ServeState();
    if (!s) return XTED_ENOMEM;
    const int rc = load(c, s, trees, ntrees);
    if (rc) {
        if (s->worker.joinable()) stop_worker(s);
        free_all(s);
        delete s;
        return rc;
    }
    c->serve = s;
    return XTED_OK;
}

int xted_query_submit(xted_ctx *c, const xted_tree *q, int32_t k, uint64_t *ticket) {
    if (!c || !q || !ticket || k < 1) return XTED_EINVAL;
    ServeState *s = c->serve;
    if (!s) return XTED_EINVAL;
    if (q->n > s->Qmax) return XTED_EINVAL;
    // every pair must fit the row scan's key range: the corpus tree is the
    // row tree (deleted at cost_ins), the query the column tree (cost_del)
    if ((int64_t)c->opts.cost_ins * s->max_tree + (int64_t)c->opts.cost_del * q->n >= XTED_COST_BOUND)
        return XTED_EINVAL;
    const int rc = validate_tree(TreeView{q->n, q->labels, q->child_off, q->child_idx});
    if (rc) return rc;
    Query Q;
    Q.n = q->n;
    Q.k = k;
    Q.lab.assign(q->labels, q->labels + q->n);
    Q.off.assign((size_t)q->n + 1, 0);
    if (q->n > 0) Q.off.assign(q->child_off, q->child_off + q->n + 1);
    if (q->n > 1) Q.idx.assign(q->child_idx, q->child_idx + q->n - 1);
    Q.t_submit = now_ms();
    {
        std::lock_guard<std::mutex> g(s->mu);
        if (s->stop) return XTED_EINVAL;
        if ((int)s->pending.size() >= kMaxPending) return XTED_EAGAIN;
        const uint64_t t = s->next_ticket++;
        s->queries.emplace(t, std::move(Q));
        s->pending.push_back(t);
        *ticket = t;
    }
    s->cv_work.notify_all();
    return XTED_OK;
}

int xted_query_poll_timed(xted_ctx *c, uint64_t ticket, int32_t *ids, int32_t *dists, int32_t *done,
                          double *queue_ms, double *total_ms) {
    if (!c || !done) return XTED_EINVAL;
    ServeState *s = c->serve;
    if (!s) return XTED_EINVAL;
    std::lock_guard<std::mutex> g(s->mu);
    auto it = s->queries.find(ticket);
    if (it == s->queries.end()) return XTED_ENOTFOUND;
    Query &q = it->second;
    *done = 0;
    if (q.state < 0) {
        const int code = q.state;
        s->queries.erase(it);
        return code;
    }
    if (q.state != 2) return XTED_OK;
    if (ids) std::memcpy(ids, q.ids.data(), 4 * q.ids.size());
    if (dists) std::memcpy(dists, q.dists.data(), 4 * q.dists.size());
    if (queue_ms) *queue_ms = q.t_admit > 0 ? q.t_admit - q.t_submit : 0.0;
    if (total_ms) *total_ms = q.t_done - q.t_submit;
    *done = 1;
    s->queries.erase(it);
    return XTED_OK;
}

int xted_query_poll(xted_ctx *c, uint64_t ticket, int32_t *ids, int32_t *dists, int32_t *done) {
    return xted_query_poll_timed(c, ticket, ids, dists, done, nullptr, nullptr);
}

int xted_serve_drain(xted_ctx *c) {
    if (!c) return XTED_EINVAL;
    ServeState *s = c->serve;
    if (!s) return XTED_EINVAL;
    std::unique_lock<std::mutex> lk(s->mu);
    s->cv_work.notify_all();
    // bounded: XTED_ETIMEOUT once no query has finished, failed or been
    // admitted for 4 x wait_timeout_s (at least 30 s)
    const double limit_ms = 1e3 * std::max(30.0, 4.0 * s->c->opts.wait_timeout_s);
    int64_t mark = -1;
    double since = now_ms();
    for (;;) {
        int64_t busy = (int64_t)s->pending.size();
        for (const Slot &sl : s->slots) busy += sl.busy;
        if (busy == 0) break;
        const int64_t m = s->served + s->pairs_served + (int64_t)s->pending.size() + 1000003 * busy;
        if (m != mark) {
            mark = m;
            since = now_ms();
        } else if (now_ms() - since > limit_ms) {
            return XTED_ETIMEOUT;
        }
        s->cv_done.wait_for(lk, std::chrono::milliseconds(5));
    }
    const int e = s->error;
    s->error = 0;
    return e;
}

int xted_serve_stats(xted_ctx *c, int64_t *out, int32_t n) {
    if (!c || !out || n < 0) return XTED_EINVAL;
    ServeState *s = c->serve;
    if (!s) return XTED_EINVAL;
    std::lock_guard<std::mutex> g(s->mu);
    const int64_t v[8] = {s->launches,     s->served,        s->pairs_served, s->cells_served,
                          s->pairs_pruned, s->second_rounds, s->bound_us,     s->plan_us};
    for (int k = 0; k < n && k < 8; k++) out[k] = v[k];
    return XTED_OK;
}

int xted_serve_options(xted_ctx *c, int32_t prune, int32_t first_round) {
    if (!c || first_round < 0) return XTED_EINVAL;
    ServeState *s = c->serve;
    if (!s) return XTED_EINVAL;
    std::lock_guard<std::mutex> g(s->mu);
    if (prune < 0 || prune > 2) return XTED_EINVAL;
    s->prune = prune;
    s->first_round = first_round > 0 ? first_round : 32;
    return XTED_OK;
}

}  // extern "C"
