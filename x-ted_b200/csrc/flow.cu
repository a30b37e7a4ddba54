// flow.cu -- the keyroot-table dynamic program on sm_100a.
//
// One persistent launch; every warp claims items (xted_internal.h: a row run
// against a column chunk, or one column stripe of a wide chunk) from one list
// and runs each to its end.
//
// Savings form. The reference's recurrence (X-TED_CPU/parallel_computing.cpp:17-43,
// its unit costs generalised to del, ins and ren) for keyroot tables (i0, j0):
//     tree cell   D[i][j] = min(D[i+1][j+1] + ren*(l(i) != l(j)), D[i+1][j] + del,
//                               D[i][j+1] + ins),  Dtree[i][j] = D[i][j]
//     forest cell D[i][j] = min(Dtree[i][j] + D[orl(i)+1][orl(j)+1], D[i+1][j] + del,
//                               D[i][j+1] + ins)
// with borders D[i][je] = (imax - i) del and D[imax][j] = (je - j) ins. With
//     S[i][j] = (imax - i) del + (je - j) ins - D[i][j],
// what the mapping saves over deleting and inserting everything, the border
// costs cancel and every add of a cost but one goes away:
//     tree cell   S[i][j] = max(S[i+1][j+1] + del + ins - ren*(l(i) != l(j)), S[i+1][j], S[i][j+1])
//     forest cell S[i][j] = max(Stree[i][j] + S[orl(i)+1][orl(j)+1], S[i+1][j], S[i][j+1])
// with all borders 0: one add-max and two maxima per cell, and row i is the
// suffix maximum of its cells' first two terms. The matrix holds Stree; the
// distance of a pair is m del + n ins - Stree[0][0]. All int32 and exact.
//
// Rows. A warp holds W consecutive columns per lane; the row above stays in
// registers, a row is a chain over the lane's columns and a warp suffix
// maximum. Columns of several segments (tables) side by side carry a key per
// segment that falls to the right by more than any value (XTED_KEY_BIG), so one
// unsegmented suffix maximum serves them all: values right of a segment always
// lose, and a segment's own border is its key. Rows that later rows use as
// S[orl(i)+1][*] go on a stack; its top rows sit in shared memory, rows that
// fall out of that window go to global scratch and come back when the stack
// unwinds to them.
//
// Waiting for data instead of levels. Nothing orders the items but the values
// they need: Stree words and the hand-off words of striped units start at -1
// and are written once, so a reader that finds -1 waits for that word. An
// item needs only items before it in the list, warps claim items in list
// order and run what they claim, so the first unfinished item can always run.
// A table thus starts as soon as its first rows' inputs exist and follows the
// tables it reads by a few rows; with one barrier per keyroot level (the
// form this replaced) a pair of 1,000-node trees took the sum over ~80 levels
// of the longest table of each.
//
// Figures (B200): see the dispatch rules below for the sizes.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/xted.h"
#include "xted_internal.h"

namespace xted {

#define FULLMASK 0xffffffffu

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ int ld_relaxed(const int32_t *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(int32_t *p, int v) {
    asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void set_error(const XKernelParams &P, int code, int a, int b, int c) {
    if (atomicCAS(P.error, 0, code) == 0) {
        P.error_info[0] = a;
        P.error_info[1] = b;
        P.error_info[2] = c;
    }
}

// Both copy `bytes` (0 up to their size) and zero the rest of the destination.
// Copies of table rows go through L2 (.cg) or, four bytes at a time, may
// allocate in L1 (.ca): a stale L1 line can only hold -1 where the value has
// since arrived, and a reader that finds -1 looks again through L2.
__device__ __forceinline__ void cp_async16(unsigned smem, const int32_t *gmem, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(unsigned smem, const int32_t *gmem, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Shared memory by 32-bit addresses: a row's accesses then cost one add each
// at most, where pointers computed in 64 bits took up to three instructions.
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ int lds(unsigned a) {
    int v;
    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ int4 lds4(unsigned a) {
    int4 v;
    asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts(unsigned a, int v) {
    asm volatile("st.shared.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts4(unsigned a, int4 v) {
    asm volatile("st.shared.v4.s32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Inclusive suffix maximum over the warp (a lane whose source is out of range
// gets its own value back).
__device__ __forceinline__ int warp_suffix_max(int v) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) v = max(v, __shfl_down_sync(FULLMASK, v, d));
    return v;
}

// A warp's shared memory: a ring of FLOW_PF table rows in flight and the stack
// window. A stack row holds column c (lane c / W, its k-th column) at 32 k + lane, so reading or writing
// every lane's k-th column touches 32 banks, then a zero word that stands for
// the border, then (W = 16) the far values a stripe takes from others. W = 16 leaves a window of 4 rows (the stack leaves it on 2.5% of
// the mixed batch's rows, against 1.7% for 8 rows), W = 8 keeps 8.
#define FLOW_PF 4
#define FLOW_RING (FLOW_PF * XTED_SW)
#define FLOW_IMPORTS 64  // far values of other stripes kept beside a stack row
template <int W>
struct StackWin {
    static constexpr int ROWS = W == 16 ? 4 : 8;
    static constexpr int PITCH = 32 * W + 4 + (W == 16 ? FLOW_IMPORTS : 0);
};
#define FLOW_STACK 2320  // the larger ROWS * PITCH
static_assert(StackWin<16>::ROWS * StackWin<16>::PITCH <= FLOW_STACK && StackWin<8>::ROWS * StackWin<8>::PITCH <= FLOW_STACK,
              "stack window");
#define FLOW_WARP_INTS (FLOW_RING + FLOW_STACK)
#define FLOW_ZERO 584  // a stack row of zeros, one per block: what tree rows read as far values
static_assert(StackWin<16>::PITCH <= FLOW_ZERO && FLOW_ZERO % 4 == 0, "row of zeros");
#define FLOW_SMEM ((FLOW_ZERO + XTED_FLOW_WARPS * FLOW_WARP_INTS) * 4)
// A row's flags in a run's row sequence, beside those of its node record.
#define ROW_NEXTTREE (1u << 26)  // the next row of the table is on its right path
#define ROW_TREE (1u << 27)      // the row is on its table's right path
#define ROW_FIRST (1u << 28)     // first row of its table (the table's last node)
#define ROW_LAST (1u << 31)      // last row of its table (the keyroot)

// The whole warp waits until every lane that needs its word at p has it (v >=
// 0); false once the launch has failed or nothing has finished anywhere for
// timeout_ns. The loop's exit is a vote and no function is called, so the
// compiler sees the warp leave it together: behind a wait on one lane every
// later shuffle of the row compiled to a check and a slow path (2.3 KB of
// code for the five of a row's suffix maximum, times every use).
__device__ __forceinline__ bool warp_wait(const XKernelParams &P, const int32_t *p, bool need, int &v) {
    uint64_t t0 = global_ns();
    int pg = ld_relaxed(P.progress);
    unsigned ns = 32;
    for (;;) {
        if (need) v = ld_relaxed(p);
        if (!__any_sync(FULLMASK, need && v < 0)) return true;
        bool out = ld_relaxed(P.error) != 0;
        const uint64_t now = global_ns();
        if (now - t0 > P.timeout_ns) {
            const int q = ld_relaxed(P.progress);
            if (q == pg) {
                set_error(P, XTED_ETIMEOUT, 1, 0, 0);
                out = true;
            }
            pg = q;
            t0 = now;
        }
        if (__any_sync(FULLMASK, out)) return false;
        __nanosleep(ns);
        if (ns < 512) ns <<= 1;
    }
}

// One item on one warp. MULTI: the chunk holds several segments (copied word
// by word; at most 32 W columns), else one segment (16-byte copies). W = 16:
// stripe s of K of a segment (K = 1: all of it).
//
// A few columns of a segment need more than the common step: those on its
// right path (on tree rows they take the diagonal and their value goes out),
// those that stripes further left read, and those whose far column lies in
// another stripe. LISTS: there are at most 64 of each, and lane q takes the
// q-th and (q + 32)-th through shared memory; otherwise (LISTS = false, and
// for several segments, where most columns are on a path) every lane tests its
// own W columns. Testing them all on every row cost 100-200 of a row's 400
// instructions, and code: the instruction cache is what the first form of this
// kernel, with six unrolled bodies, ran out of (15.6 of 24.5 cycles per issued
// instruction waited for instructions on a 256-pair mixed batch).
// What a row rarely needs (waiting, the stack leaving its window) is marked
// unlikely. Returns 0, FLOW_FAILED once the launch has failed, or FLOW_LISTS
// (nothing done) if LISTS is set and a list would be longer than 64.
#define FLOW_FAILED 1
#define FLOW_LISTS 2
template <int W, bool MULTI, bool LISTS>
__device__ __forceinline__ int run_item(const XKernelParams &P, const XItem &it, const XPair &pr, const XRun &run,
                                     const XChunk &ch, unsigned zeros, int32_t *ring, int32_t *gstk) {
    constexpr bool STRIPE = W == 16;
    static_assert(!(MULTI && (STRIPE || LISTS)), "a stripe is part of one segment");
    constexpr int SLOT = 32 * W, PF = FLOW_PF;
    constexpr int SC = StackWin<W>::ROWS, PITCH = StackWin<W>::PITCH, ZERO = 32 * W, IMP = ZERO + 4;
    constexpr int NG = W / 4;  // 16-byte pieces a lane copies per row
    const int lane = threadIdx.x & 31;
    const int2 *rows = P.rowinfo + pr.row_base, *nodes = P.rowinfo + pr.col_base;
    int32_t *dt = P.dt + pr.dt_off;
    const int pitch = pr.pitch;
    // what mapping two nodes saves: equal labels, others (a rename dearer than
    // delete + insert saves nothing: the maximum then takes another term)
    const int bm = P.c_del + P.c_ins, bn = max(bm - P.c_ren, 0);
    const int R = run.rows;
    const unsigned ring_a = smem_addr(ring), stk_a = ring_a + 4 * FLOW_RING;  // stack rows are PITCH ints apart
    constexpr unsigned SLOT_B = 4 * SLOT, RING_B = PF * SLOT_B, PITCH_B = 4 * PITCH;
    // single segment: where column c of a row lies in its ring slot (piece p at
    // p ^ ((p >> 3) & (NG - 1)): eight lanes reading their g-th pieces touch
    // eight different bank groups)
    auto swz = [](int c) { return 4 * ((c >> 2) ^ ((c >> 5) & (NG - 1))) + (c & 3); };

    // ---- columns ----
    int key[W], node[W];
    int lab[LISTS ? 1 : W];
    int fb[W];                       // far column: byte offset in a stack row (not LISTS, another stripe's: export index)
    unsigned tcol = 0;               // bit k: column k is on its segment's right path
    unsigned xfar = 0, expm = 0;     // STRIPE: far column in another stripe; exported column
    int ebase = 0;                   // STRIPE: export index of this lane's (LISTS: the stripe's) first exported column
    int sbase = 0, cend = ch.width;  // single: node of local column 0; columns [.., cend) exist
    int lead = 0, K = 1, X = 0, s = 0;
    __syncwarp();
    if (MULTI) {
        // segment of the lane's first column by binary search, then a walk over the keyroots
        int q = ch.k_lo, j = 0, j0 = 0, je = 0;
        const int c0 = lane * W;
        if (c0 < ch.width) {
            const int pos0 = P.cumw[ch.k_lo] + c0;
            int lo = ch.k_lo, hi = ch.k_lo + ch.nseg - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (P.cumw[mid] <= pos0) lo = mid;
                else hi = mid - 1;
            }
            q = lo;
            j0 = P.krd[q];
            je = (nodes[j0].y & XTED_ROW_ORL_MASK) + 1;
            j = j0 + (pos0 - P.cumw[q]);
        }
#pragma unroll
        for (int k = 0; k < W; k++) {
            const int c = c0 + k;
            fb[k] = 4 * ZERO;
            node[k] = key[k] = 0;
            if (!LISTS) lab[k] = 0;
            if (c < ch.width) {
                if (j >= je) {
                    q++;
                    j0 = P.krd[q];
                    je = (nodes[j0].y & XTED_ROW_ORL_MASK) + 1;
                    j = j0;
                }
                const int2 nd = nodes[j];
                const int f = (nd.y & XTED_ROW_ORL_MASK) + 1;  // far column's node
                node[k] = j;
                if (!LISTS) lab[k] = nd.x;
                key[k] = (ch.k_lo + ch.nseg - 1 - q) * XTED_KEY_BIG;
                if (f == je) {
                    tcol |= 1u << k;
                } else {
                    const int fc = c + f - j;
                    fb[k] = 4 * ((fc & (W - 1)) * 32 + fc / W);
                }
                j++;
            }
        }
    } else {
        const int j0 = P.krd[ch.k_lo], je = j0 + ch.width;
        lead = j0 & (XTED_PITCH - 1);
        const int base = j0 - lead;
        const int32_t *map = nullptr;
        if (STRIPE) {
            const XChunkX cx = P.chunkx[it.chunk];
            K = cx.K;
            X = cx.X;
            s = it.stripe;
            map = P.smap + cx.map;
        }
        sbase = base + s * XTED_SW;
        cend = min(je - sbase, 32 * W);
        if (STRIPE && s > 0) lead = 0;
#pragma unroll
        for (int k = 0; k < W; k++) {
            const int c = lane * W + k, j = sbase + c;
            fb[k] = 4 * ZERO;
            key[k] = node[k] = 0;
            if (!LISTS) lab[k] = 0;
            if (c >= lead && c < cend) {
                const int2 nd = nodes[j];
                const int f = (nd.y & XTED_ROW_ORL_MASK) + 1;
                if (!LISTS) lab[k] = nd.x;
                if (f == je) {
                    tcol |= 1u << k;
                } else if (!STRIPE || f - sbase < 32 * W) {
                    const int fc = f - sbase;
                    fb[k] = 4 * ((fc & (W - 1)) * 32 + fc / W);
                } else {
                    xfar |= 1u << k;
                    fb[k] = map[f - j0];
                }
                if (STRIPE && K > 1) {
                    const int e = map[j - j0];  // exports are numbered in column order
                    if (e >= 0) {
                        if (expm == 0) ebase = e;
                        expm |= 1u << k;
                    }
                }
            }
        }
    }
    // LISTS: the q-th such column of the stripe, q = lane and lane + 32
    int tq[2] = {0, 0}, tlab[2] = {0, 0};  // right path: column | its word in a ring slot << 10 | the next column's << 20
    bool tlast = false;                    // one of them is the stripe's last column
    int xq[2] = {0, 0}, iv[2] = {0, 0};    // far column elsewhere: export index; its value for the next row
    int eq[2] = {0, 0};                    // exported: its word in a stack row
    int nt = 0, nx = 0, ne = 0;
    if (LISTS) {
        auto listed = [&](unsigned mask, int &first) {  // this lane's first place in the list; the list's length
            int n = __popc(mask);
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int o = __shfl_up_sync(FULLMASK, n, d);
                if (lane >= d) n += o;
            }
            first = n - __popc(mask);
            return __shfl_sync(FULLMASK, n, 31);
        };
        int tf, xf, ef;
        nt = listed(tcol, tf);
        if (STRIPE) {
            nx = listed(xfar, xf);
            ne = listed(expm, ef);
        }
        if (nt > 64 || nx > 64 || ne > 64) return FLOW_LISTS;
        int32_t *tl = ring, *xl = ring + 64, *el = ring + 128;
#pragma unroll
        for (int k = 0; k < W; k++) {
            const int c = lane * W + k;
            if ((tcol >> k) & 1u) tl[tf++] = c;
            if (STRIPE && ((xfar >> k) & 1u)) {
                xl[xf] = fb[k];
                fb[k] = 4 * (IMP + xf++);
            }
            if (STRIPE && ((expm >> k) & 1u)) el[ef++] = k * 32 + lane;
        }
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int q = lane + 32 * h;
            if (q < nt) {
                const int c = tl[q];
                tlab[h] = nodes[sbase + c].x;
                tq[h] = c | (swz(c) << 10) | ((c + 1 < 32 * W ? swz(c + 1) : 0) << 20);
                tlast |= c + 1 == 32 * W;
            }
            if (STRIPE && q < nx) xq[h] = xl[q];
            if (STRIPE && q < ne) eq[h] = el[q];
        }
        if (STRIPE) ebase = __reduce_min_sync(FULLMASK, (unsigned)(expm ? ebase : 0x7fffffff));
    }
    const bool right = STRIPE && s + 1 < K, left = STRIPE && s > 0;
    const int32_t *Hin = P.buf + it.buf + (int64_t)s * R;          // the right neighbour's first column, per row
    int32_t *Hout = P.buf + it.buf + (int64_t)(s - 1) * R;         // this stripe's, for the left one
    int32_t *E = P.buf + it.buf + (int64_t)(K - 1) * R;            // exported columns, per row
    const bool xwarp = STRIPE && __any_sync(FULLMASK, xfar != 0);
    const bool lead_any = __any_sync(FULLMASK, lead != 0);

    // ---- shared memory ----
    __syncwarp();
    if (lane < SC) sts(stk_a + lane * PITCH_B + 4 * ZERO, 0);
    int cpn[MULTI ? W : 1], csz[MULTI ? W : NG];  // the lane's copies of a row: multi, node of column lane + 32 k; bytes
    if (MULTI) {
        // the lane's copy plan through the ring (nothing is under way there)
#pragma unroll
        for (int k = 0; k < W; k++) ring[lane * W + k] = node[k];
        __syncwarp();
#pragma unroll
        for (int k = 0; k < W; k++) {
            const bool v = lane + 32 * k < ch.width;
            cpn[MULTI ? k : 0] = v ? ring[lane + 32 * k] : 0;
            csz[MULTI ? k : 0] = v ? 4 : 0;  // past the chunk: zeroed
        }
    } else {
#pragma unroll
        for (int g = 0; g < NG; g++) csz[MULTI ? 0 : g] = 4 * max(0, min(4, cend - 4 * (lane + 32 * g)));
    }
    unsigned coff[NG];  // where the lane's own columns lie in a slot
#pragma unroll
    for (int g = 0; g < NG; g++) coff[g] = MULTI ? 4 * (lane * W + 4 * g) : 4 * swz(lane * W + 4 * g);
    __syncwarp();

    // ---- row sequence: the run's tables one after another, each from its last row up ----
    // Lane l holds row tb + l of the sequence (its node, its record with the
    // table flags, its label) and, loaded 32 rows ahead, row tb + 32 + l.
    int bi = 0, by = 0, bl = 0, ni = 0, ny = 0, nl = 0;
    auto load_rows = [&](int f, int &i, int &y, int &l) {
        f = min(f, R - 1);
        int q = run.kr_lo;
        int off = f;
        if (run.kr_hi - run.kr_lo > 1) {  // the table of row f: the last keyroot whose rows start at or before it
            const int p0 = P.cumw[run.kr_lo];
            int hi = run.kr_hi - 1;
            while (q < hi) {
                const int mid = (q + hi + 1) >> 1;
                if (P.cumw[mid] - p0 <= f) q = mid;
                else hi = mid - 1;
            }
            off = f - (P.cumw[q] - p0);
        }
        const int i0 = P.krd[q], e0 = rows[i0].y & XTED_ROW_ORL_MASK;
        i = e0 - off;
        const int2 r = rows[i];
        l = r.x;
        unsigned fl = off == 0 ? ROW_FIRST : 0u;
        if ((r.y & XTED_ROW_ORL_MASK) == e0) fl |= ROW_TREE;
        if (i == i0) fl |= ROW_LAST;
        else if ((rows[i - 1].y & XTED_ROW_ORL_MASK) == e0) fl |= ROW_NEXTTREE;
        y = (int)((unsigned)r.y | fl);
    };
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
        bi = ni, by = ny, bl = nl;
        load_rows(32 * h + lane, ni, ny, nl);
    }
    // row PF - 1 places on, by lane as above
    int ai = __shfl_sync(FULLMASK, bi, (lane + PF - 1) & 31);
    {
        const int o = __shfl_sync(FULLMASK, ni, (lane + PF - 1) & 31);
        if (lane + PF - 1 >= 32) ai = o;
    }
    const int32_t *src0 = MULTI ? dt : dt + sbase + 4 * lane;
    const unsigned dst0 = ring_a + (MULTI ? 4 * lane : 16 * (lane ^ ((lane >> 3) & (NG - 1))));
    auto copy_row = [&](unsigned so, int r) {  // row r into the slot at byte so of the ring
        const int32_t *src = src0 + (unsigned long long)(unsigned)r * (unsigned)pitch;
        const unsigned d = dst0 + so;
        if (MULTI) {
#pragma unroll
            for (int k = 0; k < W; k++) cp_async4(d + 128 * k, src + (unsigned)cpn[MULTI ? k : 0], csz[MULTI ? k : 0]);
        } else {
#pragma unroll
            for (int g = 0; g < NG; g++) cp_async16(d + 512 * g, src + 128 * g, csz[MULTI ? 0 : g]);
        }
    };
#pragma unroll 1
    for (int q = 0; q < PF - 1; q++) {
        copy_row(q * SLOT_B, __shfl_sync(FULLMASK, bi, q));  // (past the run's end: its last row again)
        cp_async_commit();
    }

    int prev[W];
#pragma unroll
    for (int k = 0; k < W; k++) prev[k] = key[k];
    int sp = 0, lo = 0;      // stack depth; lowest position held in the shared window
    int c0 = 0, c1 = 0, cprev = 0;  // stripes: the right neighbour's first column in this row, the next, the one above
    if (right) {
        c0 = ld_relaxed(Hin);
        c1 = R > 1 ? ld_relaxed(Hin + 1) : 0;
    }
    int pfw[STRIPE && !LISTS ? W : 1];  // far values of other stripes for this row (-1: not there yet)
    if (STRIPE && !LISTS) {
#pragma unroll
        for (int k = 0; k < W; k++) pfw[k] = 0;
    }

#pragma unroll 1
    for (int t = 0; t < R; t++) {
        const unsigned so = (unsigned)(t & (PF - 1)) * SLOT_B, slot = ring_a + so;
        if (!LISTS) {
            // the masks' bits are tested where they are used: kept apart in
            // registers over the whole loop they would spill it
            asm volatile("" : "+r"(tcol), "+r"(xfar), "+r"(expm));
        }
        cp_async_wait<PF - 2>();  // row t has landed
        __syncwarp();             // ... every lane's copies; row t - 1's readers are done
        const int tl = t & 31;
        const int i = __shfl_sync(FULLMASK, bi, tl);
        const unsigned y = (unsigned)__shfl_sync(FULLMASK, by, tl);
        const bool trow = (y & ROW_TREE) != 0;
        int rl = 0;
        if (trow) rl = __shfl_sync(FULLMASK, bl, tl);
        if (LISTS && trow) {  // tree rows: the path columns' words become what the diagonal gives
            const unsigned above = ring_a + ((so + RING_B - SLOT_B) & (RING_B - 1));  // the row above, if the table's
#pragma unroll
            for (int h = 0; h < 2; h++)
                if (lane + 32 * h < nt) {
                    int x = lds(above + (((unsigned)tq[h] >> 18) & 0xffcu));
                    if (y & ROW_FIRST) x = 0;
                    if (tlast && (tq[h] & 1023) + 1 == 32 * W) x = cprev;
                    sts(slot + (((unsigned)tq[h] >> 8) & 0xffcu), x + (rl == tlab[h] ? bm : bn));
                }
            __syncwarp();  // (and every lane has read the row above, whose slot is copied into next)
        }
        copy_row((so + RING_B - SLOT_B) & (RING_B - 1), __shfl_sync(FULLMASK, ai, tl));  // into row t - 1's slot
        cp_async_commit();
        int c2 = 0;
        if (right && t + 2 < R) c2 = ld_relaxed(Hin + t + 2);
        int a[W];
        for (;;) {
#pragma unroll
            for (int g = 0; g < NG; g++) {
                const int4 v = lds4(slot + coff[g]);
                a[4 * g] = v.x, a[4 * g + 1] = v.y, a[4 * g + 2] = v.z, a[4 * g + 3] = v.w;
            }
            if (!MULTI && lead_any) {  // words left of the segment
#pragma unroll
                for (int k = 0; k < 3; k++)
                    if (lane == 0 && k < lead) a[k] = 0;
            }
            if (!LISTS && trow) {
                int dn = __shfl_down_sync(FULLMASK, prev[0], 1);
                if (lane == 31) dn = cprev;
#pragma unroll
                for (int k = 0; k < W; k++) {
                    int x = k == W - 1 ? dn : prev[k + 1];
                    if (MULTI) x = max(x, key[k]) - key[k];  // past a segment's end: its border
                    x += rl == lab[k] ? bm : bn;
                    if ((tcol >> k) & 1u) a[k] = x;
                }
            }
            // a word that is still -1: another item has yet to write it
            int m = a[0];
#pragma unroll
            for (int k = 1; k < W; k++) m |= a[k];
            const unsigned who = __ballot_sync(FULLMASK, m < 0);
            if (__builtin_expect(who == 0, 1)) break;
            // the leftmost missing word is the last to come: wait for it, then
            // fetch this row and those already under way again
            int kk = 0, v = 0;
#pragma unroll
            for (int k = W - 1; k >= 0; k--)
                if (a[k] < 0) kk = MULTI ? node[k] : sbase + lane * W + k;
            kk = __shfl_sync(FULLMASK, kk, __ffs(who) - 1);
            if (!warp_wait(P, dt + (int64_t)i * pitch + kk, true, v)) return FLOW_FAILED;
            int td[2] = {0, 0};  // a tree row's path words do not change
            if (LISTS && trow) {
#pragma unroll
                for (int h = 0; h < 2; h++)
                    if (lane + 32 * h < nt) td[h] = lds(slot + (((unsigned)tq[h] >> 8) & 0xffcu));
            }
            cp_async_wait<0>();
            __syncwarp();
#pragma unroll 1
            for (int q = 0; q < PF; q++) {
                const int r = __shfl_sync(FULLMASK, tl + q < 32 ? bi : ni, (tl + q) & 31);
                const unsigned sq = (so + q * SLOT_B) & (RING_B - 1);
                if (MULTI) {  // through L2, past whatever an L1 line holds
                    const int32_t *src = dt + (int64_t)r * pitch;
#pragma unroll
                    for (int k = 0; k < W; k++)
                        if (csz[MULTI ? k : 0] > 0) sts(dst0 + sq + 128 * k, ld_relaxed(src + cpn[MULTI ? k : 0]));
                } else {
                    copy_row(sq, r);
                }
            }
            cp_async_commit();
            cp_async_wait<0>();
            __syncwarp();
            if (LISTS && trow) {
#pragma unroll
                for (int h = 0; h < 2; h++)
                    if (lane + 32 * h < nt) sts(slot + (((unsigned)tq[h] >> 8) & 0xffcu), td[h]);
                __syncwarp();
            }
        }
        if (right) {
            // (lanes reading one word at the same time need not see the same value)
            if (__builtin_expect(__any_sync(FULLMASK, c0 < 0), 0)) {
                if (!warp_wait(P, Hin + t, true, c0)) return FLOW_FAILED;
                if (t + 1 < R) c1 = ld_relaxed(Hin + t + 1);
                if (t + 2 < R) c2 = ld_relaxed(Hin + t + 2);
            }
        }
        // ---- the row's cells, before the suffix maximum ----
        unsigned top = zeros;  // a tree row's far row is the table's border
        if (!trow) {
            top = stk_a + ((sp - 1) & (SC - 1)) * PITCH_B;
            if (__builtin_expect(sp - 1 < lo, 0)) {  // the top of the stack left the window: bring it back
                lo = sp - 1;
                const int32_t *g = gstk + (int64_t)lo * ZERO + lane;
#pragma unroll 1
                for (int k = 0; k < W; k++) sts(top + 4 * lane + 128 * k, g[32 * k]);
                __syncwarp();
            }
            if (xwarp) {  // some far columns lie in stripes to the right: the far row's exports
                const int32_t *erow = E + (int64_t)(t - ((int)(y & XTED_ROW_ORL_MASK) + 1 - i)) * X;
                if (LISTS) {
                    if (__builtin_expect(__any_sync(FULLMASK, (iv[0] | iv[1]) < 0), 0)) {
                        if (!warp_wait(P, erow + xq[0], iv[0] < 0, iv[0]) || !warp_wait(P, erow + xq[1], iv[1] < 0, iv[1]))
                            return FLOW_FAILED;
                    }
                    sts(top + 4 * (IMP + lane), iv[0]);
                    if (nx > 32) sts(top + 4 * (IMP + 32 + lane), iv[1]);
                    __syncwarp();
                } else if (STRIPE) {
#pragma unroll
                    for (int k = 0; k < W; k++) {
                        const bool lack = ((xfar >> k) & 1u) && pfw[k] < 0;
                        if (__any_sync(FULLMASK, lack) && !warp_wait(P, erow + (lack ? fb[k] : 0), lack, pfw[k]))
                            return FLOW_FAILED;
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < W; k++) {
            int far;
            if (STRIPE && !LISTS) {
                const bool x = (xfar >> k) & 1u;
                far = lds(top + (x ? 4 * ZERO : fb[k]));
                if (x && !trow) far = pfw[k];
            } else {
                far = lds(top + fb[k]);
            }
            if (MULTI) far = max(far, key[k]);  // a path column's far value is its segment's border
            a[k] = __viaddmax_s32(a[k], far, prev[k]);
        }
        // ---- suffix maximum: the lane's columns (two chains when there are 16), then the lanes ----
        constexpr int H = W > 8 ? W / 2 : W;
#pragma unroll
        for (int k = W - 2; k >= 0; k--)
            if (k != H - 1) a[k] = max(a[k], a[k + 1]);
        int mine = W > 8 ? max(a[0], a[H]) : a[0];
        if (STRIPE && lane == 31) mine = max(mine, c0);
        const int incl = warp_suffix_max(mine);
        int carry = __shfl_down_sync(FULLMASK, incl, 1);
        if (lane == 31) carry = STRIPE ? c0 : 0;
        const int carry_lo = W > 8 ? max(carry, a[H]) : carry;
#pragma unroll
        for (int k = 0; k < W; k++) prev[k] = max(a[k], k < H ? carry_lo : carry);
        // ---- what others read ----
        if (left && lane == 0) st_relaxed(Hout + t, prev[0]);
        if (LISTS && (y & (ROW_TREE | ROW_NEXTTREE))) {
            // the row goes into its own ring slot (free until the next row's
            // copies): the next row's diagonal, and this row's path columns
#pragma unroll
            for (int g = 0; g < NG; g++)
                sts4(slot + coff[g], make_int4(prev[4 * g], prev[4 * g + 1], prev[4 * g + 2], prev[4 * g + 3]));
            if (trow) {
                __syncwarp();
                int32_t *o = dt + (int64_t)i * pitch + sbase;
#pragma unroll
                for (int h = 0; h < 2; h++)
                    if (h == 0 || nt > 32)
                        if (lane + 32 * h < nt) st_relaxed(o + (tq[h] & 1023), lds(slot + (((unsigned)tq[h] >> 8) & 0xffcu)));
            }
        }
        if (!LISTS && trow) {
            int32_t *o = dt + (int64_t)i * pitch + (MULTI ? 0 : sbase + lane * W);
#pragma unroll
            for (int k = 0; k < W; k++)
                if ((tcol >> k) & 1u) st_relaxed(o + (MULTI ? node[k] : k), prev[k] - key[k]);
        }
        if (y & ROW_LAST) {  // the table is done
#pragma unroll
            for (int k = 0; k < W; k++) prev[k] = key[k];
            sp = lo = 0;
            cprev = 0;
        } else {
            cprev = c0;
            if (y & XTED_ROW_ISKR) sp--;
            if (y & XTED_ROW_PREVLEAF) {
                if (__builtin_expect((unsigned)(sp - lo) >= (unsigned)SC, 0)) {
                    if (sp < lo) {
                        lo = sp - 1;
                    } else if (lo < P.stack_rows) {  // the window is full: its lowest row moves out
                        int32_t *g = gstk + (int64_t)lo * ZERO + lane;
                        const unsigned d = stk_a + (lo & (SC - 1)) * PITCH_B + 4 * lane;
#pragma unroll 1
                        for (int k = 0; k < W; k++) g[32 * k] = lds(d + 128 * k);
                    } else if (lane == 0) {
                        set_error(P, XTED_ENOMEM, 2, lo, P.stack_rows);
                    }
                    lo++;
                }
                // (every lane's reads of the slot's old row came before the shuffles above)
                const unsigned d = stk_a + (sp & (SC - 1)) * PITCH_B;
#pragma unroll
                for (int k = 0; k < W; k++) sts(d + 4 * lane + 128 * k, prev[k]);
                sp++;
                if (LISTS && ne > 0) {
                    __syncwarp();
                    int32_t *e = E + (int64_t)t * X + ebase + lane;
                    if (lane < ne) st_relaxed(e, lds(d + 4 * eq[0]));
                    if (lane + 32 < ne) st_relaxed(e + 32, lds(d + 4 * eq[1]));
                }
                if (STRIPE && !LISTS && expm) {
                    int32_t *e = E + (int64_t)t * X + ebase;
#pragma unroll
                    for (int k = 0; k < W; k++)
                        if ((expm >> k) & 1u) st_relaxed(e + __popc(expm & ((1u << k) - 1u)), prev[k]);
                }
            }
            if (xwarp && !(y & ROW_NEXTTREE)) {  // the next row's far values in other stripes
                const int nro = __shfl_sync(FULLMASK, tl + 1 < 32 ? by : ny, (tl + 1) & 31) & XTED_ROW_ORL_MASK;
                const int32_t *e = E + (int64_t)(t + 1 - (nro + 1 - (i - 1))) * X;
                if (LISTS) {
                    if (lane < nx) iv[0] = ld_relaxed(e + xq[0]);
                    if (lane + 32 < nx) iv[1] = ld_relaxed(e + xq[1]);
                } else if (STRIPE) {
#pragma unroll
                    for (int k = 0; k < W; k++)
                        if ((xfar >> k) & 1u) pfw[k] = ld_relaxed(e + fb[k]);
                }
            }
        }
        c0 = c1;
        c1 = c2;
        if (tl == 31) {
            bi = ni, by = ny, bl = nl;
            load_rows(t + 33 + lane, ni, ny, nl);
            ai = __shfl_sync(FULLMASK, bi, (lane + PF - 1) & 31);
            const int o = __shfl_sync(FULLMASK, ni, (lane + PF - 1) & 31);
            if (lane + PF - 1 >= 32) ai = o;
        }
    }
    cp_async_wait<0>();
    __syncwarp();
    return 0;
}

// Trace record of an item (XTED_TRACE): claim, start and end time, and
// stripe(8) | warp's sm(8) | columns(16) | rows(32).
__device__ void trace_item(const XKernelParams &P, int g, uint64_t claim, uint64_t start, int stripe, int width,
                           int rows) {
    unsigned sm;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    P.trace[4 * (int64_t)g] = claim;
    P.trace[4 * (int64_t)g + 1] = start;
    P.trace[4 * (int64_t)g + 2] = global_ns();
    P.trace[4 * (int64_t)g + 3] = (unsigned long long)(stripe & 255) | ((unsigned long long)(sm & 255) << 8) |
                                  ((unsigned long long)(width & 0xffff) << 16) | ((unsigned long long)(unsigned)rows << 32);
}

// The next item of a serving session (a whole warp): the lists of the queries
// in flight, the oldest query's first. -1: leave the launch. Warps leave once
// every one of them has been idle for a while (then the launch is closed and
// the host starts another when work arrives); an item claimed meanwhile
// runs to its end, the rest of its list waits for the next launch.
__device__ __noinline__ int claim_served(const XKernelParams &P, int lane, int *slot) {
    const int total = (int)(gridDim.x * (blockDim.x >> 5));
    bool idle = false;
    uint64_t t0 = 0;
    unsigned ns = 32;
    for (;;) {
        int stop = 0;
        if (lane == 0) stop = ld_relaxed(P.error) != 0 || ld_relaxed(P.ctl + XTED_CTL_CLOSED) != 0;
        stop = __shfl_sync(FULLMASK, stop, 0);
        unsigned age = 0xffffffffu;
        if (!stop && lane < XTED_SERVE_SLOTS) {
            const unsigned long long w = *(volatile unsigned long long *)&P.lists[lane];
            if ((unsigned)w < (unsigned)(w >> 32)) age = (unsigned)ld_relaxed(P.ages + lane);
        }
        const unsigned oldest = __reduce_min_sync(FULLMASK, age);
        if (oldest != 0xffffffffu) {
            const int q = __ffs(__ballot_sync(FULLMASK, age == oldest)) - 1;
            int g = -1;
            if (lane == 0) {
                const unsigned long long w = atomicAdd(&P.lists[q], 1ull);
                if ((unsigned)w < (unsigned)(w >> 32)) g = (int)(unsigned)w;
                if (g >= 0 && idle) atomicSub(&P.ctl[XTED_CTL_IDLE], 1);
            }
            g = __shfl_sync(FULLMASK, g, 0);
            if (g >= 0) {
                __threadfence();  // acquire: the query's plan and its cleared tables are visible from here on
                *slot = q;
                return g;
            }
            continue;
        }
        if (lane == 0 && !stop) {
            if (!idle) atomicAdd(&P.ctl[XTED_CTL_IDLE], 1);
            const uint64_t now = global_ns();
            if (t0 == 0) t0 = now;
            if (ld_relaxed(P.ctl + XTED_CTL_STOP) != 0) stop = 1;
            else if (now - t0 > P.idle_exit_ns && ld_relaxed(P.ctl + XTED_CTL_IDLE) >= total) stop = 1;
            if (stop) atomicExch(&P.ctl[XTED_CTL_CLOSED], 1);
        }
        idle = true;
        if (__shfl_sync(FULLMASK, stop, 0)) return -1;
        __nanosleep(ns);
        __syncwarp();
        if (ns < 1024) ns <<= 1;
    }
}

// An item of a serving query is done: the root table's item leaves the
// pair's distance in host memory, the last item of the round raises the
// slot's flag to the round's generation.
__device__ void finish_served(const XKernelParams &P, const XPair &pr, const XItem &it, bool root, int slot) {
    if (root) {
        const int d = pr.m * P.c_del + pr.n * P.c_ins - ld_relaxed(P.dt + pr.dt_off);
        ((volatile int32_t *)P.results)[it.pair] = d;
    }
    __threadfence_system();  // this item's results and table writes, before it is counted
    const int done = atomicAdd(&P.slot_done[slot], 1) + 1;
    if (done == __ldcg(&P.slot_need[slot])) {
        P.slot_done[slot] = 0;
        __threadfence_system();
        ((volatile int32_t *)P.flags)[slot] = __ldcg(&P.slot_gen[slot]);
    }
}

// Three blocks of four warps per SM: 73 KB of shared memory and up to 168
// registers a thread each (16 columns a lane hold the row above, far indices
// and, in a stripe, the far values of other stripes in registers).
__global__ void __launch_bounds__(32 * XTED_FLOW_WARPS, 3) xted_flow_kernel(const __grid_constant__ XKernelParams P) {
    extern __shared__ __align__(16) int32_t s_dyn[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t *ring = s_dyn + FLOW_ZERO + warp * FLOW_WARP_INTS;
    int32_t *gstk = P.scratch + (int64_t)(blockIdx.x * XTED_FLOW_WARPS + warp) * P.scratch_per_warp;
    for (int x = lane; x < FLOW_WARP_INTS; x += 32) ring[x] = 0;
    for (int x = threadIdx.x; x < FLOW_ZERO; x += blockDim.x) s_dyn[x] = 0;
    __syncthreads();
    for (;;) {
        int g = -1, slot = 0;
        uint64_t t_claim = P.trace ? global_ns() : 0;
        if (P.serve) {
            g = claim_served(P, lane, &slot);
        } else {
            if (lane == 0 && ld_relaxed(P.error) == 0) {
                g = atomicAdd(P.next, 1);
                if (g >= P.nitems) g = -1;
            }
            g = __shfl_sync(FULLMASK, g, 0);
        }
        if (g < 0) break;
        const uint64_t t_start = P.trace ? global_ns() : 0;
        const XItem it = P.items[g];
        const XPair pr = P.pairs[it.pair];
        const XRun run = P.runs[it.run];
        const XChunk ch = P.chunks[it.chunk];
        int rc = 0;
        if (it.pair == P.hold_pair && run.depth + ch.depth == 0) {
            // test hook: nothing that reads this table's values becomes ready
        } else if (ch.nseg > 1) {
            rc = run_item<8, true, false>(P, it, pr, run, ch, smem_addr(s_dyn), ring, gstk);
        } else if ((P.krd[ch.k_lo] & (XTED_PITCH - 1)) + ch.width <= 256) {
            rc = run_item<8, false, true>(P, it, pr, run, ch, smem_addr(s_dyn), ring, gstk);
            if (rc == FLOW_LISTS) rc = run_item<8, false, false>(P, it, pr, run, ch, smem_addr(s_dyn), ring, gstk);
        } else {
            rc = run_item<16, false, true>(P, it, pr, run, ch, smem_addr(s_dyn), ring, gstk);
            if (rc == FLOW_LISTS) rc = run_item<16, false, false>(P, it, pr, run, ch, smem_addr(s_dyn), ring, gstk);
        }
        if (rc) break;
        if (lane == 0) {
            // run and chunk of the two roots: the pair's last table (its leftmost stripe ends last)
            if (P.serve) {
                const bool root = it.stripe == 0 && run.rows == pr.m && ch.width == pr.n && run.kr_hi - run.kr_lo == 1 &&
                                  ch.nseg == 1;
                finish_served(P, pr, it, root, slot);
            }
            atomicAdd(P.progress, 1);
            if (P.trace) trace_item(P, g, t_claim, t_start, it.stripe, ch.width, run.rows);
        }
        __syncwarp();
    }
    cp_async_wait<0>();
}

// Result of pair p: m del + n ins - Stree[0][0] (X-TED_CPU/TED.cpp:188), or for
// a pair with an empty tree the cost of inserting (m = 0) or deleting (n = 0)
// the other one (TED.cpp:181-186, with unit costs there). A pair whose root
// value never came (only after a failed or held launch) reports a timeout.
__global__ void xted_gather_kernel(const XPair *pairs, const int32_t *trivial, const int32_t *dt, int npairs,
                                   int32_t *out, int c_del, int c_ins, int32_t *error) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npairs) return;
    const XPair pr = pairs[p];
    if (trivial[p] >= 0) {
        out[p] = pr.m == 0 ? pr.n * c_ins : pr.m * c_del;
        return;
    }
    const int v = __ldcg(dt + pr.dt_off);
    if (v < 0) atomicCAS(error, 0, XTED_ETIMEOUT);
    out[p] = pr.m * c_del + pr.n * c_ins - v;
}

// ---- host-side launch helpers ----
int dp_occupancy(int *blocks_per_sm) {
    cudaError_t e = cudaFuncSetAttribute(xted_flow_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FLOW_SMEM);
    if (e != cudaSuccess) return (int)e;
    return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, xted_flow_kernel, 32 * XTED_FLOW_WARPS,
                                                              FLOW_SMEM);
}

// Cooperative launch (every warp resident at once: a waiting warp never keeps
// the one it waits for off the GPU), expressed as a launch attribute so that
// the same call also records into a CUDA graph.
cudaError_t launch_dp(const XKernelParams &P, int grid, cudaStream_t s) {
    XKernelParams p = P;
    void *args[] = {&p};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(32 * XTED_FLOW_WARPS);
    cfg.dynamicSmemBytes = FLOW_SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, (const void *)xted_flow_kernel, args);
}

cudaError_t launch_gather(const XPair *pairs, const int32_t *trivial, const int32_t *dt, int npairs, int32_t *out,
                          int c_del, int c_ins, int32_t *error, cudaStream_t s) {
    if (npairs <= 0) return cudaSuccess;
    xted_gather_kernel<<<(npairs + 255) / 256, 256, 0, s>>>(pairs, trivial, dt, npairs, out, c_del, c_ins, error);
    return cudaGetLastError();
}

}  // namespace xted
