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
__device__ __forceinline__ void st_relaxed4(int32_t *p, int4 v) {  // (16-byte aligned; each word a store of its own)
    asm volatile("st.relaxed.gpu.global.v4.s32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void set_error(const XKernelParams &P, int code, int a, int b, int c) {
    if (atomicCAS(P.error, 0, code) == 0) {
        P.error_info[0] = a;
        P.error_info[1] = b;
        P.error_info[2] = c;
    }
}

// Copies of table rows go through L2 (.cg) or, four bytes at a time, may
// allocate in L1 (.ca): a stale L1 line can only hold -1 where the value has
// since arrived, and a reader that finds -1 looks again through L2. Whole
// pieces only: with a size operand (to zero what lies past a segment) a row's
// copies cost some 50 more instructions.
__device__ __forceinline__ void cp_async16(unsigned smem, const int32_t *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(unsigned smem, const int32_t *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem), "l"(gmem) : "memory");
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

// A warp's shared memory: a ring of FLOW_PF table rows in flight, the stack
// window, and lists of the chunk's special columns. A stack row holds column c
// (lane c / W, its k-th column) at 32 k + lane, so reading or writing every
// lane's k-th column touches 32 banks, then a zero word that stands for the
// border, then the far values a stripe takes from other stripes. The stack
// leaves a window of 4 rows on 2.5% of the mixed batch's rows, one of 8 on 1.7%.
#define FLOW_W 8                   // columns per lane
#define FLOW_PF 4
#define FLOW_IMPORTS 48            // far values of other stripes kept beside a stack row
#define FLOW_STACK_ROWS 4
#define FLOW_ZERO (32 * FLOW_W)    // place of the zero word in a stack row
#define FLOW_PITCH (FLOW_ZERO + 4 + FLOW_IMPORTS)
#define FLOW_RING (FLOW_PF * XTED_SW)
#define FLOW_STACK (FLOW_STACK_ROWS * FLOW_PITCH)
// path columns (column | segment << 8 | node << 16), their labels, exported columns (8 bits each)
#define FLOW_LISTS (XTED_SW + XTED_SW + XTED_SW / 4)
#define FLOW_WARP_INTS (FLOW_RING + FLOW_STACK + FLOW_LISTS)
#define FLOW_SMEM (XTED_FLOW_WARPS * FLOW_WARP_INTS * 4)
#define FLOW_SERVE_SMEM (FLOW_SMEM + XTED_FLOW_WARPS * 4)  // and each warp's generation
static_assert(XTED_SW == 32 * FLOW_W && XTED_MAX_NODES < 65536 && FLOW_PITCH % 4 == 0, "list entries and row places");
// A row's flags in a run's row sequence, beside orl (20 bits) and the flags of
// its node record (bits 29, 30). The ITEM_ flags are the same for every row of
// an item: what the row loop asks of the item. They come with the row, through
// the same shuffle, because the compiler would make a copy of the loop for
// every answer it can tell to be constant.
#define ITEM_MULTI (1u << 20)    // a chunk of several segments
#define ITEM_RIGHT (1u << 21)    // a stripe has a right neighbour
#define ITEM_LEFT (1u << 22)     // ... a left one
#define ITEM_IMPORTS (1u << 23)  // it takes far values from other stripes
#define ITEM_EXPORTS (1u << 24)  // it has columns that other stripes take
#define ITEM_EDGE (1u << 25)     // its first or last 16-byte piece holds words of other segments
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
    uint64_t t0 = 0;
    int pg = 0;
#pragma unroll 1
    for (unsigned n = 1;; n++) {
        if (need) v = ld_relaxed(p);
        if (!__any_sync(FULLMASK, need && v < 0)) return true;
        __nanosleep(n < 8 ? 40 * n : 320);
        if ((n & 31) == 0) {  // every few microseconds: has the launch failed, or stopped?
            bool out = ld_relaxed(P.error) != 0;
            const uint64_t now = global_ns();
            if (t0 == 0 || now - t0 > P.timeout_ns) {
                const int q = ld_relaxed(P.progress);
                if (t0 != 0 && q == pg) {
                    set_error(P, XTED_ETIMEOUT, 1, 0, 0);
                    out = true;
                }
                pg = q;
                t0 = now;
            }
            if (__any_sync(FULLMASK, out)) return false;
        }
    }
}

// One item on one warp: a chunk of several segments (multi, copied word by
// word), a segment one warp holds, or stripe s of K of a wider one (both
// copied in 16-byte pieces).
//
// There is one row loop for all of them, of 8 columns a lane. What bounds it
// is the instruction cache and the latency of a row: with a loop per kind of
// chunk and width (six, unrolled) 15.6 of 24.5 cycles per issued instruction
// went on waiting for instructions, with three (8 columns, 8 of several
// segments, 16 a lane) 3.6 of 9.6. So the few columns that need more than the
// common step are listed and taken by whole warps, not tested on every lane:
// those on their segment's right path (on tree rows they take the diagonal
// and their value goes out), those that stripes further left read, and those
// whose far column lies in another stripe. What a row rarely needs (waiting,
// the stack leaving its window) is marked unlikely.
//
// RARE is a second copy of the loop, for items that the lists do not serve:
// - A stripe that takes more far values from other stripes than have a place
//   beside the usual four stack rows keeps two rows, with a place for all, filled
//   when a row first needs them. 200 pairs of zigzags of 500 nodes, whose stripes
//   take up to 90 values: 1,207 ms with those past 48 loaded column by column on
//   every row, 822 ms so.
// - Many path columns and many tree rows (paths, combs, runs and chunks of single
//   nodes): path columns take the diagonal from the row above in registers, eight
//   a lane, where the lists take two passes of up to eight steps through shared
//   memory; where every column is on its path a tree row reads nothing at all. Two
//   paths of 8,000 nodes: 17.3 -> 5.9 ms, 1,024 mixed pairs 13.1 -> 12.6.
// Returns 0, FLOW_FAILED once the launch has failed, or FLOW_RARE (nothing
// done) if RARE is needed.
#define FLOW_FAILED 1
#define FLOW_RARE 2
// Path columns from which lists lose, on items of 64 rows and more of which half or more of the first 64 are tree rows.
// At 16 / 32 / 64 / 128 columns: 4,500 pairs of 20-250 nodes 12.13 / 11.95 / 11.86 / 11.84 ms, 1,024 mixed ones 12.69 /
// 12.60 / 12.59 / 12.63, 200 random ones of 500 2.14 / 2.10 / 2.06 / 2.05, a star of 600 0.70 / 0.71 / 0.70 / 0.72. From
// 32 / 64 / 128 / 256 rows: 4,500 pairs 11.97 / 11.86 / 11.84 / 11.85, 300 mixed 4.98 / 4.97 / 5.07 / 5.25, a pair of
// paths of 100 nodes 0.123 / 0.123 / 0.174 / 0.173. (The setup before the choice is made is done twice.)
#define FLOW_DENSE_COLS 64
#define FLOW_DENSE_ROWS 64
template <bool RARE>
__device__ __forceinline__ int run_item(const XKernelParams &P, const XItem &it, const XPair &pr, const XRun &run,
                                         const XChunk &ch, int32_t *ring, int32_t *gstk) {
    constexpr int W = FLOW_W, PF = FLOW_PF, ZERO = FLOW_ZERO, IMP = ZERO + 4;
    // RARE: a stack window of two rows, with a place for every column's far value, and the places' export indices
    constexpr int SC = RARE ? 2 : FLOW_STACK_ROWS, PLACES = RARE ? XTED_SW : FLOW_IMPORTS;
    constexpr unsigned SLOT_B = 4 * XTED_SW, RING_B = PF * SLOT_B, PITCH_B = 4 * (IMP + PLACES);
    static_assert(SC * PITCH_B + (RARE ? 2 * PLACES : 0) <= 4 * FLOW_STACK, "the window's room");
    const int lane = threadIdx.x & 31;
    const int2 *rows = P.rowinfo + pr.row_base, *nodes = P.rowinfo + pr.col_base;
    int32_t *dt = P.dt + pr.dt_off;
    const int pitch = pr.pitch;
    // what mapping two nodes saves: equal labels, others (a rename dearer than
    // delete + insert saves nothing: the maximum then takes another term)
    const int bm = P.c_del + P.c_ins, bn = max(bm - P.c_ren, 0);
    const int R = run.rows;
    const bool multi = ch.nseg > 1;
    const unsigned ring_a = smem_addr(ring), stk_a = ring_a + 4 * FLOW_RING;  // (stack rows are PITCH_B apart)
    const unsigned tl_a = stk_a + 4 * FLOW_STACK, lab_a = tl_a + 4 * XTED_SW, el_a = lab_a + 4 * XTED_SW;
    // where column c of a row lies in its ring slot (piece p of four words at
    // p ^ ((p >> 3) & 1): eight lanes reading their first or second pieces touch
    // eight different bank groups)
    auto swz = [](int c) { return 4 * ((c >> 2) ^ ((c >> 5) & 1)) + (c & 3); };

    // ---- columns ----
    int key[W];           // its segment's key
    int fb[W];            // its far column: byte offset in a stack row
    unsigned tcol = 0;    // bit k: column k is on its segment's right path
    unsigned xfar = 0;    // bit k: its far column is in another stripe
    unsigned expm = 0;    // bit k: stripes further left read it
    int ebase = 0x7fffffff;
    int sbase = 0, cend = ch.width, lead = 0, K = 1, X = 0, s = 0;
    __syncwarp();
    // multi: the columns' nodes, through the ring (nothing is under way there)
    if (multi) {
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
            key[k] = 0;
            int nd_j = -1;
            if (c < ch.width) {
                if (j >= je) {
                    q++;
                    j0 = P.krd[q];
                    je = (nodes[j0].y & XTED_ROW_ORL_MASK) + 1;
                    j = j0;
                }
                const int f = (nodes[j].y & XTED_ROW_ORL_MASK) + 1;  // far column's node
                nd_j = j;
                key[k] = (ch.k_lo + ch.nseg - 1 - q) * XTED_KEY_BIG;
                if (f == je) {
                    tcol |= 1u << k;
                } else {
                    const int fc = c + f - j;
                    fb[k] = 4 * ((fc & (W - 1)) * 32 + fc / W);
                }
                j++;
            }
            ring[c] = nd_j;
        }
    } else {
        const int j0 = P.krd[ch.k_lo], je = j0 + ch.width;
        lead = j0 & (XTED_PITCH - 1);
        sbase = j0 - lead;
        const int32_t *map = nullptr;
        if (lead + ch.width > XTED_SW) {
            const XChunkX cx = P.chunkx[it.chunk];
            K = cx.K;
            X = cx.X;
            s = it.stripe;
            map = P.smap + cx.map;
            sbase += s * XTED_SW;
            if (s > 0) lead = 0;
        }
        cend = min(je - sbase, XTED_SW);
#pragma unroll
        for (int k = 0; k < W; k++) {
            const int c = lane * W + k, j = sbase + c;
            fb[k] = 4 * ZERO;
            key[k] = 0;
            if (c >= lead && c < cend) {
                const int f = (nodes[j].y & XTED_ROW_ORL_MASK) + 1, fc = f - sbase;
                if (f == je) {
                    tcol |= 1u << k;
                } else if (fc < XTED_SW) {
                    fb[k] = 4 * ((fc & (W - 1)) * 32 + fc / W);
                } else {
                    xfar |= 1u << k;
                    fb[k] = map[f - j0];  // (its export index, until it has a place beside the stack row)
                }
                if (K > 1) {
                    const int e = map[j - j0];  // exports are numbered in column order
                    if (e >= 0) {
                        if (expm == 0) ebase = e;
                        expm |= 1u << k;
                    }
                }
            }
            ring[c] = j;
        }
    }
    __syncwarp();
    // ---- the lists: path columns, exported columns, far columns elsewhere ----
    auto first_of = [&](unsigned mask, int &n) {  // the lane's first place in a list; the list's length
        int v = __popc(mask);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(FULLMASK, v, d);
            if (lane >= d) v += o;
        }
        n = __shfl_sync(FULLMASK, v, 31);
        return v - __popc(mask);
    };
    int nt, nx, ne;
    int tf = first_of(tcol, nt), xf = first_of(xfar, nx), ef = first_of(expm, ne);
    ebase = (int)__reduce_min_sync(FULLMASK, (unsigned)ebase);
    unsigned char *el = (unsigned char *)(ring + FLOW_RING + FLOW_STACK + 2 * XTED_SW);
    int32_t *tlist = ring + FLOW_RING + FLOW_STACK, *tlab = tlist + XTED_SW;
    // far columns elsewhere, in column order, then the places of their values
    int32_t *xl = ring + FLOW_RING, *xplace = xl + XTED_SW, *xd = xplace + XTED_SW;  // (in the stack window, empty as yet)
    int x1 = xf;
#pragma unroll
    for (int k = 0; k < W; k++) {
        const int c = lane * W + k;
        if (RARE && ((tcol >> k) & 1u)) {  // by column, each read by its own lane only
            const int j = ring[c];
            tlab[swz(c)] = nodes[j].x;
            tlist[swz(c)] = j;
        } else if ((tcol >> k) & 1u) {
            const int j = ring[c];
            tlab[tf] = nodes[j].x;
            tlist[tf++] = (int)((unsigned)c | ((unsigned)(key[k] / XTED_KEY_BIG) << 8) | ((unsigned)j << 16));
        }
        if ((expm >> k) & 1u) el[ef++] = (unsigned char)(k * 32 + lane);
        if ((xfar >> k) & 1u) xl[x1++] = fb[k];
    }
    __syncwarp();
    int xq[2] = {0, 0};  // export index of the value in place q, q = lane, lane + 32
    int iv[2] = {0, 0};  // ... and the value for the next row
    unsigned short *xs = (unsigned short *)((char *)(ring + FLOW_RING) + SC * PITCH_B);  // RARE: of all places
    bool imported = false;  // RARE: the top row's places hold its values
    if (nx > 0) {
        // columns with one far column follow each other (subtrees across a
        // boundary are nested): they share a place
        int places = 0;
#pragma unroll 1
        for (int q0 = 0; q0 < nx; q0 += 32) {
            const int q = q0 + lane;
            const bool first = q < nx && (q == 0 || xl[q] != xl[q - 1]);
            const unsigned m = __ballot_sync(FULLMASK, first);
            const int place = places + __popc(m & (0xffffffffu >> (31 - lane))) - 1;
            if (q < nx) xplace[q] = place;
            if (first && place < PLACES) xd[place] = xl[q];
            places += __popc(m);
        }
        nx = places;
        if (!RARE && nx > FLOW_IMPORTS) return FLOW_RARE;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < W; k++)
            if ((xfar >> k) & 1u) {
                fb[k] = 4 * (IMP + xplace[xf++]);
            }
        if (RARE) {
#pragma unroll 1
            for (int q = lane; q < nx; q += 32) xs[q] = (unsigned short)xd[q];
        } else {
            if (lane < nx) xq[0] = xd[lane];
            if (lane + 32 < nx) xq[1] = xd[lane + 32];
        }
    }
    // the lane's copies of a row. multi: word lane + 32 k from column cpn[k] (-1: none); else pieces lane and lane + 32
    int cpn[W];
#pragma unroll
    for (int k = 0; k < W; k++) cpn[k] = multi ? ring[lane + 32 * k] : 4 * (lane + 32 * k) < cend ? 0 : -1;
    __syncwarp();
    if (lane < SC) sts(stk_a + lane * PITCH_B + 4 * ZERO, 0);
    // words past the chunk's copies stay zero; those that come with its first
    // or last piece are zeroed row by row, by lanes 0-2 and 3-5
    const int copied = multi ? ch.width : (cend + XTED_PITCH - 1) & ~(XTED_PITCH - 1);
#pragma unroll
    for (int k = 0; k < W; k++)
        if (lane * W + k >= copied)
            for (int q = 0; q < PF; q++) ring[q * XTED_SW + swz(lane * W + k)] = 0;
    const int ec = lane < 3 ? lane : cend + lane - 3;
    const bool edge = !multi && (lane < 3 ? lane < lead : lane < 6 && ec < copied);
    const unsigned edge_o = 4 * swz(edge ? ec : 0);
    const unsigned coff0 = 4 * swz(lane * W), coff1 = 4 * swz(lane * W + 4);  // the lane's columns in a slot
    const bool right = s + 1 < K, left = s > 0;
    const unsigned ask = (multi ? ITEM_MULTI : 0u) | (right ? ITEM_RIGHT : 0u) | (left ? ITEM_LEFT : 0u) |
                         (nx > 0 ? ITEM_IMPORTS : 0u) | (ne > 0 ? ITEM_EXPORTS : 0u) |
                         (__any_sync(FULLMASK, edge) ? ITEM_EDGE : 0u);
    const int32_t *Hin = P.buf + it.buf + (int64_t)s * R;   // the right neighbour's first column, per row
    int32_t *Hout = P.buf + it.buf + (int64_t)(s - 1) * R;  // this stripe's, for the left one
    int32_t *E = P.buf + it.buf + (int64_t)(K - 1) * R;     // exported columns, per row
    __syncwarp();

    // ---- row sequence: the run's tables one after another, each from its last row up ----
    // Lane l holds row tb + l of the sequence (its node, its record with the
    // table flags, its label) and, loaded 32 rows ahead, row tb + 32 + l.
    int bi = 0, by = 0, bl = 0, ni = 0, ny = 0, nl = 0;
    auto load_rows = [&](int f) {
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
        ni = e0 - off;
        const int2 r = rows[ni];
        nl = r.x;
        unsigned fl = off == 0 ? ROW_FIRST : 0u;
        if ((r.y & XTED_ROW_ORL_MASK) == e0) fl |= ROW_TREE;
        if (ni == i0) fl |= ROW_LAST;
        else if ((rows[ni - 1].y & XTED_ROW_ORL_MASK) == e0) fl |= ROW_NEXTTREE;
        ny = (int)((unsigned)r.y | fl | ask);
    };
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
        bi = ni, by = ny, bl = nl;
        load_rows(32 * h + lane);
    }
    const bool allp = nt == (multi ? ch.width : cend - lead);  // every column is on its segment's path
    if (!RARE && R >= FLOW_DENSE_ROWS && (allp || nt > FLOW_DENSE_COLS)) {
        const int trees = __popc(__ballot_sync(FULLMASK, by & ROW_TREE)) + __popc(__ballot_sync(FULLMASK, ny & ROW_TREE));
        if (trees >= 32) return FLOW_RARE;
    }
    int ci = bi;  // the rows being copied, PF - 1 ahead
    const int32_t *src0 = multi ? dt : dt + sbase + 4 * lane;
    const unsigned dst0 = ring_a + (multi ? 4 * lane : 16 * (lane ^ ((lane >> 3) & 1)));
    const unsigned dst1 = ring_a + (4 * lane ^ 16);  // multi: odd words of the lane (swz(lane + 32 k))
    auto copy_row = [&](unsigned so, int r, unsigned y) {  // row r into the slot at byte so of the ring
        const int32_t *src = src0 + (unsigned long long)(unsigned)r * (unsigned)pitch;
        const unsigned d = dst0 + so, d1 = dst1 + so;
        if (y & ITEM_MULTI) {
#pragma unroll
            for (int k = 0; k < W; k++)
                if (cpn[k] >= 0) cp_async4((k & 1 ? d1 : d) + 128 * k, src + (unsigned)cpn[k]);
        } else {
            if (cpn[0] >= 0) cp_async16(d, src);
            if (cpn[1] >= 0) cp_async16(d + 512, src + 128);
        }
    };
#pragma unroll 1
    for (int q = 0; q < PF - 1; q++) {
        const bool skip = RARE && allp && (__shfl_sync(FULLMASK, by, q) & ROW_TREE);
        if (!skip) copy_row(q * SLOT_B, __shfl_sync(FULLMASK, bi, q), ask);  // (past the run's end: its last row again)
        cp_async_commit();
    }

    int prev[W];
#pragma unroll
    for (int k = 0; k < W; k++) prev[k] = key[k];
    int sp = 0, lo = 0;             // stack depth; lowest position held in the shared window
    int c0 = 0, c1 = 0, cprev = 0;  // stripes: the right neighbour's first column in this row, the next, the one above
    if (right) {
        c0 = ld_relaxed(Hin);
        c1 = ld_relaxed(Hin + min(1, R - 1));
    }

#pragma unroll 1
    for (int t = 0; t < R; t++) {
        const unsigned so = (unsigned)(t & (PF - 1)) * SLOT_B, slot = ring_a + so;
        const unsigned above = ring_a + ((so + RING_B - SLOT_B) & (RING_B - 1));  // the slot of row t - 1
        const int tl = t & 31;
        cp_async_wait<PF - 2>();  // row t has landed
        __syncwarp();             // ... every lane's copies; row t - 1's readers are done
        const unsigned y = (unsigned)__shfl_sync(FULLMASK, by, tl);
        const bool trow = (y & ROW_TREE) != 0;
        int rl = 0;
        if (RARE && trow) rl = __shfl_sync(FULLMASK, bl, tl);
        if (!RARE && trow) {  // the path columns' words become what the diagonal gives
            rl = __shfl_sync(FULLMASK, bl, tl);
#pragma unroll 1
            for (int q0 = 0; q0 < nt; q0 += 32) {
                const int q = q0 + lane;
                if (q >= nt) continue;
                const unsigned e = (unsigned)lds(tl_a + 4 * q);
                const int c = e & 255, kc = (int)((e >> 8) & 255) * XTED_KEY_BIG;
                int x = c + 1 < XTED_SW ? lds(above + 4 * swz(c + 1)) : cprev;
                x = y & ROW_FIRST ? 0 : max(x - kc, 0);  // past a segment's end: its border
                sts(slot + 4 * swz(c), x + (rl == lds(lab_a + 4 * q) ? bm : bn));
            }
            __syncwarp();  // (and every lane has read the row above, whose slot is copied into next)
        }
        if (tl == 32 - (PF - 1)) ci = ni;
        const bool skip = RARE && allp && (__shfl_sync(FULLMASK, tl < 32 - (PF - 1) ? by : ny, (t + PF - 1) & 31) & ROW_TREE);
        if (!skip) copy_row(above - ring_a, __shfl_sync(FULLMASK, ci, (t + PF - 1) & 31), y);
        cp_async_commit();
        int a[W];
        auto path_values = [&]() {  // RARE: the path columns take what the diagonal gives, from the row above in registers
            const int4 l0 = lds4(lab_a + coff0), l1 = lds4(lab_a + coff1);
            const int lab[W] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
            int next = __shfl_down_sync(FULLMASK, prev[0], 1);
            if (lane == 31) next = cprev;
#pragma unroll
            for (int k = 0; k < W; k++) {
                const int x = y & ROW_FIRST ? 0 : max((k + 1 < W ? prev[k + 1] : next) - key[k], 0);
                if ((tcol >> k) & 1u) a[k] = x + (rl == lab[k] ? bm : bn);
            }
        };
        if (RARE && trow && allp) {  // nothing of the row comes from elsewhere
#pragma unroll
            for (int k = 0; k < W; k++) a[k] = 0;
            path_values();
        } else for (;;) {
            if (y & ITEM_EDGE) {
                if (edge) sts(slot + edge_o, 0);
                __syncwarp();
            }
            const int4 u = lds4(slot + coff0), v = lds4(slot + coff1);
            a[0] = u.x, a[1] = u.y, a[2] = u.z, a[3] = u.w, a[4] = v.x, a[5] = v.y, a[6] = v.z, a[7] = v.w;
            if (RARE && trow) path_values();
            // a word that is still -1: another item has yet to write it
            const unsigned who = __ballot_sync(FULLMASK, (a[0] | a[1] | a[2] | a[3] | a[4] | a[5] | a[6] | a[7]) < 0);
            if (__builtin_expect(who == 0, 1)) break;
            // the leftmost missing word is the last to come: wait for it, then
            // fetch this row and those already under way again
            int kk = 0, w = 0;
#pragma unroll
            for (int k = W - 1; k >= 0; k--)
                if (a[k] < 0) kk = k;
            kk = lane * W + kk;
            int j = sbase + kk;
            if (y & ITEM_MULTI) {  // its node: that of the keyroot's segment it lies in
                const int pos = P.cumw[ch.k_lo] + min(kk, ch.width - 1);
                int l2 = ch.k_lo, h2 = ch.k_lo + ch.nseg - 1;
                while (l2 < h2) {
                    const int mid = (l2 + h2 + 1) >> 1;
                    if (P.cumw[mid] <= pos) l2 = mid;
                    else h2 = mid - 1;
                }
                j = P.krd[l2] + pos - P.cumw[l2];
            }
            const int i = __shfl_sync(FULLMASK, bi, tl);
            if (!warp_wait(P, dt + (int64_t)i * pitch + __shfl_sync(FULLMASK, j, __ffs(who) - 1), true, w)) return FLOW_FAILED;
            cp_async_wait<0>();
            __syncwarp();
            if (!RARE && trow) {  // its path words stay: kept where the labels are while the row is copied again
#pragma unroll 1
                for (int q0 = 0; q0 < nt; q0 += 32) {
                const int q = q0 + lane;
                if (q >= nt) continue;
                    const int c = lds(tl_a + 4 * q) & 255, o = 4 * swz(c);
                    sts(lab_a + 4 * q, lds(slot + o));
                }
                __syncwarp();
            }
#pragma unroll 1
            for (int q = 0; q < PF; q++) {
                const int r = __shfl_sync(FULLMASK, tl + q < 32 ? bi : ni, (tl + q) & 31);
                const unsigned sq = (so + q * SLOT_B) & (RING_B - 1);
                if (y & ITEM_MULTI) {  // through L2, past whatever an L1 line holds
                    const int32_t *src = dt + (int64_t)r * pitch;
#pragma unroll
                    for (int k = 0; k < W; k++)
                        if (cpn[k] >= 0) sts((k & 1 ? dst1 : dst0) + sq + 128 * k, ld_relaxed(src + cpn[k]));
                } else {
                    copy_row(sq, r, y);
                }
            }
            cp_async_commit();
            cp_async_wait<0>();
            __syncwarp();
            if (!RARE && trow) {
#pragma unroll 1
                for (int q0 = 0; q0 < nt; q0 += 32) {
                const int q = q0 + lane;
                if (q >= nt) continue;
                    const unsigned e = (unsigned)lds(tl_a + 4 * q);
                    const int c = e & 255;
                    sts(slot + 4 * swz(c), lds(lab_a + 4 * q));
                    sts(lab_a + 4 * q, nodes[e >> 16].x);
                }
                __syncwarp();
            }
        }
        int c2 = 0;
        if (y & ITEM_RIGHT) {
            // (lanes reading one word at the same time need not see the same value)
            if (__builtin_expect(__any_sync(FULLMASK, c0 < 0), 0)) {
                if (!warp_wait(P, Hin + t, true, c0)) return FLOW_FAILED;
                c1 = ld_relaxed(Hin + min(t + 1, R - 1));
            }
            c2 = ld_relaxed(Hin + min(t + 2, R - 1));
        }
        // ---- the row's cells, before the suffix maximum ----
        int far[W];  // a tree row's far row is the table's border
#pragma unroll
        for (int k = 0; k < W; k++) far[k] = 0;
        if (!trow) {
            const unsigned top = stk_a + ((sp - 1) & (SC - 1)) * PITCH_B;
            if (__builtin_expect(sp - 1 < lo, 0)) {  // the top of the stack left the window: bring it back
                lo = sp - 1;
                const int32_t *g = gstk + (int64_t)lo * ZERO + lane;
#pragma unroll 1
                for (int k = 0; k < W; k++) sts(top + 4 * lane + 128 * k, g[32 * k]);
                __syncwarp();
            }
            if (RARE && (y & ITEM_IMPORTS) && !imported) {
                // (loaded a row ahead, into registers as the usual two, they gained 1%)
                const int i = __shfl_sync(FULLMASK, bi, tl);
                const int32_t *erow = E + (unsigned)(t - ((int)(y & XTED_ROW_ORL_MASK) + 1 - i)) * (unsigned)X;  // (R X < 2^32)
                int v[W];
#pragma unroll
                for (int k = 0; k < W; k++) v[k] = lane + 32 * k < nx ? ld_relaxed(erow + xs[lane + 32 * k]) : 0;
                for (;;) {
                    int x = -1, w = 0;
#pragma unroll
                    for (int k = 0; k < W; k++)
                        if (v[k] < 0) x = lane + 32 * k;
                    if (!__any_sync(FULLMASK, x >= 0)) break;
                    if (!warp_wait(P, erow + xs[max(x, 0)], x >= 0, w)) return FLOW_FAILED;
#pragma unroll
                    for (int k = 0; k < W; k++)
                        if (v[k] < 0) v[k] = ld_relaxed(erow + xs[lane + 32 * k]);
                }
#pragma unroll
                for (int k = 0; k < W; k++) sts(top + 4 * (IMP + lane + 32 * k), v[k]);
                __syncwarp();
                imported = true;
            }
            if (!RARE && (y & ITEM_IMPORTS)) {  // some far columns lie in stripes to the right: the far row's exports
                if (__builtin_expect(__any_sync(FULLMASK, (iv[0] | iv[1]) < 0), 0)) {
                    const int i = __shfl_sync(FULLMASK, bi, tl);
                    const int32_t *erow = E + (unsigned)(t - ((int)(y & XTED_ROW_ORL_MASK) + 1 - i)) * (unsigned)X;  // (R X < 2^32)
                    if (!warp_wait(P, erow + xq[0], iv[0] < 0, iv[0]) || !warp_wait(P, erow + xq[1], iv[1] < 0, iv[1]))
                        return FLOW_FAILED;
                }
                sts(top + 4 * (IMP + lane), iv[0]);
                if (lane < FLOW_IMPORTS - 32) sts(top + 4 * (IMP + 32 + lane), iv[1]);
                __syncwarp();
            }
#pragma unroll
            for (int k = 0; k < W; k++) far[k] = lds(top + fb[k]);
        }
#pragma unroll
        for (int k = 0; k < W; k++)  // a path column's far value is its segment's border
            a[k] = __viaddmax_s32(a[k], max(far[k], key[k]), prev[k]);
        // ---- suffix maximum: the lane's columns, then the lanes ----
#pragma unroll
        for (int k = W - 2; k >= 0; k--) a[k] = max(a[k], a[k + 1]);
        const int incl = warp_suffix_max(lane == 31 ? max(a[0], c0) : a[0]);
        int carry = __shfl_down_sync(FULLMASK, incl, 1);
        if (lane == 31) carry = c0;
#pragma unroll
        for (int k = 0; k < W; k++) prev[k] = max(a[k], carry);
        // ---- what others read ----
        if ((y & ITEM_LEFT) && lane == 0) st_relaxed(Hout + t, prev[0]);
        if (RARE && trow) {
            int32_t *o = dt + (int64_t)__shfl_sync(FULLMASK, bi, tl) * pitch;
            if (!(y & ITEM_MULTI) && tcol == (1u << W) - 1) {
                o += sbase + lane * W;
                st_relaxed4(o, make_int4(prev[0], prev[1], prev[2], prev[3]));
                st_relaxed4(o + 4, make_int4(prev[4], prev[5], prev[6], prev[7]));
            } else if (tcol) {
                const int4 n0 = lds4(tl_a + coff0), n1 = lds4(tl_a + coff1);
                const int nd[W] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
#pragma unroll
                for (int k = 0; k < W; k++)
                    if ((tcol >> k) & 1u) st_relaxed(o + nd[k], prev[k] - key[k]);
            }
        }
        if (!RARE && (y & (ROW_TREE | ROW_NEXTTREE))) {
            // the row goes into its own ring slot (free until the next row's
            // copies): the next row's diagonal, and this row's path columns
            sts4(slot + coff0, make_int4(prev[0], prev[1], prev[2], prev[3]));
            sts4(slot + coff1, make_int4(prev[4], prev[5], prev[6], prev[7]));
            if (trow) {
                __syncwarp();
                int32_t *o = dt + (int64_t)__shfl_sync(FULLMASK, bi, tl) * pitch;
#pragma unroll 1
                for (int q0 = 0; q0 < nt; q0 += 32) {
                const int q = q0 + lane;
                if (q >= nt) continue;
                    const unsigned e = (unsigned)lds(tl_a + 4 * q);
                    const int c = e & 255;
                    st_relaxed(o + (e >> 16), lds(slot + 4 * swz(c)) - (int)((e >> 8) & 255) * XTED_KEY_BIG);
                }
            }
        }
        if (y & ROW_LAST) {  // the table is done
#pragma unroll
            for (int k = 0; k < W; k++) prev[k] = key[k];
            sp = lo = 0;
            if (RARE) imported = false;
            cprev = 0;
        } else {
            cprev = c0;
            if (RARE && (y & (XTED_ROW_ISKR | XTED_ROW_PREVLEAF))) imported = false;
            if (y & XTED_ROW_ISKR) sp--;
            if (y & XTED_ROW_PREVLEAF) {
                if (__builtin_expect((unsigned)(sp - lo) >= (unsigned)SC, 0)) {
                    if (sp < lo) {
                        lo = sp - 1;
                    } else if (lo < (P.plan ? P.plan->stack_rows : P.stack_rows)) {  // the window is full: its lowest row moves out
                        int32_t *g = gstk + (int64_t)lo * ZERO + lane;
                        const unsigned d = stk_a + (lo & (SC - 1)) * PITCH_B + 4 * lane;
#pragma unroll 1
                        for (int k = 0; k < W; k++) g[32 * k] = lds(d + 128 * k);
                    } else if (lane == 0) {
                        set_error(P, XTED_ENOMEM, 2, lo, 0);
                    }
                    lo++;
                }
                // (every lane's reads of the slot's old row came before the shuffles above)
                const unsigned d = stk_a + (sp & (SC - 1)) * PITCH_B;
#pragma unroll
                for (int k = 0; k < W; k++) sts(d + 4 * lane + 128 * k, prev[k]);
                sp++;
                if (y & ITEM_EXPORTS) {  // the pushed row's exported columns
                    __syncwarp();
                    int32_t *e = E + (unsigned)t * (unsigned)X + ebase;
#pragma unroll 1
                    for (int q0 = 0; q0 < ne; q0 += 32)
                        if (q0 + lane < ne) st_relaxed(e + q0 + lane, lds(d + 4 * el[q0 + lane]));
                }
            }
            if (!RARE && (y & ITEM_IMPORTS) && !(y & ROW_NEXTTREE)) {  // the next row's far values in other stripes
                const int r = __shfl_sync(FULLMASK, tl < 31 ? bi : ni, (tl + 1) & 31);
                const int nro = __shfl_sync(FULLMASK, tl < 31 ? by : ny, (tl + 1) & 31) & XTED_ROW_ORL_MASK;
                const int32_t *e = E + (unsigned)(t - nro + r) * (unsigned)X;
                if (lane < nx) iv[0] = ld_relaxed(e + xq[0]);
                if (lane + 32 < nx) iv[1] = ld_relaxed(e + xq[1]);
            }
        }
        c0 = c1;
        c1 = c2;
        if (tl == 31) {
            bi = ni, by = ny, bl = nl;
            load_rows(t + 33 + lane);
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

// Before a warp's first item of a list (a whole warp): clears pieces of the
// list's tables and hand-off words while there are any, then waits for the
// pieces of others; false once the launch has failed. The launch clears them
// itself because it leaves an SM no registers: a memset beside it waited for all
// work in flight to end and for the idle exit (a lone query of 20-100 nodes with
// a second round took 4.1 ms against 0.9 so). The fences also order what was
// posted before the list, and drop whatever this SM's L1 holds of it: once a list
// and warp, where the claim of every item had one. (The claims' loop is tested
// at its top: left by a break behind the shuffle, it made the compiler guard
// every shuffle of the launch and spill, 16% of a query's time.)
__device__ __noinline__ bool open_list(const XKernelParams &P, int slot, int lane) {
    __threadfence();
    XServeClear *c = P.clears + slot;
    const int pieces = ld_relaxed(&c->pieces);
    const int64_t off = ((volatile XServeClear *)c)->off, n = ((volatile XServeClear *)c)->n;
    int k = 0;
    if (lane == 0) k = atomicAdd(&c->claimed, 1);
    k = __shfl_sync(FULLMASK, k, 0);
    while (__any_sync(FULLMASK, k < pieces)) {
        const int64_t lo = (int64_t)k * XTED_CLEAR_INTS;
        const int len = (int)min(n - lo, (int64_t)XTED_CLEAR_INTS);
        int32_t *p = P.dt + off + lo;
        for (int i = 4 * lane; i + 4 <= len; i += 128) *(int4 *)(p + i) = make_int4(-1, -1, -1, -1);
        if (lane < (len & 3)) p[(len & ~3) + lane] = -1;
        __threadfence();
        __syncwarp();
        if (lane == 0) {
            atomicAdd(&c->done, 1);
            k = atomicAdd(&c->claimed, 1);
        }
        k = __shfl_sync(FULLMASK, k, 0);
    }
    uint64_t t0 = 0;
    while (__any_sync(FULLMASK, ld_relaxed(&c->done) < pieces)) {
        __nanosleep(100);
        bool out = ld_relaxed(P.error) != 0;
        const uint64_t now = global_ns();
        if (t0 == 0) t0 = now;
        if (now - t0 > P.timeout_ns) {
            set_error(P, XTED_ETIMEOUT, 3, slot, 0);
            out = true;
        }
        if (__any_sync(FULLMASK, out)) return false;
    }
    __threadfence();
    return true;
}

// The next item of a serving session (a whole warp): the lists of the queries
// in flight, the oldest query's first. -1: leave the launch. Warps leave once
// every one of them has been idle for a while (then the launch is closed and
// the host starts another when work arrives); an item claimed meanwhile
// runs to its end, the rest of its list waits for the next launch. opened: the
// generation of the list whose item the warp had last (through L2: L1 may hold
// an item of an earlier list).
__device__ __noinline__ int claim_served(const XKernelParams &P, int lane, int *slot, int *opened) {
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
                *slot = q;
                const int gen = __ldcg(&P.items[g].gen);
                if (__any_sync(FULLMASK, gen != *(volatile int *)opened)) {
                    if (!open_list(P, q, lane)) return -1;
                    if (lane == 0) *(volatile int *)opened = gen;
                    __syncwarp();
                }
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

// Blocks of four warps, 45 KB of shared memory each: four per SM with 128
// registers a thread, or five with 96 (seven of them spilled). A row waits on
// fixed latencies for three of four cycles, so a launch of long rows that always
// has items to claim runs faster with the fifth block, one bound by its pairs'
// longest chains, or by the items' setup, runs slower: 1,023 mixed pairs 36.7 /
// 35.5 ms with four / five, 1,000 of 50-300 nodes 3.17 / 3.24, 20,000 random 46.5 /
// 49.0. The rule and more of its two sides are at XTED_FULL_PAIRS.
//
// SERVE: a serving session's launch, which claims from the lists of its queries.
template <int BLOCKS, bool SERVE>
__global__ void __launch_bounds__(32 * XTED_FLOW_WARPS, BLOCKS) xted_flow_kernel(const __grid_constant__ XKernelParams P) {
    extern __shared__ __align__(16) int32_t s_dyn[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t *ring = s_dyn + warp * FLOW_WARP_INTS;
    const XPlanOut *plan = SERVE ? nullptr : P.plan;
    const int nitems = plan ? plan->items : P.nitems;
    const int64_t per = plan ? (int64_t)plan->stack_rows * XTED_SW : P.scratch_per_warp;
    const int64_t gwarp = (int64_t)blockIdx.x * XTED_FLOW_WARPS + warp;
    int32_t *gstk = P.scratch + (plan ? -(gwarp + 1) * per : gwarp * per);
    for (int x = lane; x < FLOW_WARP_INTS; x += 32) ring[x] = 0;
    __syncwarp();
    if (plan && (gwarp + 1) * per > plan->scratch) return;
    int *opened = s_dyn + XTED_FLOW_WARPS * FLOW_WARP_INTS + warp;  // SERVE: the generation of the list that the warp is on
    if (SERVE && lane == 0) *opened = 0;
    for (;;) {
        int g = -1, slot = 0;
        const uint64_t t_claim = !SERVE && P.trace ? global_ns() : 0;
        if (SERVE) {
            g = claim_served(P, lane, &slot, opened);
        } else {
            if (lane == 0 && ld_relaxed(P.error) == 0) {
                g = atomicAdd(P.next, 1);
                if (g >= nitems) g = -1;
            }
            g = __shfl_sync(FULLMASK, g, 0);
        }
        if (g < 0) break;
        const uint64_t t_start = !SERVE && P.trace ? global_ns() : 0;
        const XItem it = P.items[g];
        const XPair pr = P.pairs[it.pair];
        const XRun run = P.runs[it.run];
        const XChunk ch = P.chunks[it.chunk];
        // (test hook: of a held pair, nothing that reads its level 0 becomes ready)
        const bool held = it.pair == P.hold_pair && run.depth + ch.depth == 0;
        if (!held) {
            // (tables of single nodes against segments of single nodes: every row and column is on its path)
            int rc = FLOW_RARE;
            if (run.kr_hi - run.kr_lo < run.rows || ch.nseg < ch.width || ch.width <= FLOW_DENSE_COLS)
                rc = run_item<false>(P, it, pr, run, ch, ring, gstk);
            if (rc == FLOW_RARE) rc = run_item<true>(P, it, pr, run, ch, ring, gstk);
            if (rc) break;
        }
        if (lane == 0) {
            // run and chunk of the two roots: the pair's last table (its leftmost stripe ends last)
            if (SERVE) {
                const bool root = it.stripe == 0 && run.rows == pr.m && ch.width == pr.n && run.kr_hi - run.kr_lo == 1 &&
                                  ch.nseg == 1;
                finish_served(P, pr, it, root, slot);
            }
            atomicAdd(P.progress, 1);
            if (!SERVE && P.trace) trace_item(P, g, t_claim, t_start, it.stripe, ch.width, run.rows);
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
template <int BLOCKS, bool SERVE>
static int occupancy_of(int *blocks_per_sm) {
    const int smem = SERVE ? FLOW_SERVE_SMEM : FLOW_SMEM;
    cudaError_t e = cudaFuncSetAttribute(xted_flow_kernel<BLOCKS, SERVE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, xted_flow_kernel<BLOCKS, SERVE>,
                                                              32 * XTED_FLOW_WARPS, smem);
}
int dp_occupancy(int *blocks_per_sm, bool full) {
    return full ? occupancy_of<5, false>(blocks_per_sm) : occupancy_of<4, false>(blocks_per_sm);
}
int serve_occupancy(int *blocks_per_sm) { return occupancy_of<4, true>(blocks_per_sm); }

// A plain launch: a block that is not resident has claimed nothing, and what
// the resident warps have claimed needs only items claimed before.
cudaError_t launch_dp(const XKernelParams &P, int grid, bool full, cudaStream_t s) {
    if (P.serve) xted_flow_kernel<4, true><<<grid, 32 * XTED_FLOW_WARPS, FLOW_SERVE_SMEM, s>>>(P);
    else if (full) xted_flow_kernel<5, false><<<grid, 32 * XTED_FLOW_WARPS, FLOW_SMEM, s>>>(P);
    else xted_flow_kernel<4, false><<<grid, 32 * XTED_FLOW_WARPS, FLOW_SMEM, s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_gather(const XPair *pairs, const int32_t *trivial, const int32_t *dt, int npairs, int32_t *out,
                          int c_del, int c_ins, int32_t *error, cudaStream_t s) {
    if (npairs <= 0) return cudaSuccess;
    xted_gather_kernel<<<(npairs + 255) / 256, 256, 0, s>>>(pairs, trivial, dt, npairs, out, c_del, c_ins, error);
    return cudaGetLastError();
}

}  // namespace xted
