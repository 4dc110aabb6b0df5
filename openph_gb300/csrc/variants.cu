// The standard, twist and row reductions as GPU kernels.
//
// The reference runs them column by column or row by row, on the host
// (standard.cu:1-57, twist.cu:10-87, ph_row.cu:38-121) or as one to five
// full-grid kernel launches per column/row with a single working thread
// (standard_parallel.cu:1-51, twist_parallel.cu:13-96,
// ph_row_parallel.cu:20-89).  Here:
//   * standard / twist: warps take the columns in the algorithm's order and
//     reduce them side by side (k_claim), each column by pivots to its left as
//     the algorithm has it; a column that holds a low which one to its left
//     comes to as well gives it up and goes on.  The lows of a reduced matrix
//     are unique, so they are those of the walk, and twist clears, dimension
//     by dimension, the columns it would.
//   * row: the lows are the same ones.  The CPU form's running essential
//     estimate follows from every column's own additions, replayed side by
//     side once the pairs are known (k_row_exact).
//   * standard / twist with trackers, which follow the walk itself, and twist
//     on matrices whose dimensions do not separate, where the clearing depends
//     on the order: one launch in which a single warp walks the columns in
//     the algorithm's order.  A 32-column window is inspected at once (lows,
//     pivot-table hits, repeated lows, twist clears landing inside the window)
//     so that columns needing no addition are retired 32 at a time; a column
//     that needs additions is reduced by the whole warp with the column kept
//     in shared memory across its chain of additions.
//   * row with trackers, or where the replay finds no room: one CTA walks the
//     rows from the bottom; a warp finds the next row with two or more columns
//     on it (per-row buckets), and the CTA's 32 warps add the row's pivot into
//     all of that row's other columns in parallel (mark_neighbours /
//     left_to_right_neighbours, ph_row_parallel.cu:3-18).
// Columns too wide for the shared buffers continue in pool-allocated global
// buffers.
#include <algorithm>
#include <climits>
#include <vector>

#include "oph_host.h"

namespace oph {

struct SeqArgs {
    int64_t m;
    int32_t *low;
    int32_t *arglow;   // standard/twist pivot table; row: pivots[] (first column ever holding each low)
    const int8_t *dim;
    int64_t *seg;
    int *pool;
    DevStatus *st;
    int32_t *ess;      // row (reference CPU form): the running essential estimate
    int32_t *bhead;    // row: bucket heads (columns whose low is the row)
    int32_t *bnext;    // row: bucket links
    int32_t *bcnt;     // row: bucket sizes
    int32_t *blist;    // row: the current row's bucket, gathered
    int start_dim;
    long long start_pos;
    int max_dim;
    int twist;         // standard (0) or twist (1)
    int row_quirk;     // row: keep the reference CPU form's running ess estimate
    long long *it_ns;  // standard / twist with trackers: end of every iteration (globaltimer), or nullptr
    long long it_base; //   the iteration this launch starts at (1, or where an interrupted walk stopped)
    // row with trackers: a log of the rows that had additions, each as
    // {row, pivot, neighbours k, end time (ns, two ints)} then k pairs
    // {column, its new low}; ev_cap ints, the length in ev[-2..-1] (int64),
    // nullptr without trackers
    int *ev;
    long long ev_cap;
};

__device__ __forceinline__ long long global_ns() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Chain of additions into column j by one warp, `next(low)` giving the column
// to add next (or -1 to stop).  The column stays in shared memory (sA/sB/sC,
// `cap` ints each) while it fits and moves to pool-allocated buffers when it
// does not.  j is written back once.  Returns the new low of j, or -2 when
// the pool is exhausted (j unchanged).
template <class Tile, class Next>
__device__ int chain(const Tile &tile, const SeqArgs &a, int j, int *sA, int *sB, int *sC, int cap, Next next,
                     long long &adds, long long &slots) {
    const int lane = tile.thread_rank();
    int lj = a.low[j];
    int p = next(lj);
    if (p < 0) return lj;
    const long long sj = a.seg[j];
    int n = a.pool[sj];
    const int capj = a.pool[sj + 1];
    int *A, *X = nullptr, *Y = nullptr;
    int bcap;
    bool smem_mode = n <= cap;
    if (smem_mode) {
        group_copy<32>(tile, sA, a.pool + sj + SEG_HDR, n);
        A = sA;
        bcap = cap;
    } else {
        bcap = round4(max(2 * n, 1024));
        long long off = 0;
        if (lane == 0) off = pool_alloc(a.st, 2ll * bcap);
        off = tile.shfl(off, 0);
        if (off < 0) return -2;
        X = a.pool + off; Y = X + bcap;
        group_copy<32>(tile, X, a.pool + sj + SEG_HDR, n);
        A = X;
    }
    while (p >= 0) {
        const long long sp = a.seg[p];
        const int np = a.pool[sp];
        if (n + np > bcap) {
            int ncap = round4(max(2 * (n + np), 1024));
            long long off = 0;
            if (lane == 0) off = pool_alloc(a.st, 2ll * ncap);
            off = tile.shfl(off, 0);
            if (off < 0) return -2;
            int *NX = a.pool + off;
            group_copy<32>(tile, NX, A, n);
            A = NX; X = NX; Y = NX + ncap; bcap = ncap; smem_mode = false;
        }
        const int *P = a.pool + sp + SEG_HDR;
        int *out;
        if (smem_mode) {
            group_copy<32>(tile, sC, P, np);
            P = sC;
            out = (A == sA) ? sB : sA;
        } else {
            out = (A == X) ? Y : X;
        }
        const int nn = merge_xor<32>(tile, A, n, P, np, out);
        slots += n + np + nn;
        adds++;
        n = nn;
        A = out;
        lj = n ? A[n - 1] : -1;
        p = next(lj);
    }
    long long dst = sj;
    int dcap = capj;
    if (n > capj) {
        dcap = round4(max(2 * n, 16));
        long long off = 0;
        if (lane == 0) off = pool_alloc(a.st, SEG_HDR + dcap);
        off = tile.shfl(off, 0);
        if (off < 0) return -2;
        dst = off;
    }
    group_copy<32>(tile, a.pool + dst + SEG_HDR, A, n);
    if (lane == 0) {
        a.pool[dst] = n;
        a.pool[dst + 1] = dcap;
        a.seg[j] = dst;
        a.low[j] = lj;
    }
    tile.sync();
    return lj;
}

constexpr int SEQ_CAP = 4096;

// standard (reduce_col_host, kernels_host.cu:62-75, for j = 0..m-1) and
// twist (the same per dimension from the top down, dimensions >= 1 only,
// then low[low_j] := -1; twist.cu:10-87).
__global__ void __launch_bounds__(32) k_seq_walk(SeqArgs a) {
    extern __shared__ int smem[];
    int *sA = smem, *sB = smem + SEQ_CAP, *sC = smem + 2 * SEQ_CAP;
    auto tile = cg::tiled_partition<32>(cg::this_thread_block());
    const int lane = tile.thread_rank();
    long long adds = 0, slots = 0;
    // iterations (the reference's, one per visited column) and their end
    // times, when trackers are kept: columns retired together in a window
    // share its time evenly
    long long it = a.it_base;
    long long tprev = global_ns();
    if (a.it_ns && it == 1 && lane == 0) a.it_ns[0] = tprev;
    const int d_end = a.twist ? 1 : a.start_dim;
    for (int d = a.start_dim; d >= d_end; d--) {
        long long j0 = (d == a.start_dim) ? a.start_pos : 0;
        while (j0 < a.m) {
            const long long j = j0 + lane;
            const bool in = j < a.m && (!a.twist || a.dim[j] == d);
            const int lj = in ? a.low[j] : -1;
            const int pj = lj >= 0 ? a.arglow[lj] : -1;
            bool dup = false, hit = false;
            for (int q = 0; q < 31; q++) {
                int lq = tile.shfl(lj, q);
                if (q < lane && lq >= 0) {
                    if (lq == lj) dup = true;
                    if (a.twist && lq == (int)j) hit = true;
                }
            }
            const bool stop = (in && ((lj >= 0 && pj != -1) || dup)) || (j < a.m && hit);
            const unsigned sb = tile.ballot(stop);
            const int fs = sb ? __ffs(sb) - 1 : 32;
            if (lane < fs && in && lj >= 0) {
                a.arglow[lj] = (int)j;
                if (a.twist) a.low[lj] = -1;
            }
            {
                const unsigned retired = tile.ballot(in) & (fs == 32 ? 0xffffffffu : (1u << fs) - 1u);
                const int cnt = __popc(retired);
                if (a.it_ns && lane == 0 && cnt) {
                    const long long t = global_ns();
                    for (int q = 0; q < cnt; q++) a.it_ns[it + q] = tprev + (t - tprev) * (q + 1) / cnt;
                    tprev = t;
                }
                it += cnt;
            }
            tile.sync();
            if (fs == 32) { j0 += 32; continue; }
            const long long jj = j0 + fs;
            const bool jj_hit = tile.shfl(hit, fs);
            if (jj_hit) { j0 = jj; continue; }  // its low was just cleared: look at it again
            auto next = [&](int l) { return l >= 0 ? a.arglow[l] : -1; };
            const int nl = chain(tile, a, (int)jj, sA, sB, sC, SEQ_CAP, next, adds, slots);
            if (nl == -2) {
                if (lane == 0) { a.st->resume_dim = d; a.st->resume_pos = jj; a.st->resume_iter = it; }
                goto out;
            }
            if (nl >= 0 && lane == 0) {
                a.arglow[nl] = (int)jj;
                if (a.twist) a.low[nl] = -1;
            }
            if (a.it_ns && lane == 0) a.it_ns[it] = tprev = global_ns();
            it++;
            tile.sync();
            j0 = jj + 1;
        }
    }
    if (lane == 0) a.st->resume_pos = -1;
out:
    if (lane == 0) {
        a.st->additions += adds;
        a.st->slots += slots;
    }
}

// ------------------------------------------------- columns side by side
constexpr int CL_WARPS = 8, CL_THREADS = 32 * CL_WARPS;
constexpr int CL_CAP = 768;                     // rows of a list that a warp keeps in shared memory
constexpr int CL_ALONE = 2;                     // additions a column makes one at a time; then 2, 4, ... 32 together
constexpr int CL_BITS = 3 * CL_CAP;             // words of a warp's bitmap (73,728 rows), at most

// The holder of a low, read and swapped as one 16-byte word: the column (-1: none yet),
// its segment / 4, and its next two rows down (-1: none), or -2 and its
// length when it has more than three.
struct __align__(16) Holder {
    int col, seg4, b, c;
};
// A launch's next column, and how many it gave up.
struct ClaimCount {
    unsigned long long next;
    int failed, pad;
};
struct ClaimArgs {
    int64_t m;
    int32_t *low;
    Holder *holder;
    const int8_t *dim;
    int64_t *seg;            // a column's segment: what it last published
    int *pool;
    DevStatus *st;
    int want_dim;            // only columns of this dimension (-1: all)
    int words;               // of a warp's bitmap
    const int32_t *redo;     // only the columns an earlier launch gave up for want of room, or nullptr
    int64_t n;               // columns to look at: of redo, or m
    int32_t *failed;         // columns this launch gives up
    ClaimCount *count;       // this launch's
    const ClaimCount *above; // of the dimensions before it, `n_above` of them: nothing to do while one has failed
    int n_above;
};
using Tile32 = cg::thread_block_tile<32>;

__device__ __forceinline__ Holder holder_load(const Holder *h) {
    long long v0, v1;
    asm volatile("{ .reg .b128 t; ld.acquire.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(v0), "=l"(v1)
                 : "l"(h)
                 : "memory");
    return Holder{(int)v0, (int)(v0 >> 32), (int)v1, (int)(v1 >> 32)};
}
__device__ __forceinline__ Holder holder_of(const Tile32 &tile, const Holder &h, int lane) {
    return Holder{tile.shfl(h.col, lane), tile.shfl(h.seg4, lane), tile.shfl(h.b, lane), tile.shfl(h.c, lane)};
}
__device__ __forceinline__ int holder_rows(const Holder &h) { return h.b == -2 ? h.c : 1 + (h.b >= 0) + (h.c >= 0); }
__device__ __forceinline__ long long pack2(int lo, int hi) { return (long long)(unsigned)lo | ((long long)hi << 32); }
// True when `was` stood there and `now` does.
__device__ __forceinline__ bool holder_swap(const Tile32 &tile, Holder *h, const Holder &was, const Holder &now) {
    tile.sync();
    bool ok = false;
    if (tile.thread_rank() == 0) {
        const long long w0 = pack2(was.col, was.seg4), w1 = pack2(was.b, was.c);
        long long g0, g1;
        asm volatile(
            "{ .reg .b128 t, w, n; mov.b128 w, {%3, %4}; mov.b128 n, {%5, %6};"
            " atom.acq_rel.gpu.global.cas.b128 t, [%2], w, n; mov.b128 {%0, %1}, t; }"
            : "=l"(g0), "=l"(g1)
            : "l"(h), "l"(w0), "l"(w1), "l"(pack2(now.col, now.seg4)), "l"(pack2(now.b, now.c))
            : "memory");
        ok = g0 == w0 && g1 == w1;
    }
    ok = tile.shfl((int)ok, 0);
    tile.sync();
    return ok;
}

// A warp's column as a bitmap of all rows: an addition flips bits, the next
// low is found 1,024 rows at a time.
struct BitColumn {
    static constexpr bool WAVES = true;
    unsigned *bits;
    int *pick;
    int n, low, bottom, top;  // rows, the highest, words that may hold bits
    __device__ void init(const Tile32 &tile, const ClaimArgs &a, int *own, int *own_pick) {
        bits = reinterpret_cast<unsigned *>(own);
        pick = own_pick;
        for (int q = tile.thread_rank(); q < a.words; q += 32) bits[q] = 0;
        tile.sync();
    }
    __device__ void start() { n = 0, low = -1, bottom = 1 << 30, top = -1; }
    __device__ void end(const Tile32 &tile) {
        for (int q = bottom + (int)tile.thread_rank(); q <= top; q += 32) bits[q] = 0;
        tile.sync();
    }
    // rows P (np >= 1 ascending, the first 32 also held one a lane in pv)
    __device__ bool add(const Tile32 &tile, const ClaimArgs &, int pv, const int *P, int np) {
        const int lane = tile.thread_rank();
        int both = 0, last = 0;
        for (int base = 0; base < np; base += 32) {
            const int q = base + lane;
            bool was = false;
            if (q < np) {
                last = base ? P[q] : pv;
                was = atomicXor(&bits[last >> 5], 1u << (last & 31)) >> (last & 31) & 1u;
            }
            both += __popc(tile.ballot(was));
        }
        n += np - 2 * both;
        bottom = min(bottom, tile.shfl(pv, 0) >> 5);
        const int high = tile.shfl(last, (np - 1) & 31);
        top = max(top, high >> 5);
        tile.sync();
        find_low(tile, max(low, high) >> 5);
        return true;
    }
    // the highest row, in word w or below
    __device__ void find_low(const Tile32 &tile, int w) {
        const int lane = tile.thread_rank();
        low = -1;
        for (; w >= bottom; w -= 32) {
            const unsigned x = w - lane >= bottom ? bits[w - lane] : 0u;
            const unsigned b = tile.ballot(x != 0);
            if (b) {
                const int f = __ffs(b) - 1;
                low = (w - f) * 32 + 31 - __clz(tile.shfl(x, f));
                break;
            }
        }
    }
    // Of its highest rows, a lane each (up to `most`, of 1,024 places): -1
    // beyond them.  Lane 0 has the low.
    __device__ int rows_at(const Tile32 &tile, int most) const {
        const int lane = tile.thread_rank(), w = (low >> 5) - lane;
        unsigned x = w >= bottom ? bits[w] : 0u;
        int upto = __popc(x), at = upto;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = tile.shfl_up(upto, o);
            if (lane >= o) upto += u;
        }
        at = upto - at;
        for (; x && at < most; at++) {
            const int b = 31 - __clz(x);
            pick[at] = w * 32 + b;
            x ^= 1u << b;
        }
        tile.sync();
        const int r = lane < min(most, tile.shfl(upto, 31)) ? pick[lane] : -1;
        tile.sync();
        return r;
    }
    // Add the columns h of the lanes that `have` one, whose low is row r; all
    // at once, which no order of additions matters to.
    __device__ void add_all(const Tile32 &tile, const ClaimArgs &a, const Holder &h, int r, bool have) {
        const int lane = tile.thread_rank(), np = have ? holder_rows(h) : 0;
        int both = 0, lowest = 1 << 30;
        auto flip = [&](int row) {
            both += atomicXor(&bits[row >> 5], 1u << (row & 31)) >> (row & 31) & 1u;
            lowest = min(lowest, row);
        };
        if (np >= 1 && np <= 3) {
            flip(r);
            if (np > 1) flip(h.b);
            if (np > 2) flip(h.c);
        }
        for (unsigned todo = tile.ballot(np > 3); todo;) {
            // four at a time, their rows loaded together
            const int *P[4];
            int pn[4], v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int f = todo ? __ffs(todo) - 1 : 0;
                pn[u] = todo ? tile.shfl(np, f) : 0;
                P[u] = a.pool + ((long long)(unsigned)tile.shfl(h.seg4, f) << 2) + SEG_HDR;
                v[u] = lane < pn[u] ? P[u][lane] : 0;
                todo &= todo - 1;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (lane < pn[u]) flip(v[u]);
                for (int q = 32 + lane; q < pn[u]; q += 32) flip(P[u][q]);
            }
        }
        n += __reduce_add_sync(0xffffffffu, np - 2 * both);
        bottom = min(bottom, __reduce_min_sync(0xffffffffu, lowest) >> 5);
        tile.sync();
        find_low(tile, low >> 5);
    }
    __device__ void write(const Tile32 &tile, int *out) const {
        const int lane = tile.thread_rank();
        int at = 0;
        for (int w = bottom; w <= (low >> 5); w += 32) {
            unsigned x = w + lane <= (low >> 5) ? bits[w + lane] : 0u;
            if (!tile.any(x != 0)) continue;
            int k = __popc(x), upto = k;
            for (int o = 1; o < 32; o <<= 1) {
                const int u = tile.shfl_up(upto, o);
                if (lane >= o) upto += u;
            }
            int *o = out + at + upto - k;
            for (; x; x &= x - 1) *o++ = (w + lane) * 32 + __ffs(x) - 1;
            at += tile.shfl(upto, 31);
        }
    }
};

// A warp's column as an ascending list, in its shared buffers while it fits,
// else in two halves of a pool allocation; for matrices too large for the
// bitmaps.
struct ListColumn {
    static constexpr bool WAVES = false;
    int *home, *A, *B, *C;  // rows, the next sum, the staged pivot
    int n, low, cap;
    __device__ void init(const Tile32 &, const ClaimArgs &, int *own, int *) { home = own; }
    __device__ void start() {
        A = home, B = home + CL_CAP, C = home + 2 * CL_CAP;
        n = 0, low = -1, cap = CL_CAP;
    }
    __device__ void end(const Tile32 &) {}
    __device__ bool add(const Tile32 &tile, const ClaimArgs &a, int pv, const int *P, int np) {
        const int lane = tile.thread_rank();
        if (n + np > cap) {
            const int ncap = round4(2 * (n + np));
            long long off = 0;
            if (lane == 0) off = pool_alloc(a.st, 2ll * ncap);
            off = tile.shfl(off, 0);
            if (off < 0) return false;
            int *N = a.pool + off;
            group_copy<32>(tile, N, A, n);
            A = N;
            B = N + ncap;
            cap = ncap;
        }
        if (np <= 4) {
            n = merge_xor_seg<32>(tile, A, n, pv, np, B);
        } else if (np <= 32) {
            n = merge_xor_thr<32>(tile, A, n, pv, np, B);
        } else {
            if (np <= CL_CAP) {  // searched in shared memory
                group_copy<32>(tile, C, P, np);
                P = C;
            }
            n = merge_xor<32>(tile, A, n, P, np, B);
        }
        int *t = A;
        A = B;
        B = t;
        low = n ? A[n - 1] : -1;
        tile.sync();
        return true;
    }
    __device__ void write(const Tile32 &tile, int *out) const { group_copy<32>(tile, out, A, n); }
};

// standard and twist, a warp per column, the columns taken in order.  A
// column adds the holder of its low while that is a column to its left
// (reduce_col_host, kernels_host.cu:62-75).  Else it publishes its rows and
// claims the low by compare-and-swap; a low held by a column to the right is
// taken from it, and the warp goes on with that column, which has the taker
// to add.  Published rows are never written again (a column that changes gets
// a new segment), so a reader sees some whole column of an index to its left
// whatever the others do meanwhile.  No warp waits for another: a swap that
// fails means that another column has taken the low.
// Bound by the chain of loads of the columns with the most additions, one
// after the other: the holder (with the rows of a holder of three) is one
// load, a longer one's rows a second.  Such a column also adds the holders,
// where they are columns to its left, of the 2, 4, ... 32 rows below its low
// in one wave.  Additions, and so the counters, vary with who came first.
// Device time (setup and reading back included), the walk by one warp first:
// twist on a 64 x 64 image 8.0 ms -> 0.18 (0.31 without waves), standard on
// 24 points 17-20 ms -> 0.08; 0.52 and 0.10 with sorted lists and holders of
// one column index.
template <class Column>
__global__ void __launch_bounds__(CL_THREADS) k_claim(ClaimArgs a) {
    extern __shared__ __align__(16) int smem[];  // a.words a warp
    const Tile32 tile = cg::tiled_partition<32>(cg::this_thread_block());
    const int lane = tile.thread_rank();
    Column c;
    __shared__ int s_pick[CL_WARPS][32];
    for (int d = 0; d < a.n_above; d++)
        if (a.above[d].failed) return;
    c.init(tile, a, smem + (size_t)(threadIdx.x >> 5) * a.words, s_pick[threadIdx.x >> 5]);
    long long adds = 0, slots = 0;
    for (;;) {
        long long idx = 0;
        if (lane == 0) idx = (long long)atomicAdd(&a.count->next, 1ull);
        idx = tile.shfl(idx, 0);
        if (idx >= a.n) break;
        int j = (int)idx;
        if (a.redo) {
            j = a.redo[idx];
        } else {
            const int d = a.dim[j], l0 = a.low[j];
            if (a.want_dim >= 0 && d != a.want_dim) continue;
            if (l0 < 0) continue;  // zero, or cleared
        }
        // the column as it was last published: header, then rows
        long long seg = a.seg[j];
        const int h = a.pool[seg + lane];
        int n = tile.shfl(h, 0);
        const int *R = a.pool + seg + SEG_HDR;
        auto row = [&](int k) { return n <= 32 - SEG_HDR ? tile.shfl(h, SEG_HDR + max(k, 0)) : R[max(k, 0)]; };
        int l = row(n - 1), rb = row(n - 2), rc = row(n - 3);
        if (n < 1) l = -1;
        bool loaded = false, changed = false, room = true;
        int wave = 0;  // additions so far, and waves of them
        c.start();
        while (l >= 0) {
            // the low's holder, and in a long chain those of the rows below it
            int r = lane == 0 ? l : -1;
            if constexpr (Column::WAVES)
                if (wave > CL_ALONE) r = c.rows_at(tile, 1 << min(wave - CL_ALONE, 5));
            Holder mine{-1, 0, 0, 0};
            if (r >= 0) mine = holder_load(a.holder + r);
            tile.sync();
            const Holder p = holder_of(tile, mine, 0);
            if constexpr (Column::WAVES)
                if (wave > CL_ALONE && p.col >= 0 && p.col < j) {
                    const bool have = mine.col >= 0 && mine.col < j;
                    const int before = c.n;
                    c.add_all(tile, a, mine, r, have);
                    changed = true;
                    wave++;
                    adds += __popc(tile.ballot(have));
                    slots += before + c.n + __reduce_add_sync(0xffffffffu, have ? holder_rows(mine) : 0);
                    l = c.low;
                    continue;
                }
            const bool take = p.col < 0 || p.col > j;
            if (take) {
                if (changed) {
                    n = c.n;
                    if (lane == 0) seg = pool_alloc(a.st, SEG_HDR + round4(n));
                    seg = tile.shfl(seg, 0);
                    if (seg < 0) {
                        room = false;
                        break;
                    }
                    int *out = a.pool + seg + SEG_HDR;
                    c.write(tile, out);
                    if (lane == 0) {
                        a.pool[seg] = n;
                        a.pool[seg + 1] = round4(n);
                        a.seg[j] = seg;
                    }
                    tile.sync();
                    if (n <= 3) {
                        rb = out[max(n - 2, 0)];
                        rc = out[max(n - 3, 0)];
                    }
                    changed = false;
                }
                if (lane == 0) a.low[j] = l;
                const Holder now = n > 3 ? Holder{j, (int)(seg >> 2), -2, n}
                                         : Holder{j, (int)(seg >> 2), n > 1 ? rb : -1, n > 2 ? rc : -1};
                if (!holder_swap(tile, a.holder + l, p, now)) continue;  // look again
                if (p.col < 0) break;  // done, for all that is known
            }
            if (!loaded) {
                loaded = true;
                const int v = tile.shfl_down(h, SEG_HDR);
                if (!c.add(tile, a, n <= 32 - SEG_HDR ? v : lane < n ? R[lane] : 0, R, n)) room = false;
            }
            // column j += column p; having taken the low, column p += column j
            const int np = holder_rows(p);
            const int *P = a.pool + ((long long)(unsigned)p.seg4 << 2) + SEG_HDR;
            int pv = 0;
            if (np > 3) {
                if (lane < np) pv = P[lane];
            } else {
                pv = lane == np - 1 ? l : lane == np - 2 ? p.b : p.c;
            }
            if (take) j = p.col;
            const int before = c.n;
            if (!room || !c.add(tile, a, pv, P, np)) {
                room = false;  // column j goes on, from what it last published, when there is more
                break;
            }
            changed = true;
            wave++;
            adds++;
            slots += before + np + c.n;
            l = c.low;
        }
        c.end(tile);
        if (lane == 0) {
            if (!room) a.failed[atomicAdd(&a.count->failed, 1)] = j;
            else if (l < 0) a.low[j] = -1;
        }
        tile.sync();
    }
    if (lane == 0 && adds) {
        atomicAdd(&a.st->additions, (unsigned long long)adds);
        atomicAdd(&a.st->slots, (unsigned long long)slots);
    }
}

// twist's clearing after a dimension: the columns whose row is a low.
__global__ void k_claim_clear(ClaimArgs a) {
    for (int d = 0; d <= a.n_above; d++)
        if (a.above[d].failed) return;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < a.m; j += (int64_t)gridDim.x * blockDim.x)
        if (a.dim[j] == a.want_dim && a.low[j] >= 0) a.low[a.low[j]] = -1;
}

// ------------------------------------- the row form's running estimate
// The row algorithm adds the first column with low i into the others with that
// low, so each column goes through the lows that it meets when it adds the
// reduced columns to its left one by one, whatever the order of the rows; the
// running estimate (ph_row.cu:2-31) follows from who met which low, and over
// which row.  With the pairs known (k_claim), k_row_exact takes the columns in
// order, a warp each, and waits for the reduced columns it adds: all to its
// left, so the first unfinished one never waits.  Every low met is an event;
// k_row_marks finds, for a low, the columns that were the first ever to hold
// it when they came to it.
// Bound by the longest chain of columns that wait for one another.  One CTA
// walking the rows takes a few microseconds a row: 6.6 ms for an image of some
// 40 x 40, now 0.32 to the call's end; 205 ms of device time on 128 x 128, now
// 3.5 (1.2 of it k_claim).
struct RowArgs {
    int64_t m;
    const int64_t *colptr;
    const Holder *holder;     // final
    unsigned long long *done; // a reduced column: segment / 4 << 32 | rows; 0: not yet
    int32_t *ess;
    int *first;               // the first column to start with each low
    int *count, *place;       // events of each low, and where they go
    int *ev_low;              // the events: low met, from which row, by which column
    int2 *ev;
    int2 *sorted;
    unsigned *n_ev;
    unsigned cap;
    int *quit;                // no room, or a wait that did not end: the walk does it
    ClaimArgs c;              // for the columns' additions
};

constexpr int ROW_WAIT = 1 << 22;  // looks at a column to the left, a few seconds
template <class Column>
__global__ void __launch_bounds__(CL_THREADS) k_row_exact(RowArgs a) {
    extern __shared__ __align__(16) int smem[];  // a.c.words a warp
    const Tile32 tile = cg::tiled_partition<32>(cg::this_thread_block());
    const int lane = tile.thread_rank();
    __shared__ int s_pick[CL_WARPS][32];
    Column c;
    c.init(tile, a.c, smem + (size_t)(threadIdx.x >> 5) * a.c.words, s_pick[threadIdx.x >> 5]);
    long long adds = 0, slots = 0;
    int *const pool = a.c.pool;
    bool quit = false;
    while (!quit) {
        long long idx = 0;
        if (lane == 0) idx = *(volatile int *)a.quit ? a.m : (long long)atomicAdd(&a.c.count->next, 1ull);
        idx = tile.shfl(idx, 0);
        if (idx >= a.m) break;
        const int j = (int)idx;
        const int64_t c0 = a.colptr[j];
        const int n = (int)(a.colptr[j + 1] - c0);
        if (n == 0) continue;
        long long seg = 8ll * j + 4 * ((c0 + 3) >> 2);  // as k_setup_columns put it
        const int *R = pool + seg + SEG_HDR;
        int l = R[n - 1];
        if (lane == 0) atomicMin(a.first + l, j);
        int q = a.holder[l].col, rows = n;
        c.start();
        if (q != j && !c.add(tile, a.c, lane < n ? R[lane] : 0, R, n)) quit = true;
        while (!quit && l >= 0 && q != j) {
            // the reduced column with this low, to the left
            unsigned long long d = 0;
            if (lane == 0 && q >= 0 && q < j)
                for (int tries = 0; tries < ROW_WAIT; tries++) {
                    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(d) : "l"(a.done + q) : "memory");
                    if (d || ((tries & 255) == 255 && *(volatile int *)a.quit)) break;
                    if (tries > 16) __nanosleep(100);
                }
            d = tile.shfl(d, 0);
            tile.sync();
            const int np = (int)(unsigned)d, before = c.n;
            const int *P = pool + (long long)(d >> 32 << 2) + SEG_HDR;
            if (!d || !c.add(tile, a.c, lane < np ? P[lane] : 0, P, np)) {
                quit = true;
                break;
            }
            adds++;
            slots += before + np + c.n;
            const int nl = c.low;
            if (lane == 0) {
                a.ess[l] = 0;
                a.ess[q] = 0;
                if (nl >= 0) {
                    const unsigned e = atomicAdd(a.n_ev, 1u);
                    if (e < a.cap) {
                        a.ev_low[e] = nl;
                        a.ev[e] = make_int2(l, j);
                        atomicAdd(a.count + nl, 1);
                    }
                    quit = e >= a.cap;
                }
            }
            quit = tile.any(quit);
            l = nl;
            if (l >= 0) q = a.holder[l].col;
            rows = c.n;
        }
        if (!quit && l >= 0) {  // a pivot: its reduced rows for those to its right
            if (c.n) {
                if (lane == 0) seg = pool_alloc(a.c.st, SEG_HDR + round4(rows));
                seg = tile.shfl(seg, 0);
                if (seg < 0) quit = true;
                else c.write(tile, pool + seg + SEG_HDR);
            }
            tile.sync();
            if (!quit && lane == 0)
                asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(a.done + j),
                             "l"((unsigned long long)(seg >> 2) << 32 | (unsigned)rows)
                             : "memory");
        }
        c.end(tile);
    }
    if (lane == 0) {
        if (quit) atomicExch(a.quit, 1);
        if (adds) {
            atomicAdd(&a.c.st->additions, (unsigned long long)adds);
            atomicAdd(&a.c.st->slots, (unsigned long long)slots);
        }
    }
}

// place[r] = events of the lows before r.  One CTA.
__global__ void __launch_bounds__(1024) k_row_places(RowArgs a) {
    __shared__ int s_sum[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    int run = 0;
    for (int64_t r0 = 0; r0 < a.m; r0 += 1024) {
        const int64_t r = r0 + tid;
        const int x = r < a.m ? a.count[r] : 0;
        int incl = x;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) s_sum[wid] = incl;
        __syncthreads();
        const int w = s_sum[lane];
        const int before = __reduce_add_sync(0xffffffffu, lane < wid ? w : 0);
        if (r < a.m) a.place[r] = run + before + incl - x;
        run += __reduce_add_sync(0xffffffffu, w);
        __syncthreads();
    }
}
__global__ void k_row_scatter(RowArgs a) {
    if (*a.quit) return;
    const unsigned n = *a.n_ev;
    for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
        a.sorted[atomicAdd(a.place + a.ev_low[e], 1)] = a.ev[e];
}
// A low a warp.  Rows come in descending order, so the columns that are first
// when they come are found by steps: of those left of the first so far, the
// ones over the largest row, and the leftmost of them.
__global__ void __launch_bounds__(256) k_row_marks(RowArgs a) {
    if (*a.quit) return;
    const int lane = threadIdx.x & 31;
    for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < a.m;
         r += (int64_t)gridDim.x * blockDim.x >> 5) {
        const int n = a.count[r];
        const int2 *const ev = a.sorted + (a.place[r] - n);  // place: past them, after the scatter
        for (int first = a.first[r];;) {
            int row = -1, col = INT_MAX;
            for (int i = lane; i < n; i += 32) {
                const int2 e = ev[i];
                if (e.y < first && (e.x > row || (e.x == row && e.y < col))) row = e.x, col = e.y;
            }
            const int top = __reduce_max_sync(0xffffffffu, row);
            if (top < 0) break;
            first = __reduce_min_sync(0xffffffffu, row == top ? col : INT_MAX);
            if (lane == 0) a.ess[first] = a.ess[r] = 0;
        }
    }
}
__global__ void k_row_ones(int64_t m, int32_t *ess) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) ess[j] = 1;
}

// Row buckets: every column with a low joins the bucket of that row;
// pivots[r] = the first column holding low r (ph_row.cu:56-59).
__global__ void k_row_buckets(SeqArgs a) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < a.m; j += (int64_t)gridDim.x * blockDim.x) {
        int lj = a.low[j];
        if (lj >= 0) {
            a.bnext[j] = atomicExch(&a.bhead[lj], (int)j);
            atomicAdd(&a.bcnt[lj], 1);
            atomicMin(&a.arglow[lj], (int)j);
        }
    }
}

constexpr int ROW_THREADS = 1024;
constexpr int ROW_CAP = 512;

// The row algorithm (ph_row.cu:38-121 / ph_row_parallel.cu:20-89): for rows
// i = m-1 .. 0, the first column with low i is added into every other column
// with low i; those move to the buckets of their new lows.  With row_quirk
// the running ess estimate of the reference CPU form is kept: before each
// addition the row and the pivot pair are marked non-essential, and after it
// a column that is now the first ever to hold its new low is marked
// non-essential together with that low (ph_row.cu:2-31).
__global__ void __launch_bounds__(ROW_THREADS) k_row_walk(SeqArgs a) {
    extern __shared__ int smem[];
    __shared__ long long s_row;
    __shared__ int s_n, s_piv;
    const int wid = threadIdx.x >> 5;
    auto tile = cg::tiled_partition<32>(cg::this_thread_block());
    const int lane = tile.thread_rank();
    int *sA = smem + (size_t)wid * 3 * ROW_CAP, *sB = sA + ROW_CAP, *sC = sB + ROW_CAP;
    long long adds = 0, slots = 0;
    long long i = a.start_pos;
    __shared__ int s_fail;
    if (threadIdx.x == 0) s_fail = 0;
    if (a.ev && threadIdx.x == 0) {
        long long *t0 = reinterpret_cast<long long *>(a.ev) - 2;
        if (*t0 == 0) *t0 = global_ns();  // the first launch of the walk
    }
    while (i >= 0) {
        if (wid == 0) {
            long long r = i, found = -1;
            while (r >= 0) {
                long long rr = r - lane;
                int c = rr >= 0 ? a.bcnt[rr] : 0;
                unsigned b = tile.ballot(c >= 2);
                if (b) { found = r - (__ffs(b) - 1); break; }
                r -= 32;
            }
            if (lane == 0) {
                s_row = found;
                if (found >= 0) {
                    int n = 0, piv = 0x7fffffff;
                    for (int c = a.bhead[found]; c != -1; c = a.bnext[c]) {
                        a.blist[n++] = c;
                        piv = min(piv, c);
                    }
                    s_n = n;
                    s_piv = piv;
                    a.bhead[found] = -1;
                    a.bcnt[found] = 0;
                    if (a.row_quirk) { a.ess[found] = 0; a.ess[piv] = 0; }
                }
            }
        }
        __syncthreads();
        i = s_row;
        if (i < 0) break;
        const int n = s_n, piv = s_piv;
        for (int k = wid; k < n; k += ROW_THREADS / 32) {
            const int j = a.blist[k];
            if (j == piv) continue;
            bool once = true;
            auto next = [&](int) { int p = once ? piv : -1; once = false; return p; };
            const int nl = chain(tile, a, j, sA, sB, sC, ROW_CAP, next, adds, slots);
            if (nl == -2) {
                if (lane == 0) s_fail = 1;
                continue;
            }
            if (nl >= 0 && lane == 0) {
                a.bnext[j] = atomicExch(&a.bhead[nl], j);
                atomicAdd(&a.bcnt[nl], 1);
                atomicMin(&a.arglow[nl], j);
            }
        }
        __syncthreads();
        if (s_fail) break;
        if (a.ev && threadIdx.x == 0) {
            // the row's additions, for the host's tracker replay (a row that
            // failed is walked again after the regrow, and logged then)
            long long *len = reinterpret_cast<long long *>(a.ev) - 1;
            const long long at = *len, need = 5 + 2ll * (n - 1);
            if (at >= 0 && at + need <= a.ev_cap) {
                int *e = a.ev + at;
                const long long t = global_ns();
                e[0] = (int)i;
                e[1] = piv;
                e[2] = n - 1;
                e[3] = (int)(t & 0xffffffffll);
                e[4] = (int)(t >> 32);
                int q = 5;
                for (int k = 0; k < n; k++) {
                    const int j = a.blist[k];
                    if (j == piv) continue;
                    e[q++] = j;
                    e[q++] = a.low[j];
                }
                *len = at + need;
            } else {
                *len = -1;  // out of room: the host keeps the final entry only
            }
        }
        if (a.row_quirk) {
            for (int k = threadIdx.x; k < n; k += ROW_THREADS) {
                const int j = a.blist[k];
                if (j == piv) continue;
                const int nl = a.low[j];
                if (nl >= 0 && a.arglow[nl] == j) { a.ess[j] = 0; a.ess[nl] = 0; }
            }
        }
        __syncthreads();
        i--;
    }
    if (threadIdx.x == 0) {
        // a failed addition leaves its column unchanged but the row's bucket
        // was consumed; report the row so the host restarts the whole walk
        a.st->resume_pos = s_fail ? i : -1;
    }
    if (lane == 0 && adds) {
        atomicAdd(&a.st->additions, (unsigned long long)adds);
        atomicAdd(&a.st->slots, (unsigned long long)slots);
    }
}

// For twist, into the status: the largest dimension, the columns of dimension
// >= 1, and whether the dimensions from 1 up separate: each has its rows in
// one lower dimension, no two in the same.  seen[d], seen[128 + d]: 128 - the
// smallest and 2 + the largest dimension of a row in a column of dimension d;
// the last block looks at them.
__global__ void __launch_bounds__(256) k_dim_stats(const int8_t *dim, const int64_t *colptr, const int32_t *rows,
                                                   int64_t m, int *seen, DevStatus *st) {
    __shared__ int s_seen[256], s_last;
    if (st->error) return;
    for (int q = threadIdx.x; q < 256; q += blockDim.x) s_seen[q] = 0;
    __syncthreads();
    int mx = -1, cnt = 0;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
        const int d = dim[j];
        mx = max(mx, d);
        if (d < 1) continue;
        cnt++;
        int lo = 126, hi = -1;
        for (int64_t k = colptr[j]; k < colptr[j + 1]; k++) {
            const int r = dim[rows[k]];
            lo = min(lo, r);
            hi = max(hi, r);
        }
        if (128 - lo > s_seen[d]) atomicMax(&s_seen[d], 128 - lo);
        if (hi + 2 > s_seen[128 + d]) atomicMax(&s_seen[128 + d], hi + 2);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&st->seq_top, mx + 2);
        if (cnt) atomicAdd(&st->seq_cols, cnt);
    }
    __syncthreads();
    if (s_seen[threadIdx.x]) atomicMax(&seen[threadIdx.x], s_seen[threadIdx.x]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&st->seq_blocks, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    s_seen[threadIdx.x] = 0;
    __syncthreads();
    bool ok = true;
    const int d = threadIdx.x;
    if (d >= 1 && d < 128) {
        const int lo = __ldcg(seen + d), hi = __ldcg(seen + 128 + d);
        if (hi) ok = 128 - lo == hi - 2 && hi - 2 < d && atomicAdd(&s_seen[hi - 1], 1) == 0;
    }
    if (__syncthreads_and(ok) && threadIdx.x == 0) st->seq_separate = 1;
}

int dim_stats(Context *ctx, const Work &w) {
    if (w.m == 0) return OPH_OK;
    int *seen = (int *)ctx_alloc(ctx, S_SEQNS, sizeof(int) * 256);
    if (!seen) return OPH_ERR_OOM;
    OPH_CUDA_TRY(cudaMemsetAsync(seen, 0, sizeof(int) * 256, ctx->stream));
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((w.m + 255) / 256, (int64_t)ctx->sm_count * 16));
    k_dim_stats<<<grid, 256, 0, ctx->stream>>>(w.dim, w.colptr, w.rows, w.m, seen, w.st);
    ctx->launches++;
    OPH_CUDA_TRY(cudaGetLastError());
    return OPH_OK;
}

// standard (all columns at once) or twist (dimension top down to 1) by
// k_claim; the store grown and the given-up columns redone when it runs out.
template <class Column>
static int claim_columns_as(Context *ctx, Work &w, int words, int top, bool twist, int *regrows) {
    cudaStream_t s = ctx->stream;
    const int64_t m = w.m;
    static PerDevice attr;
    if (!allow_shared(attr, ctx->device, k_claim<Column>, sizeof(int) * CL_WARPS * CL_BITS)) return OPH_ERR_CUDA;
    const size_t smem = sizeof(int) * CL_WARPS * (size_t)words;
    ClaimArgs a{};
    a.m = m; a.low = w.low; a.dim = w.dim; a.pool = w.pool; a.st = w.st; a.seg = w.seg; a.words = words;
    static_assert(sizeof(Holder) <= sizeof(PivRec), "the holders stand in the pivot records' buffer");
    a.holder = reinterpret_cast<Holder *>(w.rec);
    OPH_CUDA_TRY(cudaMemsetAsync(a.holder, 0xff, sizeof(Holder) * (size_t)m, s));
    const int dims = twist ? top : 1;  // launches: one for all columns, or a dimension each from the top
    if (dims < 1) return OPH_OK;       // twist leaves dimensions 0 and below as they are
    const size_t head = (sizeof(ClaimCount) * (size_t)dims + 255) & ~(size_t)255;
    char *tmp = (char *)ctx_alloc(ctx, S_TMP, head + sizeof(int32_t) * 2 * (size_t)m);
    if (!tmp) return OPH_ERR_OOM;
    ClaimCount *count = reinterpret_cast<ClaimCount *>(tmp);
    int32_t *lists[2] = {reinterpret_cast<int32_t *>(tmp + head), reinterpret_cast<int32_t *>(tmp + head) + m};
    a.above = count;
    const int64_t per_sm = std::min<int64_t>(2048 / CL_THREADS, (220 << 10) / (smem + 2048));
    const int grid = (int)std::min<int64_t>((m + CL_WARPS - 1) / CL_WARPS, ctx->sm_count * per_sm);
    const int grid_m = (int)std::max<int64_t>(1, std::min<int64_t>((m + 255) / 256, (int64_t)ctx->sm_count * 16));
    // in the context's second pinned status block where it holds them
    std::vector<ClaimCount> many(sizeof(ClaimCount) * (size_t)dims > sizeof(DevStatus) ? dims : 0);
    ClaimCount *const seen = many.empty() ? reinterpret_cast<ClaimCount *>(ctx->h_status + 1) : many.data();
    int turn = 0, d = 0, redo = 0;
    for (;;) {
        OPH_CUDA_TRY(cudaMemsetAsync(count, 0, sizeof(ClaimCount) * (size_t)dims, s));
        for (int e = d; e < dims; e++) {
            a.want_dim = twist ? top - e : -1;
            a.redo = e == d && redo ? lists[turn ^ 1] : nullptr;
            a.n = a.redo ? redo : m;
            a.failed = lists[turn];
            a.count = count + e;
            a.n_above = e;
            k_claim<Column><<<grid, CL_THREADS, smem, s>>>(a);
            ctx->launches++;
            if (twist) {
                k_claim_clear<<<grid_m, 256, 0, s>>>(a);
                ctx->launches++;
            }
        }
        OPH_CUDA_TRY(cudaGetLastError());
        OPH_CUDA_TRY(cudaMemcpyAsync(seen, count, sizeof(ClaimCount) * (size_t)dims, cudaMemcpyDeviceToHost, s));
        OPH_CUDA_TRY(cudaMemcpyAsync(ctx->h_status, w.st, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
        OPH_CUDA_TRY(cudaStreamSynchronize(s));
        while (d < dims && !seen[d].failed) d++;
        if (d == dims) return OPH_OK;
        redo = seen[d].failed;
        const int rc = grow_pool(ctx, w);
        if (rc != OPH_OK) return rc;
        a.pool = w.pool;
        turn ^= 1;
        (*regrows)++;
    }
}

// Bitmaps where a warp's holds every row, else lists.
static int claim_columns(Context *ctx, Work &w, int top, bool twist, int *regrows) {
    const int64_t words = ((w.m + 31) / 32 + 31) / 32 * 32;
    if (words <= CL_BITS) return claim_columns_as<BitColumn>(ctx, w, (int)words, top, twist, regrows);
    return claim_columns_as<ListColumn>(ctx, w, 3 * CL_CAP, top, twist, regrows);
}

// The row form's running estimate in ess[], after claim_columns; *done false
// (ess as it was) when events or columns find no room.
template <class Column>
static int row_estimate(Context *ctx, Work &w, int words, int32_t *ess, bool *done) {
    cudaStream_t s = ctx->stream;
    const int64_t m = w.m;
    *done = false;
    const int64_t cap = std::min<int64_t>(16 * m + (1 << 16), 1ll << 30);
    auto r256 = [](size_t n) { return (n + 255) & ~(size_t)255; };
    const size_t at[] = {r256(256 + sizeof(ClaimCount)), r256(8 * (size_t)m), r256(4 * (size_t)m), r256(4 * (size_t)m),
                         r256(4 * (size_t)m), r256(4 * (size_t)cap), r256(8 * (size_t)cap), r256(8 * (size_t)cap)};
    size_t off[9] = {};
    for (int q = 0; q < 8; q++) off[q + 1] = off[q] + at[q];
    char *tmp = (char *)ctx_alloc(ctx, S_ROWEST, off[8]);
    if (!tmp) return OPH_OK;
    RowArgs a{};
    a.m = m; a.colptr = w.colptr; a.ess = ess; a.cap = (unsigned)cap;
    a.holder = reinterpret_cast<const Holder *>(w.rec);
    a.n_ev = reinterpret_cast<unsigned *>(tmp);
    a.quit = reinterpret_cast<int *>(tmp + 64);
    a.c.count = reinterpret_cast<ClaimCount *>(tmp + 128);
    a.done = reinterpret_cast<unsigned long long *>(tmp + off[1]);
    a.count = reinterpret_cast<int *>(tmp + off[2]);
    a.first = reinterpret_cast<int *>(tmp + off[3]);
    a.place = reinterpret_cast<int *>(tmp + off[4]);
    a.ev_low = reinterpret_cast<int *>(tmp + off[5]);
    a.ev = reinterpret_cast<int2 *>(tmp + off[6]);
    a.sorted = reinterpret_cast<int2 *>(tmp + off[7]);
    a.c.m = m; a.c.pool = w.pool; a.c.st = w.st; a.c.words = words;
    OPH_CUDA_TRY(cudaMemsetAsync(tmp, 0, off[3], s));
    OPH_CUDA_TRY(cudaMemsetAsync(a.first, 0x7f, 4 * (size_t)m, s));
    OPH_CUDA_TRY(cudaMemsetAsync(&w.st->additions, 0, 2 * sizeof(unsigned long long), s));  // these are the row form's
    static PerDevice attr;
    if (!allow_shared(attr, ctx->device, k_row_exact<Column>, sizeof(int) * CL_WARPS * CL_BITS)) return OPH_ERR_CUDA;
    const size_t smem = sizeof(int) * CL_WARPS * (size_t)words;
    const int64_t per_sm = std::min<int64_t>(2048 / CL_THREADS, (220 << 10) / (smem + 2048));
    const int grid = (int)std::min<int64_t>((m + CL_WARPS - 1) / CL_WARPS, ctx->sm_count * per_sm);
    const int grid_m = (int)std::max<int64_t>(1, std::min<int64_t>((m + 255) / 256, (int64_t)ctx->sm_count * 16));
    k_row_exact<Column><<<grid, CL_THREADS, smem, s>>>(a);
    k_row_places<<<1, 1024, 0, s>>>(a);
    k_row_scatter<<<ctx->sm_count * 4, 256, 0, s>>>(a);
    k_row_marks<<<ctx->sm_count * 8, 256, 0, s>>>(a);
    ctx->launches += 4;
    OPH_CUDA_TRY(cudaGetLastError());
    int *const quit = reinterpret_cast<int *>(ctx->h_status + 1);
    OPH_CUDA_TRY(cudaMemcpyAsync(quit, a.quit, sizeof(int), cudaMemcpyDeviceToHost, s));
    OPH_CUDA_TRY(cudaMemcpyAsync(ctx->h_status, w.st, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
    OPH_CUDA_TRY(cudaStreamSynchronize(s));
    *done = !*quit;
    if (*quit) {
        k_row_ones<<<grid_m, 256, 0, s>>>(m, ess);
        ctx->launches++;
    }
    return OPH_OK;
}
static int row_estimate(Context *ctx, Work &w, int32_t *ess, bool *done) {
    const int64_t words = ((w.m + 31) / 32 + 31) / 32 * 32;
    if (words <= CL_BITS) return row_estimate<BitColumn>(ctx, w, (int)words, ess, done);
    return row_estimate<ListColumn>(ctx, w, 3 * CL_CAP, ess, done);
}

// The columns as they came, for a walk after columns side by side did not fit.
static int restart_store(Context *ctx, Work &w, SeqArgs &a) {
    const int rc = setup_store(ctx, w, false);
    if (rc) return rc;
    ctx->launches++;
    a.low = w.low; a.dim = w.dim; a.seg = w.seg; a.pool = w.pool; a.st = w.st;
    return OPH_OK;
}

int run_sequential(Context *ctx, Work &w, int algo, int32_t *d_ess, oph_info *info) {
    cudaStream_t s = ctx->stream;
    const int64_t m = w.m;
    SeqArgs a{};
    a.m = m; a.low = w.low; a.dim = w.dim; a.seg = w.seg; a.pool = w.pool; a.st = w.st;
    a.arglow = w.first;  // reuse: int32[m]
    const bool row = algo == OPH_ALGO_PH_ROW || algo == OPH_ALGO_PH_ROW_PARALLEL;
    const int grid_m = (int)std::max<int64_t>(1, std::min<int64_t>((m + 255) / 256, (int64_t)ctx->sm_count * 16));
    cudaEventRecord(ctx->ev[0], s);
    int regrows = 0;
    long long iters = m + 1;
    if (!row) {
        a.twist = (algo == OPH_ALGO_TWIST || algo == OPH_ALGO_TWIST_PARALLEL);
        const DevStatus set_up = *ctx->h_status;  // as the set-up left it (dim_stats)
        const int maxdim = a.twist ? set_up.seq_top - 2 : 0;
        a.max_dim = maxdim;
        a.start_dim = a.twist ? maxdim : 0;
        a.start_pos = 0;
        if (a.twist && maxdim < 1) a.start_dim = 0;  // nothing to reduce: the loop below runs no dimension
        // the reference counts one iteration per column visited
        // (twist.cu:36-86 visits the columns of dimension >= 1)
        if (a.twist) iters = 1 + (long long)set_up.seq_cols;
        SeqTracking *tk = ctx->seq_track;
        a.it_base = 1;
        // side by side, unless the walk itself is asked for, or twist's
        // clearing could depend on its order
        bool side_by_side = !tk && (!a.twist || set_up.seq_separate);
        if (side_by_side) {
            int rc = claim_columns(ctx, w, a.twist ? maxdim : -1, a.twist != 0, &regrows);
            if (rc == OPH_ERR_OOM || rc == OPH_ERR_OVERFLOW) {  // the walk writes less: it may still fit
                side_by_side = false;
                ctx_release(ctx, S_TMP);
                rc = restart_store(ctx, w, a);
            }
            if (rc) return rc;
        }
        if (tk) {
            // the state the host replays from, and a stamp per iteration
            tk->iters = iters;
            tk->low0.resize(m);
            tk->dim.resize(m);
            a.it_ns = (long long *)ctx_alloc(ctx, S_SEQNS, sizeof(long long) * (size_t)(iters + 1));
            if (!a.it_ns) return OPH_ERR_OOM;
            OPH_CUDA_TRY(cudaMemsetAsync(a.it_ns, 0, sizeof(long long) * (size_t)(iters + 1), s));
            OPH_CUDA_TRY(cudaMemcpyAsync(tk->low0.data(), w.low, sizeof(int32_t) * m, cudaMemcpyDeviceToHost, s));
            OPH_CUDA_TRY(cudaMemcpyAsync(tk->dim.data(), w.dim, (size_t)m, cudaMemcpyDeviceToHost, s));
            OPH_CUDA_TRY(cudaStreamSynchronize(s));
        }
        if (!side_by_side) OPH_CUDA_TRY(cudaMemsetAsync(a.arglow, 0xff, sizeof(int32_t) * m, s));
        static PerDevice attr;
        const size_t smem = 3 * SEQ_CAP * sizeof(int);
        if (!allow_shared(attr, ctx->device, k_seq_walk, smem)) return OPH_ERR_CUDA;
        if (!side_by_side && !(a.twist && maxdim < 1)) {
            for (;;) {
                k_seq_walk<<<1, 32, smem, s>>>(a);
                ctx->launches++;
                OPH_CUDA_TRY(cudaGetLastError());
                OPH_CUDA_TRY(cudaMemcpyAsync(ctx->h_status, w.st, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
                OPH_CUDA_TRY(cudaStreamSynchronize(s));
                if (ctx->h_status->resume_pos < 0) break;
                int g = grow_pool(ctx, w);
                if (g != OPH_OK) return g;
                a.pool = w.pool;
                a.start_dim = ctx->h_status->resume_dim;
                a.start_pos = ctx->h_status->resume_pos;
                a.it_base = ctx->h_status->resume_iter;
                regrows++;
            }
        }
        if (tk) {
            tk->ns.resize(iters);
            if (a.twist && maxdim < 1) {
                std::fill(tk->ns.begin(), tk->ns.end(), 0ll);
            } else {
                OPH_CUDA_TRY(cudaMemcpyAsync(tk->ns.data(), a.it_ns, sizeof(long long) * iters, cudaMemcpyDeviceToHost, s));
                OPH_CUDA_TRY(cudaStreamSynchronize(s));
            }
        }
    } else {
        a.bhead = (int32_t *)ctx_alloc(ctx, S_TMP, sizeof(int32_t) * (3 * m + 1));
        if (!a.bhead) return OPH_ERR_OOM;
        a.bnext = a.bhead + m; a.bcnt = a.bnext + m;
        a.blist = w.worklist;
        a.ess = d_ess;
        a.row_quirk = (algo == OPH_ALGO_PH_ROW) && d_ess != nullptr;
        SeqTracking *tk = ctx->seq_track;
        long long *ev_base = nullptr;
        // without trackers: the lows, which are those of the columns side by
        // side, and the running estimate where it is asked for
        bool side_by_side = !tk;
        if (side_by_side) {
            int rc = claim_columns(ctx, w, -1, false, &regrows);
            bool done = rc == OPH_OK;
            if (done && a.row_quirk && w.nnz > 0) rc = row_estimate(ctx, w, d_ess, &done);
            if (rc && rc != OPH_ERR_OOM && rc != OPH_ERR_OVERFLOW) return rc;
            if (!done) {
                side_by_side = false;
                ctx_release(ctx, S_ROWEST);
                if ((rc = restart_store(ctx, w, a))) return rc;
                // the columns side by side used this slot
                a.bhead = (int32_t *)ctx_alloc(ctx, S_TMP, sizeof(int32_t) * (3 * m + 1));
                if (!a.bhead) return OPH_ERR_OOM;
                a.bnext = a.bhead + m; a.bcnt = a.bnext + m;
            }
        }
        if (tk) {
            // the initial lows and a log of the walk's additions for the
            // host's replay: {start ns, length} then the records
            tk->iters = iters;
            tk->low0.resize(m);
            OPH_CUDA_TRY(cudaMemcpyAsync(tk->low0.data(), w.low, sizeof(int32_t) * m, cudaMemcpyDeviceToHost, s));
            a.ev_cap = 8 * (long long)m + (1 << 20);
            ev_base = (long long *)ctx_alloc(ctx, S_SEQNS, 16 + sizeof(int) * (size_t)a.ev_cap);
            if (!ev_base) return OPH_ERR_OOM;
            OPH_CUDA_TRY(cudaMemsetAsync(ev_base, 0, 16, s));
            a.ev = reinterpret_cast<int *>(ev_base + 2);
        }
        static PerDevice attr;
        const size_t smem = (size_t)(ROW_THREADS / 32) * 3 * ROW_CAP * sizeof(int);
        if (!allow_shared(attr, ctx->device, k_row_walk, smem)) return OPH_ERR_CUDA;
        while (!side_by_side) {
            OPH_CUDA_TRY(cudaMemsetAsync(a.bhead, 0xff, sizeof(int32_t) * m, s));
            OPH_CUDA_TRY(cudaMemsetAsync(a.bcnt, 0, sizeof(int32_t) * m, s));
            OPH_CUDA_TRY(cudaMemsetAsync(a.arglow, 0x7f, sizeof(int32_t) * m, s));
            k_row_buckets<<<grid_m, 256, 0, s>>>(a);
            a.start_pos = m - 1;
            k_row_walk<<<1, ROW_THREADS, smem, s>>>(a);
            ctx->launches += 2;
            OPH_CUDA_TRY(cudaGetLastError());
            OPH_CUDA_TRY(cudaMemcpyAsync(ctx->h_status, w.st, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
            OPH_CUDA_TRY(cudaStreamSynchronize(s));
            if (ctx->h_status->resume_pos < 0) break;
            // rows are consumed as they are walked, so an interrupted walk
            // restarts from the (consistent) column state with rebuilt buckets
            int g = grow_pool(ctx, w);
            if (g != OPH_OK) return g;
            a.pool = w.pool;
            regrows++;
        }
        if (tk) {
            long long hdr[2] = {0, 0};
            OPH_CUDA_TRY(cudaMemcpyAsync(hdr, ev_base, 16, cudaMemcpyDeviceToHost, s));
            OPH_CUDA_TRY(cudaStreamSynchronize(s));
            tk->ev_t0 = hdr[0];
            tk->rows_ok = hdr[1] >= 0;
            tk->ev.resize(hdr[1] > 0 ? (size_t)hdr[1] : 0);
            if (!tk->ev.empty()) {
                OPH_CUDA_TRY(cudaMemcpyAsync(tk->ev.data(), a.ev, sizeof(int) * tk->ev.size(), cudaMemcpyDeviceToHost, s));
                OPH_CUDA_TRY(cudaStreamSynchronize(s));
            }
        }
    }
    cudaEventRecord(ctx->ev[1], s);
    OPH_CUDA_TRY(cudaEventSynchronize(ctx->ev[1]));
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
    DevStatus hs = *ctx->h_status;
    if (info) {
        info->sweeps = 0;
        info->num_iters = (int32_t)iters;
        info->additions = (int64_t)hs.additions;
        info->slots_moved = (int64_t)hs.slots;
        info->pool_bytes = (int64_t)hs.pool_used * 4;
        info->regrows = regrows;
        info->device_ms = ms;
    }
    return OPH_OK;
}

}  // namespace oph
