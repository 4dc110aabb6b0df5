// pms on filtered simplicial complexes of dimension <= 2, block by block,
// without the column store.
//
// The boundary matrix of such a complex has two blocks, which reduce
// independently but for clearing (a column only ever adds columns of its own
// dimension): the edges (two rows, both vertices) and the triangles (three
// rows, all edges).  low is unique for a reduced matrix, so any exact
// reduction of a block gives the lows the sweeps of pms.cu give.
//
// A block whose columns hold at most two rows is the incidence matrix of a
// graph, a column of one row an edge to a ground node.  Its reduction is the
// elder rule: the columns in order, each joining two components, the younger
// component's oldest node dying there; the reduced column is the two
// components' oldest nodes, its low the younger of them.  Edges are such a
// block of D; the triangles are one of the anti-transpose D' (dual.cu: a
// column per edge, holding its triangles) when no edge has more than two
// triangles (a triangulated surface with or without boundary: lower-star
// images).  The sweeps walk those unions one addition at a time, a chain of
// dependent loads; here every component finds its first outgoing edge at
// once and joins over it when that leads to an older component
// (k_c2_graph), which takes a dozen rounds.
//
// Triangles with more on an edge (Rips complexes) are reduced on D' too, but
// D' is never built column by column.  A Rips filtration puts the triangles
// right after their last edge, third vertices ascending, so a bit per edge and
// vertex names them all (runs; the whole complex is checked against that).
// Triangles in any other order are found through a table that holds, for
// every edge and vertex, the triangle they span, written with no count, scan,
// cursor or sort.  The edges that the graph of edges on vertices pairs are
// cleared (c2_kruskal); an edge whose first triangle has it as its last edge
// is paired with it at once, as nothing can be added to either (an apparent
// pair: 98-99% of a Rips complex's edges).  What is left (107 of 58,988 edges
// on the 5M-column torus) is reduced a column per CTA (k_c2_residual).
//
// Rips complexes that fit a CTA's shared memory go from colptr to runs in one
// launch, a CTA each (k_c2_inst; the larger ones of a batch in pieces,
// k_c2_inst_more); others by a launch per step over all columns.
//
// Which form (reduce_complex2): a single matrix of at most 2^15 columns, or a
// batch of at least 128 or of that size on average, as whole instances; else,
// or where one of them does not fit, the graph when three triangles come to
// at most two edges, the runs (unless the whole instances were found not to
// come in runs), the table.  A column of other width, found by the first kernel
// that looks, ends the attempt at once.
//
// What is accepted is checked on the device before it is reported: every
// column has 0, 2 or 3 rows, ascending and in range, the rows of an edge are
// vertices, the rows of a triangle are the three edges of a triangle (so
// D D = 0, which clearing relies on).  A column may come before its rows'
// columns (rows above the diagonal are accepted input): the graph takes any
// order, the runs know theirs, vertices first and every triangle in its last
// edge's run, and the table wants triangles after their edges.  Anything else,
// malformed input included, is left to the general path and its own checks.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <mutex>

#include "oph_host.h"

namespace oph {

// 32 columns: which are vertices (no rows) and edges (two rows), and how many
// vertices and edges come before them.  One 16-byte load gives a column's
// kind and its rank among its kind; half a byte a column, so the table of a
// complex stays in L1 / L2 where a rank per column would not.
struct C2Word {
    unsigned v, e;
    int vpre, epre;
};
// An instance of a batch (a single matrix is one): its vertices and edges
// among all, and its first column.
struct __align__(16) C2Inst {
    int voff, eoff, nv, ne;
    long long base, cols;
    long long coff, roff;  // its part of the table (cells) and of the runs' bits
    // words, lists and bitmaps hold its columns relative to wbase, its words
    // from woff on (0 where the words run through the whole batch)
    long long wbase, woff;
};
struct C2Status {
    int bad;         // a column or row that is none of the accepted kinds
    int crowded;     // an edge with more than two triangles
    int unfinished;  // the rounds ran out
    int rounds;
    long long nnz;
    int nv, ne;
    int live[3];     // edges left, by round modulo three
    unsigned arrived;  // blocks at the graph's meetings
    unsigned long long joins;
    int max_nv, max_cols;  // the largest instance's vertices, columns
    int unsorted;    // the triangles do not come in runs
    int next;        // whole instances: the CTAs' queue
    int refused;     //   an instance is too large, or no complex in runs
    int no_room;     //   the tables' bounds were too small
    int items, next_item;  // pieces of theirs, and their queue
    int nres, cursor, overflow;      // residual edges; the CTAs' queue; a list ran out of room
    int maps;                        // windows kept of published columns
    long long cells;                 // entries of the edge-vertex table
    long long pairs, run_words;      // entries of the edge-id table, words of the runs' bits
    unsigned long long cells_set;    // entries of the edge-vertex table that a triangle wrote
    unsigned long long arena;        // entries of published lists
    unsigned long long adds, slots;  // additions of the residual columns, entries toggled
};

constexpr int C2_THREADS = 256, C2_TILE = 2048;
constexpr int C2_MAX_ROUNDS = 512;
constexpr unsigned long long C2_FIRST_ROUND = 0xffffffffull << 32;  // the round in a key's upper half, counting down
constexpr int C2_MAX_NV = 8192;                   // vertices of an instance the dense form takes
// residual columns: pivots added at a time, at first and at most; a torus of
// 200K columns took 279 us with 32 at most, 264 with 64, 252 with 128, batches
// of 1,024 (columns of 2.6 waves) 1,646 us with 4 at first and 1,607 with 2
__host__ __device__ constexpr int rs_first(int threads) { return threads >= 1024 ? 4 : 2; }
__host__ __device__ constexpr int rs_wave(int threads) { return threads >= 1024 ? 128 : 32; }
// edges a column under reduction may be the sum of (2,700 on the torus, 600 on 120 points)
__host__ __device__ constexpr int rs_list(int threads) { return threads >= 1024 ? 16384 : 4096; }
constexpr int RS_FLAG = 1 << 30;
// Many vertices: long rows and few, long residual columns, so large CTAs and
// windows; below, more CTAs.  The table form takes large ones always: its
// columns, of random orders above all, are sums of sums, whose lists grow with
// every addition, while published windows add at once.  Up to 2^18 columns an
// instance (RS_XL_WORDS: 1.3M) one window holds them all and no list is kept.  A
// random order of all simplices on 40 points took 1,905 us with small CTAs, 452
// with large ones, 388 without lists; on 60 points the lists ran out after 430
// us (and the column store took 1,700), now 615.  Where all columns are short, on
// a grid of 125 points, small CTAs took 303 us, large ones take 325.
constexpr int RS_MAPS = 512;  // windows of published columns kept, 16 MB
constexpr int RS_SMALL_NV = 160, RS_SMALL = 256, RS_SMALL_WORDS = 4096, RS_LARGE = 1024, RS_LARGE_WORDS = 8192, RS_XL_WORDS = 40960;

struct C2Args {
    int64_t m;
    const int64_t *colptr;
    const int32_t *rows;
    const int64_t *inst_off;  // nullptr: one matrix
    int count;
    C2Word *words;
    int2 *tiles;
    int *winst;               // per word: the instance of its first column (batches)
    C2Inst *inst;
    C2Status *st;
    int32_t *vlist, *elist;   // column of each vertex, edge
    int4 *erec;               // per edge: its vertices (ranks), its instance
    // the graph of both blocks: nodes are the vertices by rank, the ground,
    // then the triangles from the last to the first (ids ascend from the
    // oldest node of each block); slot s < ne is edge s of D, slot
    // 2 ne - 1 - k edge k of D' (slots ascend in each block's column order)
    int2 *ends;
    int *parent;
    unsigned long long *best;
    int32_t *list[2];
    int32_t *tlist;           // column of each triangle
    int32_t *low, *ess;       // outputs
    int one_based;
    // dense forms: the vertex that dies at each edge (-1: none) and which
    // vertices die; the edge-vertex table or, with runs, the edge-id table
    // (vertices by vertices), its rows in edge order, the same table of edge
    // columns, and the runs (per edge and 32 vertices: which have a triangle,
    // and the first one's column); which triangles have an
    // owner (low[] names it), and which for good; the residual edges, and the
    // list each is the sum of (offset << 24 | length)
    int32_t *neg;
    uint8_t *dead;
    int32_t *cells, *adj, *tab;
    uint2 *runs;
    uint32_t *owned, *fixed;
    int32_t *res;
    unsigned long long *sum;
    int32_t *arena;
    long long arena_cap;
    int32_t *lists;           // per CTA: rs_list() edges
    uint32_t *maps;           // large CTAs: windows of published columns, map_cap of map_words
    int map_cap, map_words;
    int whole;                // table: a window holds every column of an instance, and no list is kept
    // whole instances: what the tables hold (edges, vertices, table entries, run words)
    long long cap_e, cap_v, cap_c, cap_r;
    long long nnz;            //   and the entries rows[] holds (-1: colptr[m], one matrix)
    int *order;               //   the order they are taken in (nullptr: as they come)
    int2 *items;              //   pieces left to k_c2_inst_more: instance, first edge
    int split_cols;           //   of instances of more columns
    int chunk;                //   edges of a piece, a multiple of 8 (0: nothing is left to it)
};

__device__ __forceinline__ unsigned below(int bit) { return (1u << bit) - 1u; }

// One pass over colptr: the kind of every column, ranks within the tile.
// Bound by HBM (8 bytes a column in, half a byte out).  A warp takes 256
// consecutive columns, 32 a step, so the loads are coalesced and the bits
// come from ballots.
__global__ void __launch_bounds__(C2_THREADS) k_c2_words(C2Args a) {
    __shared__ int s_v[C2_THREADS / 32], s_e[C2_THREADS / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t nwords = (a.m + 31) >> 5;
    bool bad = false;
    if (blockIdx.x == 0 && threadIdx.x == 0 && a.colptr[0] != 0) bad = true;
    for (int64_t tile = blockIdx.x; tile * C2_TILE < a.m; tile += gridDim.x) {
        const int64_t j0 = tile * C2_TILE + wid * 256;
        unsigned vb = 0, eb = 0;  // lane i keeps step i's bits
        int64_t c[9];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int64_t j = j0 + i * 32 + lane;
            c[i] = a.colptr[j < a.m ? j : a.m];
        }
        c[8] = j0 + 256 <= a.m ? a.colptr[j0 + 256] : a.colptr[a.m];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int64_t j = j0 + i * 32 + lane;
            const int64_t first = i < 7 ? __shfl_sync(0xffffffffu, c[i + 1], 0) : c[8];
            int64_t next = __shfl_down_sync(0xffffffffu, c[i], 1);
            if (lane == 31) next = first;
            const int64_t n = next - c[i];
            const bool in = j < a.m;
            if (in && n != 0 && n != 2 && n != 3) bad = true;
            const unsigned v = __ballot_sync(0xffffffffu, in && n == 0), e = __ballot_sync(0xffffffffu, in && n == 2);
            if (lane == i) {
                vb = v;
                eb = e;
            }
        }
        const int nv = __popc(vb), ne = __popc(eb);
        int iv = nv, ie = ne;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, iv, o), w = __shfl_up_sync(0xffffffffu, ie, o);
            if (lane >= o) {
                iv += u;
                ie += w;
            }
        }
        if (lane == 7) {
            s_v[wid] = iv;
            s_e[wid] = ie;
        }
        __syncthreads();
        int pv = 0, pe = 0, tv = 0, te = 0;
#pragma unroll
        for (int w = 0; w < C2_THREADS / 32; w++) {
            if (w < wid) {
                pv += s_v[w];
                pe += s_e[w];
            }
            tv += s_v[w];
            te += s_e[w];
        }
        const int64_t w = (j0 >> 5) + lane;
        if (lane < 8 && w < nwords)
            *reinterpret_cast<int4 *>(a.words + w) = make_int4((int)vb, (int)eb, pv + iv - nv, pe + ie - ne);
        if (threadIdx.x == 0) a.tiles[tile] = make_int2(tv, te);
        __syncthreads();
    }
    if (bad) a.st->bad = 1;
}

// The pitch of an instance's rows over its vertices: whole words of them.
__host__ __device__ __forceinline__ int c2_pitch(int nv) { return (nv + 31) & ~31; }

// Exclusive prefix over the block of 1024 threads; red holds 33 values.
__device__ __forceinline__ long long c2_block_excl(long long v, long long *red, long long *total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) red[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        const long long t = red[lane];
        long long ti = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, ti, o);
            if (lane >= o) ti += u;
        }
        red[lane] = ti - t;
        if (lane == 31) red[32] = ti;
    }
    __syncthreads();
    const long long out = red[wid] + incl - v;
    *total = red[32];
    __syncthreads();
    return out;
}

// Vertices and edges before column j (tile prefixes and in-tile ranks).
__device__ __forceinline__ int2 c2_rank_tiled(const C2Args &a, int64_t j) {
    if (j >= a.m) return make_int2(a.st->nv, a.st->ne);
    const int2 t = a.tiles[j / C2_TILE];
    const C2Word w = a.words[j >> 5];
    const unsigned lt = below((int)(j & 31));
    return make_int2(t.x + w.vpre + __popc(w.v & lt), t.y + w.epre + __popc(w.e & lt));
}

// One block: the tiles' prefixes (vertices in the low, edges in the high half
// of one 64-bit scan), the totals, and the instances' shares.
__global__ void __launch_bounds__(1024) k_c2_scan(C2Args a, int64_t ntiles) {
    __shared__ long long red[33];
    constexpr int ITEMS = 8;
    long long carry = 0;
    for (int64_t t0 = 0; t0 < ntiles; t0 += 1024 * ITEMS) {
        long long v[ITEMS], sum = 0, total;
#pragma unroll
        for (int q = 0; q < ITEMS; q++) {
            const int64_t t = t0 + (int64_t)threadIdx.x * ITEMS + q;
            const int2 x = t < ntiles ? a.tiles[t] : make_int2(0, 0);
            v[q] = ((long long)x.y << 32) + x.x;
            sum += v[q];
        }
        long long run = carry + c2_block_excl(sum, red, &total);
#pragma unroll
        for (int q = 0; q < ITEMS; q++) {
            const int64_t t = t0 + (int64_t)threadIdx.x * ITEMS + q;
            if (t < ntiles) a.tiles[t] = make_int2((int)(run & 0xffffffffll), (int)(run >> 32));
            run += v[q];
        }
        carry += total;
    }
    if (threadIdx.x == 0) {
        a.st->nv = (int)(carry & 0xffffffffll);
        a.st->ne = (int)(carry >> 32);
        a.st->nnz = a.colptr[a.m];
        if (!a.inst_off) {
            C2Inst s{};
            s.nv = a.st->nv;
            s.ne = a.st->ne;
            s.cols = a.m;
            a.inst[0] = s;
            a.st->max_nv = s.nv;
            a.st->max_cols = (int)a.m;
            a.st->cells = (long long)c2_pitch(s.nv) * s.ne;
            a.st->pairs = (long long)c2_pitch(s.nv) * s.nv;
            a.st->run_words = (long long)((s.nv + 31) >> 5) * s.ne;
        }
    }
    __syncthreads();
    if (!a.inst_off) return;
    long long cells = 0, pairs = 0, words = 0;
    for (int b0 = 0; b0 < a.count; b0 += 1024) {
        const int b = b0 + (int)threadIdx.x;
        C2Inst s{};
        if (b < a.count) {
            const int64_t o0 = a.inst_off[b], o1 = a.inst_off[b + 1];
            if (o0 < 0 || o1 < o0 || o1 > a.m || (b == 0 && o0 != 0) || (b == a.count - 1 && o1 != a.m)) {
                a.st->bad = 1;
            } else {
                const int2 r0 = c2_rank_tiled(a, o0), r1 = c2_rank_tiled(a, o1);
                s.voff = r0.x;
                s.eoff = r0.y;
                s.nv = r1.x - r0.x;
                s.ne = r1.y - r0.y;
                s.base = o0;
                s.cols = o1 - o0;
                atomicMax(&a.st->max_nv, s.nv);
                atomicMax(&a.st->max_cols, (int)s.cols);
                if (s.ne == 0 && s.nv != s.cols) a.st->bad = 1;  // triangles, but no edges for their rows
            }
        }
        // coff serves the form tried first (runs); the table's is k_c2_cells'
        long long total;
        s.coff = pairs + c2_block_excl((long long)c2_pitch(s.nv) * s.nv, red, &total);
        pairs += total;
        s.roff = words + c2_block_excl((long long)((s.nv + 31) >> 5) * s.ne, red, &total);
        words += total;
        c2_block_excl((long long)c2_pitch(s.nv) * s.ne, red, &total);
        cells += total;
        if (b < a.count) a.inst[b] = s;
    }
    if (threadIdx.x == 0) {
        a.st->cells = cells;
        a.st->pairs = pairs;
        a.st->run_words = words;
    }
}

// The instances' parts of the edge-vertex table (one block).
__global__ void __launch_bounds__(1024) k_c2_cells(C2Args a) {
    __shared__ long long red[33];
    long long cells = 0, total;
    for (int b0 = 0; b0 < a.count; b0 += 1024) {
        const int b = b0 + (int)threadIdx.x;
        const long long n = b < a.count ? (long long)c2_pitch(a.inst[b].nv) * a.inst[b].ne : 0;
        const long long off = cells + c2_block_excl(n, red, &total);
        cells += total;
        if (b < a.count) a.inst[b].coff = off;
    }
}

// A thread per word: absolute ranks, the lists of vertices and edges, the
// instance of the word's first column.
__global__ void __launch_bounds__(C2_THREADS) k_c2_lists(C2Args a) {
    const int64_t nwords = (a.m + 31) >> 5;
    for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < nwords; w += (int64_t)gridDim.x * blockDim.x) {
        const int2 t = a.tiles[(w << 5) / C2_TILE];
        C2Word x = a.words[w];
        x.vpre += t.x;
        x.epre += t.y;
        a.words[w].vpre = x.vpre;
        a.words[w].epre = x.epre;
        int k = x.vpre;
        for (unsigned b = x.v; b; b &= b - 1) a.vlist[k++] = (int32_t)(w << 5) + __ffs(b) - 1;
        k = x.epre;
        for (unsigned b = x.e; b; b &= b - 1) a.elist[k++] = (int32_t)(w << 5) + __ffs(b) - 1;
        if (a.inst_off) {
            int lo = 0, hi = a.count;
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (a.inst_off[mid] <= (w << 5)) lo = mid;
                else hi = mid;
            }
            a.winst[w] = lo;
        }
    }
}

// The instance of column j: its word's, or one of the next ones.
__device__ __forceinline__ int c2_inst_of(const C2Args &a, int64_t j) {
    if (!a.inst_off) return 0;
    int b = a.winst[j >> 5];
    while (b + 1 < a.count && a.inst_off[b + 1] <= j) b++;
    return b;
}

// The triangle's third vertex seen from each edge, when three edges (their
// vertex pairs) are the edges of one triangle.
__device__ __forceinline__ bool c2_opposite(const int4 &e0, const int4 &e1, const int4 &e2, int &w0, int &w1, int &w2) {
    const int a = e0.x, b = e0.y;
    const int p = (e1.x == a || e1.x == b) ? e1.x : e1.y;  // the vertex of e0 and e1
    const int o = e1.x ^ e1.y ^ p, q = a ^ b ^ p;
    w0 = o;
    w1 = q;
    w2 = p;
    return (p == a || p == b) && o != a && o != b && ((e2.x == q && e2.y == o) || (e2.x == o && e2.y == q));
}

// A thread per edge: its rows checked, its vertices, and its two slots of
// the graph (the D' slot empty until its triangles arrive).
__global__ void __launch_bounds__(C2_THREADS) k_c2_edges(C2Args a) {
    if (a.st->bad) return;
    const int ne = a.st->ne;
    bool bad = false;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < ne; k += gridDim.x * blockDim.x) {
        const int j = a.elist[k];
        const int b = c2_inst_of(a, j);
        const C2Inst &in = a.inst[b];
        const int64_t s = a.colptr[j];
        const int r0 = a.rows[s], r1 = a.rows[s + 1];
        int u = 0, v = 0;
        if (r0 < 0 || r1 <= r0 || r1 >= in.cols) {
            bad = true;
        } else {
            const int64_t g0 = in.base + r0, g1 = in.base + r1;
            const C2Word x0 = a.words[g0 >> 5], x1 = a.words[g1 >> 5];
            const int b0 = (int)(g0 & 31), b1 = (int)(g1 & 31);
            if (!((x0.v >> b0) & 1u) || !((x1.v >> b1) & 1u)) bad = true;
            u = x0.vpre + __popc(x0.v & below(b0));
            v = x1.vpre + __popc(x1.v & below(b1));
        }
        a.erec[k] = make_int4(u, v, b, 0);
        if (a.neg) a.neg[k] = -1;
        if (a.runs && !bad) {
            // the edge on two vertices (its rank in the instance), from either side
            int32_t *t = a.cells + in.coff;
            const int pitch = c2_pitch(in.nv), x = u - in.voff, y = v - in.voff;
            const C2Word w = a.words[j >> 5];
            // a second edge on them, a vertex to come, or triangles before the first edge (in no edge's run)
            if (atomicCAS(t + (int64_t)x * pitch + y, -1, k - in.eoff) != -1 ||
                w.vpre + __popc(w.v & below(j & 31)) != in.voff + in.nv || (k == in.eoff && j - in.base != in.nv))
                a.st->unsorted = 1;
            t[(int64_t)y * pitch + x] = k - in.eoff;
            int32_t *const c = a.tab + in.coff;
            c[(int64_t)x * pitch + y] = c[(int64_t)y * pitch + x] = j - (int)in.base;
        }
        if (a.ends) {
            a.ends[k] = make_int2(u, v);
            a.ends[2 * (int64_t)ne - 1 - k] = make_int2(-1, -1);
            // a vertex's first edge (the reads spare most of the atomics)
            const unsigned long long key = C2_FIRST_ROUND | (unsigned)k;
            if (__ldcg(a.best + u) > key) atomicMin(a.best + u, key);
            if (__ldcg(a.best + v) > key) atomicMin(a.best + v, key);
        }
    }
    if (bad) a.st->bad = 1;
}

// The three edges (ranks) of triangle column j, its rows checked.  The column
// starts at 2 (edges before it) + 3 (triangles before it): colptr is not read
// again.  false: not a triangle's boundary.
__device__ __forceinline__ bool c2_triangle(const C2Args &a, int64_t j, const C2Word &w, const C2Inst &in, int *k) {
    const unsigned lt = below((int)(j & 31));
    const int64_t eb = w.epre + __popc(w.e & lt), vb = w.vpre + __popc(w.v & lt);
    const int32_t *r = a.rows + 2 * eb + 3 * (j - vb - eb);
    const int r0 = r[0], r1 = r[1], r2 = r[2];
    if (r0 < 0 || r1 <= r0 || r2 <= r1 || r2 >= in.cols) return false;
    const int64_t g[3] = {in.base + r0, in.base + r1, in.base + r2};
    bool ok = true;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const C2Word x = a.words[g[q] >> 5];
        const int b = (int)(g[q] & 31);
        ok &= ((x.e >> b) & 1u) != 0;
        k[q] = x.epre + __popc(x.e & below(b));
    }
    return ok;
}

// A thread per column, triangles only: checked, and entered as a node at the
// D' slots of its three edges.
__global__ void __launch_bounds__(C2_THREADS) k_c2_surface(C2Args a) {
    if (a.st->bad) return;
    const int nv = a.st->nv, ne = a.st->ne, nt = (int)(a.m - nv - ne);
    bool bad = false, crowded = false;
    // an instance's oldest vertex never dies, and most edges come to lead to
    // it: nothing is kept for it in best[]
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < a.count; b += gridDim.x * blockDim.x)
        if (a.inst[b].nv > 0) a.best[a.inst[b].voff] = 0;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < a.m; j += (int64_t)gridDim.x * blockDim.x) {
        const C2Word w = a.words[j >> 5];
        const int bit = (int)(j & 31);
        if (((w.v | w.e) >> bit) & 1u) continue;
        const C2Inst &in = a.inst[c2_inst_of(a, j)];
        int k[3], o[3];
        if (!c2_triangle(a, j, w, in, k)) {
            bad = true;
            continue;
        }
        if (!c2_opposite(a.erec[k[0]], a.erec[k[1]], a.erec[k[2]], o[0], o[1], o[2])) {
            bad = true;
            continue;
        }
        const int t = (int)(j - (w.vpre + __popc(w.v & below(bit))) - (w.epre + __popc(w.e & below(bit))));
        a.tlist[t] = (int32_t)j;
        const int id = nv + 1 + (nt - 1 - t);
        a.best[id] = C2_FIRST_ROUND | (unsigned)(2 * ne - 1 - k[2]);  // its last edge is its first column of D'
#pragma unroll
        for (int q = 0; q < 3; q++) {
            int *e = reinterpret_cast<int *>(a.ends + (2 * (int64_t)ne - 1 - k[q]));
            if (atomicCAS(e, -1, id) != -1 && atomicCAS(e + 1, -1, id) != -1) crowded = true;
        }
    }
    if (bad) a.st->bad = 1;
    if (crowded) a.st->crowded = 1;
}

// Components are trees: a node's parent is older, its root the component's
// oldest node.  N nodes' roots at once, so that a step up every path is one
// trip to memory (x < 0 stands for the ground); the nodes are then hung on
// them (racing writers all write ancestors).  The way up may go through L1:
// what it holds of an earlier round is an ancestor too, and half of all paths
// end at the same few nodes; that the end is a root is read from L2.
template <int N>
__device__ __forceinline__ void c2_roots(int *parent, int ground, const int (&x)[N], int (&r)[N]) {
    int p[N];
#pragma unroll
    for (int q = 0; q < N; q++) p[q] = r[q] = x[q] < 0 ? ground : parent[x[q]];
    for (;;) {
        for (;;) {
            bool more = false;
            int up[N];
#pragma unroll
            for (int q = 0; q < N; q++) up[q] = parent[r[q]];
#pragma unroll
            for (int q = 0; q < N; q++) {
                more |= up[q] != r[q];
                r[q] = up[q];
            }
            if (!more) break;
        }
        bool more = false;
        int up[N];
#pragma unroll
        for (int q = 0; q < N; q++) up[q] = __ldcg(parent + r[q]);
#pragma unroll
        for (int q = 0; q < N; q++) {
            more |= up[q] != r[q];
            r[q] = up[q];
        }
        if (!more) break;
    }
#pragma unroll
    for (int q = 0; q < N; q++)
        if (x[q] >= 0 && p[q] != r[q]) parent[x[q]] = r[q];
}

// Every node hung eight steps up (or on its root): three such passes shorten
// paths of up to 512.
__device__ __forceinline__ void c2_shorten(int *parent, int nodes, int i0, int stride) {
    constexpr int N = 4;
    for (int b = i0; b < nodes; b += N * stride) {
        int p[N], r[N];
#pragma unroll
        for (int q = 0; q < N; q++) p[q] = r[q] = parent[min(b + q * stride, nodes - 1)];
        bool more = true;
        for (int h = 1; more && h < 8; h++) {
            more = false;
#pragma unroll
            for (int q = 0; q < N; q++) {
                const int up = parent[r[q]];
                more |= up != r[q];
                r[q] = up;
            }
        }
#pragma unroll
        for (int q = 0; q < N; q++)
            if (b + q * stride < nodes && r[q] != p[q]) parent[b + q * stride] = r[q];
    }
}

// The blocks of a resident grid meet: the count of arrivals only grows, `goal`
// is the grid's size times the meetings so far.  False when the others do not
// come (never, while the grid is resident as a whole; about a second).
__device__ __forceinline__ bool c2_meet(unsigned *arrived, unsigned goal) {
    __shared__ int s_late;
    __syncthreads();
    if (threadIdx.x == 0) {
        s_late = 0;
        __threadfence();
        atomicAdd(arrived, 1u);
        int tries = 0;
        while ((unsigned)ld_acquire_i32(reinterpret_cast<const int *>(arrived)) < goal)
            if (++tries > (1 << 22)) {
                s_late = 1;
                break;
            }
        __threadfence();
    }
    __syncthreads();
    return !s_late;
}

// The elder rule on the whole graph, in rounds over the edges that still join
// two components: every component takes its first such edge (atomicMin on
// best[], the round in the key's upper half so that nothing is reset), and a
// component whose first edge leads to an older one dies there.
//
// Why that is exact: let r be the oldest node of component C, s its first
// outgoing edge, q the oldest node on the other side, q < r.  When column s
// is reduced, the component of its end in C is made of edges before s inside
// C and reaches r (a part of C joined over a later edge would have had s as
// an earlier way out), so r is its oldest node; the other side holds q or an
// older node; r is the younger, the low of column s.  An edge found inside a
// component closes a cycle of earlier edges: its column reduces to zero.
//
// The first round goes over the nodes, whose first edges k_c2_edges and
// k_c2_surface left in best[]; a node's last best[] is where it died, so the
// pairs are written at the end, a thread per node.  The paths of the first
// two rounds are long (on a smooth image they run downhill for a hundred
// pixels and more), so they are shortened for all nodes at once before roots
// are looked for edge by edge.  A round is two passes over the live edges,
// each followed by a meeting of the grid.  Bound by the latency of its
// dependent loads and the meetings (2-3 us): 11 rounds on a smooth 512 x 512
// lower-star image (1.57M slots, then 320K, 76K, ...), 17 on white noise of
// that size.
__global__ void __launch_bounds__(C2_THREADS) k_c2_graph(C2Args a, int max_rounds) {
    if (a.st->bad || a.st->crowded) return;  // written by earlier kernels: the same for every block
    const int nv = a.st->nv, ne = a.st->ne, nt = (int)(a.m - nv - ne), ground = nv, nodes = nv + 1 + nt;
    const int stride = gridDim.x * blockDim.x, i0 = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned goal = 0;
    auto meet = [&] { return c2_meet(&a.st->arrived, goal += gridDim.x); };
    // round 0, and the outputs before any pair is known
    const int none = a.one_based ? 0 : -1;
    for (int j = i0; j < a.m; j += stride) {
        a.low[j] = none;
        if (a.ess) a.ess[j] = 1;
    }
    for (int x = i0; x < nodes; x += stride) {
        const unsigned long long b = __ldcg(a.best + x);
        int p = x;
        if (x != ground && b != ~0ull && b != 0) {
            const int2 e = __ldcg(a.ends + (unsigned)b);
            int y = e.x == x ? e.y : e.x;
            if (y < 0) y = ground;
            p = min(x, y);
        }
        a.parent[x] = p;
    }
    bool met = meet();
    for (int q = 0; met && q < 3; q++) {
        c2_shorten(a.parent, nodes, i0, stride);
        met = meet();
    }
    constexpr int PER = 4, NW = C2_THREADS / 32;
    __shared__ int s_cnt[NW], s_at;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    int n = 2 * ne, round = 1;
    for (; met; round++) {
        const unsigned long long tag = (unsigned long long)(~(unsigned)round) << 32;
        const int32_t *in = a.list[(round + 1) & 1];
        int32_t *out = a.list[round & 1];
        int *count = &a.st->live[round % 3];
        // up to four edges a thread, fewer where that fills more blocks; the
        // block appends those that live together
        const int per = min(PER, (n + stride - 1) / stride);
        for (int b0 = blockIdx.x * per * C2_THREADS; b0 < n; b0 += per * stride) {
            int s[PER], x[2 * PER], r[2 * PER];
#pragma unroll
            for (int q = 0; q < PER; q++) {
                const int i = b0 + q * C2_THREADS + tid;
                s[q] = i >= n || q >= per ? -1 : round > 1 ? __ldcg(in + i) : i;
            }
#pragma unroll
            for (int q = 0; q < PER; q++) {
                const int2 e = s[q] >= 0 ? __ldcg(a.ends + s[q]) : make_int2(-1, -1);
                if (e.x < 0) s[q] = -1;  // an edge without triangles: an empty column of D'
                x[2 * q] = e.x;
                x[2 * q + 1] = e.y;
            }
            c2_roots<2 * PER>(a.parent, ground, x, r);
            unsigned live[PER];
            int mine = 0;
#pragma unroll
            for (int q = 0; q < PER; q++) {
                const int u = r[2 * q], v = r[2 * q + 1];
                const bool l = s[q] >= 0 && u != v;
                if (l) {
                    if (u != x[2 * q] || v != x[2 * q + 1]) __stcg(a.ends + s[q], make_int2(u, v));
                    const unsigned long long key = tag | (unsigned)s[q];
                    // (an old value of best[] only costs the atomic)
                    if (u != ground && a.best[u] > key) atomicMin(a.best + u, key);
                    if (v != ground && a.best[v] > key) atomicMin(a.best + v, key);
                }
                live[q] = __ballot_sync(0xffffffffu, l);
                mine += __popc(live[q]);
            }
            if (lane == 0) s_cnt[wid] = mine;
            __syncthreads();
            const int c = lane < NW ? s_cnt[lane] : 0;
            const int before = __reduce_add_sync(0xffffffffu, lane < wid ? c : 0);
            if (tid < 32) {
                const int total = __reduce_add_sync(0xffffffffu, c);
                if (lane == 0) s_at = total ? atomicAdd(count, total) : 0;
            }
            __syncthreads();
            int at = s_at + before;
#pragma unroll
            for (int q = 0; q < PER; q++) {
                if ((live[q] >> lane) & 1u) out[at + __popc(live[q] & below(lane))] = s[q];
                at += __popc(live[q]);
            }
        }
        if (!(met = meet())) break;
        n = __ldcg(count);
        if (i0 == 0) a.st->live[(round + 1) % 3] = 0;  // last read two rounds ago
        if (n == 0 || round >= max_rounds) break;
        for (int i = i0; i < n; i += stride) {
            const int s = __ldcg(out + i);
            const int2 e = __ldcg(a.ends + s);
            const int x = max(e.x, e.y), y = min(e.x, e.y);  // only the younger end can die here
            if (x != ground && __ldcg(a.best + x) == (tag | (unsigned)s)) a.parent[x] = y;
        }
        met = meet();
        for (int q = 0; round == 1 && met && q < 2; q++) {
            c2_shorten(a.parent, nodes, i0, stride);
            met = meet();
        }
    }
    if (i0 == 0) a.st->rounds = round;
    if (!met || n > 0) {
        if (threadIdx.x == 0) a.st->unfinished = 1;
        return;
    }
    // the pairs: node x died at the slot in its best[]
    unsigned long long joins = 0;
    for (int x = i0; x < nodes; x += stride) {
        if (x == ground || __ldcg(a.parent + x) == x) continue;
        const int s = (int)(unsigned)__ldcg(a.best + x), k = s < ne ? s : 2 * ne - 1 - s, e = a.elist[k];
        const int base = a.inst_off ? (int)a.inst[a.erec[k].z].base : 0;
        // an edge of D: its low is the vertex; of D': the triangle's low is the edge
        const int v = x < ground ? a.vlist[x] : a.tlist[nt - 1 - (x - ground - 1)];
        const int col = x < ground ? e : v, lo = x < ground ? v : e;
        a.low[col] = lo - base + a.one_based;
        if (a.ess) {
            a.ess[col] = 0;
            a.ess[lo] = 0;
        }
        joins++;
    }
    for (int o = 16; o > 0; o >>= 1) joins += __shfl_xor_sync(0xffffffffu, joins, o);
    if ((threadIdx.x & 31) == 0 && joins) atomicAdd(&a.st->joins, joins);
}

// -------------------------------------------------------------- dense form
// The edges on vertices of one instance, by the elder rule, a CTA: 1024 edges
// at a time in column order, each lot resolved in the rounds of k_c2_graph
// before the next, with the components in shared memory (a lot's pairs
// depend on no later edge).  It stops when one component is left: on the
// torus after 1,788 of 58,988 edges.  Bound by the latency of its rounds (a
// few hundred cycles each, some ten to a lot), and hidden behind the
// triangles of the same launch.
__device__ __forceinline__ int kr_find(uint16_t *parent, int x) {
    for (;;) {
        const int p = ((volatile uint16_t *)parent)[x];
        if (p == x) return x;
        const int g = ((volatile uint16_t *)parent)[p];
        ((volatile uint16_t *)parent)[x] = (uint16_t)g;
        x = g;
    }
}
template <int THREADS, class Ends, class Die>
__device__ void c2_kruskal(int nv, int ne, Ends ends, Die die, uint32_t *best, uint16_t *parent, int *s_parts) {
    constexpr int ITEMS = 1024 / THREADS;
    const int tid = threadIdx.x;
    for (int x = tid; x < nv; x += THREADS) {
        parent[x] = (uint16_t)x;
        best[x] = 0xffffffffu;
    }
    if (tid == 0) *s_parts = nv;
    __syncthreads();
    unsigned tag = 0x3fffff;  // counts down by rounds: nothing in best[] is reset
    for (int c0 = 0; c0 < ne && *s_parts > 1; c0 += 1024) {
        int2 e[ITEMS];
#pragma unroll
        for (int q = 0; q < ITEMS; q++) {
            const int i = c0 + q * THREADS + tid;
            e[q] = i < ne ? ends(i) : make_int2(0, 0);
        }
        for (;; tag--) {
            bool live = false;
#pragma unroll
            for (int q = 0; q < ITEMS; q++) {
                if (e[q].x == e[q].y) continue;
                e[q].x = kr_find(parent, e[q].x);
                e[q].y = kr_find(parent, e[q].y);
                if (e[q].x == e[q].y) continue;
                live = true;
                const unsigned key = tag << 10 | (unsigned)(q * THREADS + tid);
                atomicMin(best + e[q].x, key);
                atomicMin(best + e[q].y, key);
            }
            if (!__syncthreads_or(live)) break;
#pragma unroll
            for (int q = 0; q < ITEMS; q++) {
                const int young = max(e[q].x, e[q].y), old = min(e[q].x, e[q].y);
                if (young == old || best[young] != (tag << 10 | (unsigned)(q * THREADS + tid))) continue;
                parent[young] = (uint16_t)old;
                die(c0 + q * THREADS + tid, young);
                atomicSub(s_parts, 1);
            }
            __syncthreads();
        }
    }
}

// One vertex's row of the edge-id table in the order of its edges: each entry
// written at the number of smaller ones, by THREADS threads (a warp or a
// CTA; `row` holds the row in shared memory, absent edges as the largest id).
// An entry is the edge's rank and the other vertex.
constexpr int ADJ_SHIFT = 10;
template <int THREADS>
__device__ void c2_sort_row(const int32_t *src, int32_t *dst, int nv, int pitch, int32_t *row) {
    const int t = threadIdx.x & (THREADS - 1);
    auto meet = [] {
        if (THREADS == 32) __syncwarp();
        else __syncthreads();
    };
    for (int i = t; i < pitch; i += THREADS) {
        const int x = __ldcg(src + i);
        row[i] = x < 0 ? INT_MAX : x;
        dst[i] = INT_MAX;
    }
    meet();
    for (int i = t; i < nv; i += THREADS) {
        const int x = row[i];
        if (x == INT_MAX) continue;
        int at = 0;
        for (int q = 0; q < pitch; q += 4) {
            const int4 y = *reinterpret_cast<const int4 *>(row + q);
            at += (y.x < x) + (y.y < x) + (y.z < x) + (y.w < x);
        }
        dst[at] = x << ADJ_SHIFT | i;
    }
    meet();
}

// Runs.  A Rips complex is the flag complex of its edges, and its filtration
// puts the triangles right after their last edge, third vertices ascending
// (they carry that edge's length and come after it).  So the run of edge
// f = (u, v) must be the vertices w joined to u and to v by earlier edges, in
// order, and the rows of each triangle are those two edges' columns and f's.
// Nothing is looked up: a warp takes an edge, its lanes the vertices; two
// rows of the table of edge columns (vertices by vertices) say which have a
// triangle (a ballot is the run's word), and the triangles' rows are compared
// with what they must be.  The first edge must come right after the vertices,
// so that every column with three rows is in some edge's run.  A matrix that
// passes is a complex in such runs.
//
// One word of 32 vertices: its set bits, the columns of the two edges.
// VW > 0: that many words (else vw); four words' rows are in flight at a
// time, for one word at a time is a trip to HBM each.  Columns are the
// instance's, `run` holds them plus `shift`.  True where the run is not what
// it must be; the last edge of an instance may have been cut off inside its
// run (`cut`).
constexpr int NO_EDGE = 0x7f7f7f7f;  // past every column, and a byte pattern
template <int VW, bool GLOBAL>
__device__ __forceinline__ bool flag_run(const int32_t *tu, const int32_t *tv, int vw, int fc, int len, bool cut,
                                         const int32_t *src, uint2 *run, int shift) {
    const int lane = threadIdx.x & 31;
    constexpr int U = VW > 0 && VW < 4 ? VW : 4;
    unsigned diff = 0;
    int n = 0;
    for (int wb = 0; wb < (VW > 0 ? VW : vw); wb += U) {
        int x[U], y[U], t[U][3];
        bool tri[U];
        uint2 mine = make_uint2(0u, 0u);
#pragma unroll
        for (int q = 0; q < U; q++) {
            const bool on = VW > 0 || wb + q < vw;
            const int at = 32 * (wb + q) + lane;
            x[q] = on ? (GLOBAL ? __ldg(tu + at) : tu[at]) : NO_EDGE;
            y[q] = on ? (GLOBAL ? __ldg(tv + at) : tv[at]) : NO_EDGE;
        }
#pragma unroll
        for (int q = 0; q < U; q++) {
            tri[q] = max(x[q], y[q]) < fc;
            unsigned bits = __ballot_sync(0xffffffffu, tri[q]);
            const int i = n + __popc(bits & below(lane));
            tri[q] = tri[q] && i < len;
            if (cut) bits = __ballot_sync(0xffffffffu, tri[q]);
            if (lane == q) mine = make_uint2(bits, (unsigned)(fc + 1 + n + shift));
            n += __popc(bits);
            const int32_t *p = src + 3 * i;
#pragma unroll
            for (int c = 0; c < 3; c++) t[q][c] = tri[q] ? __ldg(p + c) : 0;
        }
        if (lane < U && (VW > 0 || wb + lane < vw)) run[wb + lane] = mine;
#pragma unroll
        for (int q = 0; q < U; q++)
            if (tri[q])
                diff |= (unsigned)(t[q][0] ^ min(x[q], y[q])) | (unsigned)(t[q][1] ^ max(x[q], y[q])) |
                        (unsigned)(t[q][2] ^ fc);
    }
    return diff != 0 || n != len;
}

// The first blocks pair the edges with vertices (an instance each).
// RUNS: the next ones sort the vertices' edges (a CTA each), the rest check
// the runs, a warp per edge; what fails sets `unsorted`, and the edge-vertex
// table is built instead.  Table: the rest check the triangles, a thread
// each, which also must come after their edges, and write each at its three
// entries, bound by those scattered writes.
template <bool RUNS>
__global__ void __launch_bounds__(C2_THREADS) k_c2_triangles(C2Args a, int kruskal_blocks, int sort_blocks, int max_nv) {
    extern __shared__ __align__(16) uint32_t tri_smem[];
    __shared__ int s_parts;
    // other blocks set these flags meanwhile: a block's threads leave together, or those that stay
    // would work on components and rows that nobody set up
    if (__syncthreads_or(a.st->bad || (RUNS && a.st->unsorted))) return;
    const int lane = threadIdx.x & 31;
    if ((int)blockIdx.x < kruskal_blocks) {
        for (int b = blockIdx.x; b < a.count; b += kruskal_blocks) {
            const C2Inst in = a.inst[b];
            c2_kruskal<C2_THREADS>(
                in.nv, in.ne,
                [&](int i) {
                    const int4 e = a.erec[in.eoff + i];
                    return make_int2(e.x - in.voff, e.y - in.voff);
                },
                [&](int i, int v) {
                    a.neg[in.eoff + i] = v;
                    a.dead[in.voff + v] = 1;
                },
                tri_smem, reinterpret_cast<uint16_t *>(tri_smem + max_nv), &s_parts);
            __syncthreads();
        }
        return;
    }
    if (RUNS && (int)blockIdx.x < kruskal_blocks + sort_blocks) {
        for (int v = blockIdx.x - kruskal_blocks; v < a.st->nv; v += sort_blocks) {
            const C2Inst &in = a.inst[c2_inst_of(a, a.vlist[v])];
            const int pitch = c2_pitch(in.nv);
            const int64_t at = in.coff + (int64_t)(v - in.voff) * pitch;
            c2_sort_row<C2_THREADS>(a.cells + at, a.adj + at, in.nv, pitch, reinterpret_cast<int32_t *>(tri_smem));
        }
        return;
    }
    const int others = kruskal_blocks + sort_blocks;
    if (RUNS) {
        bool wrong = false;
        const int ne = a.st->ne, warps = (gridDim.x - others) * (C2_THREADS / 32);
        for (int k = (blockIdx.x - others) * (C2_THREADS / 32) + (threadIdx.x >> 5); k < ne; k += warps) {
            const int4 e = a.erec[k];
            const C2Inst &in = a.inst[e.z];
            const int kl = k - in.eoff, fc = a.elist[k];  // columns of the whole batch
            const bool cut = kl + 1 == in.ne;
            const int len = (cut ? (int)(in.base + in.cols) : a.elist[k + 1]) - fc - 1;
            // vertices come first, so the triangles before f are the columns that are neither
            const int64_t start = a.colptr[fc] + 2;
            const int pitch = c2_pitch(in.nv), vw = pitch / 32, base = (int)in.base;
            const int32_t *tab = a.tab + in.coff;
            wrong |= flag_run<0, true>(tab + (int64_t)(e.x - in.voff) * pitch, tab + (int64_t)(e.y - in.voff) * pitch, vw,
                                       fc - base, len, cut, a.rows + start, a.runs + in.roff + (long long)kl * vw, base);
        }
        if (wrong) a.st->unsorted = 1;
        return;
    }
    bool bad = false;
    const int64_t stride = (int64_t)(gridDim.x - others) * C2_THREADS;
    for (int64_t j0 = (int64_t)(blockIdx.x - others) * C2_THREADS + (threadIdx.x - lane); j0 < a.m; j0 += stride) {
        const int64_t j = j0 + lane;
        const C2Word w = a.words[j0 >> 5];
        if (j >= a.m || ((w.v | w.e) >> lane) & 1u) continue;
        const C2Inst &in = a.inst[c2_inst_of(a, j)];
        int k[3], o[3];
        // a triangle before one of its edges is left to the general path: a residual
        // column is looked at from its edge on, where its triangles must be
        if (!c2_triangle(a, j, w, in, k) || k[2] >= w.epre + __popc(w.e & below(lane)) ||
            !c2_opposite(a.erec[k[0]], a.erec[k[1]], a.erec[k[2]], o[0], o[1], o[2])) {
            bad = true;
            continue;
        }
#pragma unroll
        for (int q = 0; q < 3; q++)
            a.cells[in.coff + (int64_t)(k[q] - in.eoff) * c2_pitch(in.nv) + (o[q] - in.voff)] = (int32_t)j;
    }
    if (bad) a.st->bad = 1;
}

// Column `col` has row `row` as its low (columns of the whole batch).
__device__ __forceinline__ void c2_pair(const C2Args &a, const C2Inst &in, int col, int row) {
    a.low[col] = row - (int)in.base + a.one_based;
    if (a.ess) {
        a.ess[col] = 0;
        a.ess[row] = 0;
    }
}

// RUNS: a thread per column writes its outputs, from the bits alone.  An
// edge with a run has it start with its first triangle, which no other
// column holds before: an apparent pair.  An edge that kills a vertex (its
// column of D' is cleared) has no run.  An edge with neither is residual.
__global__ void __launch_bounds__(C2_THREADS) k_c2_runs_out(C2Args a) {
    if (a.st->bad || a.st->unsorted) return;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, nwords = (a.m + 31) >> 5;
    const int none = a.one_based ? 0 : -1, lane = threadIdx.x & 31;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < a.m; j += stride) {
        const int64_t wi = j >> 5;
        const C2Word w = a.words[wi];
        const unsigned prev = wi > 0 ? a.words[wi - 1].e >> 31 : 0u;  // the column before the word
        const unsigned open = w.e << 1 | prev, notri = w.v | w.e;
        const bool edge = (w.e >> lane) & 1u, vertex = (w.v >> lane) & 1u;
        int low = none, ess = 1;
        if (edge) {
            const int k = w.epre + __popc(w.e & below(lane));
            const C2Inst &in = a.inst[a.erec[k].z];
            const int y = a.neg[k];
            bool run;
            if (lane < 31) run = j + 1 < a.m && !((notri >> (lane + 1)) & 1u);
            else run = wi + 1 < nwords && !((a.words[wi + 1].v | a.words[wi + 1].e) & 1u) && j + 1 < a.m;
            // the next instance starts with no triangle: a run stays inside
            if (y >= 0) low = a.vlist[in.voff + y] - (int)in.base + a.one_based;
            if (y >= 0 || run) ess = 0;
            else a.res[atomicAdd(&a.st->nres, 1)] = k;
        } else if (vertex) {
            if (a.dead[w.vpre + __popc(w.v & below(lane))]) ess = 0;
        } else if ((open >> lane) & 1u) {
            const int k = w.epre + __popc(w.e & below(lane)) - 1;
            low = (int)(j - 1 - a.inst[a.erec[k].z].base) + a.one_based;
            ess = 0;
        }
        a.low[j] = low;
        if (a.ess) a.ess[j] = ess;
        if (lane == 0) {
            a.owned[wi] = open & ~notri;
            a.fixed[wi] = open & ~notri;
        }
    }
}

// Table: outputs and owners before any pair is known.
__global__ void __launch_bounds__(C2_THREADS) k_c2_table_init(C2Args a) {
    if (a.st->bad) return;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, nwords = ((a.m + 31) >> 5) + 4;
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int none = a.one_based ? 0 : -1;
    for (int64_t j = i0; j < a.m; j += stride) {
        a.low[j] = none;
        if (a.ess) a.ess[j] = 1;
    }
    for (int64_t w = i0; w < nwords; w += stride) a.owned[w] = a.fixed[w] = 0u;
}

// Table: a warp per edge, its row of the table read once, for the entries set
// and its first triangle t.  An edge that kills a vertex is paired with it
// (its column of D' is cleared); one that is the last edge of t is t's low
// and t the low of its column of D', finally: an apparent pair.  The others
// are residual.  Bound by reading the table.
__global__ void __launch_bounds__(C2_THREADS) k_c2_table_pairs(C2Args a) {
    if (a.st->bad) return;
    const int lane = threadIdx.x & 31, ne = a.st->ne;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    unsigned long long set = 0;
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < ne; k += nw) {
        const C2Inst in = a.inst[a.erec[k].z];
        const int pitch = c2_pitch(in.nv);
        const uint4 *row = reinterpret_cast<const uint4 *>(a.cells + in.coff + (int64_t)(k - in.eoff) * pitch);
        unsigned t = 0xffffffffu;  // an empty entry is the largest
        for (int i = lane; i < pitch / 4; i += 32) {
            const uint4 x = row[i];
            set += (x.x != 0xffffffffu) + (x.y != 0xffffffffu) + (x.z != 0xffffffffu) + (x.w != 0xffffffffu);
            t = min(min(min(t, x.x), min(x.y, x.z)), x.w);
        }
        t = __reduce_min_sync(0xffffffffu, t);
        if (lane == 0) {
            const int e = a.elist[k], y = a.neg[k];
            if (y >= 0) {
                c2_pair(a, in, e, a.vlist[in.voff + y]);
            } else if (t != 0xffffffffu) {
                if (a.rows[a.colptr[t] + 2] + in.base == e) {
                    c2_pair(a, in, (int)t, e);
                    atomicOr(a.owned + (t >> 5), 1u << (t & 31));
                    atomicOr(a.fixed + (t >> 5), 1u << (t & 31));
                } else {
                    a.res[atomicAdd(&a.st->nres, 1)] = k;
                }
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) set += __shfl_xor_sync(0xffffffffu, set, o);
    if (lane == 0 && set) atomicAdd(&a.st->cells_set, set);
}

// The edges before column `col` (relative to the instance's wbase): the rank
// of an edge.
__device__ __forceinline__ int c2_edge_rank(const C2Args &a, const C2Inst &in, int col) {
    const C2Word w = a.words[in.woff + (col >> 5)];
    return w.epre + __popc(w.e & below(col & 31));
}

__device__ __forceinline__ void rs_flip(uint32_t *bits, int r) {
    asm volatile("red.shared.xor.b32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(bits + (r >> 5))),
                 "r"(1u << (r & 31))
                 : "memory");
}

__device__ __forceinline__ void rs_xor(uint32_t *word, uint32_t x) {
    asm volatile("red.shared.xor.b32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(word)), "r"(x) : "memory");
}

// The triangles on edge k toggled in the window of WORDS words from w0, by a
// warp.  RUNS: the triangle with vertex w belongs to the run of the last of
// its three edges; runs from edge `hi` on lie past the window, so the edges of
// one end are taken in order only that far (a residual column's window is
// early: a tenth of a row), the other end's ids and the runs are a gather
// each.  `later` keeps a bound on what lies past the window: an edge whose
// run may hold a triangle.  Table: the row, `later` the first triangle past.
template <bool RUNS, int WORDS>
__device__ __forceinline__ void rs_toggle(const C2Args &a, const C2Inst &in, int k, int w0, int hi, uint32_t *bits,
                                          int &later) {
    const int lane = threadIdx.x & 31, pitch = c2_pitch(in.nv);
    if (RUNS) {
        const int4 e = __ldg(a.erec + k);
        const int u = e.x - in.voff, v = e.y - in.voff, nw = (in.nv + 31) >> 5, kl = k - in.eoff;
        const int32_t *au = a.adj + in.coff + (int64_t)u * pitch, *iv = a.cells + in.coff + (int64_t)v * pitch;
        const uint2 *runs = a.runs + in.roff;
        constexpr int U = 4;
        for (int i = lane; i - lane < pitch; i += 32 * U) {
            int key[U], f[U], z[U];
            bool ok[U];
            uint2 r[U];
#pragma unroll
            for (int q = 0; q < U; q++) key[q] = i + 32 * q < pitch ? __ldg(au + i + 32 * q) : INT_MAX;
#pragma unroll
            for (int q = 0; q < U; q++) {
                const int x = key[q] >> ADJ_SHIFT, w = key[q] & ((1 << ADJ_SHIFT) - 1);
                ok[q] = x < hi && key[q] != INT_MAX;
                if (!ok[q] && key[q] != INT_MAX) later = min(later, max(x, kl));
                const int y = ok[q] ? __ldg(iv + w) : -1;
                f[q] = max(max(x, y), kl);
                z[q] = f[q] == kl ? w : f[q] == x ? v : u;
                ok[q] = y >= 0;
                if (ok[q] && f[q] >= hi) {
                    later = min(later, f[q]);
                    ok[q] = false;
                }
            }
#pragma unroll
            for (int q = 0; q < U; q++)
                r[q] = ok[q] ? __ldg(runs + (long long)f[q] * nw + (z[q] >> 5)) : make_uint2(0u, 0u);
#pragma unroll
            for (int q = 0; q < U; q++) {
                if (!((r[q].x >> (z[q] & 31)) & 1u)) continue;
                const int d = (int)r[q].y + __popc(r[q].x & below(z[q] & 31)) - w0;
                if (d < 0) continue;  // cancelled already
                if (d < 32 * WORDS) rs_flip(bits, d);
                else later = min(later, f[q]);
            }
            if (__any_sync(0xffffffffu, (key[U - 1] >> ADJ_SHIFT) >= hi)) break;
        }
    } else {
        const int4 *row = reinterpret_cast<const int4 *>(a.cells + in.coff + (int64_t)(k - in.eoff) * pitch);
        for (int i = lane; i < pitch / 4; i += 64) {
            const int4 A = __ldg(row + i);
            const int4 B = i + 32 < pitch / 4 ? __ldg(row + i + 32) : make_int4(-1, -1, -1, -1);
            const int t[8] = {A.x, A.y, A.z, A.w, B.x, B.y, B.z, B.w};
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int d = t[q] - w0;  // below the window: an empty entry, or cancelled already
                if (t[q] < 0 || d < 0) continue;
                if (d < 32 * WORDS) rs_flip(bits, d);
                else later = min(later, t[q]);
            }
        }
    }
}

// Residual columns of D', a CTA at a time.  Column k is held as the list of
// edges whose D' columns it is the sum of (a column of the matrix V with
// R = D' V) and, as bits in shared memory, the part of that sum in a window
// of triangles; a window left behind is never needed again, a later one is
// built from the list.  Its low is the first set bit.
//
// * Waves: not only the low's pivot is added but those of the first rs_wave()
//   set bits that have one.  Every column added comes before k in D' (a row
//   of the sum lies in a column of the sum, and its owner is the first column
//   that can hold it), so this is a reduction like any other, and the longest
//   column of the 5M-column torus (some 1,200 additions) takes 17 waves of up
//   to 128.
// * Owners: low[t] names the owner of triangle t.  A residual column claims
//   its low by compare-and-swap once its list is published.  Found claimed by
//   an earlier column, that column is added; by a later one, the claim is
//   taken over and this CTA goes on with the later column plus its own.  No
//   CTA waits for another, and the lows are those of any complete reduction.
//
// * Published windows: a large CTA publishes its window with its list.  Added
//   later, the window is xored word by word, where it reaches as far as the
//   adder's (the windows lie on a common grid, and nothing comes before a
//   low), instead of the 25 columns or so of the list one by one.
//
// Bound by the longest column, on one SM: of 14K cycles a wave (of 32) on the
// torus 9.7K went into some 77 columns, 126 cycles each (240 instructions a warp),
// 2.7K into the search of the window and 1.5K into the owners.  With published
// windows 28 columns are left to a wave: 250 us -> 190, with wider waves 165
// (a device call on 200K columns 337 -> 278 -> 252).  Flattening the lists of
// a wave into one, sharing a column among warps and leaving out the parts of a
// row past the window cost as much as they saved.  Complexes on many vertices,
// with few long columns, take large CTAs and windows (4,096 words instead of
// 8,192: 356 us, 16,384: 272); batches of small ones as many CTAs as fit: six
// an SM, at 40 registers with some spills, took 1,556-1,581 us for 1,024
// complexes, five 1,607-1,628, four 1,618-1,644.
// Table: where lists run out (`overflow`; past RS_XL_WORDS), or windows, all
// CTAs stop: the general path's time comes on top.
template <bool RUNS, int THREADS, int WORDS>
__global__ void __launch_bounds__(THREADS, THREADS == RS_SMALL ? 6 : 1) k_c2_residual(C2Args a) {
    if (a.st->bad || (RUNS && (a.st->unsorted || a.st->refused || a.st->no_room))) return;
    extern __shared__ __align__(16) uint32_t bits[];  // WORDS
    constexpr int NW = THREADS / 32, RS_LIST = rs_list(THREADS);
    constexpr bool MAPS = THREADS > RS_SMALL;
    constexpr int WAVE = rs_wave(THREADS);
    constexpr int HEAD = MAPS ? 4 : 0;  // of a published list: its window's place (-1: none), start, and what lies past it
    __shared__ int s_low[NW], s_cnt[NW], s_wave[WAVE];
    __shared__ int s_i, s_later, s_act, s_other, s_stop;
    __shared__ unsigned long long s_sum, s_sums[WAVE];
    enum { ACT_DONE, ACT_ADD, ACT_STEAL, ACT_FAIL };
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nres = a.st->nres, none = a.one_based ? 0 : -1;
    const bool whole = !RUNS && MAPS && a.whole;
    const int map_words = whole ? a.map_words : WORDS;
    int32_t *list = a.lists + (size_t)blockIdx.x * RS_LIST;
    unsigned long long adds = 0, slots = 0;
    for (;;) {
        if (tid == 0) {
            s_i = atomicAdd(&a.st->cursor, 1);
            if (!RUNS) s_stop = *(volatile int *)&a.st->overflow;
            s_later = INT_MAX;
        }
        __syncthreads();
        const int i = s_i;
        if (i >= nres || (!RUNS && s_stop)) break;
        int k = a.res[i];
        const C2Inst in = a.inst[a.erec[k].z];
        // columns here are relative to in.wbase; an owner's value in low[] is col - shift
        const int shift = (int)(in.base - in.wbase) - a.one_based, cols = (int)(in.base + in.cols - in.wbase);
        int32_t *const out_low = a.low + in.wbase, *const out_ess = a.ess ? a.ess + in.wbase : nullptr;
        uint32_t *const owned = a.owned + in.woff;
        const uint32_t *const fixed = a.fixed + in.woff;
        int n = 1, pos = a.elist[k] + 1, w0 = 0, hi = 0, later = INT_MAX;  // triangles come after their edges
        if (tid == 0) __stcg(list, k);
        // The published column of `sum` added: its edges to the list, its rows to
        // the window, from the window it was published with where that reaches
        // as far as this one, else edge by edge.
        auto add_list = [&](unsigned long long sum, int4 head) {
            const int len = (int)(sum & 0xffffffu);
            const int32_t *const from = a.arena + (sum >> 24) + HEAD;
            if (n + len > RS_LIST) return false;
            if (MAPS && head.x >= 0 && head.y >= w0) {
                const uint32_t *const map = a.maps + (size_t)head.x * map_words;
                const int off = (head.y - w0) >> 5;
                for (int q = off + 4 * tid; q < map_words; q += 4 * THREADS) {
                    const uint4 x = __ldcg(reinterpret_cast<const uint4 *>(map + (q - off)));
                    if (x.x) rs_xor(bits + q, x.x);
                    if (x.y) rs_xor(bits + q + 1, x.y);
                    if (x.z) rs_xor(bits + q + 2, x.z);
                    if (x.w) rs_xor(bits + q + 3, x.w);
                }
                if (off == 0) later = min(later, head.z);
                else if (w0 + 32ll * WORDS < cols) later = min(later, RUNS ? max(hi - 1, 0) : w0 + 32 * WORDS);
            } else {
                for (int x = wid; x < len; x += NW)
                    rs_toggle<RUNS, WORDS>(a, in, __ldcg(from + x), w0, hi, bits, later);
            }
            for (int v = tid; v < len; v += THREADS) __stcg(list + n + v, __ldcg(from + v));
            n += len;
            return true;
        };
        bool fresh = true;  // a new window, from pos
        int wave = rs_first(THREADS);       // most columns take a wave or two: long ones get the full width
        for (;;) {
            if (fresh) {
                // on a grid of half windows, so that published ones fit each other
                w0 = whole ? (int)(in.base - in.wbase) & ~127 : MAPS ? pos & ~(16 * WORDS - 1) : pos & ~127;
                if (RUNS)
                    hi = (w0 + 32ll * WORDS >= cols ? in.eoff + in.ne : c2_edge_rank(a, in, w0 + 32 * WORDS)) - in.eoff;
                for (int q = 4 * tid; q < WORDS; q += 4 * THREADS)
                    *reinterpret_cast<uint4 *>(bits + q) = make_uint4(0u, 0u, 0u, 0u);
                if (tid == 0) s_later = INT_MAX;
                later = INT_MAX;
                __syncthreads();
                for (int x = wid; x < n; x += NW)
                    rs_toggle<RUNS, WORDS>(a, in, __ldcg(list + x), w0, hi, bits, later);
                __syncthreads();
                fresh = false;
            }
            // the low, and the set bits with owners, from pos up
            int low = INT_MAX, before = 0, total = 0, mine = 0, at = 0;
            uint4 c = make_uint4(0u, 0u, 0u, 0u), fx = c;
            for (int base = ((pos - w0) >> 5) & ~3; base < WORDS; base += 4 * THREADS) {
                at = base + 4 * tid;
                uint4 t = make_uint4(0u, 0u, 0u, 0u);
                if (at < WORDS) t = *reinterpret_cast<const uint4 *>(bits + at);
                int fl = INT_MAX;
                c = make_uint4(0u, 0u, 0u, 0u);
                if (t.x | t.y | t.z | t.w) {
                    const uint4 p = __ldcg(reinterpret_cast<const uint4 *>(owned + (w0 >> 5) + at));
                    fx = __ldg(reinterpret_cast<const uint4 *>(fixed + (w0 >> 5) + at));
                    c = make_uint4(t.x & p.x, t.y & p.y, t.z & p.z, t.w & p.w);
                    fl = w0 + 32 * at +
                         (t.x ? __ffs(t.x) - 1 : t.y ? 31 + __ffs(t.y) : t.z ? 63 + __ffs(t.z) : 95 + __ffs(t.w));
                }
                mine = __popc(c.x) + __popc(c.y) + __popc(c.z) + __popc(c.w);
                int incl = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += u;
                }
                const int wl = __reduce_min_sync(0xffffffffu, fl);
                if (lane == 31) {
                    s_cnt[wid] = incl;
                    s_low[wid] = wl;
                }
                __syncthreads();
                const int wc = lane < NW ? s_cnt[lane] : 0;
                before = incl - mine + __reduce_add_sync(0xffffffffu, lane < wid ? wc : 0);
                total = __reduce_add_sync(0xffffffffu, wc);
                low = __reduce_min_sync(0xffffffffu, lane < NW ? s_low[lane] : INT_MAX);
                if (low != INT_MAX) break;
                __syncthreads();
            }
            if (low == INT_MAX) {  // nothing left in the window
                if (later != INT_MAX) atomicMin(&s_later, later);
                __syncthreads();
                const int next = s_later;
                __syncthreads();
                if (next == INT_MAX) {  // the column is zero: edge k is essential
                    if (tid == 0 && out_ess) out_ess[a.elist[k]] = 1;
                    break;
                }
                pos = RUNS ? a.elist[in.eoff + next] + 1 : next;
                fresh = true;
                continue;
            }
            if (mine && before < wave) {
                const unsigned cw[4] = {c.x, c.y, c.z, c.w}, fw[4] = {fx.x, fx.y, fx.z, fx.w};
                int r = before;
#pragma unroll
                for (int q = 0; q < 4; q++)
                    for (unsigned b = cw[q]; b && r < wave; b &= b - 1, r++) {
                        const int bit = __ffs(b) - 1, t = w0 + 32 * (at + q) + bit;
                        s_wave[r] = (fw[q] >> bit) & 1u ? t : t | RS_FLAG;
                    }
            }
            __syncthreads();
            int cnt = min(total, wave);
            const bool have = cnt > 0 && (s_wave[0] & ~RS_FLAG) == low;
            wave = min(2 * wave, WAVE);
            __syncthreads();
            if (!RUNS && tid == 0) s_stop = *(volatile int *)&a.st->overflow;
            if (tid < cnt) {  // the owners, all at once
                const int t = s_wave[tid] & ~RS_FLAG, fl = s_wave[tid] & RS_FLAG;
                int o;
                if (RUNS && !fl) o = c2_edge_rank(a, in, t) - 1;  // the last edge before t
                else o = c2_edge_rank(a, in, ld_acquire_i32(out_low + t) + shift);
                s_wave[tid] = o | fl;
            }
            __syncthreads();
            const int p0 = have ? s_wave[0] : -1;
            if ((!whole && n + WAVE > RS_LIST) || (!RUNS && s_stop)) {
                if (tid == 0) a.st->overflow = 1;
                break;
            }
            if (!have || ((p0 & RS_FLAG) && (p0 & ~RS_FLAG) < k)) {
                // claim the low: the list first, then the owner
                if (tid == 0) {
                    const int room = (HEAD + (whole ? 0 : n) + 3) & ~3;
                    const unsigned long long off = atomicAdd(&a.st->arena, (unsigned long long)room);
                    s_sum = off;
                    s_act = off + room > (unsigned long long)a.arena_cap ? ACT_FAIL : ACT_DONE;
                    if (MAPS) s_other = atomicAdd(&a.st->maps, 1);
                    if (whole && s_other >= a.map_cap) s_act = ACT_FAIL;
                }
                if (MAPS && later != INT_MAX) atomicMin(&s_later, later);
                __syncthreads();
                const unsigned long long off = s_sum;
                if (s_act == ACT_FAIL) {
                    if (tid == 0) a.st->overflow = 1;
                    break;
                }
                if (MAPS) {
                    const int place = s_other < a.map_cap ? s_other : -1;
                    if (place >= 0)
                        for (int q = 4 * tid; q < map_words; q += 4 * THREADS)
                            __stcg(reinterpret_cast<uint4 *>(a.maps + (size_t)place * map_words + q),
                                   *reinterpret_cast<const uint4 *>(bits + q));
                    if (tid == 0) __stcg(reinterpret_cast<int4 *>(a.arena + off), make_int4(place, w0, s_later, 0));
                }
                for (int v = tid; !whole && v < n; v += THREADS) __stcg(a.arena + off + HEAD + v, __ldcg(list + v));
                __threadfence();
                __syncthreads();
                if (tid == 0) {
                    *(volatile unsigned long long *)(a.sum + k) = (off << 24) | (unsigned)(whole ? 0 : n);
                    const int e = a.elist[k];
                    if (out_ess) {
                        out_ess[low] = 0;
                        out_ess[e] = 0;
                    }
                    __threadfence();
                    int want = p0 < 0 ? none : a.elist[p0 & ~RS_FLAG] - shift, act = ACT_FAIL, other = -1;
                    for (int tries = 0; tries < (1 << 20); tries++) {
                        const int got = atomicCAS(out_low + low, want, e - shift);
                        other = want == none ? -1 : c2_edge_rank(a, in, want + shift);
                        if (got == want) {
                            atomicOr(owned + (low >> 5), 1u << (low & 31));
                            act = want == none ? ACT_DONE : ACT_STEAL;
                            break;
                        }
                        other = c2_edge_rank(a, in, got + shift);
                        if (other > k) {  // an earlier column's by now
                            act = ACT_ADD;
                            break;
                        }
                        want = got;
                    }
                    __threadfence();
                    if (act == ACT_STEAL) s_sum = *(volatile unsigned long long *)(a.sum + other);
                    if (act == ACT_FAIL) a.st->overflow = 1;
                    s_act = act;
                    s_other = other;
                }
                __syncthreads();
                const int act = s_act;
                if (act == ACT_DONE || act == ACT_FAIL) break;
                if (act == ACT_STEAL) {
                    // its rows join those in the window (below their common low both have none left).
                    // Batches of small complexes start the window afresh instead: their lists are short,
                    // and joining cost 1,888 us against 1,843 on 1,024 of them; a torus of 5M columns took
                    // 395-423 us afresh and 378 joining.
                    const unsigned long long sum = s_sum;
                    bool room = true;
                    if constexpr (MAPS) {
                        room = add_list(sum, __ldcg(reinterpret_cast<const int4 *>(a.arena + (sum >> 24))));
                    } else {
                        const int len = (int)(sum & 0xffffffu);
                        room = n + len <= RS_LIST;
                        for (int v = tid; room && v < len; v += THREADS)
                            __stcg(list + n + v, __ldcg(a.arena + (sum >> 24) + v));
                        n += len;
                        fresh = true;
                    }
                    if (!room) {
                        if (tid == 0) a.st->overflow = 1;
                        break;
                    }
                    k = s_other;
                    pos = low;
                    __syncthreads();
                    continue;
                }
                if (tid == 0) s_wave[0] = s_other | RS_FLAG;
                cnt = 1;
                __syncthreads();
            }
            // the wave, 32 pivots a lane each (what the residual ones
            // published is read once for all warps: it may be published anew meanwhile)
            int app = 0, nres_w = 0;
#pragma unroll
            for (int h = 0; h < WAVE; h += 32) {
                const int p = h + lane < cnt ? s_wave[h + lane] : -1;
                const bool res = p >= 0 && (p & RS_FLAG) && (p & ~RS_FLAG) > k;
                const unsigned m_app = __ballot_sync(0xffffffffu, p >= 0 && !(p & RS_FLAG));
                nres_w += __popc(__ballot_sync(0xffffffffu, res));
                if (wid == h / 32) {
                    if (!whole && ((m_app >> lane) & 1u)) __stcg(list + n + app + __popc(m_app & below(lane)), p);
                    if (res) s_sums[h + lane] = *(volatile unsigned long long *)(a.sum + (p & ~RS_FLAG));
                }
                app += __popc(m_app);
            }
            for (int q = wid; q < cnt; q += NW)
                if (!(s_wave[q] & RS_FLAG)) rs_toggle<RUNS, WORDS>(a, in, s_wave[q], w0, hi, bits, later);
            if (!whole) n += app;
            adds += app + nres_w;
            slots += (unsigned long long)app * in.nv;
            bool full = false;
            if (nres_w) {
                __syncthreads();
#pragma unroll
                for (int h = 0; h < WAVE; h += 32) {
                    const int p = h + lane < cnt ? s_wave[h + lane] : -1;
                    const bool res = p >= 0 && (p & RS_FLAG) && (p & ~RS_FLAG) > k;
                    int4 head = make_int4(-1, 0, 0, 0);
                    if (MAPS && res) head = __ldcg(reinterpret_cast<const int4 *>(a.arena + (s_sums[h + lane] >> 24)));
                    for (unsigned m = __ballot_sync(0xffffffffu, res); m && !full; m &= m - 1) {
                        const int q = __ffs(m) - 1;
                        const int4 at = make_int4(__shfl_sync(0xffffffffu, head.x, q), __shfl_sync(0xffffffffu, head.y, q),
                                                  __shfl_sync(0xffffffffu, head.z, q), 0);
                        full = !add_list(s_sums[h + q], at);
                        slots += (unsigned long long)(s_sums[h + q] & 0xffffffu) * in.nv;
                    }
                }
            }
            if (full) {
                if (tid == 0) a.st->overflow = 1;
                break;
            }
            pos = low;
            __syncthreads();
        }
        __syncthreads();
    }
    if (tid == 0 && adds) {
        atomicAdd(&a.st->adds, adds);
        atomicAdd(&a.st->slots, slots);
    }
}

// ---------------------------------------------------------- whole instances
// Small Rips complexes (a batch of them, or one): an instance to a CTA, from
// its colptr to its runs in one launch, with its edges in shared memory.
//
// Against a launch per step over all columns this saves the launches, which
// are all that the smallest complexes cost, and the trips to L2 for tables
// that fit a CTA: 47 instructions a warp for 32 vertices of an edge are what
// bounds it.  Whatever is no flag complex in runs, vertices first (`unsorted`),
// or does not fit (`refused`, as the others) is left to the grid-wide kernels;
// columns that none of the forms takes (`bad`) to the general path at once.
// The CTAs stop where one instance is refused.
//
// The tables that the residual columns read later are carved from common
// arrays by counters; when those turn out too small the host makes them
// larger and starts again.  The outputs are written (k_c2_inst_out) once
// every instance has passed.
constexpr int IN_THREADS = 512;
constexpr int IN_SMEM = 112 * 1024;  // two CTAs an SM
// Where the instances have this many columns on average, those with more than
// three quarters of a CTA's share are split (k_c2_inst_more).  Below, the two
// launches cost more than they give: 64 complexes of 9 to 20 points took 85 us
// without and 98 with, one of 30 points 82 and 85, of 36 points 95 and 85.
constexpr int IN_SPLIT = 6144;
constexpr int IN_MAX_NV = 192;       // sorting the vertices' rows takes nv^3 comparisons of one CTA
// Words of an instance start at a multiple of four (16-byte windows).
__device__ __forceinline__ long long in_woff(long long o0, int b) { return 4 * ((o0 >> 7) + b); }

// The triangles of edges k0 ... k0 + own of an instance (col, ends: theirs), a
// warp per edge (flag_run); true where a run is not what it must be.
template <int VW>
__device__ bool in_triangles(const int32_t *col, const int32_t *tab, const uint16_t *ends, const int32_t *rows,
                             uint2 *runs, int k0, int own, int ne, int nv, int cols) {
    const int vw = VW > 0 ? VW : (nv + 31) >> 5, idp = 32 * vw;
    bool wrong = false;
    for (int q = threadIdx.x >> 5; q < own; q += IN_THREADS / 32) {
        const int k = k0 + q;
        const bool cut = k + 1 == ne;
        const int fc = col[q], len = (cut ? cols : col[q + 1]) - fc - 1, u = ends[q] & 0xff, v = ends[q] >> 8;
        wrong |= tab[u * idp + v] != fc;  // a second edge on these vertices
        wrong |= flag_run<VW, false>(tab + u * idp, tab + v * idp, vw, fc, len, cut,
                                     rows + (2 * (k + 1) + 3 * (fc - nv - k)), runs + (long long)k * vw, 0);
    }
    return wrong;
}

// The outputs of a whole instance, as k_c2_runs_out writes them, by a CTA: a
// word a thread, from word `first` on and every `step` words, filled with what
// a positive triangle gets, 16 bytes a store; then the few vertices, edges and
// paired triangles are corrected.  Bound by the writes where there are many
// instances (157 us for 684 MB), by the chain of a word's edges where there are
// few: up to 32 at the start of an instance, so there (EACH) the vertices and
// edges take a thread each.  50 points through openph() 213-226 us -> 205-216, 40
// of 20 to 60 points from the host 286-291 -> 276-282; 1,024
// complexes would take 0.7-1.4% longer.
template <int THREADS, bool EACH>
__device__ __forceinline__ void in_out(const C2Args &a, const C2Inst &in, int first, int step) {
    const int none = a.one_based ? 0 : -1, tid = threadIdx.x;
    auto fill = [&](int32_t *p, int n, int value) {
        const int head = min(n, (int)((16 - ((uintptr_t)p & 15)) & 15) / 4), body = (n - head) / 4;
        if (tid < head) p[tid] = value;
        int4 *q = reinterpret_cast<int4 *>(p + head);
        for (int i = tid; i < body; i += THREADS) q[i] = make_int4(value, value, value, value);
        const int at = head + 4 * body + tid;
        if (at < n) p[at] = value;
    };
    const C2Word *const words = a.words + in.woff;
    const int nw = (int)((in.cols + 31) >> 5);
    int32_t *const low = a.low + in.base, *const ess = a.ess ? a.ess + in.base : nullptr;
    for (int c0 = 32 * first; c0 < in.cols; c0 += 32 * step) {
        const int n = min(32 * THREADS, (int)in.cols - c0), w_next = (c0 >> 5) + THREADS;
        int k0 = 0, k1 = 0;  // its edges
        if (EACH) {
            k0 = words[c0 >> 5].epre;
            k1 = w_next < nw ? words[w_next].epre : in.eoff + in.ne;
        }
        fill(low + c0, n, none);
        if (ess) fill(ess + c0, n, 1);
        __syncthreads();
        const int wi = (c0 >> 5) + tid;
        if (wi < nw) {
            const C2Word w = words[wi];
            const unsigned prev = wi > 0 ? words[wi - 1].e >> 31 : 0u, notri = w.v | w.e;
            const int end = min(32, (int)in.cols - 32 * wi);
            const unsigned here = end == 32 ? ~0u : below(end);
            const unsigned open = (w.e << 1 | prev) & ~notri & here;  // first triangles: paired with the edge before
            a.owned[in.woff + wi] = open;
            a.fixed[in.woff + wi] = open;
            for (unsigned x = open; x; x &= x - 1) {
                const int j = 32 * wi + __ffs(x) - 1;
                low[j] = j - 1 + a.one_based;
                if (ess) ess[j] = 0;
            }
            if (!EACH) {
                if (ess)
                    for (unsigned x = w.v; x; x &= x - 1) {
                        const int j = 32 * wi + __ffs(x) - 1;
                        if (a.dead[in.voff + j]) ess[j] = 0;
                    }
                // bit x: the column after x is no triangle, or past the instance's end
                const unsigned next =
                    notri >> 1 | (wi + 1 < nw ? (words[wi + 1].v | words[wi + 1].e) << 31 : ~(here >> 1));
                int k = w.epre;
                for (unsigned x = w.e; x; x &= x - 1, k++) {
                    const int bit = __ffs(x) - 1, j = 32 * wi + bit, y = a.neg[k];
                    const bool run = !((next >> bit) & 1u);
                    if (y >= 0) low[j] = y + a.one_based;
                    if (y < 0 && !run) a.res[atomicAdd(&a.st->nres, 1)] = k;
                    else if (ess) ess[j] = 0;
                }
            }
        }
        if (EACH && ess)
            for (int v = c0 + tid; v < min(in.nv, c0 + n); v += THREADS)
                if (a.dead[in.voff + v]) ess[v] = 0;
        for (int k = k0 + tid; k < k1; k += THREADS) {
            const int j = a.elist[k], y = a.neg[k];
            bool run = j + 1 < in.cols;  // a triangle follows
            if (run) {
                const C2Word next = words[(j + 1) >> 5];
                run = !(((next.v | next.e) >> ((j + 1) & 31)) & 1u);
            }
            if (y >= 0) low[j] = y + a.one_based;
            if (y < 0 && !run) a.res[atomicAdd(&a.st->nres, 1)] = k;
            else if (ess) ess[j] = 0;
        }
        __syncthreads();
    }
}

// The order instances are taken in when there are more than CTAs: the largest
// first (to 2,048 columns), or the last to start may be one of 300 us when the
// others are done.  One CTA; its 6 us are those of its chain of steps.
constexpr int IO_CLASSES = 512;
__global__ void __launch_bounds__(1024) k_c2_inst_order(C2Args a) {
    __shared__ int s_at[IO_CLASSES];
    auto cls = [&](int b) {
        const int64_t n = a.inst_off[b + 1] - a.inst_off[b];
        return n <= 0 ? IO_CLASSES - 1 : (int)max((int64_t)0, IO_CLASSES - 1 - (n >> 11));
    };
    for (int q = threadIdx.x; q < IO_CLASSES; q += 1024) s_at[q] = 0;
    __syncthreads();
    for (int b = threadIdx.x; b < a.count; b += 1024) atomicAdd(&s_at[cls(b)], 1);
    __syncthreads();
    if (threadIdx.x < 32) {
        int run = 0;
        for (int q = threadIdx.x; q < IO_CLASSES; q += 32) {
            const int n = s_at[q];
            int incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)threadIdx.x >= o) incl += u;
            }
            s_at[q] = run + incl - n;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < a.count; b += 1024) a.order[atomicAdd(&s_at[cls(b)], 1)] = b;
}

template <bool OUT>
__global__ void __launch_bounds__(IN_THREADS, 2) k_c2_inst(C2Args a) {
    extern __shared__ __align__(16) unsigned char in_smem[];  // IN_SMEM
    constexpr int NW = IN_THREADS / 32;
    __shared__ int s_b, s_nv, s_ne, s_no, s_parts, s_wsum[NW];
    __shared__ C2Inst s_in;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (blockIdx.x == 0 && tid == 0) {
        a.st->nnz = a.colptr[a.m];
        if (a.colptr[0] != 0 || (a.nnz >= 0 && a.st->nnz != a.nnz) ||
            (a.inst_off && (a.inst_off[0] != 0 || a.inst_off[a.count] != a.m)))
            a.st->bad = a.st->refused = 1;
    }
    for (;;) {
        if (tid == 0) {
            const int stop = *(volatile int *)&a.st->refused, next = atomicAdd(&a.st->next, 1);
            s_b = stop ? a.count : next;
            s_nv = s_ne = 0;
            s_no = 0;
        }
        __syncthreads();
        if (s_b >= a.count) break;
        const int b = a.order ? a.order[s_b] : s_b;
        const int64_t o0 = a.inst_off ? a.inst_off[b] : 0, o1 = a.inst_off ? a.inst_off[b + 1] : a.m;
        const int64_t cols64 = o1 - o0;
        // 6 bytes a word (bits, edges before it), and room for some edges
        if (o0 < 0 || o1 > a.m || cols64 < 0 || (cols64 + 31) / 32 * 6 > IN_SMEM - 1024) {
            if (tid == 0) a.st->refused = 1;
            __syncthreads();
            continue;
        }
        const int cols = (int)cols64, nw = (cols + 31) >> 5, nw2 = (nw + 1) & ~1;
        uint32_t *ebit = reinterpret_cast<uint32_t *>(in_smem);
        uint16_t *epre = reinterpret_cast<uint16_t *>(ebit + nw2);
        const int64_t *cp = a.colptr + o0;
        const int64_t c_first = cp[0];
        // no row is read outside [0, nnz): an instance's columns lie between its ends (checked below)
        const bool outside = c_first < 0 || (a.nnz >= 0 ? cp[cols] > a.nnz : c_first != 0);
        // the kinds of the columns, eight words a warp in flight
        bool no = false;
        int nv = 0, ne = 0;
        for (int w0 = 8 * wid; w0 < nw; w0 += 8 * NW) {
            int64_t c0[8], c1[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int j = (w0 + q) * 32 + lane;
                c0[q] = cp[min(j, cols)];
                c1[q] = cp[min(j + 1, cols)];
            }
#pragma unroll
            for (int q = 0; q < 8; q++) {
                if (w0 + q >= nw) break;
                const bool in = (w0 + q) * 32 + lane < cols;
                const int64_t n = c1[q] - c0[q];
                if (in && n != 2 && n != 3 && (n != 0 || c0[q] != c_first)) no = true;  // vertices come first
                const unsigned e = __ballot_sync(0xffffffffu, in && n == 2);
                nv += __popc(__ballot_sync(0xffffffffu, in && n == 0));
                ne += __popc(e);
                if (lane == 0) ebit[w0 + q] = e;
            }
        }
        if (lane == 0) {
            atomicAdd(&s_nv, nv);
            atomicAdd(&s_ne, ne);
        }
        if (no) s_no = 1;
        __syncthreads();
        nv = s_nv;
        ne = s_ne;
        const int pitch = c2_pitch(nv), vw = pitch / 32;
        // shared memory once the words are written out: in their place the
        // table of edge columns and the edges' columns; the edges' vertices
        // (bytes) behind; the rest is scratch
        const int ends_at = (max(6 * nw2, 4 * pitch * nv + 4 * ne) + 15) & ~15;
        const int scratch_at = (ends_at + 2 * ne + 15) & ~15, left = IN_SMEM - scratch_at;
        // (without edges there are vertices only: a triangle has rows)
        if (outside || (ne == 0 && nv != cols) || ne > 65535 || nv > IN_MAX_NV || left < max(6 * nv, 4 * pitch)) {
            if (tid == 0) a.st->refused = 1;
            s_no = 1;
        }
        if (tid == 0) {
            C2Inst in{};
            in.nv = nv;
            in.ne = ne;
            in.base = in.wbase = o0;
            in.cols = cols;
            in.woff = in_woff(o0, b);
            in.eoff = atomicAdd(&a.st->ne, ne);
            in.voff = atomicAdd(&a.st->nv, nv);
            in.coff = (long long)atomicAdd((unsigned long long *)&a.st->pairs, (unsigned long long)pitch * nv);
            in.roff = (long long)atomicAdd((unsigned long long *)&a.st->run_words, (unsigned long long)ne * vw);
            atomicMax(&a.st->max_nv, nv);
            if (in.eoff + ne > a.cap_e || in.voff + nv > a.cap_v || in.coff + (long long)pitch * nv > a.cap_c ||
                in.roff + (long long)ne * vw > a.cap_r) {
                a.st->no_room = 1;
                s_no = 1;
            }
            s_in = in;
            a.inst[b] = in;
        }
        __syncthreads();
        if (s_no) {
            if (no) a.st->refused = 1;
            // (why: a column that no form takes, or a vertex after other columns)
            for (int j = tid; j < cols; j += IN_THREADS) {
                const int64_t n = cp[j + 1] - cp[j];
                if (n != 0 && n != 2 && n != 3) a.st->bad = 1;
                if (n == 0 && cp[j] != c_first) a.st->unsorted = 1;
            }
            __syncthreads();
            continue;
        }
        const C2Inst in = s_in;
        {  // edges before each word
            const int per = (nw + IN_THREADS - 1) / IN_THREADS, w1 = min(tid * per + per, nw);
            int sum = 0;
            for (int w = tid * per; w < w1; w++) sum += __popc(ebit[w]);
            int incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
            if (lane == 31) s_wsum[wid] = incl;
            __syncthreads();
            int run = incl - sum + __reduce_add_sync(0xffffffffu, lane < wid && lane < NW ? s_wsum[lane] : 0);
            for (int w = tid * per; w < w1; w++) {
                epre[w] = (uint16_t)run;
                run += __popc(ebit[w]);
            }
        }
        int32_t *const elist = a.elist + in.eoff;
        for (int i = tid; i < nv; i += IN_THREADS) a.dead[in.voff + i] = 0;
        __syncthreads();
        for (int w = tid; w < nw; w += IN_THREADS) {
            const unsigned e = ebit[w];
            const int k0 = epre[w], v0 = min(nv, 32 * w);
            *reinterpret_cast<int4 *>(a.words + in.woff + w) =
                make_int4((int)(nv - v0 >= 32 ? ~0u : below(nv - v0)), (int)e, in.voff + v0, in.eoff + k0);
            int k = k0;
            for (unsigned x = e; x; x &= x - 1) elist[k++] = 32 * w + __ffs(x) - 1;
        }
        __syncthreads();
        int32_t *const tab = reinterpret_cast<int32_t *>(in_smem), *const col = tab + pitch * nv;
        uint16_t *const ends = reinterpret_cast<uint16_t *>(in_smem + ends_at);
        uint32_t *const scratch = reinterpret_cast<uint32_t *>(in_smem + scratch_at);
        int32_t *const ids = a.cells + in.coff, *const adj = a.adj + in.coff;
        for (int i = tid; i < pitch * nv; i += IN_THREADS) {
            tab[i] = NO_EDGE;
            ids[i] = -1;
        }
        __syncthreads();
        // the edges: a column starts at 2 (edges before it) + 3 (triangles before it)
        const int32_t *const rows = a.rows + c_first;
        for (int k = tid; k < ne; k += IN_THREADS) {
            const int j = __ldcg(elist + k), s = 2 * k + 3 * (j - nv - k);
            int r0 = rows[s], r1 = rows[s + 1];
            if (k == 0 && j != nv) s_no = a.st->unsorted = 1;  // triangles before the first edge are in no edge's run
            if (r0 < 0 || r1 <= r0 || r1 >= nv) {
                s_no = 1;
                r0 = r1 = 0;
            } else {
                tab[r0 * pitch + r1] = tab[r1 * pitch + r0] = j;
                ids[r0 * pitch + r1] = ids[r1 * pitch + r0] = k;
            }
            col[k] = j;
            ends[k] = (uint16_t)(r0 | r1 << 8);
            a.erec[in.eoff + k] = make_int4(in.voff + r0, in.voff + r1, b, 0);
            a.neg[in.eoff + k] = -1;
        }
        __syncthreads();
        c2_kruskal<IN_THREADS>(
            nv, ne, [&](int i) { return make_int2(ends[i] & 0xff, ends[i] >> 8); },
            [&](int i, int v) {
                a.neg[in.eoff + i] = v;
                a.dead[in.voff + v] = 1;
            },
            scratch, reinterpret_cast<uint16_t *>(scratch + nv), &s_parts);
        __syncthreads();
        if (a.chunk > 0 && ne > 2 * a.chunk && cols > a.split_cols && !s_no) {
            // the rest in pieces, to whichever CTAs
            int4 *const out = reinterpret_cast<int4 *>(a.tab + in.coff);
            for (int i = tid; i < pitch * nv / 4; i += IN_THREADS) out[i] = reinterpret_cast<const int4 *>(tab)[i];
            const int pieces = (ne + a.chunk - 1) / a.chunk;
            if (tid == 0) s_b = atomicAdd(&a.st->items, pieces);
            __syncthreads();
            for (int i = tid; i < pieces; i += IN_THREADS) a.items[s_b + i] = make_int2(b, i * a.chunk);
            __syncthreads();
            continue;
        }
        // the vertices' edges in order, for the residual columns (as many
        // warps as the scratch has rows for)
        const int warps = min(NW, left / (4 * pitch));
        if (wid < warps)
            for (int v = wid; v < nv; v += warps)
                c2_sort_row<32>(ids + v * pitch, adj + v * pitch, nv, pitch,
                            reinterpret_cast<int32_t *>(scratch) + wid * pitch);
        uint2 *const runs = a.runs + in.roff;
        bool wrong;
        switch (vw) {
            case 1: wrong = in_triangles<1>(col, tab, ends, rows, runs, 0, ne, ne, nv, cols); break;
            case 2: wrong = in_triangles<2>(col, tab, ends, rows, runs, 0, ne, ne, nv, cols); break;
            case 3: wrong = in_triangles<3>(col, tab, ends, rows, runs, 0, ne, ne, nv, cols); break;
            case 4: wrong = in_triangles<4>(col, tab, ends, rows, runs, 0, ne, ne, nv, cols); break;
            default: wrong = in_triangles<0>(col, tab, ends, rows, runs, 0, ne, ne, nv, cols); break;
        }
        if (wrong) s_no = a.st->unsorted = 1;
        __syncthreads();
        if (tid == 0 && s_no) a.st->refused = 1;
        // a single small one's outputs at once: 12 points 54 us -> 46-50 in all
        if constexpr (OUT)
            if (!s_no && !a.st->refused) in_out<IN_THREADS, true>(a, in, 0, IN_THREADS);
        __syncthreads();
    }
}

// What k_c2_inst left of larger instances, a CTA a piece: a stretch of edges
// with their runs, and its share of the vertices' rows.  One CTA takes 330 us
// over the triangles of 120 points, while the smaller complexes of a batch are
// long done.  Instructions bound it as in k_c2_inst (47 a word of an edge, 70%
// of the issue slots); fetching rows to L2 ahead of use, and checking the
// triangles packed by a list of third vertices, gave nothing or cost 8%.
// 1,024 complexes of 20 to 120 points 1,909 us -> 1,640 in all, 40 of 20 to 60
// 182 -> 149, one of 50 points 135 -> 109.
__global__ void __launch_bounds__(IN_THREADS, 2) k_c2_inst_more(C2Args a) {
    extern __shared__ __align__(16) unsigned char in_smem[];  // IN_SMEM
    constexpr int NW = IN_THREADS / 32;
    __shared__ int s_i;
    const int tid = threadIdx.x, wid = tid >> 5;
    // other blocks set `refused` meanwhile: a block's threads leave together (thread 0 hands out the items)
    if (__syncthreads_or(a.st->refused || a.st->no_room)) return;
    const int n_items = a.st->items;
    for (int i = blockIdx.x; i < n_items; i = s_i) {
        const int2 item = a.items[i];
        const C2Inst in = a.inst[item.x];
        const int nv = in.nv, ne = in.ne, pitch = c2_pitch(nv), vw = pitch / 32;
        const int k0 = item.y, k1 = min(ne, k0 + a.chunk), own = k1 - k0;
        const int32_t *const elist = a.elist + in.eoff, *const rows = a.rows + a.colptr[in.base];
        // the piece's rows of the matrix on their way to L2
        const int f0 = __ldg(elist + k0), f1 = k1 < ne ? __ldg(elist + k1) : (int)in.cols;
        const int32_t *const r0 = rows + 2 * (k0 + 1) + 3 * (f0 - nv - k0);
        for (int q = 32 * tid; q < 2 * (own - 1) + 3 * (f1 - f0 - own); q += 32 * IN_THREADS) prefetch_l2(r0 + q);
        int32_t *const tab = reinterpret_cast<int32_t *>(in_smem), *const col = tab + pitch * nv;
        uint16_t *const ends = reinterpret_cast<uint16_t *>(col + a.chunk + 4);
        const int32_t *const src = a.tab + in.coff;
        for (int q = tid; q < pitch * nv / 4; q += IN_THREADS)
            reinterpret_cast<int4 *>(tab)[q] = __ldg(reinterpret_cast<const int4 *>(src) + q);
        for (int q = tid; q <= own; q += IN_THREADS) {
            col[q] = k0 + q < ne ? __ldg(elist + k0 + q) : (int)in.cols;
            if (q < own) {
                const int4 e = __ldg(a.erec + in.eoff + k0 + q);
                ends[q] = (uint16_t)((e.x - in.voff) | (e.y - in.voff) << 8);
            }
        }
        __syncthreads();
        bool wrong = false;
        uint2 *const runs = a.runs + in.roff;
        auto check = [&](auto words) {
            constexpr int VW = decltype(words)::value;
            wrong = in_triangles<VW>(col, tab, ends, rows, runs, k0, own, ne, nv, (int)in.cols);
        };
        switch (vw) {
            case 1: check(std::integral_constant<int, 1>()); break;
            case 2: check(std::integral_constant<int, 2>()); break;
            case 3: check(std::integral_constant<int, 3>()); break;
            case 4: check(std::integral_constant<int, 4>()); break;
            default: check(std::integral_constant<int, 0>()); break;
        }
        if (wrong) a.st->unsorted = a.st->refused = 1;
        const int pieces = (ne + a.chunk - 1) / a.chunk;
        // as many warps as there is room for rows (one at least: k_c2_inst had it beside 6 ne > 12 chunk bytes)
        int32_t *const row = reinterpret_cast<int32_t *>(ends + a.chunk);
        const int warps = min(NW, (int)(in_smem + IN_SMEM - reinterpret_cast<unsigned char *>(row)) / (4 * pitch));
        if (wid < warps)
            for (int v = k0 / a.chunk + wid * pieces; v < nv; v += warps * pieces)
                c2_sort_row<32>(a.cells + in.coff + v * pitch, a.adj + in.coff + v * pitch, nv, pitch, row + wid * pitch);
        if (tid == 0) s_i = gridDim.x + atomicAdd(&a.st->next_item, 1);
        __syncthreads();
    }
}

// The outputs, IO_COLS columns a block.
constexpr int IO_THREADS = 256, IO_COLS = 32 * IO_THREADS;
template <bool EACH>
__global__ void __launch_bounds__(IO_THREADS) k_c2_inst_out(C2Args a, int parts) {
    if (a.st->refused || a.st->no_room) return;
    for (int b = blockIdx.x / parts; b < a.count; b += gridDim.x / parts) {
        const C2Inst in = a.inst[b];
        in_out<IO_THREADS, EACH>(a, in, (int)(blockIdx.x % parts) * IO_THREADS, parts * IO_THREADS);
    }
}

// ------------------------------------------------------------------ driver
namespace {
struct Carve {
    char *p;
    size_t off = 0;
    template <class T>
    T *take(size_t n) {
        off = (off + 255) & ~(size_t)255;
        T *q = p ? reinterpret_cast<T *>(p + off) : nullptr;
        off += sizeof(T) * n;
        return q;
    }
};

int c2_grid(const Context *ctx, int64_t n, int per_sm) {
    const int64_t g = (n + C2_THREADS - 1) / C2_THREADS;
    return (int)std::max<int64_t>(1, std::min<int64_t>(g, (int64_t)ctx->sm_count * per_sm));
}

// What OPH_DUAL_AUTO's rule (dual_grade) names for these column counts.
int c2_named_matrix(int64_t m, int64_t nv, int64_t ne, int64_t nt) {
    if (m < DUAL_MIN_M) return 0;
    const int64_t lo = nv ? nv : ne ? ne : nt, hi = nt ? nt : ne ? ne : nv;
    const int kinds = (nv > 0) + (ne > 0) + (nt > 0);
    if (kinds > 1 && lo * (int64_t)DUAL_RATIO <= hi) return 1;
    const bool e_dual = ne > 0 && 2 * ne <= 2 * nv, t_dual = nt > 0 && 3 * nt <= 2 * ne;
    const bool any_dual = e_dual || t_dual, any_d = (ne > 0 && !e_dual) || (nt > 0 && !t_dual);
    return !any_dual ? 0 : any_d ? 2 : 1;
}
}  // namespace

// False when CUDA refused a launch (its resources): the form is not done,
// and the general path says what it thinks of the device.
static bool c2_launched() { return cudaGetLastError() == cudaSuccess; }

static int c2_read_status(Context *ctx, const C2Args &a, C2Status *hs) {
    OPH_CUDA_TRY(cudaMemcpyAsync(hs, a.st, sizeof(C2Status), cudaMemcpyDeviceToHost, ctx->stream));
    OPH_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return OPH_OK;
}

static int c2_run_graph(Context *ctx, C2Args a, int64_t nv, int64_t ne, int64_t nt, C2Status *hs, bool *done) {
    cudaStream_t s = ctx->stream;
    const int64_t nodes = nv + nt + 1;
    for (char *p = nullptr;;) {
        Carve c{p};
        a.tlist = c.take<int32_t>(nt + 1);
        a.ends = c.take<int2>(2 * ne);
        a.parent = c.take<int>(nodes);
        a.best = c.take<unsigned long long>(nodes);
        a.list[0] = c.take<int32_t>(2 * ne);
        a.list[1] = c.take<int32_t>(2 * ne);
        if (p) break;
        p = (char *)ctx_alloc(ctx, S_C2_MODE, c.off);
        if (!p) return OPH_OK;
    }
    // a grid that is resident as a whole, no larger than the first round's work
    static PerDevice per_sm;
    const int nb = per_sm.get(ctx->device, [] {
        int n = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_c2_graph, C2_THREADS, 0) == cudaSuccess ? n : 0;
    });
    if (nb <= 0) {
        cudaGetLastError();
        return OPH_OK;
    }
    const int gg = c2_grid(ctx, ne, std::min(nb, 4));
    a.neg = nullptr;
    OPH_CUDA_TRY(cudaMemsetAsync(a.best, 0xff, sizeof(unsigned long long) * nodes, s));
    k_c2_edges<<<c2_grid(ctx, ne, 8), C2_THREADS, 0, s>>>(a);
    k_c2_surface<<<c2_grid(ctx, a.m, 16), C2_THREADS, 0, s>>>(a);
    if (ctx->profile) cudaEventRecord(ctx->ev[2], s);
    int max_rounds = C2_MAX_ROUNDS;
    void *params[] = {&a, &max_rounds};
    // one such grid at a time on a device: its blocks wait for one another,
    // and another thread's context may have half the device's blocks
    static std::mutex alone[64];
    std::unique_lock<std::mutex> turn(alone[ctx->device & 63]);
    cudaLaunchCooperativeKernel((const void *)k_c2_graph, dim3(gg), dim3(C2_THREADS), params, 0, s);
    if (!c2_launched()) return OPH_OK;
    ctx->launches += 3;
    cudaEventRecord(ctx->ev[1], s);
    int rc = c2_read_status(ctx, a, hs);
    turn.unlock();
    *done = !rc && !hs->bad && !hs->crowded && !hs->unfinished;
    return rc;
}

template <bool RUNS, int THREADS, int WORDS>
static int c2_residual_grid(Context *ctx) {
    static PerDevice per_sm;
    constexpr int SMEM = WORDS * (int)sizeof(uint32_t);
    static PerDevice attr;
    if (!allow_shared(attr, ctx->device, k_c2_residual<RUNS, THREADS, WORDS>, SMEM)) return 0;
    const int nb = per_sm.get(ctx->device, [] {
        int n = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_c2_residual<RUNS, THREADS, WORDS>, THREADS, SMEM) ==
                       cudaSuccess
                   ? n
                   : 0;
    });
    if (nb <= 0) {
        cudaGetLastError();
        return 0;
    }
    return nb * ctx->sm_count;
}

template <bool RUNS>
static int c2_run_dense(Context *ctx, C2Args a, int64_t ne, int64_t nt, C2Status *hs, bool *done) {
    // what a form's tables may cost, in entries: a few times the matrix itself
    // (sparse complexes on many vertices are left to the general path)
    const long long room = (1ll << 24) + 8 * hs->nnz;
    const long long cells = RUNS ? hs->pairs : hs->cells, run_words = RUNS ? hs->run_words : 0;
    if (hs->max_nv > (RUNS ? 1 << ADJ_SHIFT : C2_MAX_NV) || 3 * cells > room || 2 * run_words > room) return OPH_OK;
    cudaStream_t s = ctx->stream;
    const bool small = RUNS && hs->max_nv <= RS_SMALL_NV;
    // (a window starts at a multiple of 128 columns)
    const bool xl = !RUNS && hs->max_cols > 32 * RS_LARGE_WORDS - 128 && hs->max_cols <= 32 * RS_XL_WORDS - 128;
    int gr = small ? c2_residual_grid<true, RS_SMALL, RS_SMALL_WORDS>(ctx)
             : xl  ? c2_residual_grid<false, RS_LARGE, RS_XL_WORDS>(ctx)
                   : c2_residual_grid<RUNS, RS_LARGE, RS_LARGE_WORDS>(ctx);
    if (gr == 0) return OPH_OK;
    // the components of C2_MAX_NV vertices take 48 KB beside the kernel's own shared memory
    static PerDevice roomy;
    if (!RUNS && !allow_shared(roomy, ctx->device, k_c2_triangles<RUNS>, 6 * C2_MAX_NV)) return OPH_OK;
    gr = (int)std::min<int64_t>(ne, gr);
    const int nv = hs->nv;
    a.arena_cap = (1 << 20) + 16 * ne;
    size_t head = 0;
    for (char *p = nullptr;;) {
        Carve c{p};
        a.dead = c.take<uint8_t>(nv + 1);
        head = c.off;  // zeroed
        a.runs = c.take<uint2>(run_words);
        a.owned = c.take<uint32_t>((a.m + 31) / 32 + 4);
        a.fixed = c.take<uint32_t>((a.m + 31) / 32 + 4);
        a.res = c.take<int32_t>(ne);
        a.sum = c.take<unsigned long long>(ne);
        a.arena = c.take<int32_t>(a.arena_cap);
        a.lists = c.take<int32_t>((size_t)gr * rs_list(small ? RS_SMALL : RS_LARGE));
        a.whole = !RUNS && hs->max_cols <= 32 * (xl ? RS_XL_WORDS : RS_LARGE_WORDS) - 128;
        a.map_words = a.whole ? ((hs->max_cols + 127) / 32 + 4) & ~3 : RS_LARGE_WORDS;
        a.map_cap = small ? 0
                          : (int)std::min<int64_t>(a.whole ? 2 * ne : ne,
                                                   (xl ? 4ll : 1ll) * RS_MAPS * RS_LARGE_WORDS / a.map_words);
        a.maps = c.take<uint32_t>((size_t)a.map_cap * a.map_words);
        if (p) break;
        p = (char *)ctx_alloc(ctx, S_C2_MODE, c.off);
        if (!p) return OPH_OK;
    }
    if (!RUNS) a.runs = nullptr;
    const size_t cell_bytes = sizeof(int32_t) * (size_t)std::max<long long>(cells, 1);
    a.cells = (int32_t *)ctx_alloc(ctx, S_C2_CELLS, (RUNS ? 3 : 1) * cell_bytes);
    if (!a.cells) return OPH_OK;
    a.adj = RUNS ? a.cells + cells : nullptr;  // cells is a multiple of 32
    a.tab = RUNS ? a.adj + cells : nullptr;
    a.ends = nullptr;
    const int kb = std::min(a.count, ctx->sm_count * 4);
    OPH_CUDA_TRY(cudaMemsetAsync(a.cells, 0xff, cell_bytes, s));
    if (RUNS) OPH_CUDA_TRY(cudaMemsetAsync(a.tab, NO_EDGE & 0xff, cell_bytes, s));
    OPH_CUDA_TRY(cudaMemsetAsync(ctx->bufs[S_C2_MODE].ptr, 0, head, s));
    if (!RUNS) k_c2_cells<<<1, 1024, 0, s>>>(a);
    k_c2_edges<<<c2_grid(ctx, ne, 8), C2_THREADS, 0, s>>>(a);
    // the components, or a row of vertices to sort
    const int smem = std::max(6 * hs->max_nv, RUNS ? 4 * c2_pitch(hs->max_nv) : 0);
    const int sb = RUNS ? std::min(nv, ctx->sm_count * 4) : 0;
    k_c2_triangles<RUNS><<<kb + sb + c2_grid(ctx, RUNS ? 32 * ne : a.m, 16), C2_THREADS, smem, s>>>(a, kb, sb, hs->max_nv);
    if (RUNS) {
        k_c2_runs_out<<<c2_grid(ctx, a.m, 16), C2_THREADS, 0, s>>>(a);
    } else {
        k_c2_table_init<<<c2_grid(ctx, a.m, 16), C2_THREADS, 0, s>>>(a);
        k_c2_table_pairs<<<c2_grid(ctx, 32 * ne, 8), C2_THREADS, 0, s>>>(a);
    }
    if (ctx->profile) cudaEventRecord(ctx->ev[2], s);
    if (small)
        k_c2_residual<true, RS_SMALL, RS_SMALL_WORDS><<<gr, RS_SMALL, RS_SMALL_WORDS * sizeof(uint32_t), s>>>(a);
    else if (xl)
        k_c2_residual<false, RS_LARGE, RS_XL_WORDS><<<gr, RS_LARGE, RS_XL_WORDS * sizeof(uint32_t), s>>>(a);
    else
        k_c2_residual<RUNS, RS_LARGE, RS_LARGE_WORDS><<<gr, RS_LARGE, RS_LARGE_WORDS * sizeof(uint32_t), s>>>(a);
    if (!c2_launched()) return OPH_OK;
    ctx->launches += RUNS ? 4 : 6;
    cudaEventRecord(ctx->ev[1], s);
    int rc = c2_read_status(ctx, a, hs);
    // a table entry written twice (two triangles on the same edge and vertex,
    // which no simplicial complex has) shows in the count of those set
    *done = !rc && !hs->bad && !hs->overflow && (!RUNS || !hs->unsorted) &&
            (RUNS || hs->cells_set == 3ull * (unsigned long long)nt);
    return rc;
}

// Which calls try whole instances first: a CTA each pays while the CTAs have
// instances enough (batches of at least a hundred or so), or while one is not
// much longer alone than the grid-wide kernels' launches.
constexpr int64_t IN_MAX_COLS = 1 << 15;
constexpr int IN_MIN_COUNT = 128;

static int c2_run_inst(Context *ctx, C2Args a, C2Status *hs, bool *done, bool *looked) {
    *done = *looked = false;
    cudaStream_t s = ctx->stream;
    static PerDevice one, each, more;
    if (!allow_shared(one, ctx->device, k_c2_inst<true>, IN_SMEM) ||
        !allow_shared(each, ctx->device, k_c2_inst<false>, IN_SMEM) ||
        !allow_shared(more, ctx->device, k_c2_inst_more, IN_SMEM))
        return OPH_OK;
    int gr = c2_residual_grid<true, RS_SMALL, RS_SMALL_WORDS>(ctx);
    if (gr == 0) return OPH_OK;
    // bounds for the tables: guesses from the columns, or what an earlier call needed
    const int64_t m = a.m;
    long long need[4] = {std::min<long long>(m, m / 6 + 1024), std::min<long long>(m, m / 16 + 1024), m / 2 + 65536,
                         m / 4 + 65536};
    for (int q = 0; q < 4; q++) need[q] = std::max(need[q], ctx->c2_need[q]);
    const long long nwords = 4 * (m / 128 + a.count + 1);
    const int slots = 2 * ctx->sm_count;
    // equal instances fill the CTAs by themselves, and pieces read the tables again: 304 of 60 points
    // took 394 us whole and 405-420 split, 256 of 20 to 120 points 983 us whole and 690 split
    a.split_cols = (int)std::min<int64_t>(INT_MAX, m / slots * 3 / 4);
    a.chunk = m / a.count < IN_SPLIT ? 0 : (int)std::max<int64_t>(64, std::min<int64_t>(512, m / (40 * 2 * slots))) & ~7;
    const bool out_here = a.count == 1 && !a.chunk;
    for (int tries = 0; tries < 2; tries++) {
        a.cap_e = need[0];
        a.cap_v = need[1];
        a.cap_c = (need[2] + 3) & ~3ll;
        a.cap_r = need[3];
        a.arena_cap = (1 << 20) + 16 * a.cap_e;
        for (char *p = nullptr;;) {
            Carve c{p};
            a.st = c.take<C2Status>(1);
            a.inst = c.take<C2Inst>(a.count);
            a.words = c.take<C2Word>(nwords);
            if (p) break;
            p = (char *)ctx_alloc(ctx, S_C2_TAB, c.off);
            if (!p) return OPH_OK;
        }
        for (char *p = nullptr;;) {
            Carve c{p};
            a.elist = c.take<int32_t>(a.cap_e);
            a.erec = c.take<int4>(a.cap_e);
            a.neg = c.take<int32_t>(a.cap_e);
            a.res = c.take<int32_t>(a.cap_e);
            a.sum = c.take<unsigned long long>(a.cap_e);
            a.dead = c.take<uint8_t>(a.cap_v);
            a.order = c.take<int>(a.count);
            a.items = c.take<int2>(a.chunk ? a.cap_e / a.chunk + a.count : 1);
            if (p) break;
            p = (char *)ctx_alloc(ctx, S_C2_WORK, c.off);
            if (!p) return OPH_OK;
        }
        if (a.count <= slots || !a.chunk) a.order = nullptr;
        for (char *p = nullptr;;) {
            Carve c{p};
            a.runs = c.take<uint2>(a.cap_r);
            a.owned = c.take<uint32_t>(nwords);
            a.fixed = c.take<uint32_t>(nwords);
            a.arena = c.take<int32_t>(a.arena_cap);
            a.lists = c.take<int32_t>((size_t)gr * rs_list(RS_SMALL));
            if (p) break;
            p = (char *)ctx_alloc(ctx, S_C2_MODE, c.off);
            if (!p) return OPH_OK;
        }
        a.cells = (int32_t *)ctx_alloc(ctx, S_C2_CELLS, (a.chunk ? 3 : 2) * sizeof(int32_t) * (size_t)a.cap_c);
        if (!a.cells) return OPH_OK;
        a.adj = a.cells + a.cap_c;
        a.tab = a.chunk ? a.adj + a.cap_c : nullptr;
        OPH_CUDA_TRY(cudaMemsetAsync(a.st, 0, sizeof(C2Status), s));
        if (a.order) {
            k_c2_inst_order<<<1, 1024, 0, s>>>(a);
            ctx->launches++;
        }
        if (out_here) k_c2_inst<true><<<1, IN_THREADS, IN_SMEM, s>>>(a);
        else k_c2_inst<false><<<std::min(a.count, slots), IN_THREADS, IN_SMEM, s>>>(a);
        if (a.chunk) {
            k_c2_inst_more<<<(int)std::min<int64_t>(slots, a.cap_e / a.chunk + 1), IN_THREADS, IN_SMEM, s>>>(a);
            ctx->launches++;
        }
        // enough blocks for the outputs of one instance as of many
        const int parts = (int)std::max<int64_t>(1, std::min<int64_t>(16, (m / a.count + IO_COLS - 1) / IO_COLS));
        if (!out_here) {
            const int blocks = parts * std::min(a.count, 65535);
            if (blocks <= 8 * ctx->sm_count) k_c2_inst_out<true><<<blocks, IO_THREADS, 0, s>>>(a, parts);
            else k_c2_inst_out<false><<<blocks, IO_THREADS, 0, s>>>(a, parts);
            ctx->launches++;
        }
        if (ctx->profile) cudaEventRecord(ctx->ev[2], s);
        // a residual edge or so per vertex
        const int rg = (int)std::min<int64_t>(gr, std::max<int64_t>(1, a.cap_e));
        k_c2_residual<true, RS_SMALL, RS_SMALL_WORDS><<<rg, RS_SMALL, RS_SMALL_WORDS * sizeof(uint32_t), s>>>(a);
        if (!c2_launched()) return OPH_OK;
        ctx->launches += 2;
        cudaEventRecord(ctx->ev[1], s);
        int rc = c2_read_status(ctx, a, hs);
        if (rc) return rc;
        *looked = true;
        if (hs->refused || !hs->no_room) break;
        const long long used[4] = {hs->ne, hs->nv, hs->pairs, hs->run_words};
        for (int q = 0; q < 4; q++)
            if (used[q] > need[q]) need[q] = ctx->c2_need[q] = used[q] + used[q] / 8;
    }
    *done = !hs->refused && !hs->no_room && !hs->overflow;
    return OPH_OK;
}

// Contexts that ask for something of the sweeps keep them: trackers, a forced
// matrix, a tuned narrow tier, a sweep cap or a fixed initial store, the exact
// slot counts of the store's tiers, and the switches that pick a form of the
// transpose, the tiers or the sweep loop.
bool complex2_applies(const Context *ctx, int algo) {
    for (const char *name : {"OPH_NO_INST_TRANSPOSE", "OPH_NO_CLUSTER", "OPH_HOST_LOOP", "OPH_TRACE"})
        if (getenv(name)) return false;
    return algo == OPH_ALGO_PMS && !ctx->track && ctx->dual == OPH_DUAL_AUTO && ctx->tier0 == 0 &&
           ctx->max_sweeps == 0 && ctx->initial_pool_bytes == 0 && !ctx->count_slots;
}

size_t complex2_least(const Context *ctx, int64_t m, int64_t nnz) {
    const double columns = 8.0 * m + 0.5 * m;  // outputs, words
    // a graph: three triangles to two edges at most, so the edges hold a quarter of the entries at least
    const double graph_ne = nnz / 4.0, graph = columns + 56 * graph_ne + 12 * std::max(0.0, m - nnz / 2.0);
    // dense: ne edges span at most sqrt(2)/3 ne^1.5 triangles; the arena, and a list a CTA
    const double ne = std::pow(nnz / 3.42, 2.0 / 3.0), lists = std::min(ne, 6.0 * ctx->sm_count);
    const double dense = columns + 0.25 * m + 24 * ne + sizeof(int32_t) * ((1 << 20) + lists * rs_list(RS_SMALL));
    return (size_t)(5 * nnz > 12 * m ? dense : std::min(graph, dense));
}

int reduce_complex2(Context *ctx, C2Job &job, oph_info *info, bool *taken) {
    *taken = false;
    job.nnz_read = false;
    ctx->launches = 0;
    ctx->prof = oph_profile{};
    const int64_t m = job.m;
    if (m < 1 || m >= (1 << 29)) return OPH_OK;
    if (!job.rows && job.want_nnz == 0) return OPH_OK;  // vertices only: one sweep finds nothing to do
    cudaStream_t s = ctx->stream;
    const int64_t nwords = (m + 31) / 32, ntiles = (m + C2_TILE - 1) / C2_TILE;
    const bool batch = job.inst_off != nullptr;
    C2Args a{};
    a.m = m;
    a.colptr = job.colptr;
    a.rows = job.rows;
    a.inst_off = job.inst_off;
    a.count = batch ? job.count : 1;
    a.low = job.low;
    a.ess = job.ess;
    a.one_based = job.one_based;
    a.nnz = job.want_nnz;
    static_assert(sizeof(C2Status) <= sizeof(DevStatus), "read back through the context's pinned status block");
    C2Status *hs = reinterpret_cast<C2Status *>(ctx->h_status);
    DevStatus *hb = ctx->h_status + 1;
    int rc;
    bool done = false;
    bool runs = true, counted = false;  // whether the run form may apply; whether hs holds the counts
    int64_t nv, ne, nt;
    cudaEventRecord(ctx->ev[0], s);
    if (job.rows && (!batch || job.want_nnz >= 0) && (batch ? a.count >= IN_MIN_COUNT || m / a.count <= IN_MAX_COLS : m <= IN_MAX_COLS)) {
        if (job.before) OPH_CUDA_TRY(cudaMemcpyAsync(hb, job.before, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
        bool looked = false;
        if ((rc = c2_run_inst(ctx, a, hs, &done, &looked))) return rc;
        if (looked) {
            job.nnz = hs->nnz;
            job.nnz_read = true;
            job.before_error = job.before ? hb->error : 0;
            if (job.before_error || hs->bad) return OPH_OK;
            done = done && (job.want_nnz < 0 || hs->nnz == job.want_nnz);
            runs = !hs->unsorted;
            counted = !batch;
        }
    }
    if (!done) {
    for (char *p = nullptr;;) {
        Carve c{p};
        a.st = c.take<C2Status>(1);
        a.words = c.take<C2Word>(nwords + 4);
        a.tiles = c.take<int2>(ntiles);
        a.inst = c.take<C2Inst>(a.count);
        a.winst = batch ? c.take<int>(nwords) : nullptr;
        if (p) break;
        p = (char *)ctx_alloc(ctx, S_C2_TAB, c.off);
        if (!p) return OPH_OK;  // no room: the general path decides
    }
    OPH_CUDA_TRY(cudaMemsetAsync(a.st, 0, sizeof(C2Status), s));
    k_c2_words<<<(int)std::min<int64_t>(ntiles, (int64_t)ctx->sm_count * 8), C2_THREADS, 0, s>>>(a);
    k_c2_scan<<<1, 1024, 0, s>>>(a, ntiles);
    OPH_CUDA_TRY(cudaGetLastError());
    ctx->launches += 2;
    if (counted) {  // one matrix, whose columns a CTA has counted
        C2Status st{};
        st.nnz = hs->nnz;
        st.nv = st.max_nv = hs->nv;
        st.max_cols = (int)m;
        st.ne = hs->ne;
        st.cells = (long long)c2_pitch(st.nv) * st.ne;
        st.pairs = (long long)c2_pitch(st.nv) * st.nv;
        st.run_words = (long long)((st.nv + 31) >> 5) * st.ne;
        *hs = st;
    } else {
        if (job.before) OPH_CUDA_TRY(cudaMemcpyAsync(hb, job.before, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
        if ((rc = c2_read_status(ctx, a, hs))) return rc;
        job.nnz = hs->nnz;
        job.nnz_read = true;
        job.before_error = job.before ? hb->error : 0;
        if (job.before_error) return OPH_OK;
    }
    nv = hs->nv;
    ne = hs->ne;
    nt = m - nv - ne;
    if (hs->bad || hs->nnz != 2 * ne + 3 * nt || (job.want_nnz >= 0 && hs->nnz != job.want_nnz)) return OPH_OK;
    if (ne == 0 || ne >= (1 << 29) || !job.rows) return OPH_OK;
    for (char *p = nullptr;;) {
        Carve c{p};
        a.vlist = c.take<int32_t>(nv + 1);
        a.elist = c.take<int32_t>(ne);
        a.erec = c.take<int4>(ne);
        a.neg = c.take<int32_t>(ne);
        if (p) break;
        p = (char *)ctx_alloc(ctx, S_C2_WORK, c.off);
        if (!p) return OPH_OK;
    }
    k_c2_lists<<<c2_grid(ctx, nwords, 8), C2_THREADS, 0, s>>>(a);
    ctx->launches++;
    // every edge with at most two triangles: a graph (an edge found to have
    // more leaves it to the dense form)
    if (3 * nt <= 2 * ne && (rc = c2_run_graph(ctx, a, nv, ne, nt, hs, &done))) return rc;
    if (!done && !hs->bad && runs && (rc = c2_run_dense<true>(ctx, a, ne, nt, hs, &done))) return rc;
    if (!done && !hs->bad && !hs->overflow) {
        // not in runs: the same with the table (the status as before the try)
        if (hs->unsorted) {
            OPH_CUDA_TRY(cudaMemsetAsync(&a.st->unsorted, 0, sizeof(int), s));
        }
        if ((rc = c2_run_dense<false>(ctx, a, ne, nt, hs, &done))) return rc;
    }
    if (!done) return OPH_OK;
    }
    nv = hs->nv;
    ne = hs->ne;
    nt = m - nv - ne;
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
    if (ctx->profile) {
        cudaEventElapsedTime(&ctx->prof.setup_ms, ctx->ev[0], ctx->ev[2]);
        cudaEventElapsedTime(&ctx->prof.phase2_wide_ms, ctx->ev[2], ctx->ev[1]);
        ctx->prof.tier_ms[2] = ctx->prof.phase2_wide_ms;
        ctx->prof.phase2_launches = 1;
        ctx->prof.tier_additions[3] = (int64_t)(hs->joins + hs->adds);
        ctx->prof.tier_slots[3] = (int64_t)(4 * hs->joins + hs->slots);
    }
    ctx->prof.kernel_launches = ctx->launches;
    *info = oph_info{};
    info->sweeps = std::max(1, hs->rounds);
    info->num_iters = info->sweeps + 1;
    info->additions = (int64_t)(hs->joins + hs->adds);
    info->slots_moved = (int64_t)(4 * hs->joins + hs->slots);
    for (int q : {S_C2_TAB, S_C2_WORK, S_C2_MODE, S_C2_CELLS}) info->pool_bytes += (int64_t)ctx->bufs[q].bytes;
    info->device_ms = ms;
    info->dual = c2_named_matrix(m, nv, ne, nt);
    *taken = true;
    return OPH_OK;
}

}  // namespace oph
