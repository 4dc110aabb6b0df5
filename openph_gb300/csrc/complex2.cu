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
// D' is never built column by column.  A table holds, for every edge and
// vertex, the triangle they span: a triangle writes its three entries with
// no count, scan, cursor or sort, and an edge's row of it is its column of
// D'.  The edges that the graph of edges on vertices pairs are cleared
// (c2_kruskal); an edge whose first triangle has it as its last edge is
// paired with it at once, as nothing can be added to either (an apparent
// pair: 98-99% of a Rips complex's edges).  What is left (107 of 58,988 edges
// on the 5M-column torus) is reduced a column per CTA (k_c2_residual).
//
// What is accepted is checked on the device before anything is written: every
// column has 0, 2 or 3 rows, ascending and in range, the rows of an edge are
// vertices, the rows of a triangle are the three edges of a triangle (so
// D D = 0, which clearing relies on).  Anything else, malformed input
// included, is left to the general path and its own checks.
#include <algorithm>
#include <climits>
#include <cstdlib>

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
    unsigned long long joins;
    int max_nv;      // the largest instance's vertices
    int unsorted;    // the triangles do not come in runs
    int nres, cursor, overflow;      // residual edges; the CTAs' queue; a list ran out of room
    long long cells;                 // entries of the edge-vertex table
    long long pairs, run_words;      // entries of the edge-id table, words of the runs' bits
    unsigned long long cells_set;    // entries of the edge-vertex table that a triangle wrote
    unsigned long long arena;        // entries of published lists
    unsigned long long adds, slots;  // additions of the residual columns, entries toggled
};

constexpr int C2_THREADS = 256, C2_TILE = 2048;
constexpr int C2_MAX_ROUNDS = 512;
constexpr int C2_MAX_NV = 8192;                   // vertices of an instance the dense form takes
constexpr int RS_WAVE = 32;                       // residual columns: pivots added at a time,
constexpr int RS_LIST = 16384;                    //   edges a column under reduction may be the sum of
constexpr int RS_FLAG = 1 << 30;

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
    // (vertices by vertices), its rows in edge order, and the runs (per edge
    // and 32 vertices: which have a triangle, and the first one's column); which triangles have an
    // owner (low[] names it), and which for good; the residual edges, and the
    // list each is the sum of (offset << 24 | length)
    int32_t *neg;
    uint8_t *dead;
    int32_t *cells, *adj;
    uint2 *runs;
    uint32_t *owned, *fixed;
    int32_t *res;
    unsigned long long *sum;
    int32_t *arena;
    long long arena_cap;
    int32_t *lists;           // per CTA: RS_LIST edges
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

// The pitch of an instance's rows over its vertices: whole 16-byte loads.
__host__ __device__ __forceinline__ int c2_pitch(int nv) { return (nv + 3) & ~3; }

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
            if (atomicCAS(t + (int64_t)x * pitch + y, -1, k - in.eoff) != -1 ||
                w.vpre + __popc(w.v & below(j & 31)) != in.voff + in.nv)
                a.st->unsorted = 1;
            t[(int64_t)y * pitch + x] = k - in.eoff;
        }
        if (a.ends) {
            a.ends[k] = make_int2(u, v);
            a.ends[2 * (int64_t)ne - 1 - k] = make_int2(-1, -1);
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
#pragma unroll
        for (int q = 0; q < 3; q++) {
            int *e = reinterpret_cast<int *>(a.ends + (2 * (int64_t)ne - 1 - k[q]));
            if (atomicCAS(e, -1, id) != -1 && atomicCAS(e + 1, -1, id) != -1) crowded = true;
        }
    }
    if (bad) a.st->bad = 1;
    if (crowded) a.st->crowded = 1;
}

// Outputs before any pair is known, and the graph's nodes.
__global__ void __launch_bounds__(C2_THREADS) k_c2_graph_init(C2Args a) {
    if (a.st->bad || a.st->crowded) return;
    const int64_t nodes = a.m - a.st->ne + 1, stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int none = a.one_based ? 0 : -1;
    for (int64_t j = i0; j < a.m; j += stride) {
        a.low[j] = none;
        if (a.ess) a.ess[j] = 1;
    }
    for (int64_t i = i0; i < nodes; i += stride) {
        a.parent[i] = (int)i;
        a.best[i] = ~0ull;
    }
}

// The component of a node: its oldest node.  Parents are always older than
// their children, and only grow older; the path is halved on the way (racing
// writers all write ancestors).
__device__ __forceinline__ int c2_find(int *parent, int x) {
    int cur = __ldcg(parent + x);
    if (cur == x) return x;
    int prev = x;
    for (;;) {
        const int next = __ldcg(parent + cur);
        if (next == cur) return cur;
        __stcg(parent + prev, next);
        prev = cur;
        cur = next;
    }
}

// A pair: node x dies at slot s.
__device__ __forceinline__ void c2_die(const C2Args &a, int nv, int ne, int nt, int s, int x) {
    int lo, col, k;
    if (s < ne) {  // an edge of D: its low is the vertex
        k = s;
        col = a.elist[k];
        lo = a.vlist[x];
    } else {  // an edge of D': the triangle's low is the edge
        k = 2 * ne - 1 - s;
        lo = a.elist[k];
        col = a.tlist[nt - 1 - (x - nv - 1)];
    }
    const int base = a.inst_off ? (int)a.inst[a.erec[k].z].base : 0;
    a.low[col] = lo - base + a.one_based;
    if (a.ess) {
        a.ess[col] = 0;
        a.ess[lo] = 0;
    }
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
// A round is two passes over the list of such edges, with a grid barrier
// after each.  Bound by the latency of its dependent loads (parents, best)
// and the barriers, not by bandwidth: 12 rounds on the 512 x 512 lower-star
// image (1.57M slots, then 320K, 76K, ...), 19 on white noise of that size.
__global__ void __launch_bounds__(C2_THREADS) k_c2_graph(C2Args a, int max_rounds) {
    if (a.st->bad || a.st->crowded) return;  // written by earlier kernels: the same for every block
    cg::grid_group grid = cg::this_grid();
    const int nv = a.st->nv, ne = a.st->ne, nt = (int)(a.m - nv - ne), ground = nv;
    const int stride = gridDim.x * blockDim.x, i0 = blockIdx.x * blockDim.x + threadIdx.x;
    int n = 2 * ne;
    unsigned long long joins = 0;
    for (int round = 0;; round++) {
        const unsigned long long tag = (unsigned long long)(~(unsigned)round) << 32;
        const int32_t *in = a.list[(round + 1) & 1];
        int32_t *out = a.list[round & 1];
        int *count = &a.st->live[round % 3];
        // the warp stays whole for the aggregated append
        for (int i1 = i0 - (threadIdx.x & 31); i1 < n; i1 += stride) {
            const int i = i1 + (threadIdx.x & 31);
            bool live = i < n;
            int s = 0;
            if (live) {
                s = round ? in[i] : i;
                int2 e = __ldcg(a.ends + s);
                if (round) {
                    const int x = c2_find(a.parent, e.x), y = c2_find(a.parent, e.y);
                    live = x != y;
                    if (live && (x != e.x || y != e.y)) __stcg(a.ends + s, make_int2(x, y));
                    e = make_int2(x, y);
                } else if (s >= ne) {
                    live = e.x >= 0;  // an edge without triangles: an empty column of D'
                    if (live && e.y < 0) {
                        e.y = ground;
                        a.ends[s] = e;
                    }
                }
                if (live) {
                    const unsigned long long key = tag | (unsigned)s;
                    if (e.x != ground && __ldcg(a.best + e.x) > key) atomicMin(a.best + e.x, key);
                    if (e.y != ground && __ldcg(a.best + e.y) > key) atomicMin(a.best + e.y, key);
                }
            }
            const unsigned b = __ballot_sync(0xffffffffu, live);
            if (b) {
                const int lane = threadIdx.x & 31, leader = __ffs(b) - 1;
                int at = 0;
                if (lane == leader) at = atomicAdd(count, __popc(b));
                at = __shfl_sync(0xffffffffu, at, leader);
                if (live) out[at + __popc(b & below(lane))] = s;
            }
        }
        grid.sync();
        n = __ldcg(count);
        if (i0 == 0) {
            a.st->live[(round + 1) % 3] = 0;  // last read two rounds ago
            a.st->rounds = round + 1;
            if (n > 0 && round + 1 >= max_rounds) a.st->unfinished = 1;
        }
        if (n == 0 || round + 1 >= max_rounds) break;
        for (int i = i0; i < n; i += stride) {
            const int s = __ldcg(out + i);
            const int2 e = __ldcg(a.ends + s);
            const unsigned long long key = tag | (unsigned)s;
            const int x = max(e.x, e.y), y = min(e.x, e.y);  // only the younger end can die here
            if (x != ground && __ldcg(a.best + x) == key) {
                __stcg(a.parent + x, y);
                c2_die(a, nv, ne, nt, s, x);
                joins++;
            }
        }
        grid.sync();
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
constexpr int KR_ITEMS = 4, KR_EDGES = KR_ITEMS * C2_THREADS;
__device__ __forceinline__ int kr_find(uint16_t *parent, int x) {
    for (;;) {
        const int p = ((volatile uint16_t *)parent)[x];
        if (p == x) return x;
        const int g = ((volatile uint16_t *)parent)[p];
        ((volatile uint16_t *)parent)[x] = (uint16_t)g;
        x = g;
    }
}
__device__ void c2_kruskal(const C2Args &a, const C2Inst &in, uint32_t *best, uint16_t *parent, int *s_parts) {
    const int tid = threadIdx.x;
    for (int x = tid; x < in.nv; x += C2_THREADS) {
        parent[x] = (uint16_t)x;
        best[x] = 0xffffffffu;
    }
    if (tid == 0) *s_parts = in.nv;
    __syncthreads();
    unsigned tag = 0x3fffff;  // counts down by rounds: nothing in best[] is reset
    for (int c0 = 0; c0 < in.ne && *s_parts > 1; c0 += KR_EDGES) {
        int u[KR_ITEMS], v[KR_ITEMS];
#pragma unroll
        for (int q = 0; q < KR_ITEMS; q++) {
            const int i = c0 + q * C2_THREADS + tid;
            const int4 e = i < in.ne ? a.erec[in.eoff + i] : make_int4(in.voff, in.voff, 0, 0);
            u[q] = e.x - in.voff;
            v[q] = e.y - in.voff;
        }
        for (;; tag--) {
            bool live = false;
#pragma unroll
            for (int q = 0; q < KR_ITEMS; q++) {
                if (u[q] == v[q]) continue;
                u[q] = kr_find(parent, u[q]);
                v[q] = kr_find(parent, v[q]);
                if (u[q] == v[q]) continue;
                live = true;
                const unsigned key = tag << 10 | (unsigned)(q * C2_THREADS + tid);
                atomicMin(best + u[q], key);
                atomicMin(best + v[q], key);
            }
            if (!__syncthreads_or(live)) break;
#pragma unroll
            for (int q = 0; q < KR_ITEMS; q++) {
                const int young = max(u[q], v[q]), old = min(u[q], v[q]);
                if (young == old || best[young] != (tag << 10 | (unsigned)(q * C2_THREADS + tid))) continue;
                parent[young] = (uint16_t)old;
                a.neg[in.eoff + c0 + q * C2_THREADS + tid] = young;
                a.dead[in.voff + young] = 1;
                atomicSub(s_parts, 1);
            }
            __syncthreads();
        }
    }
}

// One vertex's row of the edge-id table in the order of its edges: each entry
// written at the number of smaller ones (a warp; `row` holds the row in
// shared memory, absent edges as the largest id).  An entry is the edge's
// rank and the other vertex.
constexpr int ADJ_SHIFT = 10;
__device__ void c2_sort_row(const int32_t *src, int32_t *dst, int nv, int pitch, int32_t *row) {
    const int lane = threadIdx.x & 31;
    for (int i = lane; i < pitch; i += 32) {
        const int x = src[i];
        row[i] = x < 0 ? INT_MAX : x;
        dst[i] = INT_MAX;
    }
    __syncwarp();
    for (int i = lane; i < nv; i += 32) {
        const int x = row[i];
        if (x == INT_MAX) continue;
        int at = 0;
        for (int q = 0; q < pitch; q += 4) {
            const int4 y = *reinterpret_cast<const int4 *>(row + q);
            at += (y.x < x) + (y.y < x) + (y.z < x) + (y.w < x);
        }
        dst[at] = x << ADJ_SHIFT | i;
    }
    __syncwarp();
}

// The first blocks pair the edges with vertices (an instance each); with
// RUNS, the next ones sort the vertices' edges (a warp each); the rest check
// the triangles, a thread each.
//
// RUNS: in a Rips filtration every triangle follows its last edge with no
// other edge between (triangles carry their longest edge's length and come
// after it), the third vertices of an edge's triangles ascending.  A set of
// vertices per edge, one bit each, then names all of its run, and with it
// every triangle: per 32 vertices the bits and the first one's column, so
// (edge f, vertex z) is that column + the bits below z.  The triangles write
// nothing else, and the lanes of a warp on one word write together, where the table costs three scattered 4-byte
// writes each, of which 2% are ever read.  A triangle out of that order, or
// a second edge on the same two vertices, sets `unsorted`, and the table is
// built instead.
template <bool RUNS>
__global__ void __launch_bounds__(C2_THREADS) k_c2_triangles(C2Args a, int kruskal_blocks, int sort_blocks, int max_nv) {
    extern __shared__ __align__(16) uint32_t tri_smem[];
    __shared__ int s_parts;
    if (a.st->bad || (RUNS && a.st->unsorted)) return;
    const int lane = threadIdx.x & 31;
    if ((int)blockIdx.x < kruskal_blocks) {
        for (int b = blockIdx.x; b < a.count; b += kruskal_blocks) {
            c2_kruskal(a, a.inst[b], tri_smem, reinterpret_cast<uint16_t *>(tri_smem + max_nv), &s_parts);
            __syncthreads();
        }
        return;
    }
    if (RUNS && (int)blockIdx.x < kruskal_blocks + sort_blocks) {
        int32_t *row = reinterpret_cast<int32_t *>(tri_smem) + (threadIdx.x >> 5) * c2_pitch(max_nv);
        const int warps = sort_blocks * (C2_THREADS / 32);
        for (int v = (blockIdx.x - kruskal_blocks) * (C2_THREADS / 32) + (threadIdx.x >> 5); v < a.st->nv; v += warps) {
            const C2Inst &in = a.inst[c2_inst_of(a, a.vlist[v])];
            const int pitch = c2_pitch(in.nv);
            const int64_t at = in.coff + (int64_t)(v - in.voff) * pitch;
            c2_sort_row(a.cells + at, a.adj + at, in.nv, pitch, row);
        }
        return;
    }
    bool bad = false, unsorted = false;
    const int others = kruskal_blocks + sort_blocks;
    const int64_t stride = (int64_t)(gridDim.x - others) * C2_THREADS;
    for (int64_t j0 = (int64_t)(blockIdx.x - others) * C2_THREADS + (threadIdx.x - lane); j0 < a.m; j0 += stride) {
        const int64_t j = j0 + lane;
        const C2Word w = a.words[j0 >> 5];
        const bool tri = j < a.m && !(((w.v | w.e) >> lane) & 1u);
        const C2Inst &in = a.inst[tri ? c2_inst_of(a, j) : 0];
        int k[3], o[3];
        bool ok = tri && c2_triangle(a, j, w, in, k) &&
                  c2_opposite(a.erec[k[0]], a.erec[k[1]], a.erec[k[2]], o[0], o[1], o[2]);
        if (tri && !ok) bad = true;
        if (!RUNS) {
            if (ok)
#pragma unroll
                for (int q = 0; q < 3; q++)
                    a.cells[in.coff + (int64_t)(k[q] - in.eoff) * c2_pitch(in.nv) + (o[q] - in.voff)] = (int32_t)j;
            continue;
        }
        const unsigned lt = below(lane);
        const int last = w.epre + __popc(w.e & lt) - 1;  // the last edge before j
        const int z = ok ? o[2] - in.voff : 0;
        if (ok && k[2] != last) unsorted = true;
        // the third vertex of the triangle before it in the run is smaller
        int zp = __shfl_up_sync(0xffffffffu, z, 1);
        const bool okp = __shfl_up_sync(0xffffffffu, (int)ok, 1) != 0;
        bool first = true;  // of its word
        if (ok && k[2] == last && j - 1 != a.elist[last]) {
            if (lane == 0) {
                int kp[3], op[3];
                zp = c2_triangle(a, j - 1, a.words[(j - 1) >> 5], in, kp) &&
                             c2_opposite(a.erec[kp[0]], a.erec[kp[1]], a.erec[kp[2]], op[0], op[1], op[2])
                         ? op[2] - in.voff
                         : INT_MAX;
            } else if (!okp) {
                zp = INT_MAX;
            }
            if (zp >= z) unsorted = true;
            first = (zp >> 5) != (z >> 5);
        }
        // the bits of each word by one lane
        const int nw = (in.nv + 31) >> 5;
        const unsigned long long at =
            ok && k[2] == last ? (unsigned long long)in.roff + (unsigned long long)(last - in.eoff) * nw + (z >> 5)
                               : ~0ull;
        const unsigned peers = __match_any_sync(0xffffffffu, at);
        const unsigned v = __reduce_or_sync(peers, 1u << (z & 31));
        if (at != ~0ull && lane == __ffs(peers) - 1) {
            atomicOr(&a.runs[at].x, v);
            if (first) a.runs[at].y = (unsigned)j;
        }
    }
    if (bad) a.st->bad = 1;
    if (unsorted) a.st->unsorted = 1;
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
// * Waves: not only the low's pivot is added but those of the first RS_WAVE
//   set bits that have one.  Every column added comes before k in D' (a row
//   of the sum lies in a column of the sum, and its owner is the first column
//   that can hold it), so this is a reduction like any other, and the two
//   chains of 557 additions on the torus take 36 and 40 waves.
// * Owners: low[t] names the owner of triangle t.  A residual column claims
//   its low by compare-and-swap once its list is published.  Found claimed by
//   an earlier column, that column is added; by a later one, the claim is
//   taken over and this CTA goes on with the later column plus its own.  No
//   CTA waits for another, and the lows are those of any complete reduction.
//
// Bound by latency: a wave is a search of the window and four dependent trips
// to L2 (which set bits have owners, the owners, their vertices, their
// triangles) and of the instructions of one SM, so the columns of a wave are
// spread over the CTA's warps and no more of each is looked at than the window
// holds.  Complexes on many
// vertices, with few long columns, take large CTAs and windows; batches of
// small ones as many CTAs as fit.
template <bool RUNS, int THREADS, int WORDS>
__global__ void __launch_bounds__(THREADS) k_c2_residual(C2Args a) {
    if (a.st->bad || (RUNS && a.st->unsorted)) return;
    extern __shared__ __align__(16) uint32_t bits[];  // WORDS
    constexpr int NW = THREADS / 32;
    __shared__ int s_low[NW], s_cnt[NW], s_wave[RS_WAVE];
    __shared__ int s_i, s_later, s_act, s_other;
    __shared__ unsigned long long s_sum;
    enum { ACT_DONE, ACT_ADD, ACT_STEAL, ACT_FAIL };
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nres = a.st->nres, none = a.one_based ? 0 : -1;
    int32_t *list = a.lists + (size_t)blockIdx.x * RS_LIST;
    unsigned long long adds = 0, slots = 0;
    for (;;) {
        if (tid == 0) {
            s_i = atomicAdd(&a.st->cursor, 1);
            s_later = INT_MAX;
        }
        __syncthreads();
        const int i = s_i;
        if (i >= nres) break;
        int k = a.res[i];
        const C2Inst in = a.inst[a.erec[k].z];
        // columns here are relative to in.wbase; an owner's value in low[] is col - shift
        const int shift = (int)(in.base - in.wbase) - a.one_based, cols = (int)(in.base + in.cols - in.wbase);
        int32_t *const out_low = a.low + in.wbase, *const out_ess = a.ess ? a.ess + in.wbase : nullptr;
        uint32_t *const owned = a.owned + in.woff;
        const uint32_t *const fixed = a.fixed + in.woff;
        int n = 1, pos = a.elist[k] + 1, w0 = 0, hi = 0, later = INT_MAX;  // triangles come after their edges
        if (tid == 0) __stcg(list, k);
        bool fresh = true;  // a new window, from pos
        int wave = 4;       // most columns take a wave or two: long ones get the full width
        for (;;) {
            if (fresh) {
                w0 = pos & ~127;
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
            wave = min(2 * wave, RS_WAVE);
            __syncthreads();
            if (wid == 0 && lane < cnt) {  // the owners, all at once
                const int t = s_wave[lane] & ~RS_FLAG, fl = s_wave[lane] & RS_FLAG;
                int o;
                if (RUNS && !fl) o = c2_edge_rank(a, in, t) - 1;  // the last edge before t
                else o = c2_edge_rank(a, in, ld_acquire_i32(out_low + t) + shift);
                s_wave[lane] = o | fl;
            }
            __syncthreads();
            const int p0 = have ? s_wave[0] : -1;
            if (n + RS_WAVE > RS_LIST) {
                if (tid == 0) a.st->overflow = 1;
                break;
            }
            if (!have || ((p0 & RS_FLAG) && (p0 & ~RS_FLAG) < k)) {
                // claim the low: the list first, then the owner
                if (tid == 0) {
                    const unsigned long long off = atomicAdd(&a.st->arena, (unsigned long long)n);
                    s_sum = off;
                    s_act = off + n > (unsigned long long)a.arena_cap ? ACT_FAIL : ACT_DONE;
                }
                __syncthreads();
                const unsigned long long off = s_sum;
                if (s_act == ACT_FAIL) {
                    if (tid == 0) a.st->overflow = 1;
                    break;
                }
                for (int v = tid; v < n; v += THREADS) __stcg(a.arena + off + v, __ldcg(list + v));
                __threadfence();
                __syncthreads();
                if (tid == 0) {
                    *(volatile unsigned long long *)(a.sum + k) = (off << 24) | (unsigned)n;
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
                    const int len = (int)(s_sum & 0xffffffu);
                    const unsigned long long from = s_sum >> 24;
                    if (n + len > RS_LIST) {
                        if (tid == 0) a.st->overflow = 1;
                        break;
                    }
                    for (int v = tid; v < len; v += THREADS) __stcg(list + n + v, __ldcg(a.arena + from + v));
                    n += len;
                    k = s_other;
                    pos = low;
                    fresh = true;
                    __syncthreads();
                    continue;
                }
                if (tid == 0) s_wave[0] = s_other | RS_FLAG;
                cnt = 1;
                __syncthreads();
            }
            // the wave
            const int p = lane < cnt ? s_wave[lane] : -1;
            const unsigned m_app = __ballot_sync(0xffffffffu, p >= 0 && !(p & RS_FLAG));
            unsigned m_res = __ballot_sync(0xffffffffu, p >= 0 && (p & RS_FLAG) && (p & ~RS_FLAG) > k);
            for (int q = wid; q < cnt; q += NW)
                if ((m_app >> q) & 1u) rs_toggle<RUNS, WORDS>(a, in, s_wave[q], w0, hi, bits, later);
            if (wid == 0 && ((m_app >> lane) & 1u)) __stcg(list + n + __popc(m_app & below(lane)), p);
            n += __popc(m_app);
            bool full = false;
            adds += __popc(m_app);
            slots += (unsigned long long)__popc(m_app) * in.nv;
            for (; m_res; m_res &= m_res - 1) {
                const int o = s_wave[__ffs(m_res) - 1] & ~RS_FLAG;
                __syncthreads();
                if (tid == 0) s_sum = *(volatile unsigned long long *)(a.sum + o);
                __syncthreads();
                const int len = (int)(s_sum & 0xffffffu);
                const unsigned long long from = s_sum >> 24;
                if (n + len > RS_LIST) {
                    full = true;
                    break;
                }
                for (int x = wid; x < len; x += NW)
                    rs_toggle<RUNS, WORDS>(a, in, __ldcg(a.arena + from + x), w0, hi, bits, later);
                for (int v = tid; v < len; v += THREADS) __stcg(list + n + v, __ldcg(a.arena + from + v));
                n += len;
                adds++;
                slots += (unsigned long long)len * in.nv;
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

static int c2_read_status(Context *ctx, const C2Args &a, C2Status *hs) {
    OPH_CUDA_TRY(cudaGetLastError());
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
    static int per_sm[64];
    int &nb = per_sm[ctx->device & 63];
    if (!nb && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_c2_graph, C2_THREADS, 0) != cudaSuccess) {
        cudaGetLastError();
        nb = 0;
        return OPH_OK;
    }
    const int gg = c2_grid(ctx, 2 * ne, std::min(nb, 4));
    a.neg = nullptr;
    k_c2_edges<<<c2_grid(ctx, ne, 8), C2_THREADS, 0, s>>>(a);
    k_c2_surface<<<c2_grid(ctx, a.m, 16), C2_THREADS, 0, s>>>(a);
    k_c2_graph_init<<<c2_grid(ctx, a.m, 16), C2_THREADS, 0, s>>>(a);
    if (ctx->profile) cudaEventRecord(ctx->ev[2], s);
    int max_rounds = C2_MAX_ROUNDS;
    void *params[] = {&a, &max_rounds};
    OPH_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_c2_graph, dim3(gg), dim3(C2_THREADS), params, 0, s));
    ctx->launches += 4;
    cudaEventRecord(ctx->ev[1], s);
    int rc = c2_read_status(ctx, a, hs);
    *done = !rc && !hs->bad && !hs->crowded && !hs->unfinished;
    return rc;
}

template <bool RUNS, int THREADS, int WORDS>
static int c2_residual_grid(Context *ctx) {
    static int per_sm[64];
    int &nb = per_sm[ctx->device & 63];
    constexpr int SMEM = WORDS * (int)sizeof(uint32_t);
    if (!nb && (cudaFuncSetAttribute(k_c2_residual<RUNS, THREADS, WORDS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     SMEM) != cudaSuccess ||
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_c2_residual<RUNS, THREADS, WORDS>, THREADS,
                                                              SMEM) != cudaSuccess)) {
        cudaGetLastError();
        nb = 0;
    }
    return nb * ctx->sm_count;
}

// Many vertices: long rows and few, long residual columns, so large CTAs and
// windows; below, more CTAs.
constexpr int RS_SMALL_NV = 160, RS_SMALL = 256, RS_SMALL_WORDS = 4096, RS_LARGE = 1024, RS_LARGE_WORDS = 8192;

template <bool RUNS>
static int c2_run_dense(Context *ctx, C2Args a, int64_t ne, int64_t nt, C2Status *hs, bool *done) {
    // what a form's tables may cost, in entries: a few times the matrix itself
    // (sparse complexes on many vertices are left to the general path)
    const long long room = (1ll << 24) + 8 * hs->nnz;
    const long long cells = RUNS ? hs->pairs : hs->cells, run_words = RUNS ? hs->run_words : 0;
    if (hs->max_nv > (RUNS ? 1 << ADJ_SHIFT : C2_MAX_NV) || 2 * cells > room || 2 * run_words > room) return OPH_OK;
    cudaStream_t s = ctx->stream;
    const bool small = hs->max_nv <= RS_SMALL_NV;
    int gr = small ? c2_residual_grid<RUNS, RS_SMALL, RS_SMALL_WORDS>(ctx)
                   : c2_residual_grid<RUNS, RS_LARGE, RS_LARGE_WORDS>(ctx);
    if (gr == 0) return OPH_OK;
    gr = (int)std::min<int64_t>(ne, gr);
    const int nv = hs->nv;
    a.arena_cap = (1 << 22) + 16 * ne;
    size_t head = 0;
    for (char *p = nullptr;;) {
        Carve c{p};
        a.runs = c.take<uint2>(run_words);
        a.dead = c.take<uint8_t>(nv + 1);
        head = c.off;  // zeroed
        a.owned = c.take<uint32_t>((a.m + 31) / 32 + 4);
        a.fixed = c.take<uint32_t>((a.m + 31) / 32 + 4);
        a.res = c.take<int32_t>(ne);
        a.sum = c.take<unsigned long long>(ne);
        a.arena = c.take<int32_t>(a.arena_cap);
        a.lists = c.take<int32_t>((size_t)gr * RS_LIST);
        if (p) break;
        p = (char *)ctx_alloc(ctx, S_C2_MODE, c.off);
        if (!p) return OPH_OK;
    }
    if (!RUNS) a.runs = nullptr;
    const size_t cell_bytes = sizeof(int32_t) * (size_t)std::max<long long>(cells, 1);
    a.cells = (int32_t *)ctx_alloc(ctx, S_C2_CELLS, (RUNS ? 2 : 1) * cell_bytes);
    if (!a.cells) return OPH_OK;
    a.adj = RUNS ? a.cells + cells : nullptr;  // cells is a multiple of 4: whole 16-byte loads
    a.ends = nullptr;
    const int kb = std::min(a.count, ctx->sm_count * 4);
    OPH_CUDA_TRY(cudaMemsetAsync(a.cells, 0xff, cell_bytes, s));
    OPH_CUDA_TRY(cudaMemsetAsync(ctx->bufs[S_C2_MODE].ptr, 0, head, s));
    if (!RUNS) k_c2_cells<<<1, 1024, 0, s>>>(a);
    k_c2_edges<<<c2_grid(ctx, ne, 8), C2_THREADS, 0, s>>>(a);
    // rows of vertices in shared memory (sorted a warp each), or the components
    const int smem = std::max(6 * hs->max_nv, RUNS ? 4 * (C2_THREADS / 32) * c2_pitch(hs->max_nv) : 0);
    const int sb = RUNS ? c2_grid(ctx, 32 * (int64_t)nv, 4) : 0;
    k_c2_triangles<RUNS><<<kb + sb + c2_grid(ctx, a.m, 16), C2_THREADS, smem, s>>>(a, kb, sb, hs->max_nv);
    if (RUNS) {
        k_c2_runs_out<<<c2_grid(ctx, a.m, 16), C2_THREADS, 0, s>>>(a);
    } else {
        k_c2_table_init<<<c2_grid(ctx, a.m, 16), C2_THREADS, 0, s>>>(a);
        k_c2_table_pairs<<<c2_grid(ctx, 32 * ne, 8), C2_THREADS, 0, s>>>(a);
    }
    if (ctx->profile) cudaEventRecord(ctx->ev[2], s);
    if (small)
        k_c2_residual<RUNS, RS_SMALL, RS_SMALL_WORDS><<<gr, RS_SMALL, RS_SMALL_WORDS * sizeof(uint32_t), s>>>(a);
    else
        k_c2_residual<RUNS, RS_LARGE, RS_LARGE_WORDS><<<gr, RS_LARGE, RS_LARGE_WORDS * sizeof(uint32_t), s>>>(a);
    ctx->launches += RUNS ? 4 : 6;
    cudaEventRecord(ctx->ev[1], s);
    int rc = c2_read_status(ctx, a, hs);
    // a table entry written twice (two triangles on the same edge and vertex,
    // which no simplicial complex has) shows in the count of those set
    *done = !rc && !hs->bad && !hs->overflow && (!RUNS || !hs->unsorted) &&
            (RUNS || hs->cells_set == 3ull * (unsigned long long)nt);
    return rc;
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

int reduce_complex2(Context *ctx, C2Job &job, oph_info *info, bool *taken) {
    *taken = false;
    job.nnz_read = false;
    ctx->launches = 0;
    ctx->prof = oph_profile{};
    const int64_t m = job.m;
    if (m < 1 || m >= (1 << 29)) return OPH_OK;
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
    static_assert(sizeof(C2Status) <= sizeof(DevStatus), "read back through the context's pinned status block");
    C2Status *hs = reinterpret_cast<C2Status *>(ctx->h_status);
    int rc;
    cudaEventRecord(ctx->ev[0], s);
    OPH_CUDA_TRY(cudaMemsetAsync(a.st, 0, sizeof(C2Status), s));
    k_c2_words<<<(int)std::min<int64_t>(ntiles, (int64_t)ctx->sm_count * 8), C2_THREADS, 0, s>>>(a);
    k_c2_scan<<<1, 1024, 0, s>>>(a, ntiles);
    OPH_CUDA_TRY(cudaGetLastError());
    ctx->launches += 2;
    DevStatus *hb = ctx->h_status + 1;
    if (job.before) OPH_CUDA_TRY(cudaMemcpyAsync(hb, job.before, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
    if ((rc = c2_read_status(ctx, a, hs))) return rc;
    job.nnz = hs->nnz;
    job.nnz_read = true;
    job.before_error = job.before ? hb->error : 0;
    if (job.before_error) return OPH_OK;
    const int64_t nv = hs->nv, ne = hs->ne, nt = m - nv - ne;
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
    bool done = false;
    // every edge with at most two triangles: a graph (an edge found to have
    // more leaves it to the dense form)
    if (3 * nt <= 2 * ne && (rc = c2_run_graph(ctx, a, nv, ne, nt, hs, &done))) return rc;
    if (!done && !hs->bad && (rc = c2_run_dense<true>(ctx, a, ne, nt, hs, &done))) return rc;
    if (!done && !hs->bad && !hs->overflow) {
        // not in runs: the same with the table (the status as before the try)
        if (hs->unsorted) {
            OPH_CUDA_TRY(cudaMemsetAsync(&a.st->unsorted, 0, sizeof(int), s));
        }
        if ((rc = c2_run_dense<false>(ctx, a, ne, nt, hs, &done))) return rc;
    }
    if (!done) return OPH_OK;
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
