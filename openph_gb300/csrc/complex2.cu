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
    long long coff, pad;  // its part of the edge-vertex table
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
    int nres, cursor, overflow;      // residual edges; the CTAs' queue; a list ran out of room
    long long cells;                 // entries of the edge-vertex table
    unsigned long long cells_set;    // and those a triangle wrote
    unsigned long long arena;        // entries of published lists
    unsigned long long adds, slots;  // additions of the residual columns, entries toggled
};

constexpr int C2_THREADS = 256, C2_TILE = 2048;
constexpr int C2_MAX_ROUNDS = 512;
constexpr int C2_MAX_NV = 8192;                   // vertices of an instance the dense form takes
constexpr int RS_THREADS = 256, RS_WORDS = 8192;  // residual columns: a CTA, a window of 2^18 triangles
constexpr int RS_WAVE = 16;                       //   pivots added at a time
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
    // dense form: the edge-vertex table, the vertex that dies at each edge
    // (-1: none), the owner of each triangle's row (an edge's rank; with
    // RS_FLAG a residual one, which may still change; -1: none) and which
    // have one, the residual edges with their first triangles, the triangle
    // each holds, the list its column is the sum of (offset << 24 | length)
    int32_t *cells;
    int32_t *neg;
    int32_t *owner;
    uint32_t *owned;
    int2 *res;
    int32_t *death;
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
            a.st->cells = (long long)s.nv * s.ne;
        }
    }
    __syncthreads();
    if (!a.inst_off) return;
    long long cells = 0;
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
        long long total;
        s.coff = cells + c2_block_excl((long long)s.nv * s.ne, red, &total);
        cells += total;
        if (b < a.count) a.inst[b] = s;
    }
    if (threadIdx.x == 0) a.st->cells = cells;
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
// The edges on vertices of one instance, by the elder rule, a CTA in column
// order: 1024 edges at a time whose ends carry different labels (most after
// the first few hundred do not), those joined one by one by a warp, which
// relabels the younger component.  It stops when one component is left: on
// the torus after 1,788 of 58,988 edges.  Bound by the latency of its
// nv - 1 relabellings, and hidden behind the triangles of the same launch.
constexpr int KR_ITEMS = 4, KR_EDGES = KR_ITEMS * C2_THREADS;
__device__ void c2_kruskal(const C2Args &a, const C2Inst &in, uint16_t *label, uint16_t (*su)[C2_THREADS],
                           uint16_t (*sv)[C2_THREADS], unsigned (*mask)[C2_THREADS / 32], int *s_parts) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int x = tid; x < in.nv; x += C2_THREADS) label[x] = (uint16_t)x;
    if (tid == 0) *s_parts = in.nv;
    __syncthreads();
    for (int c0 = 0; c0 < in.ne && *s_parts > 1; c0 += KR_EDGES) {
        int4 e[KR_ITEMS];
#pragma unroll
        for (int q = 0; q < KR_ITEMS; q++) {
            const int i = c0 + q * C2_THREADS + tid;
            e[q] = i < in.ne ? a.erec[in.eoff + i] : make_int4(in.voff, in.voff, 0, 0);
        }
#pragma unroll
        for (int q = 0; q < KR_ITEMS; q++) {
            const int u = e[q].x - in.voff, v = e[q].y - in.voff;
            su[q][tid] = (uint16_t)u;
            sv[q][tid] = (uint16_t)v;
            const unsigned b = __ballot_sync(0xffffffffu, label[u] != label[v]);
            if (lane == 0) mask[q][wid] = b;
        }
        __syncthreads();
        if (wid == 0) {
            int parts = *s_parts;
            for (int g = 0; g < KR_ITEMS * (C2_THREADS / 32) && parts > 1; g++) {
                const int q = g / (C2_THREADS / 32), w = g % (C2_THREADS / 32);
                if (!mask[q][w]) continue;
                const int u = su[q][w * 32 + lane], v = sv[q][w * 32 + lane];
                for (;;) {
                    const int lu = label[u], lv = label[v];
                    const unsigned b = __ballot_sync(0xffffffffu, lu != lv);
                    if (!b) break;
                    const int first = __ffs(b) - 1;
                    const int young = __shfl_sync(0xffffffffu, max(lu, lv), first);
                    const int old = __shfl_sync(0xffffffffu, min(lu, lv), first);
                    for (int x = lane; x < in.nv; x += 32)
                        if (label[x] == young) label[x] = (uint16_t)old;
                    if (lane == 0) a.neg[in.eoff + c0 + g * 32 + first] = young;
                    parts--;
                    __syncwarp();
                }
            }
            if (lane == 0) *s_parts = parts;
        }
        __syncthreads();
    }
}

// The first blocks pair the edges with vertices (an instance each); the rest
// check the triangles, a thread each, and write each at its three entries of
// the table.  Bound by the table's scattered 4-byte writes.
__global__ void __launch_bounds__(C2_THREADS) k_c2_table(C2Args a, int kruskal_blocks) {
    __shared__ uint16_t label[C2_MAX_NV];
    __shared__ uint16_t su[KR_ITEMS][C2_THREADS], sv[KR_ITEMS][C2_THREADS];
    __shared__ unsigned mask[KR_ITEMS][C2_THREADS / 32];
    __shared__ int s_parts;
    if (a.st->bad) return;
    if ((int)blockIdx.x < kruskal_blocks) {
        for (int b = blockIdx.x; b < a.count; b += kruskal_blocks) {
            c2_kruskal(a, a.inst[b], label, su, sv, mask, &s_parts);
            __syncthreads();
        }
        return;
    }
    bool bad = false;
    const int64_t stride = (int64_t)(gridDim.x - kruskal_blocks) * C2_THREADS;
    for (int64_t j = (int64_t)(blockIdx.x - kruskal_blocks) * C2_THREADS + threadIdx.x; j < a.m; j += stride) {
        const C2Word w = a.words[j >> 5];
        if (((w.v | w.e) >> (j & 31)) & 1u) continue;
        const C2Inst &in = a.inst[c2_inst_of(a, j)];
        int k[3], o[3];
        if (!c2_triangle(a, j, w, in, k) ||
            !c2_opposite(a.erec[k[0]], a.erec[k[1]], a.erec[k[2]], o[0], o[1], o[2])) {
            bad = true;
            continue;
        }
#pragma unroll
        for (int q = 0; q < 3; q++)
            a.cells[in.coff + (int64_t)(k[q] - in.eoff) * in.nv + (o[q] - in.voff)] = (int32_t)j;
    }
    if (bad) a.st->bad = 1;
}

// Outputs and owners before any pair is known.
__global__ void __launch_bounds__(C2_THREADS) k_c2_dense_init(C2Args a) {
    if (a.st->bad) return;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, nwords = ((a.m + 31) >> 5) + 4;
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int none = a.one_based ? 0 : -1;
    for (int64_t j = i0; j < a.m; j += stride) {
        a.low[j] = none;
        if (a.ess) a.ess[j] = 1;
        a.owner[j] = -1;
    }
    for (int64_t w = i0; w < nwords; w += stride) a.owned[w] = 0u;
}

// Column `col` has row `row` as its low (columns of the whole batch).
__device__ __forceinline__ void c2_pair(const C2Args &a, const C2Inst &in, int col, int row) {
    a.low[col] = row - (int)in.base + a.one_based;
    if (a.ess) {
        a.ess[col] = 0;
        a.ess[row] = 0;
    }
}

// A warp per edge: its row of the table read once, for the entries set and
// its first triangle t.  An edge that kills a vertex is paired with it (its
// column of D' is cleared); one that is the last edge of t is t's low and t
// the low of its column of D', finally: an apparent pair.  The others are
// residual.  Bound by reading the table.
__global__ void __launch_bounds__(C2_THREADS) k_c2_pairs(C2Args a) {
    if (a.st->bad) return;
    const int lane = threadIdx.x & 31, ne = a.st->ne;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    unsigned long long set = 0;
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < ne; k += nw) {
        const C2Inst in = a.inst[a.erec[k].z];
        const int32_t *row = a.cells + in.coff + (int64_t)(k - in.eoff) * in.nv;
        unsigned t = 0xffffffffu;  // an empty entry is the largest
        for (int i = lane; i < in.nv; i += 32) {
            const unsigned x = (unsigned)row[i];
            set += x != 0xffffffffu;
            t = min(t, x);
        }
        t = __reduce_min_sync(0xffffffffu, t);
        if (lane == 0) {
            const int e = a.elist[k], y = a.neg[k];
            if (y >= 0) {
                c2_pair(a, in, e, a.vlist[in.voff + y]);
            } else if (t != 0xffffffffu) {
                if (a.rows[a.colptr[t] + 2] + in.base == e) {
                    c2_pair(a, in, (int)t, e);
                    a.owner[t] = k;
                    atomicOr(a.owned + (t >> 5), 1u << (t & 31));
                } else {
                    a.res[atomicAdd(&a.st->nres, 1)] = make_int2(k, (int)t);
                    a.death[k] = -1;
                }
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) set += __shfl_xor_sync(0xffffffffu, set, o);
    if (lane == 0 && set) atomicAdd(&a.st->cells_set, set);
}

// Toggle an edge's triangles in the window from w0 (a warp); `later` keeps
// the first one past the window.
__device__ __forceinline__ void rs_toggle(const int32_t *row, int nv, int w0, uint32_t *bits, int &later) {
    for (int i = threadIdx.x & 31; i < nv; i += 128) {
        int t[4];
#pragma unroll
        for (int q = 0; q < 4; q++) t[q] = i + 32 * q < nv ? __ldg(row + i + 32 * q) : -1;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int r = t[q] - w0;  // an empty entry (-1) falls below the window, as rows already cancelled do
            if (r < 0 || t[q] < 0) continue;
            if (r < 32 * RS_WORDS) atomicXor(bits + (r >> 5), 1u << (r & 31));
            else later = min(later, t[q]);
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
//   chains of 557 additions on the torus take 38 waves.  A wave is three
//   round trips to L2 (which bits have owners, the owners, their rows).
// * Owners: a residual column claims its low by compare-and-swap once its
//   list is published.  Found claimed by an earlier column, that column is
//   added; by a later one, the claim is taken over and this CTA goes on with
//   the later column plus its own.  No CTA waits for another, and the lows
//   are those of any complete reduction.
__global__ void __launch_bounds__(RS_THREADS) k_c2_residual(C2Args a) {
    if (a.st->bad) return;
    extern __shared__ __align__(16) uint32_t bits[];  // RS_WORDS
    constexpr int NW = RS_THREADS / 32;
    __shared__ int s_low[NW], s_cnt[NW], s_wave[RS_WAVE];
    __shared__ int s_i, s_first, s_later, s_act, s_other;
    __shared__ unsigned long long s_sum;
    enum { ACT_DONE, ACT_ADD, ACT_STEAL, ACT_FAIL };
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nres = a.st->nres;
    int32_t *list = a.lists + (size_t)blockIdx.x * RS_LIST;
    unsigned long long adds = 0, slots = 0;
    for (;;) {
        if (tid == 0) s_i = atomicAdd(&a.st->cursor, 1);
        __syncthreads();
        const int i = s_i;
        __syncthreads();
        if (i >= nres) break;
        int k = a.res[i].x, pos = a.res[i].y;
        const C2Inst in = a.inst[a.erec[k].z];
        const int32_t *cells = a.cells + in.coff;
        auto row = [&](int e) { return cells + (int64_t)(e - in.eoff) * in.nv; };
        int n = 1, w0 = pos & ~127, later = INT_MAX;
        if (tid == 0) list[0] = k;
        bool refill = true;
        for (;;) {
            if (refill) {
                for (int q = 4 * tid; q < RS_WORDS; q += 4 * RS_THREADS)
                    *reinterpret_cast<uint4 *>(bits + q) = make_uint4(0u, 0u, 0u, 0u);
                if (tid == 0) s_later = INT_MAX;
                later = INT_MAX;
                __syncthreads();
                for (int v = wid; v < n; v += NW) rs_toggle(row(__ldcg(list + v)), in.nv, w0, bits, later);
                __syncthreads();
                refill = false;
            }
            // the low, and the set bits with owners, from pos up
            int low = INT_MAX, before = 0, total = 0, mine = 0, at = 0;
            uint4 c = make_uint4(0u, 0u, 0u, 0u);
            for (int base = ((pos - w0) >> 5) & ~3; base < RS_WORDS; base += 4 * RS_THREADS) {
                at = base + 4 * tid;
                uint4 t = make_uint4(0u, 0u, 0u, 0u);
                if (at < RS_WORDS) t = *reinterpret_cast<const uint4 *>(bits + at);
                int fl = INT_MAX;
                c = make_uint4(0u, 0u, 0u, 0u);
                if (t.x | t.y | t.z | t.w) {
                    const uint4 p = __ldcg(reinterpret_cast<const uint4 *>(a.owned + (w0 >> 5) + at));
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
                before = incl - mine;
                total = 0;
                low = INT_MAX;
#pragma unroll
                for (int w = 0; w < NW; w++) {
                    if (w < wid) before += s_cnt[w];
                    total += s_cnt[w];
                    low = min(low, s_low[w]);
                }
                if (low != INT_MAX) break;
                __syncthreads();
            }
            if (low == INT_MAX) {  // nothing left in the window
                if (later != INT_MAX) atomicMin(&s_later, later);
                __syncthreads();
                const int next = s_later;
                __syncthreads();
                if (next == INT_MAX) {  // the column is zero: edge k is essential
                    if (tid == 0) a.death[k] = -1;
                    break;
                }
                pos = next;
                w0 = next & ~127;
                refill = true;
                continue;
            }
            if (mine && before < RS_WAVE) {
                const unsigned cw[4] = {c.x, c.y, c.z, c.w};
                int r = before;
#pragma unroll
                for (int q = 0; q < 4; q++)
                    for (unsigned b = cw[q]; b && r < RS_WAVE; b &= b - 1, r++) {
                        const int t = w0 + 32 * (at + q) + __ffs(b) - 1;
                        if (r == 0) s_first = t;
                        s_wave[r] = ld_acquire_i32(a.owner + t);
                    }
            }
            __syncthreads();
            int cnt = min(total, RS_WAVE);
            const bool have = cnt > 0 && s_first == low;
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
                for (int v = tid; v < n; v += RS_THREADS) __stcg(a.arena + off + v, __ldcg(list + v));
                __threadfence();
                __syncthreads();
                if (tid == 0) {
                    *(volatile unsigned long long *)(a.sum + k) = (off << 24) | (unsigned)n;
                    a.death[k] = low;
                    __threadfence();
                    int want = p0, act = ACT_FAIL, other = -1;
                    for (int tries = 0; tries < (1 << 20); tries++) {
                        const int got = atomicCAS(a.owner + low, want, k | RS_FLAG);
                        if (got == want) {
                            atomicOr(a.owned + (low >> 5), 1u << (low & 31));
                            act = want < 0 ? ACT_DONE : ACT_STEAL;
                            other = want & ~RS_FLAG;
                            break;
                        }
                        if (!(got & RS_FLAG) || (got & ~RS_FLAG) > k) {  // an earlier column's by now
                            act = ACT_ADD;
                            other = got;
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
                    for (int v = tid; v < len; v += RS_THREADS) __stcg(list + n + v, __ldcg(a.arena + from + v));
                    n += len;
                    k = s_other;
                    pos = low;
                    w0 = low & ~127;
                    refill = true;
                    __syncthreads();
                    continue;
                }
                if (tid == 0) s_wave[0] = s_other;
                cnt = 1;
                __syncthreads();
            }
            // the wave
            const int p = lane < cnt ? s_wave[lane] : -1;
            const unsigned m_app = __ballot_sync(0xffffffffu, p >= 0 && !(p & RS_FLAG));
            unsigned m_res = __ballot_sync(0xffffffffu, p >= 0 && (p & RS_FLAG) && (p & ~RS_FLAG) > k);
            for (int q = wid; q < cnt; q += NW)
                if ((m_app >> q) & 1u) rs_toggle(row(s_wave[q]), in.nv, w0, bits, later);
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
                for (int v = wid; v < len; v += NW) {
                    const int e = __ldcg(a.arena + from + v);
                    rs_toggle(row(e), in.nv, w0, bits, later);
                    if (lane == 0) __stcg(list + n + v, e);
                }
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

// The pairs of the residual edges.
__global__ void __launch_bounds__(C2_THREADS) k_c2_residual_pairs(C2Args a) {
    if (a.st->bad) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.st->nres; i += gridDim.x * blockDim.x) {
        const int k = a.res[i].x, t = a.death[k];
        if (t >= 0) c2_pair(a, a.inst[a.erec[k].z], t, a.elist[k]);
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

static int c2_run_dense(Context *ctx, C2Args a, int64_t nv, int64_t ne, int64_t nt, C2Status *hs, bool *done) {
    // The table costs a write and a read of its cells; past a few times the
    // matrix itself (sparse complexes on many vertices) it no longer pays.
    if (hs->max_nv > C2_MAX_NV || hs->cells > (1ll << 24) + 8 * hs->nnz) return OPH_OK;
    cudaStream_t s = ctx->stream;
    static int per_sm[64];
    int &nb = per_sm[ctx->device & 63];
    constexpr int SMEM = RS_WORDS * (int)sizeof(uint32_t);
    if (!nb && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_c2_residual, RS_THREADS, SMEM) != cudaSuccess) {
        cudaGetLastError();
        nb = 0;
        return OPH_OK;
    }
    const int gr = (int)std::max<int64_t>(1, std::min<int64_t>(ne, (int64_t)ctx->sm_count * nb));
    a.arena_cap = (1 << 22) + 16 * ne;
    for (char *p = nullptr;;) {
        Carve c{p};
        a.owner = c.take<int32_t>(a.m);
        a.owned = c.take<uint32_t>((a.m + 31) / 32 + 4);
        a.res = c.take<int2>(ne);
        a.death = c.take<int32_t>(ne);
        a.sum = c.take<unsigned long long>(ne);
        a.arena = c.take<int32_t>(a.arena_cap);
        a.lists = c.take<int32_t>((size_t)gr * RS_LIST);
        if (p) break;
        p = (char *)ctx_alloc(ctx, S_C2_MODE, c.off);
        if (!p) return OPH_OK;
    }
    const size_t cell_bytes = sizeof(int32_t) * (size_t)std::max<long long>(hs->cells, 1);
    a.cells = (int32_t *)ctx_alloc(ctx, S_C2_CELLS, cell_bytes);
    if (!a.cells) return OPH_OK;
    a.ends = nullptr;
    const int kb = std::min(a.count, ctx->sm_count * 4);
    OPH_CUDA_TRY(cudaMemsetAsync(a.cells, 0xff, cell_bytes, s));
    k_c2_edges<<<c2_grid(ctx, ne, 8), C2_THREADS, 0, s>>>(a);
    k_c2_table<<<kb + c2_grid(ctx, a.m, 16), C2_THREADS, 0, s>>>(a, kb);
    k_c2_dense_init<<<c2_grid(ctx, a.m, 16), C2_THREADS, 0, s>>>(a);
    k_c2_pairs<<<c2_grid(ctx, 32 * ne, 8), C2_THREADS, 0, s>>>(a);
    if (ctx->profile) cudaEventRecord(ctx->ev[2], s);
    k_c2_residual<<<gr, RS_THREADS, SMEM, s>>>(a);
    k_c2_residual_pairs<<<c2_grid(ctx, ne, 1), C2_THREADS, 0, s>>>(a);
    ctx->launches += 6;
    cudaEventRecord(ctx->ev[1], s);
    int rc = c2_read_status(ctx, a, hs);
    // a table entry written twice (two triangles on the same edge and vertex,
    // which no simplicial complex has) shows in the count of those set
    *done = !rc && !hs->bad && !hs->overflow && hs->cells_set == 3ull * (unsigned long long)nt;
    (void)nv;
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
    if (!done && !hs->bad && (rc = c2_run_dense(ctx, a, nv, ne, nt, hs, &done))) return rc;
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
