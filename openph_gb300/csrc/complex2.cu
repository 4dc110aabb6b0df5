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
// What is accepted is checked on the device before anything is written: every
// column has 0, 2 or 3 rows, ascending and in range, the rows of an edge are
// vertices, the rows of a triangle are the three edges of a triangle (so
// D D = 0, which clearing relies on).  Anything else, malformed input
// included, is left to the general path and its own checks.
#include <algorithm>

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
};

constexpr int C2_THREADS = 256, C2_TILE = 2048;
constexpr int C2_MAX_ROUNDS = 512;

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
        }
    }
    __syncthreads();
    if (!a.inst_off) return;
    for (int b = threadIdx.x; b < a.count; b += 1024) {
        const int64_t o0 = a.inst_off[b], o1 = a.inst_off[b + 1];
        if (o0 < 0 || o1 < o0 || o1 > a.m || (b == 0 && o0 != 0) || (b == a.count - 1 && o1 != a.m)) {
            a.st->bad = 1;
            continue;
        }
        const int2 r0 = c2_rank_tiled(a, o0), r1 = c2_rank_tiled(a, o1);
        C2Inst s;
        s.voff = r0.x;
        s.eoff = r0.y;
        s.nv = r1.x - r0.x;
        s.ne = r1.y - r0.y;
        s.base = o0;
        s.cols = o1 - o0;
        a.inst[b] = s;
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

// Contexts that ask for something of the sweeps keep them: trackers, a forced
// matrix, a tuned narrow tier, a sweep cap or a fixed initial store, and the
// exact slot counts of the store's tiers.
bool complex2_applies(const Context *ctx, int algo) {
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
    auto read_status = [&]() -> int {
        OPH_CUDA_TRY(cudaMemcpyAsync(hs, a.st, sizeof(C2Status), cudaMemcpyDeviceToHost, s));
        OPH_CUDA_TRY(cudaStreamSynchronize(s));
        return OPH_OK;
    };
    int rc;
    cudaEventRecord(ctx->ev[0], s);
    OPH_CUDA_TRY(cudaMemsetAsync(a.st, 0, sizeof(C2Status), s));
    k_c2_words<<<(int)std::min<int64_t>(ntiles, (int64_t)ctx->sm_count * 8), C2_THREADS, 0, s>>>(a);
    k_c2_scan<<<1, 1024, 0, s>>>(a, ntiles);
    OPH_CUDA_TRY(cudaGetLastError());
    ctx->launches += 2;
    DevStatus *hb = ctx->h_status + 1;
    if (job.before) OPH_CUDA_TRY(cudaMemcpyAsync(hb, job.before, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
    if ((rc = read_status())) return rc;
    job.nnz = hs->nnz;
    job.nnz_read = true;
    job.before_error = job.before ? hb->error : 0;
    if (job.before_error) return OPH_OK;
    const int64_t nv = hs->nv, ne = hs->ne, nt = m - nv - ne;
    if (hs->bad || hs->nnz != 2 * ne + 3 * nt || (job.want_nnz >= 0 && hs->nnz != job.want_nnz)) return OPH_OK;
    if (ne == 0 || ne >= (1 << 29) || !job.rows) return OPH_OK;
    if (3 * nt > 2 * ne) return OPH_OK;  // some edge has more than two triangles

    const int64_t nodes = nv + nt + 1;
    for (char *p = nullptr;;) {
        Carve c{p};
        a.vlist = c.take<int32_t>(nv + 1);
        a.elist = c.take<int32_t>(ne);
        a.erec = c.take<int4>(ne);
        a.tlist = c.take<int32_t>(nt + 1);
        a.ends = c.take<int2>(2 * ne);
        a.parent = c.take<int>(nodes);
        a.best = c.take<unsigned long long>(nodes);
        a.list[0] = c.take<int32_t>(2 * ne);
        a.list[1] = c.take<int32_t>(2 * ne);
        if (p) break;
        p = (char *)ctx_alloc(ctx, S_C2_WORK, c.off);
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
    k_c2_lists<<<c2_grid(ctx, nwords, 8), C2_THREADS, 0, s>>>(a);
    k_c2_edges<<<c2_grid(ctx, ne, 8), C2_THREADS, 0, s>>>(a);
    k_c2_surface<<<c2_grid(ctx, m, 16), C2_THREADS, 0, s>>>(a);
    k_c2_graph_init<<<c2_grid(ctx, m, 16), C2_THREADS, 0, s>>>(a);
    if (ctx->profile) cudaEventRecord(ctx->ev[2], s);
    int max_rounds = C2_MAX_ROUNDS;
    void *params[] = {&a, &max_rounds};
    OPH_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_c2_graph, dim3(gg), dim3(C2_THREADS), params, 0, s));
    OPH_CUDA_TRY(cudaGetLastError());
    ctx->launches += 5;
    cudaEventRecord(ctx->ev[1], s);
    if ((rc = read_status())) return rc;
    if (hs->bad || hs->crowded || hs->unfinished) return OPH_OK;
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
    if (ctx->profile) cudaEventElapsedTime(&ctx->prof.setup_ms, ctx->ev[0], ctx->ev[2]);
    ctx->prof.kernel_launches = ctx->launches;
    *info = oph_info{};
    info->sweeps = hs->rounds;
    info->num_iters = hs->rounds + 1;
    info->additions = (int64_t)hs->joins;
    info->slots_moved = 4 * (int64_t)hs->joins;
    info->pool_bytes = (int64_t)(ctx->bufs[S_C2_TAB].bytes + ctx->bufs[S_C2_WORK].bytes);
    info->device_ms = ms;
    info->dual = c2_named_matrix(m, nv, ne, nt);
    *taken = true;
    return OPH_OK;
}

}  // namespace oph
