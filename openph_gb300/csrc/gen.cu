// Complexes built on the device: the Vietoris-Rips complex of a point cloud
// and the lower-star filtration of an image, as the sorted CSC boundary
// matrix the reduction consumes, with no host pass over the simplices.
//
// The input stand-ins of the reference's benchmarks (Javaplex streams,
// example_factory.m:17-114, stream2cmo.m:1-26) are generated on the host by
// gen/ophgen.c; these kernels produce the identical matrix (same filtration
// values, same order, same rows) from the points or the image already in
// HBM.  The order is (value, dimension, vertex tuple).
//
// * Rips: a triangle carries its longest edge's value, so only the edges are
//   sorted (their 64-bit values; the sort is stable, and they are listed by
//   vertices).  When no two edges are equally long, the triangles of an edge
//   (u, v) follow it directly, ascending in the third vertex: the vertices
//   joined to u and to v by earlier edges.  Counting them per edge, a prefix
//   sum and one pass over the edges write the matrix.  The whole complex of
//   the 1M-column torus was sorted by 128-bit keys before, sixteen passes
//   over 16 bytes a simplex (330 us) after a walk over the triangles by a
//   warp per vertex (790 us).
// * Equally long edges mix their triangles: then every simplex gets that
//   128-bit key, the order-preserving bits of its FP64 value followed by a
//   word holding its dimension and vertex ids, and one radix sort of the keys
//   is the filtration order.  The key alone names the simplex.
// * Lower star: simplices are listed by (dimension, vertices), so a stable
//   sort of their FP32 values' 32 bits (four passes of 8 bytes) is the order.
//
// Distances are summed in the host generator's order with separately
// rounded multiplies and adds (no FMA) and a correctly rounded square root,
// so every value, and with it the order, is bit-identical to the host's.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cuda/std/tuple>

#include "oph_host.h"

namespace oph {

namespace {

struct SKey {
    unsigned long long vb;   // order-preserving bits of the filtration value
    unsigned long long lex;  // dimension << 60 | a << 40 | b << 20 | c
};
struct SKeyDecomposer {
    __host__ __device__ cuda::std::tuple<unsigned long long &, unsigned long long &> operator()(SKey &k) const {
        return {k.vb, k.lex};
    }
};

__device__ __forceinline__ unsigned long long dbits(double v) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double dvalue(unsigned long long b) {
    const unsigned long long u = (b & 0x8000000000000000ull) ? (b & 0x7fffffffffffffffull) : ~b;
    return __longlong_as_double((long long)u);
}
__device__ __forceinline__ unsigned long long lexkey(int dim, unsigned a, unsigned b, unsigned c) {
    return ((unsigned long long)dim << 60) | ((unsigned long long)a << 40) | ((unsigned long long)b << 20) | c;
}

// ------------------------------------------------------------------ Rips
// Distances of every pair (upper triangle) and the adjacency bitsets: bit c
// of row a (words of 32) is set when a != c and |p_a - p_c| <= thr.
// What the host reads of a Rips complex, and the longest edge (its bits).
struct RipsTotals {
    unsigned long long edges, triangles, longest;
    int tied, crowded;  // equally long edges; ranks not settled: too many of one coarse length, or tied
};
__global__ void __launch_bounds__(256) k_rips_dist(const double *__restrict__ pts, int n, int d, double thr,
                                                   double *__restrict__ D, unsigned *__restrict__ adj, int words,
                                                   RipsTotals *totals) {
    __shared__ unsigned long long s_longest;
    if (threadIdx.x == 0) s_longest = 0;
    __syncthreads();
    double longest = 0.0;  // edge; distances are not negative, so their bits compare like them
    const int64_t pairs = (int64_t)n * n;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < pairs; q += (int64_t)gridDim.x * blockDim.x) {
        const int a = (int)(q / n), b = (int)(q % n);
        if (b <= a) continue;
        double s = 0.0;
        for (int t = 0; t < d; t++) {
            const double x = __dsub_rn(pts[(int64_t)a * d + t], pts[(int64_t)b * d + t]);
            s = __dadd_rn(s, __dmul_rn(x, x));
        }
        const double v = __dsqrt_rn(s);
        D[(int64_t)a * n + b] = v;
        D[(int64_t)b * n + a] = v;
        if (v <= thr) {
            longest = max(longest, v);
            atomicOr(&adj[(int64_t)a * words + (b >> 5)], 1u << (b & 31));
            atomicOr(&adj[(int64_t)b * words + (a >> 5)], 1u << (a & 31));
        }
    }
    for (int o = 16; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&s_longest, dbits(longest));
    __syncthreads();
    if (threadIdx.x == 0 && s_longest) atomicMax(&totals->longest, s_longest);
}

// Bits of row r above column c (exclusive), within word w.
__device__ __forceinline__ unsigned above(int w, int c) {
    const int lo = w * 32;
    if (c < lo) return 0xffffffffu;
    if (c >= lo + 31) return 0u;
    return 0xffffffffu << ((c - lo) + 1);
}

// Edges per row (b > a), one thread per row.
__global__ void k_rips_deg(const unsigned *__restrict__ adj, int n, int words, long long *__restrict__ deg) {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x) {
        long long s = 0;
        for (int w = a >> 5; w < words; w++) s += __popc(adj[(int64_t)a * words + w] & above(w, a));
        deg[a] = s;
    }
}

// Triangles above every edge (a, b): common neighbours c > b.  One warp per
// row a walks its edges; lane-strided over the words.
__global__ void k_rips_tri_count(const unsigned *__restrict__ adj, int n, int words,
                                 const long long *__restrict__ eoff, long long *__restrict__ tcnt) {
    const int lane = threadIdx.x & 31;
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int a = wid; a < n; a += nw) {
        long long e = eoff[a];
        const unsigned *ra = adj + (int64_t)a * words;
        for (int wb = a >> 5; wb < words; wb++) {
            unsigned bits = ra[wb] & above(wb, a);
            while (bits) {
                const int b = wb * 32 + __ffs(bits) - 1;
                bits &= bits - 1;
                const unsigned *rb = adj + (int64_t)b * words;
                long long s = 0;
                for (int w = (b >> 5) + lane; w < words; w += 32) s += __popc(ra[w] & rb[w] & above(w, b));
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) tcnt[e] = s;
                e++;
            }
        }
    }
}

// Keys of every simplex: vertices at [0, n), edges at n + edge index, and
// the triangles of edge e at n + E + toff[e].
__global__ void k_rips_keys(const unsigned *__restrict__ adj, const double *__restrict__ D, int n, int words,
                            const long long *__restrict__ eoff, const long long *__restrict__ toff, long long E,
                            SKey *__restrict__ keys) {
    const int lane = threadIdx.x & 31;
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int a = wid; a < n; a += nw) {
        if (lane == 0) keys[a] = SKey{dbits(0.0), lexkey(0, a, 0, 0)};
        long long e = eoff[a];
        const unsigned *ra = adj + (int64_t)a * words;
        for (int wb = a >> 5; wb < words; wb++) {
            unsigned bits = ra[wb] & above(wb, a);
            while (bits) {
                const int b = wb * 32 + __ffs(bits) - 1;
                bits &= bits - 1;
                const double dab = D[(int64_t)a * n + b];
                if (lane == 0) keys[n + e] = SKey{dbits(dab), lexkey(1, a, b, 0)};
                const unsigned *rb = adj + (int64_t)b * words;
                long long t = n + E + toff[e];
                // common neighbours c > b in increasing c, lane-parallel by word
                for (int w0 = b >> 5; w0 < words; w0 += 32) {
                    const int w = w0 + lane;
                    const unsigned cm = w < words ? (ra[w] & rb[w] & above(w, b)) : 0u;
                    int cnt = __popc(cm);
                    int pre = cnt;
                    for (int o = 1; o < 32; o <<= 1) {
                        const int u = __shfl_up_sync(0xffffffffu, pre, o);
                        if (lane >= o) pre += u;
                    }
                    const int total = __shfl_sync(0xffffffffu, pre, 31);
                    long long slot = t + pre - cnt;
                    unsigned bitsc = cm;
                    while (bitsc) {
                        const int c = w * 32 + __ffs(bitsc) - 1;
                        bitsc &= bitsc - 1;
                        double v = dab;
                        const double dac = D[(int64_t)a * n + c], dbc = D[(int64_t)b * n + c];
                        if (dac > v) v = dac;
                        if (dbc > v) v = dbc;
                        keys[slot++] = SKey{dbits(v), lexkey(2, a, b, c)};
                    }
                    t += total;
                }
                e++;
            }
        }
    }
}

// Sorted keys -> position tables (vertex id, and edge (a, b) as a * n + b).
__global__ void k_rips_pos(const SKey *__restrict__ keys, int64_t m, int n, int32_t *__restrict__ vpos,
                           int32_t *__restrict__ epos) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < m; r += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long L = keys[r].lex;
        const int dim = (int)(L >> 60);
        const int a = (int)((L >> 40) & 0xfffff), b = (int)((L >> 20) & 0xfffff);
        if (dim == 0) vpos[a] = (int32_t)r;
        else if (dim == 1) epos[(int64_t)a * n + b] = (int32_t)r;
    }
}

// Column sizes and values.
__global__ void k_col_sizes(const SKey *__restrict__ keys, int64_t m, int64_t *__restrict__ cnt,
                            double *__restrict__ value) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < m; r += (int64_t)gridDim.x * blockDim.x) {
        const int dim = (int)(keys[r].lex >> 60);
        cnt[r] = dim > 0 ? dim + 1 : 0;
        if (value) value[r] = dvalue(keys[r].vb);
    }
}

__device__ __forceinline__ void sort3(int32_t &x, int32_t &y, int32_t &z) {
    int32_t t;
    if (x > y) { t = x; x = y; y = t; }
    if (y > z) { t = y; y = z; z = t; }
    if (x > y) { t = x; x = y; y = t; }
}

__global__ void k_rips_rows(const SKey *__restrict__ keys, int64_t m, int n, const int32_t *__restrict__ vpos,
                            const int32_t *__restrict__ epos, const int64_t *__restrict__ colptr,
                            int32_t *__restrict__ rows) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < m; r += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long L = keys[r].lex;
        const int dim = (int)(L >> 60);
        const int a = (int)((L >> 40) & 0xfffff), b = (int)((L >> 20) & 0xfffff), c = (int)(L & 0xfffff);
        const int64_t k = colptr[r];
        if (dim == 1) {
            int32_t x = vpos[a], y = vpos[b];
            rows[k] = min(x, y);
            rows[k + 1] = max(x, y);
        } else if (dim == 2) {
            int32_t x = epos[(int64_t)a * n + b], y = epos[(int64_t)a * n + c], z = epos[(int64_t)b * n + c];
            sort3(x, y, z);
            rows[k] = x;
            rows[k + 1] = y;
            rows[k + 2] = z;
        }
    }
}

// The edges in vertex order: their lengths' bits and the first 32 bits of their
// share of the longest (which order them, but for a few), their vertices,
// their place (the sort's payload).  A warp per row, a lane per vertex of a word.
__global__ void k_rips_edge_list(const unsigned *__restrict__ adj, const double *__restrict__ D, int n, int words,
                                 const long long *__restrict__ eoff, const RipsTotals *__restrict__ totals,
                                 unsigned long long *__restrict__ key, unsigned *__restrict__ coarse,
                                 unsigned *__restrict__ place, int2 *__restrict__ ends) {
    const int lane = threadIdx.x & 31;
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    const double scale = 4294967040.0 / dvalue(totals->longest);
    for (int a = wid; a < n; a += nw) {
        long long e = eoff[a];
        for (int w = a >> 5; w < words; w++) {
            const unsigned bits = adj[(int64_t)a * words + w] & above(w, a);
            if ((bits >> lane) & 1u) {
                const int b = w * 32 + lane;
                const long long at = e + __popc(bits & ((1u << lane) - 1u));
                const double v = D[(int64_t)a * n + b];
                key[at] = dbits(v);
                coarse[at] = __double2uint_rd(v * scale);
                place[at] = (unsigned)at;
                ends[at] = make_int2(a, b);
            }
            e += __popc(bits);
        }
    }
}
// Edges and triangles, counted by pairs of a vertex and 32 others, a warp each.
__global__ void __launch_bounds__(256) k_rips_total(const unsigned *__restrict__ adj, int n, int words,
                                                    RipsTotals *totals) {
    const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
    unsigned long long t = 0, edges = 0;
    for (long long q = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; q < (long long)n * words; q += nw) {
        const int a = (int)(q / words), w0 = (int)(q % words);
        unsigned bits = w0 >= a >> 5 ? adj[(int64_t)a * words + w0] & above(w0, a) : 0u;
        if (lane == 0) edges += __popc(bits);
        for (; bits; bits &= bits - 1) {
            const int b = w0 * 32 + __ffs(bits) - 1;
            for (int w = w0 + lane; w < words; w += 32)
                t += __popc(adj[(int64_t)a * words + w] & adj[(int64_t)b * words + w] & above(w, b));
        }
    }
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) {
        if (t) atomicAdd(&totals->triangles, t);
        if (edges) atomicAdd(&totals->edges, edges);
    }
}
// The edges' ranks from their order by coarse length (32 bits of the length
// over the longest, half the passes of a sort by all 64): an edge comes after
// the shorter ones of its coarse length, of which there are few or none.
// coarse == nullptr: the order is the exact one.  28K edges of a torus: 8 passes
// of 10 us by 64 bits, 4 by 32; with the host's reads between the steps (7, now
// 3) a million columns from points to pairs 659 us -> 554.
constexpr int RIPS_SAME = 64;  // edges of one coarse length
__global__ void k_rips_rank(const unsigned *__restrict__ coarse, const unsigned long long *__restrict__ key,
                            const unsigned *__restrict__ place, const int2 *__restrict__ ends, long long E, int n,
                            int32_t *__restrict__ rank, int2 *__restrict__ by_rank,
                            unsigned long long *__restrict__ sorted, RipsTotals *totals) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < E; k += (long long)gridDim.x * blockDim.x) {
        const unsigned p = place[k];
        const int2 e = ends[p];
        const unsigned long long mine = key[p];
        long long at = k;
        if (coarse) {
            const unsigned c = coarse[k];
            int same = 0;
            bool tied = false;
            for (long long q = k - 1; q >= 0 && coarse[q] == c && same < RIPS_SAME && !tied; q--, same++) {
                const unsigned long long x = key[place[q]];
                at -= x > mine;
                tied = x == mine;
            }
            for (long long q = k + 1; q < E && coarse[q] == c && same < RIPS_SAME && !tied; q++, same++) {
                const unsigned long long x = key[place[q]];
                at += x < mine;
                tied = x == mine;
            }
            if (tied) totals->tied = 1;
            if (tied || same == RIPS_SAME) totals->crowded = 1;  // (nothing more is read from these ranks)
        } else if (k > 0 && key[place[k - 1]] == mine) {
            totals->tied = 1;
        }
        by_rank[at] = e;
        sorted[at] = mine;
        rank[(int64_t)e.x * n + e.y] = rank[(int64_t)e.y * n + e.x] = (int32_t)at;
    }
}

// The triangles whose last edge is k, a warp: `body` gets, word by word of
// 32 vertices, the mask of third vertices (uniform), and each lane's own
// edges' ranks.  32 words at a time are looked over first, so that sparse
// complexes on many vertices skip those without common neighbours.
template <class Body>
__device__ __forceinline__ void rips_run(const unsigned *adj, const int32_t *rank, int n, int words, int2 e, int k,
                                         Body body) {
    const int lane = threadIdx.x & 31;
    const unsigned *ra = adj + (int64_t)e.x * words, *rb = adj + (int64_t)e.y * words;
    for (int w0 = 0; w0 < words; w0 += 32) {
        const unsigned both = w0 + lane < words ? ra[w0 + lane] & rb[w0 + lane] : 0u;
        for (unsigned some = __ballot_sync(0xffffffffu, both != 0u); some; some &= some - 1) {
            const int q = __ffs(some) - 1, c = (w0 + q) * 32 + lane;
            const unsigned m = __shfl_sync(0xffffffffu, both, q);
            int x = 0, y = 0;
            bool on = (m >> lane) & 1u;
            if (on) {
                x = rank[(int64_t)e.x * n + c];
                y = rank[(int64_t)e.y * n + c];
                on = x < k && y < k;
            }
            body(__ballot_sync(0xffffffffu, on), on, x, y);
        }
    }
}

__global__ void k_rips_run_count(const unsigned *__restrict__ adj, const int32_t *__restrict__ rank, int n, int words,
                                 const int2 *__restrict__ by_rank, long long E, const RipsTotals *__restrict__ totals,
                                 long long *__restrict__ cnt) {
    const int nw = (gridDim.x * blockDim.x) >> 5;
    if (totals->crowded) return;  // by_rank has gaps
    for (long long k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < E; k += nw) {
        long long c = 0;
        rips_run(adj, rank, n, words, by_rank[k], (int)k, [&](unsigned mask, bool, int, int) { c += __popc(mask); });
        if ((threadIdx.x & 31) == 0) cnt[k] = c;
    }
}

// The matrix: vertices first, then every edge (column n + k + the triangles
// before it, toff[k]) with its triangles.
__global__ void k_rips_write(const unsigned *__restrict__ adj, const int32_t *__restrict__ rank, int n, int words,
                             const int2 *__restrict__ by_rank, const unsigned long long *__restrict__ key, long long E,
                             const long long *__restrict__ toff, RipsTotals *totals, int64_t *__restrict__ colptr, int32_t *__restrict__ rows, double *__restrict__ value) {
    const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0) totals->triangles = (unsigned long long)toff[E];
    if (totals->tied || totals->crowded || n + E + toff[E] >= 1ll << 31) return;  // the host sees it afterwards
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        colptr[v] = 0;
        if (value) value[v] = 0.0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) colptr[n + E + toff[E]] = 2 * E + 3 * toff[E];
    auto column = [&](int r) { return (int32_t)(n + r + toff[r]); };
    for (long long k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < E; k += nw) {
        const int2 e = by_rank[k];
        const double val = dvalue(key[k]);
        const int32_t col = column((int)k);
        const int64_t start = 2 * k + 3 * toff[k];
        if (lane == 0) {
            colptr[col] = start;
            rows[start] = e.x;
            rows[start + 1] = e.y;
            if (value) value[col] = val;
        }
        int done = 0;
        rips_run(adj, rank, n, words, e, (int)k, [&](unsigned mask, bool on, int x, int y) {
            if (on) {
                const int i = done + __popc(mask & ((1u << lane) - 1u));
                const int64_t at = start + 2 + 3ll * i;
                colptr[col + 1 + i] = at;
                rows[at] = column(min(x, y));
                rows[at + 1] = column(max(x, y));
                rows[at + 2] = col;
                if (value) value[col + 1 + i] = val;
            }
            done += __popc(mask);
        });
    }
}

// ------------------------------------------------------------ lower star
// Vertex (y, x) = y * w + x; the edges of vertex a in the order of their other
// end: H to a + 1, V to a + w, D to a + w + 1, where the image goes on; per
// square the triangles upper (a, a+1, a+w+1) and lower (a, a+w, a+w+1).
__device__ __forceinline__ int64_t ls_edge(unsigned a, unsigned b, int h, int w) {
    const int y = (int)(a / w), x = (int)(a % w);
    if (y == h - 1) return (int64_t)y * (3 * w - 2) + x;
    const int sub = x == w - 1 ? 0 : b == a + 1 ? 0 : b == a + (unsigned)w ? 1 : 2;
    return (int64_t)y * (3 * w - 2) + 3 * x + sub;
}
// The vertices of simplex q (vertices, then edges, then triangles).
__device__ __forceinline__ int ls_simplex(int64_t q, int h, int w, unsigned &a, unsigned &b, unsigned &c) {
    const int64_t V = (int64_t)h * w, E = (int64_t)h * (w - 1) + (int64_t)(h - 1) * w + (int64_t)(h - 1) * (w - 1);
    a = b = c = (unsigned)q;
    if (q < V) return 0;
    q -= V;
    if (q < E) {
        const int per = 3 * w - 2, y = (int)(q / per), i = (int)(q - (int64_t)y * per);
        if (y == h - 1) {  // the last row: H only
            a = y * w + i;
            b = a + 1;
        } else {
            const int x = min(i / 3, w - 1), sub = x == w - 1 ? 1 : i - 3 * x;
            a = y * w + x;
            b = sub == 0 ? a + 1 : sub == 1 ? a + w : a + w + 1;
        }
        c = b;
        return 1;
    }
    q -= E;
    const int64_t sq = q >> 1;
    const int y = (int)(sq / (w - 1)), x = (int)(sq % (w - 1));
    a = y * w + x;
    b = (q & 1) ? a + w : a + 1;
    c = a + w + 1;
    return 2;
}
__device__ __forceinline__ unsigned fbits(float v) {
    const unsigned u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fvalue(unsigned b) {
    return __uint_as_float((b & 0x80000000u) ? (b & 0x7fffffffu) : ~b);
}

// Every simplex's value (its largest vertex's) and place.
__global__ void k_ls_keys(const float *__restrict__ img, int h, int w, int64_t m, unsigned *__restrict__ key,
                          unsigned *__restrict__ place) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < m; q += (int64_t)gridDim.x * blockDim.x) {
        unsigned a, b, c;
        const int dim = ls_simplex(q, h, w, a, b, c);
        float v = img[a];
        const float vb = img[b], vc = img[c];
        if (dim == 1) v = v > vb ? v : vb;
        if (dim == 2) {
            if (vb > v) v = vb;
            if (vc > v) v = vc;
        }
        key[q] = fbits(v);
        place[q] = (unsigned)q;
    }
}

// Sorted simplices: each one's position, its column's size, its value.
__global__ void k_ls_pos(const unsigned *__restrict__ key, const unsigned *__restrict__ place, int64_t m, int64_t V,
                         int64_t VE, int32_t *__restrict__ pos, int64_t *__restrict__ cnt, double *__restrict__ value) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < m; r += (int64_t)gridDim.x * blockDim.x) {
        const int64_t q = place[r];
        if (q < VE) pos[q] = (int32_t)r;
        cnt[r] = q < V ? 0 : q < VE ? 2 : 3;
        if (value) value[r] = (double)fvalue(key[r]);
    }
}

__global__ void k_ls_rows(const unsigned *__restrict__ place, int64_t m, int h, int w, int64_t V,
                          const int32_t *__restrict__ pos, const int64_t *__restrict__ colptr,
                          int32_t *__restrict__ rows) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < m; r += (int64_t)gridDim.x * blockDim.x) {
        unsigned a, b, c;
        const int dim = ls_simplex(place[r], h, w, a, b, c);
        const int64_t k = colptr[r];
        if (dim == 1) {
            const int32_t x = pos[a], y = pos[b];
            rows[k] = min(x, y);
            rows[k + 1] = max(x, y);
        } else if (dim == 2) {
            int32_t x = pos[V + ls_edge(a, b, h, w)], y = pos[V + ls_edge(b, c, h, w)], z = pos[V + ls_edge(a, c, h, w)];
            sort3(x, y, z);
            rows[k] = x;
            rows[k + 1] = y;
            rows[k + 2] = z;
        }
    }
}

int grid_of(Context *ctx, int64_t n) {
    const int64_t g = (n + 255) / 256, cap = (int64_t)ctx->sm_count * 16;
    return (int)std::max<int64_t>(1, std::min(g, cap));
}

// Scratch of one generator call: first from the context's own buffer, kept
// from call to call (pool allocations are given back to the driver at every
// synchronisation, and cost more than the kernels on small complexes) up to
// KEEP_MOST bytes a slot, then from the stream's memory pool, released on every
// exit.
struct Scratch {
    cudaStream_t s;
    std::vector<void *> ptrs;
    char *kept = nullptr;
    size_t room = 0, used = 0;
    explicit Scratch(cudaStream_t st) : s(st) {}
    // the context's buffer `slot`, of at least `bytes` where its budget
    // allows, for what is taken from here on (S_GEN, and those of the
    // reduction, which nothing uses now)
    static constexpr size_t KEEP_MOST = 256 << 20;
    void keep(Context *ctx, int slot, size_t bytes) {
        kept = bytes <= KEEP_MOST ? (char *)ctx_alloc(ctx, slot, bytes) : nullptr;
        room = kept ? ctx->bufs[slot].bytes : 0;
        used = 0;
    }
    void *get(size_t bytes) {
        const size_t want = ((bytes ? bytes : 16) + 255) & ~(size_t)255;
        if (used + want <= room) {
            used += want;
            return kept + used - want;
        }
        void *p = nullptr;
        if (cudaMallocAsync(&p, bytes ? bytes : 16, s) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        ptrs.push_back(p);
        return p;
    }
    ~Scratch() {
        for (void *p : ptrs) cudaFreeAsync(p, s);
    }
};

// Sort the keys, then sizes, values and column pointers; returns the
// sorted keys (in k0 or k1).
int sort_and_colptr(Context *ctx, Scratch &sc, SKey *k0, SKey *k1, int64_t m, int64_t *d_colptr, double *d_value,
                    SKey **sorted) {
    cudaStream_t s = ctx->stream;
    cub::DoubleBuffer<SKey> db(k0, k1);
    size_t tb = 0;
    OPH_CUDA_TRY(cub::DeviceRadixSort::SortKeys(nullptr, tb, db, m, SKeyDecomposer{}, 0, 128, s));
    void *tmp = sc.get(tb);
    if (!tmp) return OPH_ERR_OOM;
    OPH_CUDA_TRY(cub::DeviceRadixSort::SortKeys(tmp, tb, db, m, SKeyDecomposer{}, 0, 128, s));
    *sorted = db.Current();
    // colptr = exclusive scan of the column sizes, colptr[m] = nnz
    int64_t *cnt = (int64_t *)sc.get(sizeof(int64_t) * (size_t)(m + 1));
    if (!cnt) return OPH_ERR_OOM;
    k_col_sizes<<<grid_of(ctx, m), 256, 0, s>>>(*sorted, m, cnt, d_value);
    OPH_CUDA_TRY(cudaMemsetAsync(cnt + m, 0, sizeof(int64_t), s));
    size_t sb = 0;
    OPH_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, sb, cnt, d_colptr, m + 1, s));
    void *st = sc.get(sb);
    if (!st) return OPH_ERR_OOM;
    OPH_CUDA_TRY(cub::DeviceScan::ExclusiveSum(st, sb, cnt, d_colptr, m + 1, s));
    return OPH_OK;
}

}  // namespace

}  // namespace oph

using namespace oph;

extern "C" {

__attribute__((visibility("default"))) int oph_rips_device(oph_context *ctx, const double *d_points, int n, int d,
                                                           double threshold, int64_t *m_out, int64_t *nnz_out,
                                                           int64_t *d_colptr, int32_t *d_rows, double *d_value) {
    if (!ctx || n <= 0 || n > OPH_GEN_MAX_POINTS || d <= 0 || !d_points || threshold != threshold)
        return OPH_ERR_BAD_INPUT;
    OPH_CUDA_TRY(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    Scratch sc(s);
    const int words = (n + 31) / 32;
    const size_t nn = (size_t)n * n;
    sc.keep(ctx, S_GEN, 8 * nn + 4 * (size_t)n * words + 16 * (size_t)(n + 1) + (64 << 10));
    double *D = (double *)sc.get(sizeof(double) * nn);
    unsigned *adj = (unsigned *)sc.get(sizeof(unsigned) * (size_t)n * words);
    long long *deg = (long long *)sc.get(sizeof(long long) * (size_t)(n + 1));
    long long *eoff = (long long *)sc.get(sizeof(long long) * (size_t)(n + 1));
    RipsTotals *totals = (RipsTotals *)sc.get(sizeof(RipsTotals));
    if (!D || !adj || !deg || !eoff || !totals) return OPH_ERR_OOM;
    OPH_CUDA_TRY(cudaMemsetAsync(adj, 0, sizeof(unsigned) * (size_t)n * words, s));
    OPH_CUDA_TRY(cudaMemsetAsync(totals, 0, sizeof(RipsTotals), s));
    k_rips_dist<<<grid_of(ctx, (int64_t)n * n), 256, 0, s>>>(d_points, n, d, threshold, D, adj, words, totals);
    RipsTotals t{};
    if (!d_colptr) {  // sizes only
        k_rips_total<<<grid_of(ctx, 32 * (int64_t)n * words), 256, 0, s>>>(adj, n, words, totals);
        OPH_CUDA_TRY(cudaGetLastError());
        OPH_CUDA_TRY(cudaMemcpyAsync(&t, totals, sizeof(t), cudaMemcpyDeviceToHost, s));
        OPH_CUDA_TRY(cudaStreamSynchronize(s));
        const int64_t m = n + (int64_t)(t.edges + t.triangles);
        if (m >= (1ll << 31)) return OPH_ERR_BAD_INPUT;
        if (m_out) *m_out = m;
        if (nnz_out) *nnz_out = 2 * (int64_t)t.edges + 3 * (int64_t)t.triangles;
        return OPH_OK;
    }
    k_rips_deg<<<grid_of(ctx, n), 256, 0, s>>>(adj, n, words, deg);
    OPH_CUDA_TRY(cudaMemsetAsync(deg + n, 0, sizeof(long long), s));
    size_t sb = 0;
    OPH_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, sb, deg, eoff, n + 1, s));
    void *st = sc.get(sb);
    if (!st) return OPH_ERR_OOM;
    OPH_CUDA_TRY(cub::DeviceScan::ExclusiveSum(st, sb, deg, eoff, n + 1, s));
    long long E = 0;
    OPH_CUDA_TRY(cudaMemcpyAsync(&E, eoff + n, sizeof(long long), cudaMemcpyDeviceToHost, s));
    OPH_CUDA_TRY(cudaStreamSynchronize(s));
    const int wgrid = (int)std::max<int64_t>(1, std::min<int64_t>((n + 7) / 8, (int64_t)ctx->sm_count * 8));
    const int egrid = (int)std::max<int64_t>(1, std::min<int64_t>((E + 7) / 8, (int64_t)ctx->sm_count * 16));
    // the edges: lengths, coarse lengths and places twice (the sort's two
    // buffers), vertices in both orders, ranks, triangles before each
    const size_t e1 = (size_t)E + 1;
    sc.keep(ctx, S_C2_CELLS, 4 * nn + 72 * e1 + (8 << 20));
    unsigned long long *key[2] = {(unsigned long long *)sc.get(8 * e1), (unsigned long long *)sc.get(8 * e1)};
    unsigned *coarse[2] = {(unsigned *)sc.get(4 * e1), (unsigned *)sc.get(4 * e1)};
    unsigned *place[2] = {(unsigned *)sc.get(4 * e1), (unsigned *)sc.get(4 * e1)};
    int2 *ends = (int2 *)sc.get(8 * e1);
    int2 *by_rank = (int2 *)sc.get(8 * e1);
    int32_t *rank = (int32_t *)sc.get(4 * nn);
    long long *tcnt = (long long *)sc.get(8 * e1), *toff = (long long *)sc.get(8 * e1);
    if (!key[0] || !key[1] || !coarse[0] || !coarse[1] || !place[0] || !place[1] || !ends || !by_rank || !rank ||
        !tcnt || !toff)
        return OPH_ERR_OOM;
    size_t sb2 = 0;
    OPH_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, sb2, tcnt, toff, E + 1, s));
    void *st2 = sc.get(sb2);
    if (!st2) return OPH_ERR_OOM;
    int64_t m = 0, nnz = 0;
    for (bool exact = false;; exact = true) {
        OPH_CUDA_TRY(cudaMemsetAsync(tcnt, 0, 8 * e1, s));
        unsigned long long *sorted = key[1];
        if (E > 0) {
            k_rips_edge_list<<<wgrid, 256, 0, s>>>(adj, D, n, words, eoff, totals, key[0], coarse[0], place[0], ends);
            cub::DoubleBuffer<unsigned> dp(place[0], place[1]);
            size_t tb = 0;
            const unsigned *order = nullptr;
            const unsigned long long *lengths = key[0];
            if (!exact) {
                cub::DoubleBuffer<unsigned> dc(coarse[0], coarse[1]);
                OPH_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, dc, dp, E, 0, 32, s));
                void *tmp = sc.get(tb);
                if (!tmp) return OPH_ERR_OOM;
                OPH_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp, tb, dc, dp, E, 0, 32, s));
                order = dc.Current();
            } else {
                // too many edges of one coarse length: by the lengths themselves, beside which they stay by place
                unsigned long long *const by_place = (unsigned long long *)sc.get(8 * e1);
                if (!by_place) return OPH_ERR_OOM;
                OPH_CUDA_TRY(cudaMemcpyAsync(by_place, key[0], 8 * e1, cudaMemcpyDeviceToDevice, s));
                OPH_CUDA_TRY(cudaMemsetAsync(&totals->tied, 0, 2 * sizeof(int), s));
                cub::DoubleBuffer<unsigned long long> dk(key[0], key[1]);
                OPH_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, dk, dp, E, 0, 64, s));
                void *tmp = sc.get(tb);
                if (!tmp) return OPH_ERR_OOM;
                OPH_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp, tb, dk, dp, E, 0, 64, s));
                lengths = by_place;
                sorted = dk.Alternate();
            }
            k_rips_rank<<<grid_of(ctx, E), 256, 0, s>>>(order, lengths, dp.Current(), ends, E, n, rank, by_rank, sorted,
                                                        totals);
            k_rips_run_count<<<egrid, 256, 0, s>>>(adj, rank, n, words, by_rank, E, totals, tcnt);
        }
        OPH_CUDA_TRY(cub::DeviceScan::ExclusiveSum(st2, sb2, tcnt, toff, E + 1, s));
        if (d_rows || E == 0)
            k_rips_write<<<std::max(egrid, 1), 256, 0, s>>>(adj, rank, n, words, by_rank, sorted, E, toff, totals,
                                                            d_colptr, d_rows, d_value);
        else
            OPH_CUDA_TRY(cudaMemcpyAsync(&totals->triangles, toff + E, sizeof(long long), cudaMemcpyDeviceToDevice, s));
        OPH_CUDA_TRY(cudaGetLastError());
        OPH_CUDA_TRY(cudaMemcpyAsync(&t, totals, sizeof(t), cudaMemcpyDeviceToHost, s));
        OPH_CUDA_TRY(cudaStreamSynchronize(s));
        if (t.crowded && !t.tied && !exact) continue;
        break;
    }
    if (t.tied) {  // the triangles above every edge
        OPH_CUDA_TRY(cudaMemsetAsync(tcnt, 0, 8 * e1, s));
        k_rips_tri_count<<<wgrid, 256, 0, s>>>(adj, n, words, eoff, tcnt);
        OPH_CUDA_TRY(cub::DeviceScan::ExclusiveSum(st2, sb2, tcnt, toff, E + 1, s));
        if (t.crowded) {  // (else those by last edge have been counted, as many)
            OPH_CUDA_TRY(cudaMemcpyAsync(&t.triangles, toff + E, sizeof(long long), cudaMemcpyDeviceToHost, s));
            OPH_CUDA_TRY(cudaStreamSynchronize(s));
        }
    }
    m = n + E + (int64_t)t.triangles;
    nnz = 2 * E + 3 * (int64_t)t.triangles;
    if (m >= (1ll << 31)) return OPH_ERR_BAD_INPUT;
    if (m_out) *m_out = m;
    if (nnz_out) *nnz_out = nnz;
    if (!d_rows && nnz > 0) return OPH_ERR_BAD_INPUT;
    if (!t.tied) return OPH_OK;
    // equally long edges: one sort of every simplex
    SKey *k0 = (SKey *)sc.get(sizeof(SKey) * (size_t)m), *k1 = (SKey *)sc.get(sizeof(SKey) * (size_t)m);
    int32_t *vpos = (int32_t *)sc.get(sizeof(int32_t) * (size_t)n);
    if (!k0 || !k1 || !vpos) return OPH_ERR_OOM;
    k_rips_keys<<<wgrid, 256, 0, s>>>(adj, D, n, words, eoff, toff, E, k0);
    SKey *sorted = nullptr;
    int rc = sort_and_colptr(ctx, sc, k0, k1, m, d_colptr, d_value, &sorted);
    if (rc) return rc;
    k_rips_pos<<<grid_of(ctx, m), 256, 0, s>>>(sorted, m, n, vpos, rank);
    k_rips_rows<<<grid_of(ctx, m), 256, 0, s>>>(sorted, m, n, vpos, rank, d_colptr, d_rows);
    OPH_CUDA_TRY(cudaGetLastError());
    OPH_CUDA_TRY(cudaStreamSynchronize(s));
    return OPH_OK;
}

__attribute__((visibility("default"))) int oph_lower_star_device(oph_context *ctx, const float *d_image, int h,
                                                                 int w, int64_t *m_out, int64_t *nnz_out,
                                                                 int64_t *d_colptr, int32_t *d_rows,
                                                                 double *d_value) {
    if (!ctx || h < 2 || w < 2 || (int64_t)h * w >= (1ll << 20) || !d_image) return OPH_ERR_BAD_INPUT;
    const int64_t V = (int64_t)h * w, ED = (int64_t)(h - 1) * (w - 1);
    const int64_t E = (int64_t)h * (w - 1) + (int64_t)(h - 1) * w + ED, T = 2 * ED;
    const int64_t m = V + E + T, nnz = 2 * E + 3 * T;
    if (m_out) *m_out = m;
    if (nnz_out) *nnz_out = nnz;
    if (!d_colptr) return OPH_OK;
    if (!d_rows) return OPH_ERR_BAD_INPUT;
    OPH_CUDA_TRY(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    Scratch sc(s);
    sc.keep(ctx, S_GEN, 16 * (size_t)m + 4 * (size_t)(V + E) + 8 * (size_t)(m + 1) + (4 << 20));
    unsigned *key[2] = {(unsigned *)sc.get(4 * (size_t)m), (unsigned *)sc.get(4 * (size_t)m)};
    unsigned *place[2] = {(unsigned *)sc.get(4 * (size_t)m), (unsigned *)sc.get(4 * (size_t)m)};
    int32_t *pos = (int32_t *)sc.get(sizeof(int32_t) * (size_t)(V + E));
    int64_t *cnt = (int64_t *)sc.get(sizeof(int64_t) * (size_t)(m + 1));
    if (!key[0] || !key[1] || !place[0] || !place[1] || !pos || !cnt) return OPH_ERR_OOM;
    k_ls_keys<<<grid_of(ctx, m), 256, 0, s>>>(d_image, h, w, m, key[0], place[0]);
    cub::DoubleBuffer<unsigned> dk(key[0], key[1]), dp(place[0], place[1]);
    size_t tb = 0, sb = 0;
    OPH_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, dk, dp, m, 0, 32, s));
    OPH_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, sb, cnt, d_colptr, m + 1, s));
    void *tmp = sc.get(tb), *st = sc.get(sb);
    if (!tmp || !st) return OPH_ERR_OOM;
    OPH_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp, tb, dk, dp, m, 0, 32, s));
    k_ls_pos<<<grid_of(ctx, m), 256, 0, s>>>(dk.Current(), dp.Current(), m, V, V + E, pos, cnt, d_value);
    OPH_CUDA_TRY(cudaMemsetAsync(cnt + m, 0, sizeof(int64_t), s));
    OPH_CUDA_TRY(cub::DeviceScan::ExclusiveSum(st, sb, cnt, d_colptr, m + 1, s));
    k_ls_rows<<<grid_of(ctx, m), 256, 0, s>>>(dp.Current(), m, h, w, V, pos, d_colptr, d_rows);
    OPH_CUDA_TRY(cudaGetLastError());
    OPH_CUDA_TRY(cudaStreamSynchronize(s));
    return OPH_OK;
}

}  // extern "C"
