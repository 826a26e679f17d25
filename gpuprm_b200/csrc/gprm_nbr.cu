/*
 * gprm_nbr.cu - neighbour search on the device (gprm_nbr_* of
 * include/gprm_b200.h).
 *
 * The reference planner finds the roadmap nodes within distance D of a new
 * node by scanning the key blocks of its host map (get_near_vertices,
 * prm/src/lib/prm/prmsolver.cpp:2533-2574): squared distance accumulated
 * over the joints in order in float, kept when normsq < D*D, written until
 * the caller's buffer is full.  Here the nodes stay on the device:
 *
 *   radius   one warp per query walks the nodes in index order, 32 at a
 *            time; a ballot compacts the hits, so a query's neighbours come
 *            out in ascending index order and the first `cap` are kept
 *            (the reference's "terminate if buffer full");
 *   knn      the k nearest nodes under the same distance, ties broken by
 *            the lower index.  Nodes are bucketed into a uniform grid over
 *            all joints (counting sort by cell); a query scans the
 *            3^ndof cells around its own and keeps a sorted top-k
 *            (a warp per query); a
 *            result is accepted only when its k-th distance is below the
 *            distance to the scanned block's boundary (with slack for float
 *            rounding), otherwise the query is redone over the 5^ndof block,
 *            and if that block's test fails too, by a
 *            block that scans every node.  The result is therefore the exact
 *            top-k.
 *
 * Distances use the reference's arithmetic: d = x_j - q_j, s = s + d*d
 * (no FMA; the library is compiled with -fmad=false), dist = sqrt(s).
 */
#include <cuda_runtime.h>
#include <math.h>
#include <stdarg.h>
#include <stdio.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/gprm_b200.h"

namespace {

constexpr int NBR_MAX_GRID = GPRM_MAX_DOF;
constexpr int NBR_MAX_K = 32;
constexpr int NBR_MAX_CELLS = 1 << 21;
constexpr int NBR_MAX_JOINT_CELLS = 1 << 17;   /* the slack for rounding is then 0.13 of a cell */
/* cell size over the estimated distance of the 16th neighbour: smaller cells
 * hold fewer nodes out of reach, but more queries outgrow their 3^ndof block
 * (480,001 6-D nodes, k = 10: 3.5 ms at 1.1, 4.5 at 1.0, 8.3 at 0.9) */
constexpr double KNN_CELL = 1.1;

struct GridView {
    int ndof, G, n;
    float lo[NBR_MAX_GRID];
    float inv_cell;   /* 1 / cell */
    float cell;
    float slack;      /* rounding allowance of the exactness test */
    int nc[NBR_MAX_GRID];
    const float* xs;      /* nodes sorted by cell, SoA [ndof][n] */
    const int* id;        /* original index of each sorted node */
    const int* start;     /* cell start offsets [ncells + 1] */
};

__device__ __forceinline__ float dist2(const float* __restrict__ x, long long xstride, long long i,
                                       const float* qv, int ndof)
{
    float s = 0.0f;
    for (int j = 0; j < ndof; ++j) {
        const float d = x[i + xstride * j] - qv[j];
        s = s + d * d;
    }
    return s;
}

__device__ __forceinline__ int cell_coord(float v, float lo, float inv_cell, int nc)
{
    float c = floorf((v - lo) * inv_cell);
    int ci = isfinite(c) ? (int)fminf(fmaxf(c, 0.0f), (float)(nc - 1)) : 0;
    return ci;
}

/* dist2 of four consecutive nodes p..p+3: the same arithmetic per node,
 * the four nodes' loads issued together. */
__device__ __forceinline__ void dist2_4(const float* __restrict__ x, long long xstride, long long p, const float* qv,
                                        int ndof, float* s)
{
    s[0] = s[1] = s[2] = s[3] = 0.0f;
    for (int j = 0; j < ndof; ++j) {
        const float* xj = x + p + xstride * j;
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = xj[u];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float d = v[u] - qv[j];
            s[u] = s[u] + d * d;
        }
    }
}

/* (s, id) lexicographic order */
__device__ __forceinline__ bool less_pair(float s, int i, float t, int j)
{
    return s < t || (s == t && i < j);
}

__global__ void k_minmax(const float* __restrict__ x, int n, long long stride, int ndof, float* out)
{
    /* out[2j] = min, out[2j+1] = max of joint j; out pre-set to +inf/-inf */
    for (int j = 0; j < ndof; ++j) {
        float lo = INFINITY, hi = -INFINITY;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            const float v = x[i + stride * j];
            if (isfinite(v)) { lo = fminf(lo, v); hi = fmaxf(hi, v); }
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        /* one atomic per block: one per warp queued 4,700 of them on a word
           (480,001 points: 42 -> 13 us) */
        __shared__ float ws[2][32];
        const int lane = threadIdx.x & 31;
        __syncthreads();
        if (lane == 0) { ws[0][threadIdx.x >> 5] = lo; ws[1][threadIdx.x >> 5] = hi; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < (int)(blockDim.x >> 5); ++w) { lo = fminf(lo, ws[0][w]); hi = fmaxf(hi, ws[1][w]); }
            /* float min/max through the ordered-int trick (values are finite) */
            int* o2 = reinterpret_cast<int*>(out);
            if (lo <= hi) {
                if (lo >= 0) atomicMin(&o2[2 * j], __float_as_int(lo));
                else atomicMax((unsigned*)&o2[2 * j], __float_as_uint(lo));
                if (hi >= 0) atomicMax(&o2[2 * j + 1], __float_as_int(hi));
                else atomicMin((unsigned*)&o2[2 * j + 1], __float_as_uint(hi));
            }
        }
    }
}

__global__ void k_cell_keys(const float* __restrict__ x, int n, long long stride, GridView g, int* key, int* count)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int k = 0;
        for (int d = g.G - 1; d >= 0; --d) k = k * g.nc[d] + cell_coord(x[i + stride * d], g.lo[d], g.inv_cell, g.nc[d]);
        key[i] = k;
        atomicAdd(&count[k], 1);
    }
}

/* Exclusive scan of count[0..nc) into start[0..nc], one block: 4096 counts a
 * pass, four neighbouring ones per thread, a shuffle scan per warp and one
 * over the warps' sums.  Bound by the passes' latency (12 of them for 6^6
 * cells); a contiguous piece per thread, read one word at a time, took 111 of
 * the search's 3,500 us at 480,001 points. */
__global__ void __launch_bounds__(1024) k_scan(const int* __restrict__ count, int nc, int* start)
{
    __shared__ int part[2][32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int carry = 0, buf = 0, next[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) next[k] = 4 * t + k < nc ? count[4 * t + k] : 0;
    for (int b = 0; b < nc; b += 4096, buf ^= 1) {
        const int i = b + 4 * t;
        int v[4], s = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = next[k];
            s += v[k];
            next[k] = (long long)i + 4096 + k < nc ? count[i + 4096 + k] : 0;
        }
        int x = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) part[buf][warp] = x;
        __syncthreads();   /* the other buffer's readers are past the last one */
        int w = part[buf][lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        const int total = __shfl_sync(0xffffffffu, w, 31);
        const int before = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
        int run = carry + (warp > 0 ? before : 0) + x - s;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (i + k < nc) start[i + k] = run;
            run += v[k];
        }
        carry += total;
    }
    if (t == 0) start[nc] = carry;
}

__global__ void k_scatter(const float* __restrict__ x, int n, long long stride, int ndof, const int* __restrict__ key,
                          const int* __restrict__ start, int* cursor, float* xs, int* id)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int k = key[i];
        const int p = start[k] + atomicAdd(&cursor[k], 1);
        for (int j = 0; j < ndof; ++j) xs[p + (long long)n * j] = x[i + stride * j];
        id[p] = i;
    }
}

/* ---------------------------------------------------------------- radius */

__global__ void k_radius(const float* __restrict__ x, int n, long long xstride, const float* __restrict__ q, int m,
                         long long qstride, int ndof, float D2, int cap, int* counts, int* idx, float* dist)
{
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    for (long long w = (long long)blockIdx.x * wpb + (threadIdx.x >> 5); w < m; w += (long long)gridDim.x * wpb) {
        float qv[GPRM_MAX_DOF];
        for (int j = 0; j < ndof; ++j) qv[j] = q[w + qstride * j];
        int found = 0;
        for (int base = 0; base < n && found < cap; base += 32) {
            const int i = base + lane;
            float s = 0.0f;
            bool hit = false;
            if (i < n) {
                s = dist2(x, xstride, i, qv, ndof);
                hit = s < D2;
            }
            const unsigned hm = __ballot_sync(0xffffffffu, hit);
            if (hit) {
                const int slot = found + __popc(hm & ((1u << lane) - 1u));
                if (slot < cap) {
                    idx[w * (long long)cap + slot] = i;
                    dist[w * (long long)cap + slot] = sqrtf(s);
                }
            }
            found += __popc(hm);
        }
        if (lane == 0) counts[w] = found < cap ? found : cap;
    }
}

/* ---------------------------------------------------------------- knn */

/* The list's current k-th entry, kept in registers so that most
 * candidates are rejected by one comparison, before their index is even
 * loaded: (INFINITY, INT_MAX) until the list is full. */
struct TopkBound {
    float s;
    int i;
};

__device__ __forceinline__ void topk_bound(const float* ts, const int* ti, int len, int k, TopkBound& b)
{
    if (len == k) { b.s = ts[k - 1]; b.i = ti[k - 1]; }
}

/* Inserts (s, i) into the sorted top list (len entries used, capacity k). */
__device__ __forceinline__ void topk_insert(float* ts, int* ti, int& len, int k, float s, int i)
{
    if (len == k && !less_pair(s, i, ts[k - 1], ti[k - 1])) return;
    int p = len < k ? len : k - 1;
    while (p > 0 && less_pair(s, i, ts[p - 1], ti[p - 1])) {
        ts[p] = ts[p - 1];
        ti[p] = ti[p - 1];
        --p;
    }
    ts[p] = s;
    ti[p] = i;
    if (len < k) ++len;
}

/* The block of cells a query scans: cells c-radius..c+radius in each
 * gridded joint (clipped to the grid); guard = the distance from q to the block's faces
 * that have cells beyond them (infinite when none).  Returns false when a
 * gridded coordinate is not finite. */
__device__ __forceinline__ bool query_block(const GridView& g, const float* qv, int* lo, int* hi, float* guard,
                                            int radius = 1)
{
    bool finite = true;
    float gd = INFINITY;
    for (int d = 0; d < g.G; ++d) {
        finite &= isfinite(qv[d]);
        const int c = cell_coord(qv[d], g.lo[d], g.inv_cell, g.nc[d]);
        lo[d] = max(c - radius, 0);
        hi[d] = min(c + radius, g.nc[d] - 1);
        if (lo[d] > 0) gd = fminf(gd, qv[d] - (g.lo[d] + (float)lo[d] * g.cell));
        if (hi[d] < g.nc[d] - 1) gd = fminf(gd, (g.lo[d] + (float)(hi[d] + 1) * g.cell) - qv[d]);
    }
    for (int j = g.G; j < g.ndof; ++j) finite &= isfinite(qv[j]);
    *guard = gd;
    return finite;
}

/* Number of rows of the block (cells varying in joints 1..G-1) and the
 * sorted-node range of row r (joint 0 runs lo[0]..hi[0], contiguous). */
__device__ __forceinline__ int block_rows(const GridView& g, const int* lo, const int* hi)
{
    int r = 1;
    for (int d = 1; d < g.G; ++d) r *= hi[d] - lo[d] + 1;
    return r;
}

__device__ __forceinline__ void block_row_range(const GridView& g, const int* lo, const int* hi, int r, int* b, int* e)
{
    int cell = 0;
    int rest = r;
    int coord[NBR_MAX_GRID];
    for (int d = 1; d < g.G; ++d) {
        const int span = hi[d] - lo[d] + 1;
        coord[d] = lo[d] + rest % span;
        rest /= span;
    }
    for (int d = g.G - 1; d >= 1; --d) cell = cell * g.nc[d] + coord[d];
    const int row = cell * g.nc[0];
    *b = g.start[row + lo[0]];
    *e = g.start[row + hi[0] + 1];
}

/* The exactness test: k results strictly inside the guard ball, with slack
 * for the rounding of the cell assignment and of s. */
__device__ __forceinline__ bool knn_exact(const GridView& g, bool finite, int len, int k, float kth, float guard)
{
    const float gs = guard - g.slack;
    return finite && len == k && (!isfinite(gs) || (gs > 0.0f && kth < gs * gs * 0.99999f));
}

/* A lower bound of the squared distance to a node in a cell whose coordinate
 * range starts `gap` beyond q: shortened by the rounding of the cell
 * assignment and of the nodes' computed distances, so that a node whose cell
 * is skipped for it could not have entered the list. */
__device__ __forceinline__ float gap2(const GridView& g, float gap)
{
    const float d = fmaxf(gap - g.slack, 0.0f);
    return d * d * 0.99998f;
}

/* gap2 of coordinate v of joint d to the cells with coordinate c (the edge
 * cells hold every node beyond the grid as well). */
__device__ __forceinline__ float cell_gap2(const GridView& g, float v, int d, int c)
{
    const float below = c > 0 ? (g.lo[d] + (float)c * g.cell) - v : 0.0f;
    const float above = c < g.nc[d] - 1 ? v - (g.lo[d] + (float)(c + 1) * g.cell) : 0.0f;
    return gap2(g, fmaxf(below, above));
}

/* A thread per query, the node at sorted position t, over every cell around
 * its own (queries and nodes in the same order: neighbouring threads read
 * the same cells).  In up to three joints those are few cells, and a warp
 * that shares them among its lanes mostly idles; with many nodes and a short
 * list the threads are faster.  Uniform nodes, us, warp against thread:
 *            65,536 nodes             200,000                  1,000,000
 *   joints   k = 1    4       10      k = 1    4       10      k = 1     4        10
 *   1        53/25    69/34   103/52  118/32   167/53  270/110 506/71    754/164  1291/402
 *   2        69/34    83/51   119/86  163/48   209/80  309/193 726/138   961/264  1460/622
 *   3        91/57    111/88  159/151 225/94   285/150 428/345 1040/336  1337/549 2048/1199
 * (30,000 nodes, k = 10: 60/47, 68/78, 86/133; 30,000 crowded ones take a
 * thread twice as long as a warp.) */
constexpr int KNN_THREAD_DIM = 3, KNN_THREAD_K = 10, KNN_THREAD_NODES = 1 << 16;
template <int DIM>
__global__ void __launch_bounds__(128) k_knn_grid_thread(GridView g, int m, int k, int* out_idx, float* out_dist,
                                                         int* redo, int* nredo)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < m; t += gridDim.x * blockDim.x) {
        float qv[DIM];
        const int qid = g.id[t];
#pragma unroll
        for (int j = 0; j < DIM; ++j) qv[j] = g.xs[t + (long long)g.n * j];
        float ts[KNN_THREAD_K];
        int ti[KNN_THREAD_K];
        int len = 0;
        TopkBound bound{INFINITY, 0x7fffffff};
        int lo[NBR_MAX_GRID], hi[NBR_MAX_GRID];
        float guard;
        const bool finite = query_block(g, qv, lo, hi, &guard);
        const int rows = block_rows(g, lo, hi);
        for (int r = 0; r < rows; ++r) {
            int b, e;
            block_row_range(g, lo, hi, r, &b, &e);
            for (int p = b; p < e; p += 4) {
                float s[4];
                if (p + 4 <= e) {
                    dist2_4(g.xs, g.n, p, qv, DIM, s);
                } else {
                    for (int u = 0; u < 4; ++u) s[u] = p + u < e ? dist2(g.xs, g.n, p + u, qv, DIM) : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float sd = s[u] == s[u] ? s[u] : INFINITY;     /* NaN sorts last */
                    if (p + u >= e || p + u == t || sd > bound.s) continue;
                    const int id = g.id[p + u];
                    if (!less_pair(sd, id, bound.s, bound.i)) continue;
                    topk_insert(ts, ti, len, k, sd, id);
                    topk_bound(ts, ti, len, k, bound);
                }
            }
        }
        const float kth = len ? ts[len - 1] : INFINITY;
        if (knn_exact(g, finite, len, k, kth, guard)) {
            for (int r = 0; r < k; ++r) {
                out_idx[(long long)qid * k + r] = ti[r];
                out_dist[(long long)qid * k + r] = sqrtf(ts[r]);
            }
        } else {
            out_dist[(long long)qid * k + k - 1] = finite && len == k ? kth : INFINITY;
            redo[atomicAdd(nredo, 1)] = qid;
        }
    }
}

template <int N> struct Pow3 { static constexpr int value = 3 * Pow3<N - 1>::value; };
template <> struct Pow3<0> { static constexpr int value = 1; };

/* A warp's candidates of k_knn_grid. */
constexpr int KNN_CAND = 128;
struct KnnWarp {
    float s[KNN_CAND];
    int id[KNN_CAND];
};

/* Keeps the k smallest of the warp's n candidates (n <= KNN_CAND), sorted by
 * (distance, index): k rounds of a warp minimum over four candidates a
 * lane.  Squared distances are not negative, so their bits order like
 * them. */
__device__ __forceinline__ void knn_select(KnnWarp& W, int& n, int k)
{
    const int lane = threadIdx.x & 31;
    unsigned s[4];
    int id[4];
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int c = lane + 32 * u;
        s[u] = c < n ? __float_as_uint(W.s[c]) : 0xffffffffu;
        id[u] = c < n ? W.id[c] : 0x7fffffff;
    }
    __syncwarp();
    if (k > n) k = n;
    n = k;
#pragma unroll 1
    for (int r = 0; r < k; ++r) {
        const unsigned m = __reduce_min_sync(0xffffffffu, min(min(s[0], s[1]), min(s[2], s[3])));
        int mine = 0x7fffffff;
#pragma unroll
        for (int u = 0; u < 4; ++u) mine = s[u] == m ? min(mine, id[u]) : mine;
        const int best = __reduce_min_sync(0xffffffffu, mine);
#pragma unroll
        for (int u = 0; u < 4; ++u) s[u] = s[u] == m && id[u] == best ? 0xffffffffu : s[u];
        if (lane == 0) {
            W.s[r] = __uint_as_float(m);
            W.id[r] = best;
        }
    }
    __syncwarp();
}

/* The nodes of the lanes' rows [b, e) (sorted positions; e = b: none), one
 * after the other over the lanes: those within `reach` of q (not the node at
 * position self_at or of index self_id) join the warp's n candidates, cut
 * back to the k best, with the bound they give, when the buffer fills. */
template <int DIM>
__device__ __forceinline__ void knn_scan(const GridView& g, KnnWarp& W, const float* qv, int b, int e, int self_at,
                                         int self_id, int k, int& n, float& reach)
{
    const int lane = threadIdx.x & 31;
    int upto = e - b;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= d) upto += y;
    }
    const int total = __shfl_sync(0xffffffffu, upto, 31);
    const int shift = b - (upto - (e - b));         /* node = its number + its row's shift */
#pragma unroll 1
    for (int f0 = 0; f0 < total; f0 += 32) {
        const int f = f0 + lane;
        int row = 0;                                /* the first row with upto > f */
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) {
            const int y = __shfl_sync(0xffffffffu, upto, row + d - 1);
            if (y <= f) row += d;
        }
        const int p = f + __shfl_sync(0xffffffffu, shift, row & 31);
        bool hit = false;
        float s = 0.0f;
        int id = 0;
        if (f < total) {
#pragma unroll
            for (int j = 0; j < DIM; ++j) {
                const float d = g.xs[p + (long long)g.n * j] - qv[j];
                s = s + d * d;
            }
            if (s != s) s = INFINITY;               /* NaN sorts last */
            hit = s <= reach && p != self_at;
            if (hit) {
                id = g.id[p];
                hit = id != self_id;
            }
        }
        const unsigned hm = __ballot_sync(0xffffffffu, hit);
        if (hm) {
            if (n > KNN_CAND - 32) {
                knn_select(W, n, k);
                if (n == k) reach = fminf(reach, W.s[k - 1]);
            }
            if (hit) {
                const int at = n + __popc(hm & ((1u << lane) - 1u));
                W.s[at] = s;
                W.id[at] = id;
            }
            n += __popc(hm);
        }
    }
}

/* A warp per query, the node at sorted position t (queries are the nodes;
 * neighbouring warps hold neighbouring nodes).  Of the 3^DIM cells around
 * the query's, in rows of three along joint 0, first the own row and those
 * one cell away in one other joint are read: the k-th distance so far is
 * then a bound within which few of the other rows lie (the ball of the k-th
 * distance holds k of the block's about 3000 nodes).  A lane per row adds up
 * the gaps to its cells; the rows in reach are read eight at a time, four
 * lanes a row.  Nodes within the bound are collected and cut back to the k
 * best when the buffer fills.  A query that the block cannot settle leaves
 * its k-th squared distance in its last output slot for k_knn_wide.
 * 480,001 6-D nodes, k = 10: 7.1 ms with a thread per query reading every
 * cell, 4.5 ms with a thread per query and the bound (10 of 32 lanes
 * active), 3.7 ms
 * with four lanes a row. */
template <int DIM>
__global__ void __launch_bounds__(256) k_knn_grid(GridView g, int m, int k, int* out_idx, float* out_dist, int* redo,
                                                  int* nredo)
{
    constexpr int ROWS = Pow3<DIM - 1>::value;
    __shared__ unsigned short digits[ROWS];      /* per row two bits a joint: own, below, above; few moves first */
    __shared__ int slot[8];
    __shared__ KnnWarp ws[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 8) slot[threadIdx.x] = 0;
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass) {
        for (int r = threadIdx.x; r < ROWS; r += blockDim.x) {
            int rest = r, moved = 0, dg = 0;
            for (int d = 0; d < DIM - 1; ++d) {
                const int c = rest % 3;
                rest /= 3;
                moved += c != 0;
                dg |= c << (2 * d);
            }
            const int at = atomicAdd(&slot[moved], 1);
            if (pass == 1) digits[at] = (unsigned short)dg;
        }
        __syncthreads();
        if (pass == 0 && threadIdx.x == 0) {
            int sum = 0;
            for (int c = 0; c < 8; ++c) {
                const int n = slot[c];
                slot[c] = sum;
                sum += n;
            }
        }
        __syncthreads();
    }
    KnnWarp& W = ws[warp];
    for (int t = blockIdx.x * 8 + warp; t < m; t += gridDim.x * 8) {
        float qv[DIM];
        const int qid = g.id[t];
#pragma unroll
        for (int j = 0; j < DIM; ++j) qv[j] = g.xs[t + (long long)g.n * j];
        int lo[NBR_MAX_GRID], hi[NBR_MAX_GRID];
        float guard;
        const bool finite = query_block(g, qv, lo, hi, &guard);
        float below[DIM], above[DIM];            /* squared gaps, INFINITY: no such cell */
        int stride[DIM], own = 0, cells = 1;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const int c = cell_coord(qv[d], g.lo[d], g.inv_cell, g.nc[d]);
            own += c * cells;
            stride[d] = cells;
            cells *= g.nc[d];
            below[d] = c > lo[d] ? gap2(g, qv[d] - (g.lo[d] + (float)c * g.cell)) : INFINITY;
            above[d] = c < hi[d] ? gap2(g, (g.lo[d] + (float)(c + 1) * g.cell) - qv[d]) : INFINITY;
        }
        int n = 0;
        float reach = INFINITY;                  /* nodes beyond it cannot enter the list */
        const int first = 2 * DIM - 1;
#pragma unroll 1
        for (int r0 = 0; r0 < ROWS; r0 += r0 == 0 ? first : 32) {
            const int r1 = r0 == 0 ? (first < 32 ? first : 32) : min(ROWS, r0 + 32);
            const int r = r0 + lane;
            bool open = false;
            int b = 0, e = 0;
            if (r < r1) {
                const unsigned dg = digits[r];
                float gap = 0.0f;
                int cell = own;
#pragma unroll
                for (int d = 1; d < DIM; ++d) {
                    const unsigned c = (dg >> (2 * (d - 1))) & 3u;
                    gap = c == 0u ? gap : gap + (c == 1u ? below[d] : above[d]);
                    cell += c == 0u ? 0 : c == 1u ? -stride[d] : stride[d];
                }
                open = gap <= reach && gap != INFINITY;
                if (open) {
                    b = g.start[cell - (below[0] != INFINITY && gap + below[0] <= reach)];
                    e = g.start[cell + 1 + (above[0] != INFINITY && gap + above[0] <= reach)];
                    open = e > b;
                }
            }
            knn_scan<DIM>(g, W, qv, open ? b : 0, open ? e : 0, t, -1, k, n, reach);
            if (n > k) {
                /* a tighter bound for the rows to come */
                knn_select(W, n, k);
                reach = W.s[k - 1];
            }
        }
        knn_select(W, n, k);
        const float kth = n ? W.s[n - 1] : INFINITY;
        if (knn_exact(g, finite, n, k, kth, guard)) {
            if (lane < k) {
                out_idx[(long long)qid * k + lane] = W.id[lane];
                out_dist[(long long)qid * k + lane] = sqrtf(W.s[lane]);
            }
        } else if (lane == 0) {
            out_dist[(long long)qid * k + k - 1] = finite && n == k ? kth : INFINITY;
            redo[atomicAdd(nredo, 1)] = qid;
        }
        __syncwarp();
    }
}

/* Merges the lanes' sorted top lists into the warp's k smallest (k rounds
 * of a warp argmin); every lane gets round r's winner in (ws, wi) when
 * r == its lane. */
__device__ __forceinline__ void warp_topk_merge(const float* ts, const int* ti, int len, int k, float* my_s, int* my_i,
                                                float* kth, int* found)
{
    const int lane = threadIdx.x & 31;
    int head = 0, cnt = 0;
    float last = INFINITY;
    *my_s = INFINITY;
    *my_i = -1;
    for (int r = 0; r < k; ++r) {
        float bs = head < len ? ts[head] : INFINITY;
        int bi = head < len ? ti[head] : 0x7fffffff;
        for (int o = 16; o > 0; o >>= 1) {
            const float os = __shfl_xor_sync(0xffffffffu, bs, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (less_pair(os, oi, bs, bi)) { bs = os; bi = oi; }
        }
        if (head < len && ti[head] == bi && ts[head] == bs) ++head;
        if (bi != 0x7fffffff) { ++cnt; last = bs; }
        if (lane == r) { *my_s = bs; *my_i = bi != 0x7fffffff ? bi : -1; }
    }
    *kth = last;
    *found = cnt;
}

/* Warp per query (outside queries q): lanes split the block's nodes. */
__global__ void k_knn_grid_warp(GridView g, const float* __restrict__ q, int m, long long qstride, int k,
                                int* out_idx, float* out_dist, int* redo, int* nredo)
{
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    for (int t = blockIdx.x * wpb + (threadIdx.x >> 5); t < m; t += gridDim.x * wpb) {
        float qv[GPRM_MAX_DOF];
        for (int j = 0; j < g.ndof; ++j) qv[j] = q[t + qstride * j];
        float ts[NBR_MAX_K];
        int ti[NBR_MAX_K];
        int len = 0;
        TopkBound bound{INFINITY, 0x7fffffff};
        int lo[NBR_MAX_GRID], hi[NBR_MAX_GRID];
        float guard;
        const bool finite = query_block(g, qv, lo, hi, &guard);
        const int rows = block_rows(g, lo, hi);
        /* many short rows (every joint gridded): the lanes split the rows;
           few long rows: the lanes split each row's nodes */
        const bool by_row = rows >= 32;
        for (int r = by_row ? lane : 0; r < rows; r += by_row ? 32 : 1) {
            int b, e;
            block_row_range(g, lo, hi, r, &b, &e);
            for (int p = b + (by_row ? 0 : lane); p < e; p += by_row ? 1 : 32) {
                float sd = dist2(g.xs, g.n, p, qv, g.ndof);
                if (sd != sd) sd = INFINITY;
                if (sd > bound.s) continue;
                const int nid = g.id[p];
                if (!less_pair(sd, nid, bound.s, bound.i)) continue;
                topk_insert(ts, ti, len, k, sd, nid);
                topk_bound(ts, ti, len, k, bound);
            }
        }
        float my_s, kth;
        int my_i, found;
        warp_topk_merge(ts, ti, len, k, &my_s, &my_i, &kth, &found);
        if (knn_exact(g, finite, found, k, kth, guard)) {
            if (lane < k) {
                out_idx[(long long)t * k + lane] = my_i;
                out_dist[(long long)t * k + lane] = sqrtf(my_s);
            }
        } else if (lane == 0) {
            out_dist[(long long)t * k + k - 1] = finite && found == k ? kth : INFINITY;
            redo[atomicAdd(nredo, 1)] = t;
        }
    }
}

/* Second try for the queries the 3^ndof block could not settle: a warp per
 * query goes through the 5^ndof (1-D: 17) block around it and applies the same
 * exactness test with that block's guard; a query it cannot settle either
 * goes to the full scan (redo2).  The k-th squared distance over the 3^ndof
 * block, left in the query's last output slot, bounds the true one from the
 * start: few of the block's rows are in its reach.  (A block of threads per
 * query that read every row took 3.6 ms for 6,600 of 480,001 6-D queries,
 * with the bound 0.8 ms.) */
template <int DIM>
__global__ void __launch_bounds__(256) k_knn_wide(GridView g, const float* __restrict__ q, long long qstride, int k,
                                                  int exclude_self, const int* __restrict__ redo,
                                                  const int* __restrict__ nredo, int* redo2, int* nredo2,
                                                  int* out_idx, float* out_dist)
{
    constexpr int SPAN = DIM == 1 ? 17 : 5;   /* 1-D: 44 nodes in five cells, too few for k = 32 */
    __shared__ KnnWarp ws[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    KnnWarp& W = ws[warp];
    const int cnt = *nredo;
    for (int w = blockIdx.x * 8 + warp; w < cnt; w += gridDim.x * 8) {
        const int qid = redo[w];
        float qv[DIM];
#pragma unroll
        for (int j = 0; j < DIM; ++j) qv[j] = q[qid + qstride * j];
        int lo[NBR_MAX_GRID], hi[NBR_MAX_GRID];
        float guard;
        const bool finite = query_block(g, qv, lo, hi, &guard, SPAN / 2);
        float reach = out_dist[(long long)qid * k + k - 1];
        const int self = exclude_self ? qid : -1;
        int n = 0, rows = 1;
#pragma unroll
        for (int d = 1; d < DIM; ++d) rows *= hi[d] - lo[d] + 1;
#pragma unroll 1
        for (int r0 = 0; r0 < rows; r0 += 32) {
            const int r = r0 + lane;
            int b = 0, e = 0;
            if (r < rows) {
                float gap = 0.0f;
                int rest = r, cell = 0, cells = g.nc[0];
#pragma unroll
                for (int d = 1; d < DIM; ++d) {
                    const int span = hi[d] - lo[d] + 1;
                    const int c = lo[d] + rest % span;
                    rest /= span;
                    gap = gap + cell_gap2(g, qv[d], d, c);
                    cell += c * cells;
                    cells *= g.nc[d];
                }
                if (gap <= reach) {
                    int c0 = lo[0], c1 = hi[0];
                    while (c0 < c1 && gap + cell_gap2(g, qv[0], 0, c0) > reach) ++c0;
                    while (c1 > c0 && gap + cell_gap2(g, qv[0], 0, c1) > reach) --c1;
                    b = g.start[cell + c0];
                    e = g.start[cell + c1 + 1];
                }
            }
            if (__any_sync(0xffffffffu, e > b)) knn_scan<DIM>(g, W, qv, b, e, -1, self, k, n, reach);
        }
        knn_select(W, n, k);
        const float kth = n ? W.s[n - 1] : INFINITY;
        if (knn_exact(g, finite, n, k, kth, guard)) {
            if (lane < k) {
                out_idx[(long long)qid * k + lane] = W.id[lane];
                out_dist[(long long)qid * k + lane] = sqrtf(W.s[lane]);
            }
        } else if (lane == 0) {
            redo2[atomicAdd(nredo2, 1)] = qid;
        }
        __syncwarp();
    }
}

/* Redo of the queries the grid could not settle: one block per query scans
 * every node (each thread four consecutive nodes at a time, keeping its own
 * top-k); each warp merges its lanes' lists by k rounds of a warp argmin,
 * then warp 0 merges the eight warp lists the same way. */
__global__ void __launch_bounds__(256) k_knn_full(const float* __restrict__ x, int n, long long xstride,
                                                  const float* __restrict__ q, long long qstride, int ndof, int k,
                                                  int exclude_self, const int* __restrict__ redo,
                                                  const int* __restrict__ nredo, int* out_idx, float* out_dist)
{
    __shared__ float ms[8 * NBR_MAX_K];
    __shared__ int mi[8 * NBR_MAX_K];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cnt = *nredo;
    for (int w = blockIdx.x; w < cnt; w += gridDim.x) {
        const int qid = redo[w];
        float qv[GPRM_MAX_DOF];
        for (int j = 0; j < ndof; ++j) qv[j] = q[qid + qstride * j];
        float ts[NBR_MAX_K];
        int ti[NBR_MAX_K];
        int len = 0;
        TopkBound bound{INFINITY, 0x7fffffff};
        /* thread t takes nodes 4t.. 4t+3, 4(t+256).. : four loads in flight */
        for (int i0 = 4 * threadIdx.x; i0 < n; i0 += 4 * 256) {
            float s4[4];
            if (i0 + 4 <= n) {
                dist2_4(x, xstride, i0, qv, ndof, s4);
            } else {
                for (int u = 0; u < 4; ++u) s4[u] = i0 + u < n ? dist2(x, xstride, i0 + u, qv, ndof) : INFINITY;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u;
                if (i >= n || (exclude_self && i == qid)) continue;
                float s = s4[u];
                if (s != s) s = INFINITY;   /* NaN sorts last */
                if (!less_pair(s, i, bound.s, bound.i)) continue;
                topk_insert(ts, ti, len, k, s, i);
                topk_bound(ts, ti, len, k, bound);
            }
        }
        /* per warp: the k smallest of its lanes; then warp 0 merges the 8 lists */
        float my_s, kth;
        int my_i, found;
        warp_topk_merge(ts, ti, len, k, &my_s, &my_i, &kth, &found);
        if (lane < k) {
            ms[warp * k + lane] = my_s;
            mi[warp * k + lane] = my_i < 0 ? 0x7fffffff : my_i;
        }
        __syncthreads();
        if (warp == 0) {
            len = 0;
            bound = TopkBound{INFINITY, 0x7fffffff};
            for (int e = lane; e < 8 * k; e += 32) {
                if (mi[e] == 0x7fffffff) continue;
                if (!less_pair(ms[e], mi[e], bound.s, bound.i)) continue;
                topk_insert(ts, ti, len, k, ms[e], mi[e]);
                topk_bound(ts, ti, len, k, bound);
            }
            warp_topk_merge(ts, ti, len, k, &my_s, &my_i, &kth, &found);
            if (lane < k) {
                const bool have = my_i >= 0;
                out_idx[(long long)qid * k + lane] = have ? my_i : -1;
                out_dist[(long long)qid * k + lane] = have ? sqrtf(my_s) : INFINITY;
            }
        }
        __syncthreads();
    }
}

}  // namespace

struct gprm_nbr {
    int ndof = 0;
    int device = 0;
    int sms = 0;
    int n = 0;
    GridView g{};
    const float* x = nullptr;     /* caller's nodes (kept for radius and the redo path) */
    long long xstride = 0;
    float* xs = nullptr;
    int* id = nullptr;
    int* start = nullptr;
    int* key = nullptr;
    int* count = nullptr;
    int* cursor = nullptr;
    float* mm = nullptr;
    int* redo = nullptr;
    int* nredo = nullptr;          /* [0]: queries the 3^ndof block left, [1]: the 5^ndof block */
    int* redo2 = nullptr;
    size_t cap_xs = 0, cap_id = 0, cap_key = 0, cap_start = 0, cap_count = 0, cap_cursor = 0, cap_redo = 0,
           cap_redo2 = 0;
    std::string err = "no error";
};

namespace {

thread_local std::string g_nbr_create_error = "no error";

int nfail(gprm_nbr* h, int code, const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    if (h) h->err = buf;
    else g_nbr_create_error = buf;
    return code;
}

#define NBR_TRY(h, call)                                                                    \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess)                                                              \
            return nfail((h), e_ == cudaErrorMemoryAllocation ? GPRM_ERR_NOMEM : GPRM_ERR_CUDA, \
                         "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
    } while (0)

template <class T>
int grow(gprm_nbr* h, T** p, size_t& cap, size_t need)
{
    if (need <= cap && *p) return GPRM_OK;
    cudaFree(*p);
    *p = nullptr;
    size_t c = need + need / 4 + 16;
    NBR_TRY(h, cudaMalloc((void**)p, c * sizeof(T)));
    cap = c;
    return GPRM_OK;
}

}  // namespace

extern "C" {

int gprm_nbr_create(int ndof, gprm_nbr** out)
{
    if (!out) return nfail(nullptr, GPRM_ERR_ARG, "null output");
    *out = nullptr;
    if (ndof < 1 || ndof > GPRM_MAX_DOF) return nfail(nullptr, GPRM_ERR_ARG, "ndof %d outside 1..%d", ndof, GPRM_MAX_DOF);
    gprm_nbr* h = new gprm_nbr();
    h->ndof = ndof;
    if (cudaGetDevice(&h->device) != cudaSuccess ||
        cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, h->device) != cudaSuccess) {
        delete h;
        return nfail(nullptr, GPRM_ERR_CUDA, "no CUDA device");
    }
    *out = h;
    return GPRM_OK;
}

void gprm_nbr_destroy(gprm_nbr* h)
{
    if (!h) return;
    cudaSetDevice(h->device);
    cudaDeviceSynchronize();
    cudaFree(h->xs);
    cudaFree(h->id);
    cudaFree(h->start);
    cudaFree(h->key);
    cudaFree(h->count);
    cudaFree(h->cursor);
    cudaFree(h->mm);
    cudaFree(h->redo);
    cudaFree(h->redo2);
    cudaFree(h->nredo);
    delete h;
}

const char* gprm_nbr_last_error(const gprm_nbr* h) { return h ? h->err.c_str() : g_nbr_create_error.c_str(); }

int gprm_nbr_build(gprm_nbr* h, const float* x, int n, int stride, float cell, void* stream)
{
    if (!h) return GPRM_ERR_ARG;
    if (n < 0 || (n > 0 && !x) || stride < n) return nfail(h, GPRM_ERR_ARG, "bad x/n/stride");
    if (!(cell >= 0.0f) || !isfinite(cell)) return nfail(h, GPRM_ERR_ARG, "cell must be finite and >= 0");
    NBR_TRY(h, cudaSetDevice(h->device));
    cudaStream_t st = (cudaStream_t)stream;
    /* every joint is gridded: a query's block of 3^ndof cells then holds
       about 3^ndof x (nodes per cell) candidates, far fewer than a grid over
       some joints whose block spans the others' whole range */
    const int nd = h->ndof, G = nd < NBR_MAX_GRID ? nd : NBR_MAX_GRID;
    h->n = n;
    h->x = x;
    h->xstride = stride;
    GridView& g = h->g;
    g = GridView{};
    g.ndof = nd;
    g.G = G;
    g.n = n;
    int rc;
    if (!h->mm) NBR_TRY(h, cudaMalloc((void**)&h->mm, 2 * GPRM_MAX_DOF * sizeof(float)));
    if (!h->nredo) NBR_TRY(h, cudaMalloc((void**)&h->nredo, 2 * sizeof(int)));
    std::vector<float> mm(2 * nd);
    for (int j = 0; j < nd; ++j) { mm[2 * j] = INFINITY; mm[2 * j + 1] = -INFINITY; }
    NBR_TRY(h, cudaMemcpyAsync(h->mm, mm.data(), 2 * nd * sizeof(float), cudaMemcpyHostToDevice, st));
    if (n > 0) k_minmax<<<h->sms * 4, 256, 0, st>>>(x, n, stride, nd, h->mm);
    NBR_TRY(h, cudaGetLastError());
    NBR_TRY(h, cudaMemcpyAsync(mm.data(), h->mm, 2 * nd * sizeof(float), cudaMemcpyDeviceToHost, st));
    NBR_TRY(h, cudaStreamSynchronize(st));
    /* cell size: given, or about the distance of the 16th neighbour of
       uniformly spread nodes (full-dimensional estimate) */
    double vol = 1.0;
    for (int j = 0; j < nd; ++j) {
        double e = (n > 0 && mm[2 * j + 1] > mm[2 * j]) ? (double)mm[2 * j + 1] - mm[2 * j] : 1e-3;
        vol *= e;
    }
    double c = cell;
    if (!(c > 0.0)) {
        const double unit = pow(M_PI, nd / 2.0) / tgamma(nd / 2.0 + 1.0);
        c = KNN_CELL * pow(16.0 * vol / ((n > 0 ? n : 1) * unit), 1.0 / nd);
    }
    /* the whole range in cells of that size, coarsened until the grid fits
       (at most 1024 cells in a joint and the nodes beyond in the last one:
       91 % of 200,000 1-D nodes, 72 ms for their neighbours, 0.1 ms so) */
    double cells, most;
    for (;; c *= 1.25) {
        cells = most = 1.0;
        for (int d = 0; d < G; ++d) {
            const double e = (n > 0 && mm[2 * d + 1] > mm[2 * d]) ? (double)mm[2 * d + 1] - mm[2 * d] : 0.0;
            const double k = fmin(fmax(ceil(e / c), 1.0), NBR_MAX_CELLS);
            g.nc[d] = (int)k;
            g.lo[d] = n > 0 ? mm[2 * d] : 0.0f;
            cells *= k;
            most = fmax(most, k);
        }
        if (cells <= NBR_MAX_CELLS && most <= NBR_MAX_JOINT_CELLS) break;
    }
    const long long ncells = (long long)cells;
    g.cell = (float)c;
    g.inv_cell = (float)(1.0 / c);
    /* slack of the exactness test: rounding of the cell assignment and of
       the block faces, relative to the coordinates' magnitude */
    double mag = 0.0;
    for (int d = 0; d < G; ++d) mag = fmax(mag, fabs((double)g.lo[d]) + g.nc[d] * c);
    g.slack = (float)(1e-5 * c + 1e-6 * mag);
    /* buffers only grow, so rebuilding an index allocates nothing */
    if ((rc = grow(h, &h->xs, h->cap_xs, (size_t)n * nd + 1)) != GPRM_OK) return rc;
    if ((rc = grow(h, &h->id, h->cap_id, (size_t)n + 1)) != GPRM_OK) return rc;
    if ((rc = grow(h, &h->key, h->cap_key, (size_t)n + 1)) != GPRM_OK) return rc;
    if ((rc = grow(h, &h->start, h->cap_start, (size_t)ncells + 1)) != GPRM_OK) return rc;
    if ((rc = grow(h, &h->count, h->cap_count, (size_t)ncells)) != GPRM_OK) return rc;
    if ((rc = grow(h, &h->cursor, h->cap_cursor, (size_t)ncells)) != GPRM_OK) return rc;
    NBR_TRY(h, cudaMemsetAsync(h->count, 0, (size_t)ncells * sizeof(int), st));
    NBR_TRY(h, cudaMemsetAsync(h->cursor, 0, (size_t)ncells * sizeof(int), st));
    if (n > 0) k_cell_keys<<<h->sms * 8, 256, 0, st>>>(x, n, stride, g, h->key, h->count);
    k_scan<<<1, 1024, 0, st>>>(h->count, (int)ncells, h->start);
    if (n > 0) k_scatter<<<h->sms * 8, 256, 0, st>>>(x, n, stride, nd, h->key, h->start, h->cursor, h->xs, h->id);
    NBR_TRY(h, cudaGetLastError());
    g.xs = h->xs;
    g.id = h->id;
    g.start = h->start;
    return GPRM_OK;
}

int gprm_nbr_radius(gprm_nbr* h, const float* q, int m, int qstride, float D, int cap, int* counts, int* idx,
                    float* dist, void* stream)
{
    if (!h) return GPRM_ERR_ARG;
    if (m < 0 || (m > 0 && (!q || !counts || !idx || !dist)) || qstride < m || cap < 1)
        return nfail(h, GPRM_ERR_ARG, "bad q/m/qstride/cap/outputs");
    if (!(D >= 0.0f) || !isfinite(D)) return nfail(h, GPRM_ERR_ARG, "D must be finite and >= 0");
    if (m == 0) return GPRM_OK;
    NBR_TRY(h, cudaSetDevice(h->device));
    const float D2 = D * D;   /* D2 = D*D in float, prmsolver.cpp:71 */
    k_radius<<<h->sms * 8, 256, 0, (cudaStream_t)stream>>>(h->x, h->n, h->xstride, q, m, qstride, h->ndof, D2, cap,
                                                           counts, idx, dist);
    NBR_TRY(h, cudaGetLastError());
    return GPRM_OK;
}

int gprm_nbr_knn(gprm_nbr* h, const float* q, int m, int qstride, int k, int queries_are_nodes, int* idx,
                 float* dist, void* stream)
{
    if (!h) return GPRM_ERR_ARG;
    if (k < 1 || k > NBR_MAX_K) return nfail(h, GPRM_ERR_ARG, "k=%d outside 1..%d", k, NBR_MAX_K);
    if (queries_are_nodes) {
        q = h->x;
        m = h->n;
        qstride = (int)h->xstride;
    }
    if (m < 0 || (m > 0 && (!q || !idx || !dist)) || qstride < m) return nfail(h, GPRM_ERR_ARG, "bad q/m/qstride/outputs");
    if (m == 0) return GPRM_OK;
    NBR_TRY(h, cudaSetDevice(h->device));
    cudaStream_t st = (cudaStream_t)stream;
    int rc = grow(h, &h->redo, h->cap_redo, (size_t)m);
    if (rc) return rc;
    if ((rc = grow(h, &h->redo2, h->cap_redo2, (size_t)m))) return rc;
    NBR_TRY(h, cudaMemsetAsync(h->nredo, 0, 2 * sizeof(int), st));
    if (queries_are_nodes) {
        const int blocks = (int)std::min<long long>(((long long)m + 7) / 8, (long long)h->sms * 16);
        const int tblocks = (int)(((long long)m + 127) / 128);
        const bool by_thread = h->ndof <= KNN_THREAD_DIM && k <= KNN_THREAD_K && m >= KNN_THREAD_NODES;
        switch (by_thread ? -h->ndof : h->ndof) {
#define GPRM_KNN_THREAD(D)                                                                                    \
        case -D: k_knn_grid_thread<D><<<tblocks, 128, 0, st>>>(h->g, m, k, idx, dist, h->redo, h->nredo); break
        GPRM_KNN_THREAD(1); GPRM_KNN_THREAD(2); GPRM_KNN_THREAD(3);
#undef GPRM_KNN_THREAD
#define GPRM_KNN_GRID(D)                                                                             \
        case D: k_knn_grid<D><<<blocks, 256, 0, st>>>(h->g, m, k, idx, dist, h->redo, h->nredo); break
        GPRM_KNN_GRID(1); GPRM_KNN_GRID(2); GPRM_KNN_GRID(3); GPRM_KNN_GRID(4);
        GPRM_KNN_GRID(5); GPRM_KNN_GRID(6); GPRM_KNN_GRID(7);
#undef GPRM_KNN_GRID
        }
    } else {
        const int wpb = 8;
        const long long wblocks = ((long long)m + wpb - 1) / wpb;
        const int blocks = (int)(wblocks < (long long)h->sms * 16 ? wblocks : (long long)h->sms * 16);
        k_knn_grid_warp<<<blocks, 32 * wpb, 0, st>>>(h->g, q, m, qstride, k, idx, dist, h->redo, h->nredo);
    }
    NBR_TRY(h, cudaGetLastError());
    switch (h->ndof) {
#define GPRM_KNN_WIDE(D)                                                                                           \
    case D: k_knn_wide<D><<<h->sms * 8, 256, 0, st>>>(h->g, q, qstride, k, queries_are_nodes ? 1 : 0, h->redo, h->nredo, \
                                                      h->redo2, h->nredo + 1, idx, dist); break
        GPRM_KNN_WIDE(1); GPRM_KNN_WIDE(2); GPRM_KNN_WIDE(3); GPRM_KNN_WIDE(4);
        GPRM_KNN_WIDE(5); GPRM_KNN_WIDE(6); GPRM_KNN_WIDE(7);
#undef GPRM_KNN_WIDE
    }
    NBR_TRY(h, cudaGetLastError());
    k_knn_full<<<h->sms * 8, 256, 0, st>>>(h->x, h->n, h->xstride, q, qstride, h->ndof, k, queries_are_nodes ? 1 : 0,
                                           h->redo2, h->nredo + 1, idx, dist);
    NBR_TRY(h, cudaGetLastError());
    return GPRM_OK;
}

int gprm_nbr_redo_count(gprm_nbr* h, int* out)
{
    if (!h || !out) return GPRM_ERR_ARG;
    NBR_TRY(h, cudaSetDevice(h->device));
    NBR_TRY(h, cudaMemcpy(out, h->nredo, sizeof(int), cudaMemcpyDeviceToHost));
    return GPRM_OK;
}

}  /* extern "C" */
