/*
 * gprm_kernels.cu - sm_100a kernels of the collision checker.
 *
 * Replaces kernel_indicator2 / kernel_indicator2_1 and set_kernel
 * (prm/src/lib/robotspace/robotconfigspace.cpp:362-595) and the host loop
 * over indicator(q) (robotconfigspace.cpp:313-346, prmsolver.cpp:2611).
 *
 * Work mapping (persistent grid, warps take work from a device counter):
 *   vertex checks  a warp takes 32 configurations: FK a lane each, then one
 *                  configuration after the other swept with a lane per pair
 *                  (on short pair lists each by its lane),
 *                  and the pairs left tested 32 at a time whoever they belong
 *                  to, applied per configuration in pair order.
 *   edge checks    a warp takes one edge; its lanes hold 32 steps of that
 *                  edge (coarse-to-fine: round r, lane i -> step i*R + r with
 *                  R = ceil(testnum/32); or descending steps when every step's
 *                  code is wanted).  A sweep stage settles most pairs for all
 *                  lanes at once, the lanes step through the rest together,
 *                  and one warp vote after each exact test ends the edge at
 *                  its first colliding step.
 *   small requests a block of four warps per configuration or edge, its FP64
 *                  checks included, in one launch.
 * The scene (vertices with packed adjacency, neighbour bytes, pair table)
 * can be copied into shared memory per block where it fits.
 *
 * FP64 band: a check whose FP32 result is decided within the band (or by
 * the iteration cap) is appended to a queue; k_recheck recomputes it in
 * FP64, a thread or a warp per item, and its verdict replaces the FP32 one.
 *
 * Times in the comments are of one B200; two of them compare only within a
 * comment, since the scenes' seeds differ between comments.
 */
#include "gprm_internal.h"

#include <math.h>
#include <mutex>
#include <unordered_map>

namespace gprm {

#define FULL_MASK 0xffffffffu

/* minimum resident blocks of 128 threads the FP32 kernels are compiled for
 * (caps registers per thread; 0 = no cap) */
#ifndef GPRM_MIN_BLOCKS
#define GPRM_MIN_BLOCKS 0
#endif
#if GPRM_MIN_BLOCKS > 0
#define GPRM_BOUNDS __launch_bounds__(128, GPRM_MIN_BLOCKS)
#else
#define GPRM_BOUNDS __launch_bounds__(512)
#endif

size_t scene_smem_bytes(const DevScene& sc)
{
    /* tab | pairs | far | scan_c | scan_b */
    return (size_t)sc.ntab * 16 + (size_t)sc.npairs * 64;
}

size_t frame_smem_bytes(const DevScene& sc, int threads, bool vertex_kernel)
{
    return (size_t)(threads / 32) * lane_floats(sc, vertex_kernel) * 32 * sizeof(float);
}

struct SceneView {
    const float4* tab;
    const int4* pairs;
    const float4* far;
    const int4* scan_c;
    const float4* scan_b;
    float* frames;   /* this lane's frames (lane-interleaved, stride 32) */
    float4* sweep;   /* the warp's per-slot sweep balls */
    unsigned* bits;  /* the pairs of the sweep group left open (one bit each) */
};

/* The warp's sweep area: after the frames in a vertex kernel
 * (the start of its VertexArea), the last SWEEP_LANE_FLOATS entries of the
 * block in an edge kernel. */
template <bool VERTEX>
__device__ __forceinline__ float4* sweep_area(const DevScene& sc, float* lane_frames)
{
    const int lane = threadIdx.x & 31;
    const size_t at = VERTEX ? (size_t)sc.ndof * 12 : lane_floats(sc, false) - SWEEP_LANE_FLOATS;
    return reinterpret_cast<float4*>(lane_frames - lane + at * 32);
}

/* The open bits of the warp's sweep stage: before the sweep area in an edge
 * kernel, after the VertexArea in a vertex kernel. */
template <bool VERTEX>
__device__ __forceinline__ unsigned* open_area(const DevScene& sc, float* lane_frames)
{
    const int lane = threadIdx.x & 31;
    const size_t at = (size_t)sc.ndof * 12 + (VERTEX ? (size_t)VERTEX_LANE_FLOATS : 0);
    return reinterpret_cast<unsigned*>(lane_frames - lane + at * 32);
}

/* Copies the scene into shared memory (SMEM) and returns the pointers the
 * warp uses, including its lane's slice of the frame array (laid out for
 * the vertex or the edge kernels, VERTEX). */
template <bool SMEM, bool VERTEX>
__device__ __forceinline__ SceneView stage_scene(const DevScene& sc, unsigned char* smem)
{
    SceneView s;
    size_t off = 0;
    if (SMEM) {
        const size_t np = (size_t)sc.npairs;
        float4* t = reinterpret_cast<float4*>(smem);
        int4* p = reinterpret_cast<int4*>(smem + (size_t)sc.ntab * 16);
        float4* fr = reinterpret_cast<float4*>(smem + (size_t)sc.ntab * 16 + np * 16);
        int4* scc = reinterpret_cast<int4*>(smem + (size_t)sc.ntab * 16 + np * 32);
        float4* scb = reinterpret_cast<float4*>(smem + (size_t)sc.ntab * 16 + np * 48);
        for (int i = threadIdx.x; i < sc.ntab; i += blockDim.x) t[i] = sc.tab[i];
        for (int i = threadIdx.x; i < sc.npairs; i += blockDim.x) {
            p[i] = sc.pairs[i];
            fr[i] = sc.far[i];
            scc[i] = sc.scan_c[i];
            scb[i] = sc.scan_b[i];
        }
        s.tab = t;
        s.pairs = p;
        s.far = fr;
        s.scan_c = scc;
        s.scan_b = scb;
        off = (size_t)sc.ntab * 16 + np * 64;
    } else {
        s.tab = sc.tab;
        s.pairs = sc.pairs;
        s.far = sc.far;
        s.scan_c = sc.scan_c;
        s.scan_b = sc.scan_b;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    s.frames = reinterpret_cast<float*>(smem + off) + (size_t)warp * lane_floats(sc, VERTEX) * 32 + lane;
    s.sweep = sweep_area<VERTEX>(sc, s.frames);
    s.bits = open_area<VERTEX>(sc, s.frames);
    __syncthreads();
    return s;
}

/* Slots whose vertex 0 has a sweep ball too (the swept direction test). */
constexpr int SWEEP_V0_SLOTS = GPRM_MAX_SLOTS / 2;

/* Warp-wide minimum and maximum, NaN if any lane's value is. */
__device__ __forceinline__ float warp_min_nan(float a)
{
    float d;
    asm volatile("redux.sync.min.NaN.f32 %0, %1, 0xffffffff;" : "=f"(d) : "f"(a));
    return d;
}
__device__ __forceinline__ float warp_max_nan(float a)
{
    float d;
    asm volatile("redux.sync.max.NaN.f32 %0, %1, 0xffffffff;" : "=f"(d) : "f"(a));
    return d;
}

/* One sweep ball: PATH: centre at lane mid's point, else the midpoint of the
 * lanes' bounding box, radius over the lanes' points.  Lane p keeps the
 * squared radius as bits (NaN, which is larger than any number's bits, if a
 * point is not finite). */
template <bool PATH>
__device__ __forceinline__ void sweep_ball(float4* sweep, int mid, int p, const float* u, unsigned& r2)
{
    const int lane = threadIdx.x & 31;
    float m[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
        m[c] = PATH ? __shfl_sync(FULL_MASK, u[c], mid) : 0.5f * (warp_min_nan(u[c]) + warp_max_nan(u[c]));
    const float dx = u[0] - m[0], dy = u[1] - m[1], dz = u[2] - m[2];
    const unsigned r = __reduce_max_sync(FULL_MASK, __float_as_uint(__fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz))));
    if (lane == p) {
        r2 = r;
        sweep[p] = make_float4(m[0], m[1], m[2], 0.0f);
    }
}

/* Counts of how pair tests were settled: by a certificate (a lane's own
 * and, in lane 0, those settled for the whole warp), by the exact test. */
struct PairCounts {
    unsigned long long cert, full;
};

/* The MUFU's reciprocal square root and reciprocal, denormals as zero (no
 * scaling around them). */
__device__ __forceinline__ float rsqrt_fast(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_fast(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

/* The direction test of points_certified for every lane of the warp at
 * once.  Each polytope's ball centre lies in a ball over the lanes, and so
 * does its vertex 0 (the slot's sweep balls; radius 0 for a polytope of
 * frame 0): s = the difference of the vertex-0 ball centres, D = that of
 * the centres' (both from the same polytope to the other; the sign cancels
 * in <s, D>), rv and rc the sums of the two radii.  Every lane's s' = s -
 * alpha, |alpha| <= rv, and D' = D - gamma, |gamma| <= rc, have
 *     <s', D'> >= <s, D> - |s| rc - rv |D| - rv rc = N
 *     |s'| in [|s| - rv, |s| + rv],  |D'| <= |D| + rc,
 * so when N > 0, the G - err of the per-lane test is at least
 *     N / (|s| + rv) - R - (|D| + rc + R)(eps_dir / (|s| - rv) + 1e-6),
 * which must exceed thr_dir (with 1e-5 relative allowances for the
 * rounding of this bound, which cover the approximate root and quotient:
 * a settled pair is one that every lane's own test would certify). */
__device__ __forceinline__ bool swept_direction(float eps_dir, float thr_dir, float sx, float sy, float sz, float rv,
                                                float dx, float dy, float dz, float rc, float R)
{
    const float n2 = __fmaf_rn(sx, sx, __fmaf_rn(sy, sy, sz * sz));
    const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
    const float sn = n2 * rsqrt_fast(n2), dn = d2 * rsqrt_fast(d2);   /* NaN for 0: not settled */
    const float N = __fmaf_rn(sx, dx, __fmaf_rn(sy, dy, sz * dz)) * (1.0f - 1e-5f) -
                    __fmaf_rn(sn, rc, __fmaf_rn(rv, dn, rv * rc)) * (1.0f + 1e-5f);
    const float slo = sn * (1.0f - 1e-5f) - rv * (1.0f + 1e-5f), sup = (sn + rv) * (1.0f + 1e-5f);
    const float err = (dn + rc + R) * __fmaf_rn(eps_dir, rcp_fast(slo), 1e-6f) * (1.0f + 2e-5f);
    return N > 0.0f && slo > 1e-3f && N * (1.0f - 1e-5f) > sup * (__fmaf_rn(R, 1.0f + 1e-5f, err) + thr_dir);
}

/* Distance test of a sweep record against the warp's sweep balls: false
 * when the balls are farther apart in every lane than rc (the radii) +
 * root, with D from the moving slot's ball to the other's. */
__device__ __forceinline__ bool swept_near(float4 o, float4 m, float root, float& dx, float& dy, float& dz, float& rc)
{
    dx = o.x - m.x; dy = o.y - m.y; dz = o.z - m.z;
    rc = o.w + m.w;
    const float dd2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
    const float A = (root + rc) * (1.0f + 1e-6f);
    /* |m - o|^2 >= dd2 (1 - 1e-6) > A^2 settles; NaN does not */
    return !(dd2 * (1.0f - 1e-6f) > A * A);
}

/* A sweep entry (r: swp, v: swb) against the warp's sweep balls: true when
 * neither the distance nor the direction settles its pair for every lane.
 * Branch-free, so that two entries go side by side.  POINT: the balls have
 * radius 0 (one configuration), and the direction test is that of
 * lane_certified with a margin for the approximate roots. */
template <bool POINT>
__device__ __forceinline__ bool swept_open(const float4* sweep, const float4* v0, bool dir_on, float eps_dir,
                                           float thr_dir, float4 r, float4 v)
{
    const int w = __float_as_int(r.w);
    const int a = w & 15, b = (w >> 4) & 15;   /* a: a moving polytope's slot; b != a: the other's */
    float4 o = make_float4(r.x, r.y, r.z, 0.0f), u = make_float4(v.x, v.y, v.z, 0.0f);
    if (b != a) { o = sweep[b]; u = v0[b]; }
    const float root = __int_as_float(w | 255);   /* the slot bits round it up */
    const float4 m = v0[a];
    if constexpr (POINT) {
        const float4 c = sweep[a];
        const float dx = o.x - c.x, dy = o.y - c.y, dz = o.z - c.z;
        const float sx = u.x - m.x, sy = u.y - m.y, sz = u.z - m.z;
        const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
        const float n2 = __fmaf_rn(sx, sx, __fmaf_rn(sy, sy, sz * sz));
        const float inv = rsqrt_fast(n2);
        const float G = __fmaf_rn(sx, dx, __fmaf_rn(sy, dy, sz * dz)) * inv;
        const float err = __fmaf_rn(d2, rsqrt_fast(d2), v.w) * __fmaf_rn(eps_dir, inv, 1e-6f);
        const bool settled = d2 * (1.0f - 2e-6f) > root * root ||
                             (n2 > 1.00001e-6f && G * (1.0f - 1e-5f) > __fmaf_rn(v.w + err, 1.0f + 2e-5f, thr_dir));
        return !settled && !(root < 0.0f);
    } else {
        float dx, dy, dz, rc;
        const bool near = swept_near(o, sweep[a], root, dx, dy, dz, rc);
        const bool settled = dir_on && swept_direction(eps_dir, thr_dir, u.x - m.x, u.y - m.y, u.z - m.z, u.w + m.w, dx,
                                                       dy, dz, rc, v.w);
        return near && !settled && !(root < 0.0f);
    }
}

__device__ __forceinline__ void sweep_mark(const int* swj, unsigned* bits, int g, int i, bool open)
{
    if (open) {
        const int j = swj[i] - g * SWEEP_GROUP;
        atomicOr(&bits[j >> 5], 1u << (j & 31));
    }
}

/* The sweep stage of an edge round for the pairs of group g, against the
 * warp's sweep balls: a pair whose ball centres are farther apart in every
 * lane than rho_P + rho_Q + sqrt(T2) is settled for all lanes at once (each
 * lane's exact distance then exceeds sqrt(T2)); else the direction test is
 * bounded over all lanes at once (swept_direction).  Sets in S.bits the
 * bits of the pairs left for the lanes' own tests (bit j - g *
 * SWEEP_GROUP); share: the leaves of every 32 that this warp goes through;
 * POINT: see swept_open; dir_on, v0_at: whether, and from where, the sweep area holds balls of the
 * slots' vertex 0.
 *
 * Two levels: lane l tests leaf l of the next 32 (32 pairs of one slot whose
 * static partners lie close together) by its ball, then the warp goes
 * through the leaves left, a lane per pair, two leaves side by side without
 * branches (this stage waits on its loads: 3 % slower one leaf at a time
 * with the next one's records loaded ahead, 7 % with swb read only where
 * the distance leaves a pair open).  In pair order, with every pair of the
 * list tested, it took 108,000 of 151,000 cycles of a round on the 7-DOF
 * wall scene (129 chunks of 32 pairs; 70,001 edges 27.7 -> 15.9 ms with the
 * leaves); on 64 obstacles (two leaves a slot) the leaf level costs what it
 * saves (62.1 -> 61.7 ms). */
template <bool POINT>
__device__ __forceinline__ void sweep_leaves(const DevScene& sc, const SceneView& S, int g, unsigned share, bool dir_on,
                                             int v0_at)
{
    const int lane = threadIdx.x & 31;
    /* the descriptor's fields in registers: a batch keeps it in shared
       memory, where the bits are set */
    const float eps_dir = sc.eps_dir, thr_dir = sc.thr_dir;
    const float4 *swl = sc.swl, *swp = sc.swp, *swb = sc.swb, *sweep = S.sweep, *v0 = S.sweep + (dir_on ? v0_at : 0);
    const int* swj = sc.swj;
    unsigned* bits = S.bits;
    const int end = sc.swg[g + 1];
#pragma unroll 1
    for (int l0 = sc.swg[g]; l0 < end; l0 += 32) {
        bool open = false;
        if (l0 + lane < end) {
            const float4 r = swl[l0 + lane];
            const int w = __float_as_int(r.w);
            float dx, dy, dz, rc;
            open = swept_near(make_float4(r.x, r.y, r.z, 0.0f), sweep[w & 15], __int_as_float(w | 15), dx, dy, dz,
                              rc);
        }
        unsigned left = __ballot_sync(FULL_MASK, open) & share;
        if (!left) continue;
        /* two leaves side by side (the last one with itself: the bits are
           only ever set) */
        int ia = (l0 + __ffs(left) - 1) * 32 + lane;
        left &= left - 1u;
        int ib = left ? (l0 + __ffs(left) - 1) * 32 + lane : ia;
        left &= left - 1u;
#pragma unroll 1
        for (;;) {
            const float4 ra = swp[ia], va = swb[ia], rb = swp[ib], vb = swb[ib];
            const bool oa = swept_open<POINT>(sweep, v0, dir_on, eps_dir, thr_dir, ra, va);
            const bool ob = swept_open<POINT>(sweep, v0, dir_on, eps_dir, thr_dir, rb, vb);
            sweep_mark(swj, bits, g, ia, oa);
            sweep_mark(swj, bits, g, ib, ob);
            if (!left) break;
            ia = (l0 + __ffs(left) - 1) * 32 + lane;
            left &= left - 1u;
            ib = left ? (l0 + __ffs(left) - 1) * 32 + lane : ia;
            left &= left - 1u;
        }
    }
}

__device__ __forceinline__ void sweep_stage(const DevScene& sc, const SceneView& S, int g, int words)
{
    for (int w = threadIdx.x & 31; w < words; w += 32) S.bits[w] = 0u;
    __syncwarp();
    sweep_leaves<false>(sc, S, g, FULL_MASK, sc.nslots <= SWEEP_V0_SLOTS, SWEEP_V0_SLOTS);
    __syncwarp();
}

/* The certificates of a pair for one configuration, given the world ball
 * centres p, q and vertices 0 a, b of its polytopes (T2, R: of the pair; c:
 * its scan_c; frames: the configuration's): the ball-distance and direction
 * tests without a branch between them, then, where both miss, the box
 * test. */
__device__ __forceinline__ bool points_certified(const DevScene& sc, const float* frames, int4 c, float T2, float R,
                                                 V3<float> p, V3<float> q, V3<float> a, V3<float> b)
{
    const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
    const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
    float sx = b.x - a.x, sy = b.y - a.y, sz = b.z - a.z;
    const float n2 = __fmaf_rn(sx, sx, __fmaf_rn(sy, sy, sz * sz));
    const float inv = rsqrtf(n2);
    const float G = __fmaf_rn(sx, dx, __fmaf_rn(sy, dy, sz * dz)) * inv - R;
    /* |D| from above: d2 * rsqrt(d2) is within 3 ulp of |D| (rsqrtf <= 2
       ulp), the factor covers it; d2 = 0 gives NaN, which fails the tests */
    const float dn = d2 * rsqrtf(d2) * (1.0f + 2e-6f);
    /* direction error <= eps_dir*inv (+ rsqrt and rounding, 1e-6) */
    const float err = (dn + R) * __fmaf_rn(sc.eps_dir, inv, 1e-6f);
    const bool dir = n2 > 1e-6f;   /* |s| < 1e-3: leave it to the test */
    if (d2 > T2 || (dir && G - err > sc.thr_dir)) return true;
    if (!dir) return false;
    sx = sx * inv; sy = sy * inv; sz = sz * inv;
    const float hp = box_support(sc.box + 3 * c.y, frames, SCAN_SYS_P(c.x), sx, sy, sz);
    const float hq = box_support(sc.box + 3 * c.z, frames, SCAN_SYS_Q(c.x), sx, sy, sz);
    const float Gb = __fmaf_rn(sx, dx, __fmaf_rn(sy, dy, sz * dz)) - (hp + hq) * (1.0f + 1e-5f);
    return Gb - err > sc.thr_dir;
}

/* Point x of frame f (1..ndof) of a configuration, with the FMA chain of the
 * slot points. */
__device__ __forceinline__ V3<float> frame_point(const float* frames, int f, float4 x)
{
    const float* T = frames + (f - 1) * 12 * 32;
    V3<float> o;
    o.x = __fmaf_rn(T[0], x.x, __fmaf_rn(T[3 * 32], x.y, __fmaf_rn(T[6 * 32], x.z, T[9 * 32])));
    o.y = __fmaf_rn(T[32], x.x, __fmaf_rn(T[4 * 32], x.y, __fmaf_rn(T[7 * 32], x.z, T[10 * 32])));
    o.z = __fmaf_rn(T[2 * 32], x.x, __fmaf_rn(T[5 * 32], x.y, __fmaf_rn(T[8 * 32], x.z, T[11 * 32])));
    return o;
}

/* World ball centre and vertex 0 of a slot's polytope (in frame f) for this
 * lane, as the FK pass had them. */
__device__ __forceinline__ void slot_points(const DevScene& sc, const SceneView& S, int slot, int f, V3<float>& p,
                                            V3<float>& a)
{
    const float4* blk = S.tab + sc.slot_block[slot];
    const float4 x = blk[0], v = blk[1];
    p = frame_point(S.frames, f, x);
    a = frame_point(S.frames, f, v);
}

/* points_certified for the lane whose frames S holds: the moving polytopes'
 * points from their frames (slot_points), a static one's from the records f
 * and b.  A pair that is not SCAN_USABLE is never
 * certified here (no slot, or two static polytopes whose certificate failed
 * when the tables were uploaded). */
__device__ __forceinline__ bool lane_certified(const DevScene& sc, const SceneView& S, int4 c, float4 f, float4 b)
{
    if (c.w != SCAN_USABLE) return false;
    V3<float> P = {f.x, f.y, f.z}, Q = P, A = {b.x, b.y, b.z}, B = A;
    const int sp = SCAN_SLOT_P(c.x), sq = SCAN_SLOT_Q(c.x);
    if (sp >= 0) slot_points(sc, S, sp, SCAN_SYS_P(c.x), P, A);
    if (sq >= 0) slot_points(sc, S, sq, SCAN_SYS_Q(c.x), Q, B);
    return points_certified(sc, S.frames, c, f.w, b.w, P, Q, A, B);
}

/* points_certified of pair j from the frames alone (a vertex check keeps no
 * slot points). */
__device__ __forceinline__ bool frames_certified(const DevScene& sc, const SceneView& S, const float* frames, int j)
{
    const int4 c = S.scan_c[j];
    if (c.w != SCAN_USABLE) return false;
    const int4 pr = S.pairs[j];
    const float4 p = S.tab[pr.x], a = S.tab[pr.x + 1], q = S.tab[pr.y], b = S.tab[pr.y + 1];
    V3<float> P = {p.x, p.y, p.z}, A = {a.x, a.y, a.z}, Q = {q.x, q.y, q.z}, B = {b.x, b.y, b.z};
    if (pr.z) { P = frame_point(frames, pr.z, p); A = frame_point(frames, pr.z, a); }
    if (pr.w) { Q = frame_point(frames, pr.w, q); B = frame_point(frames, pr.w, b); }
    return points_certified(sc, frames, c, S.far[j].w, S.scan_b[j].w, P, Q, A, B);
}

/* This lane's certificates of the pairs j0 + k, k in cand (warp-uniform),
 * all order-free (a certified pair is free with its margin above the band,
 * so it changes neither a code nor a band decision).  Returns the pairs that
 * need the exact test (bit k).
 *
 * One copy of the code and the next pair's records loaded ahead, rather than
 * two pairs side by side with every case inlined for each: the edge kernel
 * waited on instruction fetches more than on anything else (2.6 of 9.5 warp
 * cycles per instruction; 2.5 M roadmap edges 86.7 -> 64.3 ms). */
__device__ __forceinline__ unsigned lane_scan(const DevScene& sc, const SceneView& S, int j0, unsigned cand,
                                              PairCounts& pc)
{
    if (!cand) return 0u;
    const unsigned all = cand;
    unsigned need = 0;
    int k = __ffs(cand) - 1;
    int4 c = S.scan_c[j0 + k];
    float4 f = S.far[j0 + k], b = S.scan_b[j0 + k];
#pragma unroll 1
    for (;;) {
        cand &= cand - 1u;
        const int kn = cand ? __ffs(cand) - 1 : k;
        const int4 cn = S.scan_c[j0 + kn];
        const float4 fn = S.far[j0 + kn], bn = S.scan_b[j0 + kn];
        if (!lane_certified(sc, S, c, f, b)) need |= 1u << k;
        if (!cand) break;
        k = kn; c = cn; f = fn; b = bn;
    }
    pc.cert += (unsigned)__popc(all & ~need);
    return need;
}

/* The exact test of pair j for this lane (its certificates failed): the pair's code, and its margin in *margin. */
template <bool FAST>
__device__ __forceinline__ int eval_pair(const DevScene& sc, const SceneView& S, int j, float* margin,
                                         PairCounts& pc);

/* The frames of a pair, from the lane's frame array (frame 0 is unused). */
__device__ __forceinline__ void pair_frames(const float* fr, int4 pr, Frame<float>& tp, Frame<float>& tq)
{
    if (pr.z) load_frame(fr, pr.z, tp);
    if (pr.w) load_frame(fr, pr.w, tq);
}

template <bool FAST>
__device__ __forceinline__ int eval_pair(const DevScene& sc, const SceneView& S, int j, float* margin,
                                         PairCounts& pc)
{
    const int4 pr = S.pairs[j];
    ++pc.full;
    Frame<float> tp, tq;
    pair_frames(S.frames, pr, tp, tq);
    if constexpr (FAST) return pair_test_fast(sc, S.tab, pr, sc.ppoly[j], tp, tq, margin);
    else return pair_test<PF32>(sc, S.tab, pr, tp, tq, margin);
}

/* Forward kinematics of a lane into its shared-memory frames, in the
 * arithmetic of the kernel variant, and (SLOTS) the warp's sweep balls:
 * sweep[slot] holds the slot's ball centre in every lane; with at most
 * SWEEP_V0_SLOTS slots, sweep[SWEEP_V0_SLOTS + slot] the slots' vertex 0,
 * for the swept direction test.  PATH: centred at lane mid's points (of an
 * edge's round the middle step: its steps lie on a path); else at the
 * middle of the points' bounding box (configurations that lie anywhere:
 * 4,096 of wall7 620 us with a configuration as the centre, 597 so; 543 when
 * the points were kept in shared memory, which the edges paid for).  Radius
 * the largest distance from there, rounded up; a non-finite point makes it
 * infinite, which disables the sweep tests for the slot.
 *
 * Nothing else of the points is kept: lane_scan takes them from the frames
 * again.  With 6 floats a slot and lane in shared memory (and the balls
 * from the rows' extremes) the 6-joint edge kernel left 28 KB to L1 and one
 * of 7 joints ran 13 warps an SM; now 92 KB and 16 warps (2.5 M hull6 edges
 * 59.9 -> 57.3 ms, 70,001 wall edges 13.6 -> 12.3, a mixed batch 26.8 -> 22.7;
 * the exact arithmetic on hull6 16.9 -> 17.4).  The extremes by
 * warp reductions instead (6 a point) took 1,900 cycles of a round more. */
template <bool FAST, bool SLOTS = true, bool PATH = true, class Joint>
__device__ __forceinline__ void lane_fk(const DevScene& sc, const SceneView& S, Joint joint, int mid = 0)
{
    const bool v0 = sc.nslots <= SWEEP_V0_SLOTS;
    unsigned r2 = 0u;
    forward_kinematics_smem<FAST, SLOTS>(sc, S.tab, joint, S.frames, [&](int slot, const float* u, const float* w) {
        sweep_ball<PATH>(S.sweep, mid, slot, u, r2);
        if (v0) sweep_ball<PATH>(S.sweep, mid, SWEEP_V0_SLOTS + slot, w, r2);
    });
    if constexpr (SLOTS) {
        __syncwarp();
        const int lane = threadIdx.x & 31;
        if (lane < GPRM_MAX_SLOTS) {
            const float rho = __fsqrt_ru(__uint_as_float(r2)) * (1.0f + 5e-6f) + 1e-30f;
            S.sweep[lane].w = rho < PF32::inf() ? rho : PF32::inf();
        }
        __syncwarp();
    }
}

__device__ __forceinline__ void flush_counts(PairCounts pc, Control* ctl)
{
    for (int o = 16; o > 0; o >>= 1) {
        pc.cert += __shfl_xor_sync(0xffffffffu, pc.cert, o);
        pc.full += __shfl_xor_sync(0xffffffffu, pc.full, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (pc.cert) atomicAdd(&ctl->certified, pc.cert);
        if (pc.full) atomicAdd(&ctl->full_tests, pc.full);
    }
}

/* Appends the items of the lanes with `want` set, one atomic per warp;
 * range: the pairs the item's FP64 recheck tests (BandQueue::pair_range). */
__device__ __forceinline__ unsigned recheck_range(int code, int jfirst, int jlast, int npairs)
{
    if (jfirst >= npairs) return (unsigned)npairs << 16;          /* not recorded: every pair */
    const int hi = code != 0 ? npairs : (jlast < npairs ? jlast + 1 : npairs);
    return (unsigned)jfirst | ((unsigned)hi << 16);
}

__device__ __forceinline__ void warp_append(bool want, uint2 item, unsigned range, BandQueue bq,
                                            Control* ctl)
{
    unsigned m = __ballot_sync(FULL_MASK, want);
    if (!m) return;
    int lane = threadIdx.x & 31;
    unsigned base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd(&ctl->qcount, (unsigned)__popc(m));
    base = __shfl_sync(FULL_MASK, base, __ffs(m) - 1);
    if (want) {
        unsigned slot = base + __popc(m & ((1u << lane) - 1));
        if (slot < bq.cap) {
            bq.items[slot] = item;
            if (bq.pair_range) bq.pair_range[slot] = range;
        } else {
            atomicOr(&ctl->flags, GPRM_DEVFLAG_QUEUE_FULL);
            const unsigned x = item.x;
            if (bq.ovf && (long long)x < bq.n) {
                const unsigned bit = 1u << (x & 31u);
                if (!(atomicOr(&bq.ovf[bq.n + (x >> 5)], bit) & bit))
                    bq.ovf[atomicAdd(&ctl->ovf_count, 1ull)] = x;
            }
        }
    }
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long x)
{
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL_MASK, x, o);
    return x;
}

/* ------------------------------------------------------------------ */
/* vertex checks                                                        */
/* ------------------------------------------------------------------ */

/* The warp's shared area of a vertex kernel (VERTEX_LANE_FLOATS per lane):
 * the balls of the configuration in the sweep stage, the queue of (lane |
 * pair << 5) items that it leaves open, per configuration the pairs that
 * need the exact test (count of them; those that found no room start at
 * pair `resume`), the first colliding pair (pair << 5 | code + 1 | 16 if
 * inside the band) and the first and last free one inside the band.  The
 * open bits of the sweep stage follow. */
constexpr int VERTEX_TESTS = 12;
struct VertexArea {
    float4 balls[2 * GPRM_MAX_SLOTS];
    unsigned open[64];
    unsigned test[VERTEX_TESTS][32];
    int count[32];
    unsigned resume[32];
    unsigned jkey[32], jfirst[32];
    int jlast[32];
};
static_assert(sizeof(VertexArea) == VERTEX_LANE_FLOATS * 32 * sizeof(float), "vertex area");
constexpr unsigned JKEY_NONE = 0xffffffffu;
constexpr unsigned PAIR_NONE = 0x7fffffffu;

/* Whether the certificates of a vertex check go a lane per configuration
 * through every pair (lane_list) instead of a configuration after the other
 * with a lane per pair.  The sweep of one configuration costs about 1,000
 * warp instructions however short its leaves are, a pair's certificates for
 * 32 configurations about 60.  400,000 configurations, fast (exact), us a
 * call, sweep against lanes: 67 pairs of the box scene 859/519 (925/612), 91
 * pairs 659/419 (748/529), 131 911/718 (1084/923), 208 1297/1118 (1523/1392),
 * 256 1298/1121 (1464/1307), 340 1741/1634 (2040/1928), 370 1889/1911
 * (2305/2296), 412 2057/2069 (2477/2494); the same order at 40,000. */
constexpr int LANE_LIST_PAIRS = 256;
__device__ __forceinline__ bool lane_lists(const DevScene& sc) { return sc.npairs <= LANE_LIST_PAIRS; }

/* The certificates of this lane's configuration (mine: it takes part) over
 * the pairs from `from` on, in pair order; the pairs that they leave go on
 * its list, those that find no room there wait from the first on. */
__device__ __forceinline__ void lane_list(const DevScene& sc, const SceneView& S, VertexArea& A, bool mine,
                                          unsigned from, PairCounts& pc)
{
    const int lane = threadIdx.x & 31;
    int at = 0;
    unsigned rest = PAIR_NONE;
#pragma unroll 1
    for (int j0 = 0; j0 < sc.npairs; j0 += 32) {
        const unsigned cand = __ballot_sync(FULL_MASK, j0 + lane < sc.npairs && S.scan_c[j0 + lane].w != SCAN_SETTLED);
        if (!mine || rest != PAIR_NONE || from >= (unsigned)j0 + 32u) continue;
        PairCounts settled = {0, 0};                /* the caller counts what is left */
        unsigned need = lane_scan(sc, S, j0, cand, settled);
        if (from > (unsigned)j0) need &= FULL_MASK << (from & 31u);
        for (; need; need &= need - 1u) {
            const unsigned j = (unsigned)(j0 + __ffs(need) - 1);
            if (at == VERTEX_TESTS) {
                rest = j;
                break;
            }
            A.test[at++][lane] = j;
            --pc.cert;
        }
    }
    A.count[lane] = at;
    A.resume[lane] = rest;
    __syncwarp();
}

/* Configurations i0 .. i0+count-1 (count <= 32), one per lane.
 *
 * Lanes hold unrelated configurations, so what one needs another does not.
 * FK runs a lane per configuration; then, but on short pair lists
 * (lane_lists), the configurations go through the
 * sweep stage one after the other, a lane per pair, with balls of radius 0
 * (whole leaves of far obstacles drop out at once); the pairs that leaves
 * open, of whichever configurations, go 32 at a time through their
 * certificates (frames_certified), and what those leave is listed per
 * configuration in pair order.  The exact tests follow in rounds: every
 * configuration without a collision gives its next tests, one while 32 take
 * part, more as fewer do, so that a colliding configuration runs few tests
 * behind the one that decides it (without that, 15 tests a configuration
 * instead of 4 on the wall scene, the larger part of the kernel).  A
 * configuration whose list is full leaves its other pairs to another sweep,
 * which resumes with them; those pairs are not looked at before.  50,000
 * configurations with a NaN joint, whose pairs all stay open, took 15 ms on
 * 5,410 pairs with all their certificates evaluated in every sweep, 2.4 ms
 * with that, 0.7 ms with their sweep left out (usual ones 2.5 ms); 100,003
 * of the wall scene 3.20 -> 2.81 ms.
 * With every pair's certificates evaluated per lane in pair order this
 * kernel took 5.3 ms for 2^20 hull6 configurations and 7.4 ms for 100,003 of
 * the wall scene (exact), nearly all of it in those tests; slot points are
 * not kept, which leaves shared memory for 16 warps per SM. */
template <bool FAST>
__device__ __forceinline__ void check_config_chunk(const DevScene& sc, const SceneView& S, const float* __restrict__ q,
                                                   long long offset, long long i0, int count, int* __restrict__ res,
                                                   int band_on, float band, BandQueue bq,
                                                   Control* ctl, PairCounts& pc, unsigned long long& exec)
{
    const int lane = threadIdx.x & 31;
    VertexArea& A = *reinterpret_cast<VertexArea*>(S.sweep);
    const long long i = i0 + lane;
    const bool valid = lane < count;
    bool active = valid;
    if (valid) {
        /* check_boundaries(q) (robotconfigspace.cpp:795-802) */
#pragma unroll 1
        for (int j = 0; j < sc.ndof; ++j) {
            const float x = q[i + offset * j];
            if (x < sc.mins[j] || x > sc.maxs[j]) active = false;
        }
    }
    bool finite = true;
    if (active) {
        lane_fk<FAST, false>(sc, S, [&](int j) { return q[i + offset * j]; });
        const float* T = S.frames + (sc.ndof - 1) * 12 * 32;
        finite = T[9 * 32] - T[9 * 32] == 0.0f && T[0] - T[0] == 0.0f;
    }
    /* a joint that is no number: no pair can be settled, the sweep is left out */
    const unsigned wild = __ballot_sync(FULL_MASK, !finite);
    /* this lane's sweep ball: slot `lane`'s ball centre, or slot lane - 16's vertex 0 */
    const int slot = lane & (GPRM_MAX_SLOTS - 1);
    float4 point = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int frame = 1;
    if (slot < sc.nslots) {
        point = S.tab[sc.slot_block[slot] + (lane >= GPRM_MAX_SLOTS)];
        frame = sc.slot_sys[slot];
    }
    A.jkey[lane] = JKEY_NONE;
    A.jfirst[lane] = PAIR_NONE;
    A.jlast[lane] = -1;
    unsigned todo = __ballot_sync(FULL_MASK, active);   /* configurations to sweep */
    if (lane == 0) pc.cert += (unsigned long long)sc.npairs * (unsigned)__popc(todo);
    unsigned from = 0u;                                 /* this lane's configuration: from this pair on */
#pragma unroll 1
    while (todo) {
        A.count[lane] = 0;
        A.resume[lane] = PAIR_NONE;
        const bool lanes = lane_lists(sc);
        if (lanes) lane_list(sc, S, A, (todo >> lane) & 1u, from, pc);
        /* the sweep in progress: configuration c, its next group of pairs
           g0, the next word row of the group's open bits, this lane's word */
        int c = 0, g0 = sc.npairs, row = 0, rows = 0, base = 0;
        unsigned word = 0u;
        int n = 0;                                      /* items in the open queue */
        bool more = !lanes;
#pragma unroll 1
        while (more || n > 0) {
            while (n < 32 && more) {
                const unsigned m = __ballot_sync(FULL_MASK, word != 0u);
                if (m) {
                    /* in pair order: the whole row where it fits, else its
                       next word */
                    int at = __popc(word);
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const int y = __shfl_up_sync(FULL_MASK, at, d);
                        if (lane >= d) at += y;
                    }
                    const int total = __shfl_sync(FULL_MASK, at, 31);
                    const bool fits = n + total <= 64;
                    const int l = fits ? 31 : __ffs(m) - 1;         /* words up to lane l */
                    const int pushed = __shfl_sync(FULL_MASK, at, l);
                    if (lane <= l) {
                        at += n - __popc(word);
                        for (; word; word &= word - 1u)
                            A.open[at++] = (unsigned)c | ((unsigned)(base + __ffs(word) - 1) << 5);
                    }
                    n += pushed;
                } else if (row < rows) {
                    const int w = row * 32 + lane;
                    base = g0 - SWEEP_GROUP + w * 32;
                    word = base < min(sc.npairs, g0) ? S.bits[w] : 0u;
                    ++row;
                    /* a resumed configuration: the pairs from there on */
                    const unsigned lo = __shfl_sync(FULL_MASK, from, c);
                    if (lo > (unsigned)base) word = lo >= (unsigned)base + 32u ? 0u : word & (FULL_MASK << (lo & 31u));
                } else if (g0 < sc.npairs) {
                    const int words = (min(sc.npairs - g0, SWEEP_GROUP) + 31) >> 5;
                    const bool sweep = !((wild >> c) & 1u);
                    __syncwarp();
                    for (int w = lane; w < words; w += 32) {
                        const int left = sc.npairs - g0 - 32 * w;
                        S.bits[w] = sweep ? 0u : left >= 32 ? FULL_MASK : (1u << left) - 1u;
                    }
                    __syncwarp();
                    if (sweep) sweep_leaves<true>(sc, S, g0 / SWEEP_GROUP, FULL_MASK, true, GPRM_MAX_SLOTS);
                    __syncwarp();
                    row = 0;
                    rows = (words + 31) >> 5;
                    g0 += SWEEP_GROUP;
                } else if (todo) {
                    c = __ffs(todo) - 1;
                    todo &= todo - 1u;
                    __syncwarp();
                    if (slot < sc.nslots) {
                        const V3<float> w = frame_point(S.frames - lane + c, frame, point);
                        A.balls[lane] = make_float4(w.x, w.y, w.z, 0.0f);
                    }
                    __syncwarp();
                    /* a resumed configuration: from the group of its pair on */
                    g0 = (int)(__shfl_sync(FULL_MASK, from, c) / SWEEP_GROUP) * SWEEP_GROUP;
                    row = rows = 0;
                } else {
                    more = false;
                }
            }
            __syncwarp();
            /* certificates of the first 32 open pairs; those left join their
               configurations' lists in order */
            unsigned own = 32u, j = 0u;
            bool need = false;
            if (lane < n) {
                own = A.open[lane] & 31u;
                j = A.open[lane] >> 5;
                need = !frames_certified(sc, S, S.frames - lane + own, (int)j);
            }
            const unsigned same = __match_any_sync(FULL_MASK, need ? own : 32u);
            if (need) {
                const int at = A.count[own] + __popc(same & ((1u << lane) - 1u));
                if (at < VERTEX_TESTS) {
                    A.test[at][own] = j;
                    --pc.cert;
                } else {
                    atomicMin(&A.resume[own], j);
                }
            }
            __syncwarp();
            if (need && (same >> lane) == 1u)   /* the last of its configuration */
                A.count[own] = min(A.count[own] + __popc(same), VERTEX_TESTS);
            const int left = n > 32 ? n - 32 : 0;       /* at most 31 */
            const unsigned mv = lane < left ? A.open[32 + lane] : 0u;
            __syncwarp();
            if (lane < left) A.open[lane] = mv;
            n = left;
            __syncwarp();
            if (more && A.count[c] == VERTEX_TESTS) {
                /* the list of the configuration in the sweep is full: its
                   pairs that are not queued wait for another sweep */
                const unsigned m = __ballot_sync(FULL_MASK, word != 0u);
                int next = row < rows ? g0 - SWEEP_GROUP + row * 1024 : g0;
                if (m) next = __shfl_sync(FULL_MASK, base + __ffs(word) - 1, __ffs(m) - 1);
                if (lane == 0 && next < sc.npairs) atomicMin(&A.resume[c], (unsigned)next);
                word = 0u;
                row = rows;
                g0 = sc.npairs;
            }
        }
        /* the exact tests in rounds */
        const int tests = A.count[lane];
        int done = 0;
#pragma unroll 1
        for (;;) {
            const bool open = done < tests && A.jkey[lane] == JKEY_NONE;
            const unsigned m = __ballot_sync(FULL_MASK, open);
            if (!m) break;
            const int per = 32 / __popc(m);             /* tests each gives */
            __syncwarp();
            A.open[lane] = PAIR_NONE;
            __syncwarp();
            if (open) {
                const int at = __popc(m & ((1u << lane) - 1u)) * per;
                for (int k = 0; k < per && done + k < tests; ++k)
                    A.open[at + k] = (unsigned)lane | (A.test[done + k][lane] << 5);
            }
            done += per;
            __syncwarp();
            const unsigned it = A.open[lane];
            if (it != PAIR_NONE) {
                const int own = (int)(it & 31u), j = (int)(it >> 5);
                const int4 pr = S.pairs[j];
                Frame<float> tp, tq;
                pair_frames(S.frames - lane + own, pr, tp, tq);
                float mg;
                int code;
                if constexpr (FAST) code = pair_test_fast(sc, S.tab, pr, sc.ppoly[j], tp, tq, &mg);
                else code = pair_test<PF32>(sc, S.tab, pr, tp, tq, &mg);
                ++pc.full;
                if (code != 0) {
                    const unsigned inb = band_on && in_band(code, mg, band) ? 16u : 0u;
                    atomicMin(&A.jkey[own], ((unsigned)j << 5) | inb | (unsigned)(code + 1));
                } else if (!(mg >= band)) {
                    atomicMin(&A.jfirst[own], (unsigned)j);
                    atomicMax(&A.jlast[own], j);
                }
            }
            __syncwarp();
        }
        from = A.resume[lane];
        const bool again = from != PAIR_NONE && A.jkey[lane] == JKEY_NONE;
        if (from != PAIR_NONE && !again) pc.cert -= sc.npairs - from;   /* not looked at */
        todo = __ballot_sync(FULL_MASK, again);
        __syncwarp();
    }
    int code = valid && !active ? 1 : 0;
    bool want = false;
    int jrec = 0x7fffffff, jlast = -1;
    if (active) {
        const unsigned jk = A.jkey[lane], jf = A.jfirst[lane];
        jrec = (int)min(jf, jk >> 5);
        if (jk != JKEY_NONE) {
            code = (int)(jk & 15u) - 1;
            want = (jk & 16u) != 0u;
        } else {
            want = band_on && jf != PAIR_NONE;
            jlast = A.jlast[lane];
        }
    }
    if (valid) {
        exec += active;
        res[i] = code;
    }
    warp_append(want, make_uint2((unsigned)i, (unsigned)(code + 1) << 27), recheck_range(code, jrec, jlast, sc.npairs),
                bq, ctl);
    __syncwarp();
}

/* 120 registers, without spills: 16 warps an SM (vertices of hull6 and of the
 * 7-DOF wall 3.41 and 2.80 ms; 112 and 18 warps 3.43 and 2.80).  The
 * edge kernel is slower with fewer than 128 (112: 57.9 -> 59.1 ms, 96: 59.9). */
template <bool SMEM, bool FAST>
__global__ void __maxnreg__(120) k_check_configs(DevScene sc, const float* __restrict__ q,
                                            long long n, long long offset,
                                            int* __restrict__ res, int band_on, float band,
                                            BandQueue bq,
                                            Control* ctl)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const SceneView S = stage_scene<SMEM, true>(sc, smem);
    const int lane = threadIdx.x & 31;
    unsigned long long exec = 0;
    PairCounts pc = {0, 0};
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&ctl->next, 32ull);
        base = __shfl_sync(FULL_MASK, base, 0);
        if (base >= (unsigned long long)n) break;
        const long long left = n - (long long)base;
        check_config_chunk<FAST>(sc, S, q, offset, (long long)base, left < 32 ? (int)left : 32, res, band_on,
                                 band, bq, ctl, pc, exec);
    }
    exec = warp_sum(exec);
    if (lane == 0 && exec) atomicAdd(&ctl->configs_exec, exec);
    flush_counts(pc, ctl);
}

/* ------------------------------------------------------------------ */
/* edge checks                                                          */
/* ------------------------------------------------------------------ */

/* Edge keys (one uint32 per edge, decoded by k_finalize_edges):
 *   early exit  min over colliding steps of (order << 4 | (code+1)),
 *               0xffffffff = free
 *   all steps   max over colliding steps of ((t+1) << 4 | (code+1)),
 *               0 = free                                                   */
__device__ __forceinline__ unsigned early_key(unsigned order, int code) { return (order << 4) | (unsigned)(code + 1); }
__device__ __forceinline__ unsigned all_key(int t, int code) { return ((unsigned)(t + 1) << 4) | (unsigned)(code + 1); }

/* Segments of an edge of R rounds when a batch splits its edges into
 * pieces of about seg_rounds rounds (at most EDGE_MAX_SEGS per edge). */
constexpr int EDGE_MAX_SEGS = 64;
__device__ __forceinline__ int edge_seg_count(int R, int seg_rounds)
{
    const int s = (R + seg_rounds - 1) / seg_rounds;
    return s < EDGE_MAX_SEGS ? s : EDGE_MAX_SEGS;
}

/* One edge e (testnum steps, rounds of 32 steps over the lanes), or with
 * seg_rounds > 0 its segment `seg`: a contiguous range of rounds, so that
 * several warps share a long edge.  The rounds keep their step order, a
 * segment's decision is merged into key[e] atomically (min for early exit,
 * max for all steps, the same merge as the FP64 recheck) and a segment
 * stops once key[e] holds a decision that none of its remaining rounds can
 * improve on. */
template <int POLICY, bool SPLIT, bool FAST>
__device__ __forceinline__ void check_edge(const DevScene& sc, const SceneView& S, const float* __restrict__ qs,
                                           const float* __restrict__ qe, long long e, long long offset, float dq,
                                           unsigned* __restrict__ key, int band_on, float band,
                                           BandQueue bq, Control* ctl, PairCounts& pc,
                                           unsigned long long& exec, unsigned long long& nominal,
                                           int seg = 0, int seg_rounds = 0)
{
    const int lane = threadIdx.x & 31;
    const int tn = edge_testnum(qs, qe, e, offset, sc.ndof, dq);
    if (tn < 0) {
        if (lane == 0 && seg == 0) atomicOr(&ctl->flags, GPRM_DEVFLAG_BAD_EDGE);
        return;
    }
    if (lane == 0 && seg == 0) nominal += tn;
    /* the edge's ends, spread over the lanes for every round: lane j holds
       joint j of qs, lane 16 + j that of qe */
    float ends = 0.0f;
    if ((lane & 15) < sc.ndof) ends = (lane < 16 ? qs : qe)[e + offset * (lane & 15)];
    const int R = (tn + 31) >> 5;
    int r_begin = 0, r_end = R;
    if constexpr (SPLIT) {
        const int ns = edge_seg_count(R, seg_rounds);
        const int rs = (R + ns - 1) / ns;
        r_begin = seg * rs;
        r_end = min(R, r_begin + rs);
    }
    bool decided = false;
#pragma unroll 1
    for (int r = r_begin; r < r_end && !decided; ++r) {
        if constexpr (SPLIT) {
            const unsigned kv = *(volatile const unsigned*)&key[e];
            const bool beaten = (POLICY == EDGE_EARLY_EXIT)
                ? (kv != 0xffffffffu && (kv >> 4) < (unsigned)(r * 32))
                : (kv != 0u && (int)(kv >> 4) - 1 > tn - 1 - r * 32);
            if (__any_sync(FULL_MASK, beaten)) break;
        }
        /* lanes past the round's last step repeat it: every lane's frames
           then belong to the round and the sweep balls need no mask */
        int t;
        unsigned order;
        bool valid;
        if (POLICY == EDGE_EARLY_EXIT) {
            const int last = (tn - 1 - r) / R;     /* lanes 0 .. last hold steps */
            valid = lane <= last;
            t = (valid ? lane : last) * R + r;
            order = (unsigned)(r * 32 + lane);
        } else {
            t = tn - 1 - (r * 32 + lane);
            valid = t >= 0;
            if (!valid) t = 0;
            order = 0;
        }
        /* the step's configuration as edge_step_config */
        const float c1 = (float)t / (float)(tn - 1), c2 = 1.0f - c1;
        const unsigned valid_mask = __ballot_sync(FULL_MASK, valid);
        lane_fk<FAST>(sc, S, [&](int j) {
            return c1 * __shfl_sync(FULL_MASK, ends, j) + c2 * __shfl_sync(FULL_MASK, ends, 16 + j);
        }, __popc(valid_mask) >> 1);
        if (lane == 0) exec += __popc(valid_mask);
        bool active = valid;
        int code = 0;
        float mmin = PF32::inf(), mdec = 0.0f;
        int cut = 32;   /* lanes above the highest-priority colliding lane no longer matter */
        int jend = 0;   /* pairs processed by the warp */
        int jrec = 0x7fffffff, jlast = -1;   /* first and last pair decided within the band */
        bool stop = false;
        /* the sweep stage for a group of pairs, then per chunk of 32 pairs
           with one left open the lanes' own certificates and the exact tests
           in the reference's order; a code can only change at such a test,
           so the vote runs only there */
        unsigned nact = __ballot_sync(FULL_MASK, active);
#pragma unroll 1
        for (int g0 = 0; g0 < sc.npairs; g0 += 1024) {     /* a word per lane */
            const int gend = min(sc.npairs, g0 + 1024);
            if (g0 % SWEEP_GROUP == 0)
                sweep_stage(sc, S, g0 / SWEEP_GROUP, (min(sc.npairs - g0, SWEEP_GROUP) + 31) >> 5);
            const int wi = ((g0 % SWEEP_GROUP) >> 5) + lane;
            const unsigned open = g0 + 32 * lane < gend ? S.bits[wi] : 0u;
            unsigned left = __ballot_sync(FULL_MASK, open != 0u);
            int pos = g0;   /* pairs before it are counted */
            while (left) {
                const int c = __ffs(left) - 1;
                left &= left - 1u;
                const unsigned cand = __shfl_sync(FULL_MASK, open, c);
                const int j0 = g0 + 32 * c, j1 = min(gend, j0 + 32);
                if (lane == 0) pc.cert += (unsigned)((j1 - pos - __popc(cand)) * __popc(nact));
                pos = j1;
                const unsigned need = active ? lane_scan(sc, S, j0, cand, pc) : 0u;
                unsigned todo = __reduce_or_sync(FULL_MASK, need);
                while (todo) {
                    const int k = __ffs(todo) - 1;
                    todo &= todo - 1u;
                    if (active && ((need >> k) & 1u)) {
                        float m;
                        const int rr = eval_pair<FAST>(sc, S, j0 + k, &m, pc);
                        if (rr != 0) { code = rr; mdec = m; active = false; jrec = min(jrec, j0 + k); }
                        else {
                            mmin = min_nan(mmin, m);
                            if (!(m >= band)) { jrec = min(jrec, j0 + k); jlast = j0 + k; }
                        }
                    }
                    jend = j0 + k + 1;
                    bool oobj = code != 0 && !(band_on && in_band(code, mdec, band));
                    unsigned hits = __ballot_sync(FULL_MASK, oobj);
                    if (hits) {
                        int Lj = __ffs(hits) - 1;
                        if (Lj < cut) cut = Lj;
                        if (POLICY == EDGE_EARLY_EXIT) { stop = true; break; }
                        if (lane > cut) active = false;
                    }
                }
                nact = __ballot_sync(FULL_MASK, active);
                if (stop || !nact) break;
            }
            if (stop || !nact) break;
            if (lane == 0) pc.cert += (unsigned)((gend - pos) * __popc(nact));
            jend = gend;
        }
        /* settle the round */
        const bool oob = code != 0 && !(band_on && in_band(code, mdec, band));
        const unsigned hits = __ballot_sync(FULL_MASK, oob && lane <= cut);
        const int L = hits ? __ffs(hits) - 1 : 32;
        const bool free_done = valid && code == 0 && active && jend == sc.npairs;
        const bool inb = band_on && ((code != 0 && !oob) || (free_done && in_band(0, mmin, band)));
        /* in-band steps earlier in order (early exit) or higher t (all steps)
           than the deciding step go to the FP64 queue */
        const bool want = inb && lane < L;
        warp_append(want, make_uint2((unsigned)e, (unsigned)t | ((unsigned)(code + 1) << 27)),
                    recheck_range(code, jrec, jlast, sc.npairs), bq, ctl);
        if (hits) {
            if (lane == L) {
                const unsigned kv = (POLICY == EDGE_EARLY_EXIT) ? early_key(order, code) : all_key(t, code);
                if constexpr (!SPLIT) key[e] = kv;
                else if (POLICY == EDGE_EARLY_EXIT) atomicMin(&key[e], kv);
                else atomicMax(&key[e], kv);
            }
            decided = true;
        }
    }
}

__device__ __forceinline__ void flush_edge_counts(unsigned long long exec, unsigned long long nominal, PairCounts pc,
                                                  Control* ctl)
{
    exec = warp_sum(exec);
    nominal = warp_sum(nominal);
    if ((threadIdx.x & 31) == 0) {
        if (exec) atomicAdd(&ctl->steps_exec, exec);
        if (nominal) atomicAdd(&ctl->steps_nominal, nominal);
    }
    flush_counts(pc, ctl);
}

/* SPLIT: the work items are the segments of the edges, edge e owning
 * items [seg_off[e], seg_off[e+1]) (seg_off from k_edge_segments);
 * otherwise one item per edge and seg_off is unused. */
template <bool SMEM, int POLICY, bool SPLIT, bool FAST>
__global__ void GPRM_BOUNDS k_check_edges(DevScene sc, const float* __restrict__ qs,
                                          const float* __restrict__ qe, long long n,
                                          long long offset, float dq, unsigned* __restrict__ key,
                                          int band_on, float band, BandQueue bq, Control* ctl,
                                          const unsigned* __restrict__ seg_off,
                                          int seg_rounds)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const SceneView S = stage_scene<SMEM, false>(sc, smem);
    const int lane = threadIdx.x & 31;
    unsigned long long exec = 0, nominal = 0;
    PairCounts pc = {0, 0};
    if constexpr (!SPLIT) {
        for (;;) {
            unsigned long long eu = 0;
            if (lane == 0) eu = atomicAdd(&ctl->next, 1ull);
            eu = __shfl_sync(FULL_MASK, eu, 0);
            if (eu >= (unsigned long long)n) break;
            check_edge<POLICY, false, FAST>(sc, S, qs, qe, (long long)eu, offset, dq, key, band_on, band, bq, ctl,
                                            pc, exec, nominal);
        }
        flush_edge_counts(exec, nominal, pc, ctl);
        return;
    }
    const unsigned long long items = (unsigned long long)seg_off[n];
    for (;;) {
        unsigned long long eu = 0;
        long long e = 0;
        int seg = 0;
        if (lane == 0) {
            eu = atomicAdd(&ctl->next, 1ull);
            if (eu < items) {
                long long lo = 0, hi = n;       /* seg_off[lo] <= eu < seg_off[hi] */
                while (hi - lo > 1) {
                    const long long mid = (lo + hi) >> 1;
                    if ((unsigned long long)seg_off[mid] <= eu) lo = mid;
                    else hi = mid;
                }
                e = lo;
                seg = (int)(eu - seg_off[lo]);
            }
        }
        eu = __shfl_sync(FULL_MASK, eu, 0);
        if (eu >= items) break;
        e = __shfl_sync(FULL_MASK, e, 0);
        seg = __shfl_sync(FULL_MASK, seg, 0);
        check_edge<POLICY, true, FAST>(sc, S, qs, qe, e, offset, dq, key, band_on, band, bq, ctl, pc,
                                       exec, nominal, seg, seg_rounds);
    }
    flush_edge_counts(exec, nominal, pc, ctl);
}

/* Segment offsets of n edges (one block): seg_off[e] = sum over e' < e of
 * the segment count of edge e', seg_off[n] = the total.  Edges the check
 * rejects (non-finite or oversized) count one segment. */
__global__ void __launch_bounds__(1024) k_edge_segments(const float* __restrict__ qs, const float* __restrict__ qe,
                                                        long long n, long long offset, int ndof, float dq,
                                                        int seg_rounds, unsigned* __restrict__ seg_off)
{
    __shared__ unsigned wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long per = (n + blockDim.x - 1) / blockDim.x;
    const long long b0 = min(n, (long long)tid * per), b1 = min(n, b0 + per);
    auto segs = [&](long long e) -> unsigned {
        const int tn = edge_testnum(qs, qe, e, offset, ndof, dq);
        return tn < 0 ? 1u : (unsigned)edge_seg_count((tn + 31) >> 5, seg_rounds);
    };
    unsigned s = 0;
    for (long long e = b0; e < b1; ++e) s += segs(e);
    unsigned x = s;                                    /* inclusive scan in the warp */
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned y = __shfl_up_sync(FULL_MASK, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        unsigned w = lane < nw ? wsum[lane] : 0u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned y = __shfl_up_sync(FULL_MASK, w, d);
            if (lane >= d) w += y;
        }
        if (lane < nw) wsum[lane] = w;                 /* inclusive warp totals */
    }
    __syncthreads();
    unsigned base = x - s + (warp > 0 ? wsum[warp - 1] : 0u);
    for (long long e = b0; e < b1; ++e) {
        seg_off[e] = base;
        base += segs(e);
    }
    if (tid == (int)blockDim.x - 1) seg_off[n] = base;
}

/* Segment count of edge e for the split kernels (a rejected edge counts
 * one segment). */
__device__ __forceinline__ unsigned edge_segs(const float* __restrict__ qs, const float* __restrict__ qe, long long e,
                                              long long offset, int ndof, float dq, int seg_rounds)
{
    const int tn = edge_testnum(qs, qe, e, offset, ndof, dq);
    return tn < 0 ? 1u : (unsigned)edge_seg_count((tn + 31) >> 5, seg_rounds);
}

/* Exclusive scan of x over the block (blockDim.x <= 1024, a multiple of
 * 32); *total gets the block's sum.  wsum: 32 words of shared memory. */
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned x, unsigned* wsum, unsigned* total)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    unsigned v = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned y = __shfl_up_sync(FULL_MASK, v, d);
        if (lane >= d) v += y;
    }
    if (lane == 31) wsum[warp] = v;
    __syncthreads();
    if (warp == 0) {
        unsigned w = lane < nw ? wsum[lane] : 0u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned y = __shfl_up_sync(FULL_MASK, w, d);
            if (lane >= d) w += y;
        }
        if (lane < nw) wsum[lane] = w;                 /* inclusive warp totals */
    }
    __syncthreads();
    const unsigned ex = v - x + (warp > 0 ? wsum[warp - 1] : 0u);
    *total = wsum[nw - 1];
    __syncthreads();
    return ex;
}

/* Segment offsets of more than EDGE_SPLIT_ONE_BLOCK edges, in three
 * passes: block b (of EDGE_SEG_BLOCKS) takes the edges [b c, (b+1) c),
 * c = ceil(n / blocks), each thread a contiguous run of them.  Pass 0
 * writes the block's segment count to bsum[b]; k_seg_scan_blocks turns
 * bsum into exclusive offsets (and seg_off[n] into the total); pass 1
 * writes seg_off[e] for the block's edges. */
template <int PASS>
__global__ void __launch_bounds__(256) k_seg_pass(const float* __restrict__ qs, const float* __restrict__ qe,
                                                  long long n, long long offset, int ndof, float dq, int seg_rounds,
                                                  unsigned* __restrict__ seg_off, unsigned* __restrict__ bsum)
{
    __shared__ unsigned wsum[32];
    const long long chunk = (n + gridDim.x - 1) / gridDim.x;
    const long long c0 = min(n, (long long)blockIdx.x * chunk), c1 = min(n, c0 + chunk);
    const long long per = (c1 - c0 + blockDim.x - 1) / blockDim.x;
    const long long b0 = min(c1, c0 + (long long)threadIdx.x * per), b1 = min(c1, b0 + per);
    unsigned s = 0;
    for (long long e = b0; e < b1; ++e) s += edge_segs(qs, qe, e, offset, ndof, dq, seg_rounds);
    unsigned total = 0;
    unsigned base = block_exclusive_scan(s, wsum, &total);
    if (PASS == 0) {
        if (threadIdx.x == 0) bsum[blockIdx.x] = total;
        return;
    }
    base += bsum[blockIdx.x];
    for (long long e = b0; e < b1; ++e) {
        seg_off[e] = base;
        base += edge_segs(qs, qe, e, offset, ndof, dq, seg_rounds);
    }
}

/* bsum[0..nb) -> exclusive offsets, *total_out = their sum (one block of
 * 1024 threads, nb <= 1024). */
__global__ void __launch_bounds__(1024) k_seg_scan_blocks(unsigned* __restrict__ bsum, int nb,
                                                          unsigned* __restrict__ total_out)
{
    __shared__ unsigned wsum[32];
    const int t = threadIdx.x;
    const unsigned x = t < nb ? bsum[t] : 0u;
    unsigned total = 0;
    const unsigned ex = block_exclusive_scan(x, wsum, &total);
    if (t < nb) bsum[t] = ex;
    if (t == 0) *total_out = total;
}

/* ------------------------------------------------------------------ */
/* FP64 recheck and finalisation                                        */
/* ------------------------------------------------------------------ */

/* The FP64 check of one configuration (in bounds): the reference's pair
 * loop in double with the FP64 certificates, over pairs [j_start, j_end)
 * (the pairs outside that range were decided separated outside the band by
 * the FP32 check, so in FP64 they are separated too, and the first
 * colliding pair, hence the code, is the same as over every pair). */
__device__ __forceinline__ int check_config64(const DevScene& sc, const float* qi, int j_start = 0, int j_end = -1)
{
    if (j_end < 0 || j_end > sc.npairs) j_end = sc.npairs;
    Frame<double> F[GPRM_MAX_FRAMES];
    forward_kinematics<PF64>(sc, qi, F);
    /* slot ball centres in FP64, once per check (the same transform the
       certificate would apply per pair) */
    double cen[GPRM_MAX_SLOTS * 3];
    for (int sl = 0; sl < sc.nslots; ++sl) {
        const float4 b = sc.tab[sc.slot_block[sl]];
        const V3<double> c = xform<double>(F[sc.slot_sys[sl]], (double)b.x, (double)b.y, (double)b.z);
        cen[3 * sl] = c.x; cen[3 * sl + 1] = c.y; cen[3 * sl + 2] = c.z;
    }
#pragma unroll 1
    for (int j = j_start; j < j_end; ++j) {
        const int4 pr = sc.pairs[j];
        if (pair_certified64(sc, sc.tab, pr, sc.pairs_b[j], F, cen, j)) continue;
        double m;
        const int r = pair_test<PF64>(sc, sc.tab, pr, F[pr.z], F[pr.w], &m);
        if (r != 0) return r;
    }
    return 0;
}

/* The item's configuration (vertex kind 0 or edge step kind 1); for an
 * edge step also its step t and the edge's step count tn. */
__device__ __forceinline__ void recheck_config(const DevScene& sc, int kind, uint2 it, const float* __restrict__ q,
                                               const float* __restrict__ qs, const float* __restrict__ qe,
                                               long long offset, float dq, float* qi, int& t, int& tn)
{
    t = 0;
    tn = 0;
    if (kind == 0) {
        for (int j = 0; j < sc.ndof; ++j) qi[j] = q[(long long)it.x + offset * j];
    } else {
        t = (int)(it.y & ((1u << 27) - 1));
        tn = edge_testnum(qs, qe, (long long)it.x, offset, sc.ndof, dq);
        edge_step_config(qs, qe, (long long)it.x, offset, sc.ndof, t, tn, qi);
    }
}

/* Writes an FP64 recheck's code: a configuration's result, or an edge
 * step's key merge (the order of the check kernel for early exit). */
__device__ __forceinline__ void recheck_store(int kind, uint2 it, int code, int t, int tn, int policy,
                                              int* __restrict__ res, unsigned* __restrict__ key)
{
    if (kind == 0) {
        res[it.x] = code;
    } else if (code != 0) {
        if (policy == EDGE_EARLY_EXIT) {
            const int R = (tn + 31) >> 5;
            const unsigned order = (unsigned)((t % R) * 32 + t / R);
            atomicMin(&key[it.x], early_key(order, code));
        } else {
            atomicMax(&key[it.x], all_key(t, code));
        }
    }
}

/* The FP32 check of one configuration (in bounds) in one thread, in the
 * arithmetic of the kernel variant (FAST), frames in registers: every
 * pair's exact test in the reference's order (the certificates only ever
 * skip pairs whose test gives 0 with a margin above the band, so the code
 * and the band decision are those of the warp kernels).  *margin: the
 * deciding pair's margin, or the minimum over the pairs of a free check;
 * *jdec (when given): the deciding pair's index, npairs for a free check. */
template <bool FAST>
__device__ __forceinline__ int check_config32(const DevScene& sc, const float* qi, float* margin,
                                              int* jdec = nullptr)
{
    Frame<float> F[GPRM_MAX_FRAMES];
    if constexpr (FAST) forward_kinematics_fast(sc, qi, F);
    else forward_kinematics<PF32>(sc, qi, F);
    float mmin = PF32::inf();
#pragma unroll 1
    for (int j = 0; j < sc.npairs; ++j) {
        const int4 pr = sc.pairs[j];
        float m;
        int r;
        if constexpr (FAST) r = pair_test_fast(sc, sc.tab, pr, sc.ppoly[j], F[pr.z], F[pr.w], &m);
        else r = pair_test<PF32>(sc, sc.tab, pr, F[pr.z], F[pr.w], &m);
        if (r != 0) {
            *margin = m;
            if (jdec) *jdec = j;
            return r;
        }
        mmin = min_nan(mmin, m);
    }
    *margin = mmin;
    if (jdec) *jdec = sc.npairs;
    return 0;
}

/* One item of the overflow list, recomputed in full by one thread: a
 * configuration (kind 0: bounds, FP32, FP64 inside the band -> res), or an
 * edge (kind 1), whose key is rebuilt from scratch as the check and recheck
 * kernels build it when nothing overflows:
 *   all steps   the max over every step (FP32, FP64 inside the band);
 *   early exit  the check kernel's rounds (round r: steps t = lane*R + r,
 *               order r*32 + lane) until the first round with a collision
 *               outside the band.  The kernel runs a round pair by pair in
 *               the reference's pair order and stops at the first pair
 *               index j* at which some step collides outside the band; its
 *               lowest such lane L decides.  Steps of lower lanes whose
 *               loop had ended by then in the band (a collision at a pair
 *               <= j*, or a free check when nothing decided) go to the FP64
 *               check, and a collision there takes the lower order. */
template <bool FAST>
__device__ __forceinline__ void overflow_item(const DevScene& sc, int kind, unsigned x, const float* __restrict__ q,
                                              const float* __restrict__ qs, const float* __restrict__ qe,
                                              long long offset, float dq, int policy, float band,
                                              int* __restrict__ res, unsigned* __restrict__ key,
                                              unsigned long long& checks, unsigned long long& flips)
{
    float qi[GPRM_MAX_FRAMES];
    if (kind == 0) {
        for (int j = 0; j < sc.ndof; ++j) qi[j] = q[(long long)x + offset * j];
        int code = 0;
        for (int j = 0; j < sc.ndof; ++j)
            if (qi[j] < sc.mins[j] || qi[j] > sc.maxs[j]) { code = 1; break; }
        if (code == 0) {
            float m;
            code = check_config32<FAST>(sc, qi, &m);
            if (in_band(code, m, band)) {
                const int c64 = check_config64(sc, qi);
                ++checks;
                flips += ((c64 != 0) != (code != 0));
                code = c64;
            }
        }
        res[x] = code;
        return;
    }
    const int tn = edge_testnum(qs, qe, (long long)x, offset, sc.ndof, dq);
    if (tn < 0) return;   /* flagged by the check kernel */
    const int R = (tn + 31) >> 5;
    if (policy != EDGE_EARLY_EXIT) {
        unsigned k = 0u;
#pragma unroll 1
        for (int t = 0; t < tn; ++t) {
            edge_step_config(qs, qe, (long long)x, offset, sc.ndof, t, tn, qi);
            float m;
            int code = check_config32<FAST>(sc, qi, &m);
            if (in_band(code, m, band)) {
                const int c64 = check_config64(sc, qi);
                ++checks;
                flips += ((c64 != 0) != (code != 0));
                code = c64;
            }
            if (code != 0) {
                const unsigned kv = all_key(t, code);
                if (kv > k) k = kv;
            }
        }
        key[x] = k;
        return;
    }
    unsigned k = 0xffffffffu;
#pragma unroll 1
    for (int r = 0; r < R; ++r) {
        /* the round's deciding pair index j* and lane L */
        int jstar = 0x7fffffff, L = 32, codeL = 0;
#pragma unroll 1
        for (int lane = 0; lane < 32; ++lane) {
            const int t = lane * R + r;
            if (t >= tn) break;
            edge_step_config(qs, qe, (long long)x, offset, sc.ndof, t, tn, qi);
            float m;
            int j;
            const int code = check_config32<FAST>(sc, qi, &m, &j);
            if (code != 0 && !in_band(code, m, band) && j < jstar) { jstar = j; L = lane; codeL = code; }
        }
        /* the in-band steps below L that the kernel queues */
#pragma unroll 1
        for (int lane = 0; lane < L; ++lane) {
            const int t = lane * R + r;
            if (t >= tn) break;
            edge_step_config(qs, qe, (long long)x, offset, sc.ndof, t, tn, qi);
            float m;
            int j;
            const int code = check_config32<FAST>(sc, qi, &m, &j);
            const bool queued = code != 0 ? (in_band(code, m, band) && j <= jstar)
                                          : (L == 32 && in_band(0, m, band));
            if (!queued) continue;
            const int c64 = check_config64(sc, qi);
            ++checks;
            flips += ((c64 != 0) != (code != 0));
            if (c64 != 0) {
                const unsigned kv = early_key((unsigned)(r * 32 + lane), c64);
                if (kv < k) k = kv;
            }
        }
        if (L < 32) {
            const unsigned kv = early_key((unsigned)(r * 32 + L), codeL);
            if (kv < k) k = kv;
            break;
        }
    }
    key[x] = k;
}

/* check_config64 by a warp, joint j's value in lane j: joint trigonometry a
 * lane per joint, the frame products an entry per lane, the pairs of the
 * range over the lanes, those that no certificate settles queued (64
 * entries) and tested 32 at a time.  Same operations as check_config64, same
 * code. */
__device__ __forceinline__ int warp_check64(const DevScene& sc, Frame<double>* F, Frame<double>* L, double* cen,
                                            unsigned* queue, float q, int j_start, int j_end)
{
    const int lane = threadIdx.x & 31;
    if (j_end > sc.npairs) j_end = sc.npairs;
    if (lane < sc.ndof) {
        float th = sc.q0[lane], d = sc.d0[lane];
        if (sc.types[lane] == 0) th = q;
        else d = q;
        double cq, sq, ca, sa;
        PF64::trig(th, cq, sq);
        PF64::trig_alpha(sc, lane, ca, sa);
        dh_frame<PF64>(L[lane], cq, sq, ca, sa, (double)sc.a[lane], (double)d);
    }
    if (lane < 12) F[0].m[lane] = lane % 4 == 0 && lane < 9 ? 1.0 : (lane == 3 || lane == 7 || lane == 10 ? -0.0 : 0.0);
    __syncwarp();
    const int c = lane / 3, r = lane - 3 * c;
#pragma unroll 1
    for (int i = 0; i < sc.ndof; ++i) {
        if (lane < 12) {
            const double* T = F[i].m;
            const double* u = L[i].m + 3 * c;
            double o = T[r] * u[0] + T[3 + r] * u[1] + T[6 + r] * u[2];
            if (c == 3) o = o + T[9 + r];
            F[i + 1].m[lane] = o;
        }
        __syncwarp();
    }
    if (lane < sc.nslots) {
        const float4 b = sc.tab[sc.slot_block[lane]];
        const V3<double> w = xform<double>(F[sc.slot_sys[lane]], (double)b.x, (double)b.y, (double)b.z);
        cen[3 * lane] = w.x; cen[3 * lane + 1] = w.y; cen[3 * lane + 2] = w.z;
    }
    __syncwarp();
    int code = 0, n = 0;
#pragma unroll 1
    for (int j0 = j_start; j0 < j_end || n > 0; j0 += 32) {
        const int j = j0 + lane;
        bool open = false;
        if (j < j_end) open = !pair_certified64(sc, sc.tab, sc.pairs[j], sc.pairs_b[j], F, cen, j);
        const unsigned m = __ballot_sync(FULL_MASK, open);
        if (open) queue[n + __popc(m & ((1u << lane) - 1u))] = (unsigned)j;
        n += __popc(m);
        __syncwarp();
        if (n < 32 && j0 + 32 < j_end) continue;
        /* the first 32 open pairs side by side, in order */
        int rr = 0;
        if (lane < n) {
            const int4 pr = sc.pairs[queue[lane]];
            double mg;
            rr = pair_test<PF64>(sc, sc.tab, pr, F[pr.z], F[pr.w], &mg);
        }
        const unsigned hit = __ballot_sync(FULL_MASK, rr != 0);
        if (hit) {
            code = __shfl_sync(FULL_MASK, rr, __ffs(hit) - 1);
            break;
        }
        const unsigned mv = lane + 32 < n ? queue[32 + lane] : 0u;
        __syncwarp();
        if (lane + 32 < n) queue[lane] = mv;
        n = n > 32 ? n - 32 : 0;
        __syncwarp();
    }
    __syncwarp();
    return code;
}

/* The FP64 recheck of the queued items: one thread per item, or, for few
 * items, one warp per item with its pairs over the lanes (warp_check64).
 * With many items their own parallelism hides the FP64 latency better; with
 * few, the longest item's chain of pairs is the kernel's time, so what
 * counts as few grows with the pair list.  Measured (thread per item ->
 * warp per item): 1 item per resident warp, 4117 pairs (vertex checks of
 * the wall scene) 1.7 -> 0.35 ms; 59 per warp, 4117 pairs (its edges) 3.0 ->
 * 1.8 ms; 10 per warp, 394 pairs (hull6 vertices) 0.34 -> 0.54 ms; 27 per
 * warp, 394 pairs (exact hull6 edges) 1.1 -> 3.0 ms. */
constexpr unsigned RECHECK_FEW = 4;
__device__ __forceinline__ bool recheck_by_warp(unsigned items, unsigned warps, int npairs)
{
    const unsigned few = RECHECK_FEW * (npairs > 512 ? (unsigned)npairs >> 8 : 1u);
    return (unsigned long long)items <= (unsigned long long)few * warps;
}
constexpr int RECHECK_THREADS = 128;

/* The pairs [lo, hi) of queue item idx: as recorded, else all of them (a
 * pair list whose indices do not fit a recorded range). */
struct PairSpan {
    int lo, hi;
};
__device__ __forceinline__ PairSpan recheck_span(const BandQueue& bq, unsigned idx, int npairs)
{
    if (!bq.pair_range) return {0, npairs};
    const unsigned range = bq.pair_range[idx];
    return {(int)(range & 0xffffu), (int)(range >> 16)};
}

__device__ __forceinline__ void recheck_item(const DevScene& sc, int kind, uint2 it, const float* __restrict__ q,
                                             const float* __restrict__ qs, const float* __restrict__ qe,
                                             long long offset, float dq, int policy, int* __restrict__ res,
                                             unsigned* __restrict__ key, unsigned long long& checks,
                                             unsigned long long& flips, PairSpan span)
{
    float qi[GPRM_MAX_FRAMES];
    int t, tn;
    recheck_config(sc, kind, it, q, qs, qe, offset, dq, qi, t, tn);
    const int code = check_config64(sc, qi, span.lo, span.hi);
    ++checks;
    flips += ((code != 0) != ((int)(it.y >> 27) - 1 != 0));
    recheck_store(kind, it, code, t, tn, policy, res, key);
}

/* Shared memory of a warp's item (warp_check64). */
struct Warp64 {
    Frame<double> F[GPRM_MAX_FRAMES], L[GPRM_MAX_FRAMES];
    double cen[GPRM_MAX_SLOTS * 3];
    unsigned queue[64];
};

/* recheck_item by a warp; lane 0 counts and stores. */
__device__ __forceinline__ void recheck_item_warp(const DevScene& sc, int kind, uint2 it, const float* __restrict__ q,
                                                  const float* __restrict__ qs, const float* __restrict__ qe,
                                                  long long offset, float dq, int policy, int* __restrict__ res,
                                                  unsigned* __restrict__ key, unsigned long long& checks,
                                                  unsigned long long& flips, PairSpan span, Warp64& W)
{
    const int lane = threadIdx.x & 31;
    int t = 0, tn = 0;
    float x = 0.0f;
    if (kind == 0) {
        if (lane < sc.ndof) x = q[(long long)it.x + offset * lane];
    } else {
        /* as recheck_config: joint j in lane j */
        t = (int)(it.y & ((1u << 27) - 1));
        tn = edge_testnum(qs, qe, (long long)it.x, offset, sc.ndof, dq);
        const float c1 = (float)t / (float)(tn - 1), c2 = 1.0f - c1;
        if (lane < sc.ndof)
            x = c1 * qs[(long long)it.x + offset * lane] + c2 * qe[(long long)it.x + offset * lane];
    }
    const int code = warp_check64(sc, W.F, W.L, W.cen, W.queue, x, span.lo, span.hi);
    if (lane == 0) {
        ++checks;
        flips += ((code != 0) != ((int)(it.y >> 27) - 1 != 0));
        recheck_store(kind, it, code, t, tn, policy, res, key);
    }
}

__global__ void __launch_bounds__(RECHECK_THREADS) k_recheck(DevScene sc, int kind, const float* __restrict__ q,
                                                             const float* __restrict__ qs,
                                                             const float* __restrict__ qe, long long offset,
                                                             float dq, int policy, int* __restrict__ res,
                                                             unsigned* __restrict__ key, const BandQueue bq,
                                                             Control* ctl)
{
    __shared__ Warp64 W[RECHECK_THREADS / 32];
    unsigned cnt = ctl->qcount;
    if (cnt > bq.cap) cnt = bq.cap;
    unsigned long long checks = 0, flips = 0;
    const unsigned warps = gridDim.x * (RECHECK_THREADS / 32), warp = threadIdx.x >> 5;
    if (recheck_by_warp(cnt, warps, sc.npairs)) {
        for (unsigned idx = warp * gridDim.x + blockIdx.x; idx < cnt; idx += warps)
            recheck_item_warp(sc, kind, bq.items[idx], q, qs, qe, offset, dq, policy, res, key, checks, flips,
                              recheck_span(bq, idx, sc.npairs), W[warp]);
    } else {
        for (unsigned idx = blockIdx.x * blockDim.x + threadIdx.x; idx < cnt; idx += gridDim.x * blockDim.x)
            recheck_item(sc, kind, bq.items[idx], q, qs, qe, offset, dq, policy, res, key, checks, flips,
                         recheck_span(bq, idx, sc.npairs));
    }
    if (checks) atomicAdd(&ctl->band_checks, checks);
    if (flips) atomicAdd(&ctl->band_flips, flips);
}

/* The overflow pass of a request: every item in the overflow list,
 * recomputed by one thread (overflow_item).  Exits at once when nothing
 * overflowed. */
template <bool FAST>
__global__ void __launch_bounds__(128) k_overflow(DevScene sc, int kind, const float* __restrict__ q,
                                                  const float* __restrict__ qs, const float* __restrict__ qe,
                                                  long long offset, float dq, int policy, float band,
                                                  int* __restrict__ res, unsigned* __restrict__ key, BandQueue bq,
                                                  Control* ctl)
{
    const unsigned long long cnt = ctl->ovf_count;
    if (cnt == 0 || !bq.ovf) return;
    unsigned long long checks = 0, flips = 0;
    for (unsigned long long idx = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; idx < cnt;
         idx += (unsigned long long)gridDim.x * blockDim.x)
        overflow_item<FAST>(sc, kind, bq.ovf[idx], q, qs, qe, offset, dq, policy, band, res, key, checks, flips);
    if (checks) atomicAdd(&ctl->band_checks, checks);
    if (flips) atomicAdd(&ctl->band_flips, flips);
}

__global__ void k_finalize_edges(long long n, int policy, const unsigned* __restrict__ key,
                                 int* __restrict__ res)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        unsigned k = key[e];
        bool none = (policy == EDGE_EARLY_EXIT) ? (k == 0xffffffffu) : (k == 0u);
        res[e] = none ? 0 : (int)(k & 15u) - 1;
    }
}

__global__ void k_fk_probe(DevScene sc, const float* q, float* out)
{
    Frame<float> F[GPRM_MAX_FRAMES];
    float qi[GPRM_MAX_FRAMES];
    for (int j = 0; j < sc.ndof; ++j) qi[j] = q[j];
    forward_kinematics<PF32>(sc, qi, F);
    for (int f = 0; f <= sc.ndof; ++f)
        for (int c = 0; c < 12; ++c) out[f * 12 + c] = F[f].m[c];
}

/* ------------------------------------------------------------------ */
/* small requests: a block per configuration or edge                    */
/* ------------------------------------------------------------------ */
/*
 * A request of few items is bound by the latency of its longest chain, not
 * by throughput: with a warp per 32 configurations or per edge most of the
 * GPU idles, the exact tests of a warp run one after the other, the FP64
 * recheck is a second launch in which one thread goes through a check's
 * pairs, and control words, keys and results pass through eight more stream
 * operations.  The kernels below run the whole request in one launch: a block
 * of four warps per configuration (up to 32 of them, one per lane, for
 * larger requests) or per edge, whose rounds of 32 steps `segs` blocks
 * share.  Per round warp 0 runs the forward kinematics and the sweep balls,
 * the warps share the sweep stage's leaves and the open pairs' words, queue
 * the exact tests that their lanes need and run them 32 at a time whoever
 * they belong to; a step's first colliding pair is the minimum over the
 * pairs that collide, so the tests need no order.  Steps decided in the
 * band get their FP64 check at once, a warp per step with its pairs over
 * the lanes.  Codes, bands and key merges are those of the kernels above.
 */
constexpr int SMALL_WARPS = 4;

struct SmallShared {
    unsigned jkey[32];            /* per lane: min over colliding pairs of j << 8 | in band << 4 | code + 1 */
    unsigned jfirst[32];          /* first free pair with a margin inside the band */
    int jlast[32];                /* last one */
    unsigned queue[SMALL_WARPS][64];
    float q[GPRM_MAX_FRAMES][32]; /* configurations: joint j of lane i */
    Frame<double> F[SMALL_WARPS][GPRM_MAX_FRAMES];
    Frame<double> L[SMALL_WARPS][GPRM_MAX_FRAMES];
    double cen[SMALL_WARPS][GPRM_MAX_SLOTS * 3];
    unsigned cut;                 /* what an out-of-band collision found so far makes needless (small_run) */
    unsigned key;                 /* the edge's merged key (all steps: max, early exit: min) */
    unsigned beaten;
    unsigned full, checks, flips;
    unsigned open;                /* pairs of the round that no certificate settles or that are left out */
};

/* What B.cut holds of a lane's collision outside the band at pair j. */
enum SmallCut { CUT_NONE, CUT_LANE, CUT_PAIR };
template <int CUT>
__device__ __forceinline__ unsigned small_cut(int lane, int j)
{
    return CUT == CUT_LANE ? (unsigned)lane : (unsigned)j;
}

/* Runs the first cnt (<= 32) of the warp's queued tests (lane | pair << 5),
 * one per lane on its owner's frames, and merges their results.  Left out:
 * pairs after one that the owner already collides at, and, with a cut (the
 * lowest lane, or the first pair, with a collision outside the band so far),
 * the lanes or pairs beyond it, which cannot change the round's decision as
 * long as that collision stands (the caller checks that it does). */
template <bool FAST, int CUT>
__device__ __forceinline__ void small_run(const DevScene& sc, const SceneView& S, SmallShared& B, unsigned* q, int cnt,
                                          bool cutting, int band_on, float band)
{
    const int lane = threadIdx.x & 31;
    __syncwarp();
    const unsigned it = q[lane];
    const int owner = (int)(it & 31u), j = (int)(it >> 5);
    bool run = lane < cnt && ((unsigned)j << 8) <= *(volatile unsigned*)&B.jkey[owner];
    if (CUT != CUT_NONE && cutting) run = run && small_cut<CUT>(owner, j) <= *(volatile unsigned*)&B.cut;
    if (run) {
        const int4 pr = S.pairs[j];
        Frame<float> tp, tq;
        pair_frames(S.frames - lane + owner, pr, tp, tq);
        float m;
        int c;
        if constexpr (FAST) c = pair_test_fast(sc, S.tab, pr, sc.ppoly[j], tp, tq, &m);
        else c = pair_test<PF32>(sc, S.tab, pr, tp, tq, &m);
        if (c != 0) {
            const unsigned inb = band_on && in_band(c, m, band) ? 16u : 0u;
            atomicMin(&B.jkey[owner], ((unsigned)j << 8) | inb | (unsigned)(c + 1));
            if (CUT != CUT_NONE && !inb) atomicMin(&B.cut, small_cut<CUT>(owner, j));
        } else if (!(m >= band)) {
            atomicMin(&B.jfirst[owner], (unsigned)j);
            atomicMax(&B.jlast[owner], j);
        }
    }
    const unsigned ran = __ballot_sync(FULL_MASK, run);
    if (lane == 0 && ran) atomicAdd(&B.full, (unsigned)__popc(ran));
}

/* Certificates and exact tests of one round for the lanes of `valid` (their
 * frames in S, ready to read by the block): fills jkey, jfirst and jlast,
 * adds the pairs that certificates settle to total's.  Every thread of the
 * block calls it; ends with a block barrier.  (The count is kept in shared
 * memory: a register for it through the tests took 500 edges of the box
 * scene from 100 to 104 us.) */
template <bool FAST, int CUT>
__device__ __forceinline__ void small_pairs(const DevScene& sc, const SceneView& S, SmallShared& B, unsigned valid,
                                            bool cutting, int band_on, float band, Control* total)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool mine = (valid >> lane) & 1u;
    unsigned* q = B.queue[warp];
    PairCounts pc = {0, 0};
    int n = 0;
#pragma unroll 1
    for (int g0 = 0; g0 < sc.npairs; g0 += SWEEP_GROUP) {
        const int words = (min(sc.npairs - g0, SWEEP_GROUP) + 31) >> 5;
        for (int w = threadIdx.x; w < words; w += SMALL_WARPS * 32) S.bits[w] = 0u;
        __syncthreads();
        sweep_leaves<false>(sc, S, g0 / SWEEP_GROUP, 0x11111111u << warp, sc.nslots <= SWEEP_V0_SLOTS, SWEEP_V0_SLOTS);
        __syncthreads();
#pragma unroll 1
        for (int w = warp; w < words; w += SMALL_WARPS) {
            const unsigned cand = S.bits[w];
            if (!cand) continue;
            const int j0 = g0 + 32 * w;
            bool scan = mine && ((unsigned)j0 << 8) <= *(volatile unsigned*)&B.jkey[lane];
            if (CUT != CUT_NONE && cutting) scan = scan && small_cut<CUT>(lane, j0) <= *(volatile unsigned*)&B.cut;
            const unsigned need = scan ? lane_scan(sc, S, j0, cand, pc) : 0u;
            const unsigned open = __reduce_add_sync(FULL_MASK, mine ? __popc(scan ? need : cand) : 0);
            if (lane == 0) atomicAdd(&B.open, open);
            unsigned todo = __reduce_or_sync(FULL_MASK, need);
            while (todo) {
                const int k = __ffs(todo) - 1;
                todo &= todo - 1u;
                const unsigned m = __ballot_sync(FULL_MASK, (need >> k) & 1u);
                if ((need >> k) & 1u) q[n + __popc(m & ((1u << lane) - 1u))] = (unsigned)lane | ((unsigned)(j0 + k) << 5);
                n += __popc(m);
                if (n >= 32) {
                    small_run<FAST, CUT>(sc, S, B, q, 32, cutting, band_on, band);
                    n -= 32;
                    const unsigned mv = lane < n ? q[32 + lane] : 0u;
                    __syncwarp();
                    if (lane < n) q[lane] = mv;
                }
            }
        }
        __syncthreads();
    }
    if (n > 0) small_run<FAST, CUT>(sc, S, B, q, n, cutting, band_on, band);
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(&total->certified, (unsigned long long)sc.npairs * (unsigned)__popc(valid) - B.open);
        B.open = 0u;
    }
}

/* The view of the block's one set of frames for this thread's lane. */
__device__ __forceinline__ SceneView small_view(const DevScene& sc, unsigned char* smem)
{
    SceneView S;
    S.tab = sc.tab; S.pairs = sc.pairs;
    S.far = sc.far; S.scan_c = sc.scan_c; S.scan_b = sc.scan_b;
    S.frames = reinterpret_cast<float*>(smem) + (threadIdx.x & 31);
    S.sweep = sweep_area<false>(sc, S.frames);
    S.bits = open_area<false>(sc, S.frames);
    return S;
}

__device__ __forceinline__ void small_reset(SmallShared& B)
{
    if (threadIdx.x < 32) {
        B.jkey[threadIdx.x] = 0xffffffffu;
        B.jfirst[threadIdx.x] = 0x7fffffffu;
        B.jlast[threadIdx.x] = -1;
    }
    if (threadIdx.x == 32) B.cut = 0xffffffffu;
}

/* Configurations: block b checks items b * per .. b * per + per - 1 (per <=
 * 32), one per lane. */
template <bool FAST>
__global__ void __launch_bounds__(SMALL_WARPS * 32, 4) k_configs_small(DevScene sc, const float* __restrict__ q, int n,
                                                                       long long offset, int per, int* __restrict__ res,
                                                                       int band_on, float band, Control* total)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SmallShared B;
    const SceneView S = small_view(sc, smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i0 = blockIdx.x * per, count = min(per, n - i0);
    small_reset(B);
    if (threadIdx.x == 0) B.full = B.checks = B.flips = B.open = 0u;
    for (int t = threadIdx.x; t < sc.ndof * 32; t += blockDim.x) {
        const int j = t >> 5, i = t & 31;
        if (i < count) B.q[j][i] = q[i0 + i + offset * j];
    }
    __syncthreads();
    /* check_boundaries(q) (robotconfigspace.cpp:795-802) */
    bool in = lane < count;
    if (in)
#pragma unroll 1
        for (int j = 0; j < sc.ndof; ++j) {
            const float x = B.q[j][lane];
            if (x < sc.mins[j] || x > sc.maxs[j]) in = false;
        }
    const unsigned valid = __ballot_sync(FULL_MASK, in);
    int code = lane < count && !in ? 1 : 0;
    bool want = false;
    if (valid) {
        if (warp == 0) {
            /* the other lanes repeat a valid one, so that the sweep balls hold no more */
            const int src = in ? lane : __ffs(valid) - 1;
            lane_fk<FAST, true, false>(sc, S, [&](int j) { return B.q[j][src]; });
            }
        small_pairs<FAST, CUT_NONE>(sc, S, B, valid, false, band_on, band, total);
        if (in) {
            const unsigned jk = B.jkey[lane];
            if (jk != 0xffffffffu) {
                code = (int)(jk & 15u) - 1;
                want = (jk & 16u) != 0u;
            } else {
                want = band_on && B.jfirst[lane] != 0x7fffffffu;
            }
        }
        unsigned todo = __ballot_sync(FULL_MASK, want);
        for (int w = 0; todo; ++w) {
            const int i = __ffs(todo) - 1;
            todo &= todo - 1u;
            if (w % SMALL_WARPS != warp) continue;
            const unsigned jk = B.jkey[i];
            const bool coll = jk != 0xffffffffu;
            const int lo = (int)min(B.jfirst[i], jk >> 8), hi = coll ? sc.npairs : B.jlast[i] + 1;
            const int c64 = warp_check64(sc, B.F[warp], B.L[warp], B.cen[warp], B.queue[warp],
                                         lane < sc.ndof ? B.q[lane][i] : 0.0f, lo, hi);
            if (lane == i) {
                atomicAdd(&B.checks, 1u);
                if ((c64 != 0) != (code != 0)) atomicAdd(&B.flips, 1u);
                res[i0 + i] = c64;
            }
        }
    }
    if (warp == 0 && lane < count && !want) res[i0 + lane] = code;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned done = (unsigned)__popc(valid);
        atomicAdd(&total->configs_exec, (unsigned long long)done);
        if (B.full) atomicAdd(&total->full_tests, (unsigned long long)B.full);
        if (B.checks) atomicAdd(&total->band_checks, (unsigned long long)B.checks);
        if (B.flips) atomicAdd(&total->band_flips, (unsigned long long)B.flips);
    }
}

/* Edges: block (e, s) of n * segs checks rounds s, s + segs, ... of edge e.
 * With segs > 1 scratch (2 n zeroed words) holds the edges' merged keys and
 * counts their finished blocks, the last of which writes the code and leaves
 * the words zeroed (a memset before a launch takes 4 us).  status:
 * gets GPRM_DEVFLAG_BAD_EDGE for a non-finite or oversized edge (or null). */
template <int POLICY, bool FAST>
__global__ void __launch_bounds__(SMALL_WARPS * 32, 4) k_edges_small(DevScene sc, const float* __restrict__ qs,
                                                                     const float* __restrict__ qe, int n,
                                                                     long long offset, float dq, int segs,
                                                                     int* __restrict__ res, unsigned* scratch,
                                                                     int band_on, float band, Control* total,
                                                                     volatile unsigned* status)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SmallShared B;
    const SceneView S = small_view(sc, smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s = blockIdx.x / n, e = blockIdx.x - s * n;   /* the edges' first rounds first */
    constexpr unsigned NONE = POLICY == EDGE_EARLY_EXIT ? 0xffffffffu : 0u;
    float ends = 0.0f;
    if ((lane & 15) < sc.ndof) ends = (lane < 16 ? qs : qe)[e + offset * (lane & 15)];
    /* edge_testnum */
    float norm = 0.0f;
#pragma unroll 1
    for (int j = 0; j < sc.ndof; ++j) {
        const float diff = __shfl_sync(FULL_MASK, ends, 16 + j) - __shfl_sync(FULL_MASK, ends, j);
        norm = norm + diff * diff;
    }
    const float x = __fsqrt_rn(norm) / dq;
    const int tn = x < 1.0e8f ? (int)x + 1 : -1;
    const int R = (tn + 31) >> 5;      /* no round for a rejected edge */
    if (s > 0 && s >= R) return;
    const int parts = min(segs, max(R, 1));   /* blocks that share the edge */
    if (threadIdx.x == 0) {
        B.key = NONE;
        B.full = B.checks = B.flips = B.open = 0u;
    }
    unsigned exec = 0;
#pragma unroll 1
    for (int r = s; r < R; r += segs) {
        if (parts > 1) {
            /* a decision that no step of this round or a later one improves on */
            if (threadIdx.x == 0) {
                unsigned kv = *(volatile unsigned*)&scratch[e];
                if (POLICY == EDGE_EARLY_EXIT) kv = ~kv;
                B.beaten = kv == NONE ? 0u
                    : (POLICY == EDGE_EARLY_EXIT) ? (kv >> 4) < (unsigned)(r * 32) : (int)(kv >> 4) - 1 > tn - 1 - r * 32;
            }
            __syncthreads();
            if (B.beaten) break;
        }
        int t;
        bool in;
        if (POLICY == EDGE_EARLY_EXIT) {
            const int last = (tn - 1 - r) / R;
            in = lane <= last;
            t = (in ? lane : last) * R + r;
        } else {
            t = tn - 1 - (r * 32 + lane);
            in = t >= 0;
            if (!in) t = 0;
        }
        const float c1 = (float)t / (float)(tn - 1), c2 = 1.0f - c1;   /* as edge_step_config */
        const unsigned valid = __ballot_sync(FULL_MASK, in);
        if (warp == 0) {
            lane_fk<FAST>(sc, S, [&](int j) {
                return c1 * __shfl_sync(FULL_MASK, ends, j) + c2 * __shfl_sync(FULL_MASK, ends, 16 + j);
            }, __popc(valid) >> 1);
            }
        exec += (unsigned)__popc(valid);
        /* settle the round as check_edge does; where the collision that the
           tests were cut by turned out to be decided by an earlier pair
           inside the band, go through the round again without the cut */
        unsigned jk;
        int code, L, jstar;
        bool oob;
#pragma unroll 1
        for (bool cutting = true;; cutting = false) {
            small_reset(B);
            small_pairs<FAST, POLICY == EDGE_EARLY_EXIT ? CUT_PAIR : CUT_LANE>(sc, S, B, valid, cutting, band_on, band,
                                                                              total);
            jk = B.jkey[lane];
            code = jk == 0xffffffffu ? 0 : (int)(jk & 15u) - 1;
            oob = in && code != 0 && !(jk & 16u);
            L = 32;
            jstar = 0x7fffffff;
            if (POLICY == EDGE_EARLY_EXIT)
                jstar = (int)__reduce_min_sync(FULL_MASK, oob ? jk >> 8 : 0x7fffffffu);
            const unsigned hits = __ballot_sync(FULL_MASK, oob && (POLICY != EDGE_EARLY_EXIT || (int)(jk >> 8) == jstar));
            if (hits) L = __ffs(hits) - 1;
            const unsigned stands = !hits ? 0xffffffffu : POLICY == EDGE_EARLY_EXIT ? (unsigned)jstar : (unsigned)L;
            if (!cutting || B.cut == stands) break;
            __syncthreads();
        }
        bool want = band_on && in && lane < L;
        if (code != 0) want = want && !oob && (POLICY != EDGE_EARLY_EXIT || (int)(jk >> 8) <= jstar);
        else want = want && B.jfirst[lane] != 0x7fffffffu &&
                    (POLICY != EDGE_EARLY_EXIT || L == 32 || jstar == sc.npairs - 1);
        if (warp == 0 && lane == L) {
            if (POLICY == EDGE_EARLY_EXIT) atomicMin(&B.key, early_key((unsigned)(r * 32 + lane), code));
            else atomicMax(&B.key, all_key(t, code));
        }
        unsigned todo = __ballot_sync(FULL_MASK, want);
        for (int w = 0; todo; ++w) {
            const int i = __ffs(todo) - 1;
            todo &= todo - 1u;
            if (w % SMALL_WARPS != warp) continue;
            const unsigned ik = B.jkey[i];
            const int lo = (int)min(B.jfirst[i], ik >> 8), hi = ik != 0xffffffffu ? sc.npairs : B.jlast[i] + 1;
            const float d1 = __shfl_sync(FULL_MASK, c1, i), d2 = __shfl_sync(FULL_MASK, c2, i);
            const float q = d1 * __shfl_sync(FULL_MASK, ends, lane & 15) + d2 * __shfl_sync(FULL_MASK, ends, 16 + (lane & 15));
            const int c64 = warp_check64(sc, B.F[warp], B.L[warp], B.cen[warp], B.queue[warp], q, lo, hi);
            if (lane == i) {
                atomicAdd(&B.checks, 1u);
                if ((c64 != 0) != (code != 0)) atomicAdd(&B.flips, 1u);
                if (c64 != 0) {
                    if (POLICY == EDGE_EARLY_EXIT) atomicMin(&B.key, early_key((unsigned)(r * 32 + i), c64));
                    else atomicMax(&B.key, all_key(t, c64));
                }
            }
        }
        __syncthreads();
        if (L < 32) break;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    unsigned key = B.key;
    bool write = true;
    if (parts > 1) {
        /* zeroed words: the larger is the better for both policies */
        if (key != NONE) atomicMax(&scratch[e], POLICY == EDGE_EARLY_EXIT ? ~key : key);
        __threadfence();
        write = atomicAdd(&scratch[n + e], 1u) == (unsigned)parts - 1u;
        if (write) {
            __threadfence();
            key = *(volatile unsigned*)&scratch[e];
            if (POLICY == EDGE_EARLY_EXIT) key = ~key;
            scratch[e] = scratch[n + e] = 0u;   /* for the next launch */
        }
    }
    if (write) res[e] = key == NONE ? 0 : (int)(key & 15u) - 1;
    if (s == 0) {
        if (tn >= 0) atomicAdd(&total->steps_nominal, (unsigned long long)tn);
        else {
            atomicOr(&total->flags, GPRM_DEVFLAG_BAD_EDGE);
            if (status) *status = GPRM_DEVFLAG_BAD_EDGE;
        }
    }
    if (exec) atomicAdd(&total->steps_exec, (unsigned long long)exec);
    if (B.full) atomicAdd(&total->full_tests, (unsigned long long)B.full);
    if (B.checks) atomicAdd(&total->band_checks, (unsigned long long)B.checks);
    if (B.flips) atomicAdd(&total->band_flips, (unsigned long long)B.flips);
}

/* Marks (SCAN_SETTLED) the pairs whose polytopes are both in frame 0 and
 * whose certificate holds: it is the same for every configuration, so the
 * checks need not evaluate it again.  A robot with a base link has one such
 * pair per obstacle (512 of 4117 pairs of the 7-DOF wall scene); evaluating
 * them lane by lane, without slots and hence past the sweep tests, took
 * 72 % of an edge round there (570,000 of 790,000 cycles): 70,001 roadmap
 * edges 135.0 -> 43.0 ms, a vertex check of 100,003 configurations 8.8 ->
 * 8.2 ms. */
__global__ void k_static_pairs(DevScene sc, int4* __restrict__ scan_c)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= sc.npairs) return;
    const int4 c = scan_c[j];
    const int4 pr = sc.pairs[j];
    if (c.w == SCAN_USABLE || pr.z != 0 || pr.w != 0) return;
    const float4 pb = sc.pairs_b[j];
    const float4 p = sc.tab[pr.x], a = sc.tab[pr.x + 1], q = sc.tab[pr.y], b = sc.tab[pr.y + 1];
    /* no frame is read: both polytopes are untransformed */
    if (points_certified(sc, nullptr, c, pb.y, pb.x, {p.x, p.y, p.z}, {q.x, q.y, q.z}, {a.x, a.y, a.z}, {b.x, b.y, b.z}))
        scan_c[j].w = SCAN_SETTLED;
}

/* ------------------------------------------------------------------ */
/* launchers                                                            */
/* ------------------------------------------------------------------ */

cudaError_t launch_static_pairs(const DevScene& sc, cudaStream_t st)
{
    if (sc.npairs < 1) return cudaSuccess;
    k_static_pairs<<<(sc.npairs + 127) / 128, 128, 0, st>>>(sc, const_cast<int4*>(sc.scan_c));
    return cudaGetLastError();
}

/* The dynamic shared-memory cap is an attribute of the kernel, shared by
 * every handle in the process: it is opened to the device's opt-in limit
 * (less the kernel's static shared memory), so that configuring one handle
 * never shrinks what another handle launches with.  Fails when `need`
 * bytes do not fit. */
static cudaError_t open_smem_cap(const void* fn, int optin, size_t need)
{
    cudaFuncAttributes fa;
    cudaError_t err = cudaFuncGetAttributes(&fa, fn);
    if (err != cudaSuccess) return err;
    const int cap = optin - (int)fa.sharedSizeBytes;
    if (cap < 0 || need > (size_t)cap) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
}

/* Occupancy of one FP32 kernel variant, in resident warps per SM. */
static cudaError_t variant_warps(const void* fn, int threads, size_t smem, int* warps_per_sm)
{
    int per_sm = 0;
    cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
    *warps_per_sm = per_sm * (threads / 32);
    return err;
}

template <bool FAST>
static const void* kernel_fn_t(int vertex_kernel, bool smem, int policy, bool split)
{
    if (vertex_kernel) return smem ? (const void*)k_check_configs<true, FAST> : (const void*)k_check_configs<false, FAST>;
    if (split) {
        if (policy == EDGE_EARLY_EXIT)
            return smem ? (const void*)k_check_edges<true, EDGE_EARLY_EXIT, true, FAST>
                        : (const void*)k_check_edges<false, EDGE_EARLY_EXIT, true, FAST>;
        return smem ? (const void*)k_check_edges<true, EDGE_ALL_STEPS, true, FAST>
                    : (const void*)k_check_edges<false, EDGE_ALL_STEPS, true, FAST>;
    }
    if (policy == EDGE_EARLY_EXIT)
        return smem ? (const void*)k_check_edges<true, EDGE_EARLY_EXIT, false, FAST>
                    : (const void*)k_check_edges<false, EDGE_EARLY_EXIT, false, FAST>;
    return smem ? (const void*)k_check_edges<true, EDGE_ALL_STEPS, false, FAST>
                : (const void*)k_check_edges<false, EDGE_ALL_STEPS, false, FAST>;
}

static const void* kernel_fn(int vertex_kernel, bool smem, int policy, bool split = false, bool fast = false)
{
    return fast ? kernel_fn_t<true>(vertex_kernel, smem, policy, split)
                : kernel_fn_t<false>(vertex_kernel, smem, policy, split);
}

/* Sets a kernel's preferred shared-memory carveout (percent of the SM's
 * maximum; -1 restores the default) when it differs from the value last
 * set for it, so that every launch runs with its own handle's split of the
 * SM's L1 and shared memory. */
static cudaError_t apply_carveout(const void* fn, int pct)
{
    static std::mutex mu;
    static std::unordered_map<const void*, int> last;
    std::lock_guard<std::mutex> lock(mu);
    auto it = last.find(fn);
    const int cur = it == last.end() ? -1 : it->second;
    if (cur == pct) return cudaSuccess;
    cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
    if (err == cudaSuccess) last[fn] = pct;
    return err;
}

cudaError_t configure_launch(const DevScene& sc, int vertex_kernel, int threads, int scene_in_smem,
                             LaunchCfg* cfg, int blocks_cap)
{
    int dev = 0, sms = 0, optin = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    size_t smem = frame_smem_bytes(sc, threads, vertex_kernel != 0) + (scene_in_smem ? scene_smem_bytes(sc) : 0);
    for (int pol = 0; pol < (vertex_kernel ? 1 : 2); ++pol)
        for (int split = 0; split < (vertex_kernel ? 1 : 2); ++split)
            for (int fast = 0; fast < 2; ++fast) {
                err = open_smem_cap(kernel_fn(vertex_kernel, scene_in_smem != 0, pol, split != 0, fast != 0), optin,
                                    smem);
                if (err != cudaSuccess) return err;
            }
    /* occupancy of the slower-to-fit of the two arithmetic variants, with
       the default carveout */
    for (int pol = 0; pol < (vertex_kernel ? 1 : 2); ++pol)
        for (int split = 0; split < (vertex_kernel ? 1 : 2); ++split)
            for (int fast = 0; fast < 2; ++fast) {
                err = apply_carveout(kernel_fn(vertex_kernel, scene_in_smem != 0, pol, split != 0, fast != 0), -1);
                if (err != cudaSuccess) return err;
            }
    int warps = 0, warps_fast = 0;
    err = variant_warps(kernel_fn(vertex_kernel, scene_in_smem != 0, 0), threads, smem, &warps);
    if (err != cudaSuccess) return err;
    err = variant_warps(kernel_fn(vertex_kernel, scene_in_smem != 0, 0, false, true), threads, smem, &warps_fast);
    if (err != cudaSuccess) return err;
    if (warps_fast < warps) warps = warps_fast;
    if (warps < 1) return cudaErrorInvalidConfiguration;
    int per_sm = warps / (threads / 32);
    int carveout = -1;
    if (blocks_cap > 0 && blocks_cap < per_sm) {
        /* fewer resident blocks: a carveout just large enough for them (each
           block also reserves 1 KB), the rest of the SM's combined L1 and
           shared memory left to L1 */
        int smem_sm = 0;
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        per_sm = blocks_cap;
        const double need = (double)per_sm * (double)(smem + 1024);
        carveout = smem_sm > 0 ? (int)ceil(100.0 * need / smem_sm) : -1;
        if (carveout > 100) carveout = 100;
    }
    cfg->threads = threads;
    cfg->smem_bytes = smem;
    cfg->scene_in_smem = scene_in_smem;
    cfg->blocks = sms * per_sm;
    cfg->blocks_per_sm = per_sm;
    cfg->warps_per_sm = per_sm * (threads / 32);
    cfg->carveout = carveout;
    return cudaSuccess;
}

cudaError_t plan_launch(const DevScene& sc, int vertex_kernel, int threads, LaunchCfg* cfg)
{
    /* default: the variant with the most resident warps, the scene in shared
       memory on ties (the autotuner times the candidates instead).  Blocks
       smaller than four warps never hold more: without the slots' points 16
       warps fit for seven joints too. */
    LaunchCfg best{};
    int best_w = -1;
    const int cand_threads[4] = {threads, 256, 384, 512};
    for (int ci = 0; ci < 4; ++ci)
        for (int sm = 1; sm >= 0; --sm) {
            LaunchCfg c{};
            if (configure_launch(sc, vertex_kernel, cand_threads[ci], sm, &c) != cudaSuccess) {
                cudaGetLastError();
                continue;
            }
            if (c.warps_per_sm > best_w) { best = c; best_w = c.warps_per_sm; }
        }
    if (best_w < 0) return cudaErrorInvalidConfiguration;
    /* re-apply the chosen variant's shared-memory attribute */
    cudaError_t err = configure_launch(sc, vertex_kernel, best.threads, best.scene_in_smem, cfg);
    return err;
}

cudaError_t launch_check_configs(const DevScene& sc, const LaunchCfg& cfg, const float* q, long long n,
                                 long long offset, int* res, int band_on, float band, BandQueue bq, Control* ctl,
                                 cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    {
        cudaError_t err = apply_carveout(kernel_fn(1, cfg.scene_in_smem != 0, 0, false, sc.fast != 0), cfg.carveout);
        if (err != cudaSuccess) return err;
    }
#define GPRM_CFG_LAUNCH(SM_, FAST_)                                                                            \
    k_check_configs<SM_, FAST_><<<cfg.blocks, cfg.threads, cfg.smem_bytes, st>>>(sc, q, n, offset, res, band_on, \
                                                                                band, bq, ctl)
    if (cfg.scene_in_smem) { if (sc.fast) GPRM_CFG_LAUNCH(true, true); else GPRM_CFG_LAUNCH(true, false); }
    else { if (sc.fast) GPRM_CFG_LAUNCH(false, true); else GPRM_CFG_LAUNCH(false, false); }
#undef GPRM_CFG_LAUNCH
    return cudaGetLastError();
}

cudaError_t launch_check_edges(const DevScene& sc, const LaunchCfg& cfg, const float* qs, const float* qe,
                               long long n, long long offset, float dq, int policy, unsigned* key,
                               int band_on, float band, BandQueue bq, Control* ctl,
                               cudaStream_t st, unsigned* seg_off, int seg_rounds)
{
    if (n <= 0) return cudaSuccess;
    if (seg_off && (seg_rounds < 1 || n > EDGE_SPLIT_MAX)) return cudaErrorInvalidValue;
    if (seg_off) {
        if (n <= EDGE_SPLIT_ONE_BLOCK) {
            k_edge_segments<<<1, 1024, 0, st>>>(qs, qe, n, offset, sc.ndof, dq, seg_rounds, seg_off);
        } else {
            static_assert(EDGE_SEG_BLOCKS <= 1024, "one block scans the block sums");
            unsigned* bsum = seg_off + n + 1;   /* EDGE_SEG_BLOCKS words after the offsets */
            k_seg_pass<0><<<EDGE_SEG_BLOCKS, 256, 0, st>>>(qs, qe, n, offset, sc.ndof, dq, seg_rounds, seg_off, bsum);
            k_seg_scan_blocks<<<1, 1024, 0, st>>>(bsum, EDGE_SEG_BLOCKS, seg_off + n);
            k_seg_pass<1><<<EDGE_SEG_BLOCKS, 256, 0, st>>>(qs, qe, n, offset, sc.ndof, dq, seg_rounds, seg_off, bsum);
        }
        cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) return err;
    }
    size_t sm = cfg.smem_bytes;
    {
        cudaError_t err = apply_carveout(kernel_fn(0, cfg.scene_in_smem != 0, policy, seg_off != nullptr, sc.fast != 0),
                                         cfg.carveout);
        if (err != cudaSuccess) return err;
    }
#define GPRM_EDGE_LAUNCH2(SM_, POL_, SPLIT_, FAST_)                                                           \
    k_check_edges<SM_, POL_, SPLIT_, FAST_><<<cfg.blocks, cfg.threads, sm, st>>>(                                 \
        sc, qs, qe, n, offset, dq, key, band_on, band, bq, ctl, seg_off, seg_rounds)
#define GPRM_EDGE_LAUNCH(SM_, POL_, SPLIT_)                                                                   \
    do { if (sc.fast) GPRM_EDGE_LAUNCH2(SM_, POL_, SPLIT_, true); else GPRM_EDGE_LAUNCH2(SM_, POL_, SPLIT_, false); } \
    while (0)
    const bool split = seg_off != nullptr;
    if (policy == EDGE_EARLY_EXIT) {
        if (cfg.scene_in_smem) { if (split) GPRM_EDGE_LAUNCH(true, EDGE_EARLY_EXIT, true); else GPRM_EDGE_LAUNCH(true, EDGE_EARLY_EXIT, false); }
        else { if (split) GPRM_EDGE_LAUNCH(false, EDGE_EARLY_EXIT, true); else GPRM_EDGE_LAUNCH(false, EDGE_EARLY_EXIT, false); }
    } else {
        if (cfg.scene_in_smem) { if (split) GPRM_EDGE_LAUNCH(true, EDGE_ALL_STEPS, true); else GPRM_EDGE_LAUNCH(true, EDGE_ALL_STEPS, false); }
        else { if (split) GPRM_EDGE_LAUNCH(false, EDGE_ALL_STEPS, true); else GPRM_EDGE_LAUNCH(false, EDGE_ALL_STEPS, false); }
    }
#undef GPRM_EDGE_LAUNCH
#undef GPRM_EDGE_LAUNCH2
    return cudaGetLastError();
}

cudaError_t launch_recheck(const DevScene& sc, int blocks, int kind, const float* q, const float* qs,
                           const float* qe, long long offset, float dq, int policy, int* res, unsigned* key,
                           BandQueue bq, Control* ctl, cudaStream_t st)
{
    k_recheck<<<blocks, RECHECK_THREADS, 0, st>>>(sc, kind, q, qs, qe, offset, dq, policy, res, key, bq, ctl);
    return cudaGetLastError();
}

cudaError_t launch_overflow(const DevScene& sc, int blocks, int kind, const float* q, const float* qs,
                            const float* qe, long long offset, float dq, int policy, float band, int* res,
                            unsigned* key, BandQueue bq, Control* ctl, cudaStream_t st)
{
    if (!bq.ovf) return cudaSuccess;
    if (sc.fast)
        k_overflow<true><<<blocks, 128, 0, st>>>(sc, kind, q, qs, qe, offset, dq, policy, band, res, key, bq, ctl);
    else
        k_overflow<false><<<blocks, 128, 0, st>>>(sc, kind, q, qs, qe, offset, dq, policy, band, res, key, bq, ctl);
    return cudaGetLastError();
}

cudaError_t launch_finalize_edges(long long n, int policy, const unsigned* key, int* res, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    long long b = (n + 255) / 256;
    if (b > 4096) b = 4096;
    k_finalize_edges<<<(int)b, 256, 0, st>>>(n, policy, key, res);
    return cudaGetLastError();
}


/* Opens the dynamic shared-memory cap of the small-request kernels for the
 * scene's frames; *bytes gets one block's, 0 where they do not fit. */
cudaError_t configure_small(const DevScene& sc, size_t* bytes)
{
    *bytes = 0;
    int dev = 0, optin = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const size_t need = lane_floats(sc, false) * 32 * sizeof(float);
    const void* fns[6] = {(const void*)k_configs_small<false>, (const void*)k_configs_small<true>,
                          (const void*)k_edges_small<EDGE_ALL_STEPS, false>,
                          (const void*)k_edges_small<EDGE_ALL_STEPS, true>,
                          (const void*)k_edges_small<EDGE_EARLY_EXIT, false>,
                          (const void*)k_edges_small<EDGE_EARLY_EXIT, true>};
    for (const void* fn : fns) {
        err = open_smem_cap(fn, optin, need);
        if (err != cudaSuccess) {
            cudaGetLastError();
            return err == cudaErrorInvalidValue ? cudaSuccess : err;
        }
    }
    *bytes = need;
    return cudaSuccess;
}

cudaError_t launch_configs_small(const DevScene& sc, size_t smem, const float* q, int n, long long offset, int per,
                                 int* res, int band_on, float band, Control* total, cudaStream_t st)
{
    const int blocks = (int)(((long long)n + per - 1) / per);
    if (sc.fast)
        k_configs_small<true><<<blocks, SMALL_WARPS * 32, smem, st>>>(sc, q, n, offset, per, res, band_on, band, total);
    else
        k_configs_small<false><<<blocks, SMALL_WARPS * 32, smem, st>>>(sc, q, n, offset, per, res, band_on, band, total);
    return cudaGetLastError();
}

cudaError_t launch_edges_small(const DevScene& sc, size_t smem, const float* qs, const float* qe, int n, long long offset,
                               float dq, int policy, int segs, int* res, unsigned* scratch, int band_on, float band,
                               Control* total, unsigned* status, cudaStream_t st)
{
#define GPRM_SMALL_LAUNCH(POL_, FAST_)                                                                            \
    k_edges_small<POL_, FAST_><<<n * segs, SMALL_WARPS * 32, smem, st>>>(sc, qs, qe, n, offset, dq, segs, res, scratch, \
                                                                        band_on, band, total, status)
    if (policy == EDGE_EARLY_EXIT) { if (sc.fast) GPRM_SMALL_LAUNCH(EDGE_EARLY_EXIT, true); else GPRM_SMALL_LAUNCH(EDGE_EARLY_EXIT, false); }
    else { if (sc.fast) GPRM_SMALL_LAUNCH(EDGE_ALL_STEPS, true); else GPRM_SMALL_LAUNCH(EDGE_ALL_STEPS, false); }
#undef GPRM_SMALL_LAUNCH
    return cudaGetLastError();
}

/* ------------------------------------------------------------------ */
/* many problems in one launch                                          */
/* ------------------------------------------------------------------ */

/* shared bytes of one warp's cached scene descriptor */
constexpr int SCENE_CACHE_BYTES = (int)((sizeof(DevScene) + 15) / 16 * 16);

/* Problem of item `it`: the p with offs[p] <= it < offs[p+1]. */
__device__ __forceinline__ int problem_of(const BatchView& B, long long it)
{
    int lo = 0, hi = B.S;   /* offs[lo] <= it < offs[hi] */
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (B.offs[mid] <= it) lo = mid;
        else hi = mid;
    }
    return lo;
}

/* Range of work item w of the shared edge launch: the k with
 * woffs[k] <= w < woffs[k+1]. */
__device__ __forceinline__ int range_of(const BatchView& B, long long w)
{
    int lo = 0, hi = B.K;
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (B.woffs[mid] <= w) lo = mid;
        else hi = mid;
    }
    return lo;
}

/* Makes problem p's descriptor the warp's current scene (warp-uniform p). */
template <bool VERTEX>
__device__ __forceinline__ void switch_scene(const BatchView& B, int p, DevScene* wsc, float* frames, SceneView& S)
{
    __syncwarp();
    const unsigned* src = reinterpret_cast<const unsigned*>(B.scenes + p);
    unsigned* dst = reinterpret_cast<unsigned*>(wsc);
    for (int k = threadIdx.x & 31; k < (int)(sizeof(DevScene) / 4); k += 32) dst[k] = src[k];
    __syncwarp();
    S.tab = wsc->tab;
    S.pairs = wsc->pairs;
    S.far = wsc->far;
    S.scan_c = wsc->scan_c;
    S.scan_b = wsc->scan_b;
    S.frames = frames;
    S.sweep = sweep_area<VERTEX>(*wsc, frames);
    S.bits = open_area<VERTEX>(*wsc, frames);
}

template <bool FAST>
__global__ void GPRM_BOUNDS k_check_configs_multi(BatchView B, const float* __restrict__ q, long long offset,
                                                  int* __restrict__ res, int band_on, float band,
                                                  BandQueue bq, Control* ctl)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    DevScene* wsc = reinterpret_cast<DevScene*>(smem + warp * SCENE_CACHE_BYTES);
    float* frames = reinterpret_cast<float*>(smem + nw * SCENE_CACHE_BYTES) + (size_t)warp * B.lane_floats * 32 + lane;
    SceneView S;
    int cur = -1;
    unsigned long long exec = 0;
    PairCounts pc = {0, 0};
    for (;;) {
        unsigned long long c = 0;
        if (lane == 0) c = atomicAdd(&ctl->next, 1ull);
        c = __shfl_sync(FULL_MASK, c, 0);
        if (c >= (unsigned long long)B.nwork) break;
        const int4 ch = B.chunks[c];
        if (ch.x != cur) { switch_scene<true>(B, ch.x, wsc, frames, S); cur = ch.x; }
        check_config_chunk<FAST>(*wsc, S, q, offset, (long long)ch.y, ch.z, res, band_on, band, bq, ctl, pc,
                                 exec);
    }
    exec = warp_sum(exec);
    if (lane == 0 && exec) atomicAdd(&ctl->configs_exec, exec);
    flush_counts(pc, ctl);
}

template <int POLICY, bool FAST>
__global__ void GPRM_BOUNDS k_check_edges_multi(BatchView B, const float* __restrict__ qs, const float* __restrict__ qe,
                                                long long offset, unsigned* __restrict__ key, int band_on, float band,
                                                BandQueue bq, Control* ctl)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    DevScene* wsc = reinterpret_cast<DevScene*>(smem + warp * SCENE_CACHE_BYTES);
    float* frames = reinterpret_cast<float*>(smem + nw * SCENE_CACHE_BYTES) + (size_t)warp * B.lane_floats * 32 + lane;
    SceneView S;
    int cur = -1;
    unsigned long long exec = 0, nominal = 0;
    PairCounts pc = {0, 0};
    for (;;) {
        unsigned long long eu = 0;
        if (lane == 0) eu = atomicAdd(&ctl->next, 1ull);
        eu = __shfl_sync(FULL_MASK, eu, 0);
        if (eu >= (unsigned long long)B.nwork) break;
        const int k = range_of(B, (long long)eu);
        const int p = B.wprob[k];
        const long long e = B.wbase[k] + ((long long)eu - B.woffs[k]);
        if (p != cur) { switch_scene<false>(B, p, wsc, frames, S); cur = p; }
        check_edge<POLICY, false, FAST>(*wsc, S, qs, qe, e, offset, wsc->dq, key, band_on, band, bq, ctl,
                                        pc, exec, nominal);
    }
    flush_edge_counts(exec, nominal, pc, ctl);
}

__global__ void __launch_bounds__(RECHECK_THREADS) k_recheck_multi(BatchView B, int kind,
                                                                   const float* __restrict__ q,
                                                                   const float* __restrict__ qs,
                                                                   const float* __restrict__ qe, long long offset,
                                                                   int policy, int* __restrict__ res,
                                                                   unsigned* __restrict__ key, BandQueue bq,
                                                                   Control* ctl)
{
    unsigned cnt = ctl->qcount;
    if (cnt > bq.cap) cnt = bq.cap;
    unsigned long long checks = 0, flips = 0;
    __shared__ Warp64 W[RECHECK_THREADS / 32];
    const unsigned warps = gridDim.x * (RECHECK_THREADS / 32), warp = threadIdx.x >> 5;
    if (recheck_by_warp(cnt, warps, 0)) {   /* the problems' pair lists differ: as for a short one */
        for (unsigned idx = warp * gridDim.x + blockIdx.x; idx < cnt; idx += warps) {
            const uint2 it = bq.items[idx];
            const DevScene& sc = B.scenes[problem_of(B, (long long)it.x)];
            recheck_item_warp(sc, kind, it, q, qs, qe, offset, sc.dq, policy, res, key, checks, flips,
                              recheck_span(bq, idx, sc.npairs), W[warp]);
        }
        cnt = 0;
    }
    for (unsigned idx = blockIdx.x * blockDim.x + threadIdx.x; idx < cnt; idx += gridDim.x * blockDim.x) {
        const uint2 it = bq.items[idx];
        const DevScene& sc = B.scenes[problem_of(B, (long long)it.x)];
        recheck_item(sc, kind, it, q, qs, qe, offset, sc.dq, policy, res, key, checks, flips,
                     recheck_span(bq, idx, sc.npairs));
    }
    if (checks) atomicAdd(&ctl->band_checks, checks);
    if (flips) atomicAdd(&ctl->band_flips, flips);
}

/* The overflow pass over many problems: each item's problem by binary
 * search over the layout's offsets. */
template <bool FAST>
__global__ void __launch_bounds__(128) k_overflow_multi(BatchView B, int kind, const float* __restrict__ q,
                                                        const float* __restrict__ qs, const float* __restrict__ qe,
                                                        long long offset, int policy, float band,
                                                        int* __restrict__ res, unsigned* __restrict__ key,
                                                        BandQueue bq, Control* ctl)
{
    const unsigned long long cnt = ctl->ovf_count;
    if (cnt == 0 || !bq.ovf) return;
    unsigned long long checks = 0, flips = 0;
    for (unsigned long long idx = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; idx < cnt;
         idx += (unsigned long long)gridDim.x * blockDim.x) {
        const unsigned x = bq.ovf[idx];
        const DevScene& sc = B.scenes[problem_of(B, (long long)x)];
        overflow_item<FAST>(sc, kind, x, q, qs, qe, offset, sc.dq, policy, band, res, key, checks, flips);
    }
    if (checks) atomicAdd(&ctl->band_checks, checks);
    if (flips) atomicAdd(&ctl->band_flips, flips);
}

cudaError_t launch_overflow_multi(const BatchView& B, int blocks, int kind, const float* q, const float* qs,
                                  const float* qe, long long offset, int policy, float band, int* res, unsigned* key,
                                  BandQueue bq, Control* ctl, cudaStream_t st)
{
    if (!bq.ovf) return cudaSuccess;
    if (B.fast)
        k_overflow_multi<true><<<blocks, 128, 0, st>>>(B, kind, q, qs, qe, offset, policy, band, res, key, bq, ctl);
    else
        k_overflow_multi<false><<<blocks, 128, 0, st>>>(B, kind, q, qs, qe, offset, policy, band, res, key, bq, ctl);
    return cudaGetLastError();
}

static const void* batch_kernel_fn(int vertex_kernel, int policy, bool fast)
{
    if (vertex_kernel) return fast ? (const void*)k_check_configs_multi<true> : (const void*)k_check_configs_multi<false>;
    if (fast)
        return policy == EDGE_EARLY_EXIT ? (const void*)k_check_edges_multi<EDGE_EARLY_EXIT, true>
                                         : (const void*)k_check_edges_multi<EDGE_ALL_STEPS, true>;
    return policy == EDGE_EARLY_EXIT ? (const void*)k_check_edges_multi<EDGE_EARLY_EXIT, false>
                                     : (const void*)k_check_edges_multi<EDGE_ALL_STEPS, false>;
}

cudaError_t configure_batch_launch(const BatchView& B, int vertex_kernel, int threads, LaunchCfg* cfg,
                                   int blocks_cap)
{
    int dev = 0, sms = 0, optin = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const int nw = threads / 32;
    size_t smem = (size_t)nw * SCENE_CACHE_BYTES + (size_t)nw * B.lane_floats * 32 * sizeof(float);
    for (int pol = 0; pol < (vertex_kernel ? 1 : 2); ++pol) {
        err = open_smem_cap(batch_kernel_fn(vertex_kernel, pol, B.fast != 0), optin, smem);
        if (err != cudaSuccess) return err;
    }
    int warps = 0;
    err = variant_warps(batch_kernel_fn(vertex_kernel, 0, B.fast != 0), threads, smem, &warps);
    if (err != cudaSuccess) return err;
    if (warps < 1) return cudaErrorInvalidConfiguration;
    int per_sm = warps / nw;
    int carveout = -1;
    if (blocks_cap > 0 && blocks_cap < per_sm) {
        int smem_sm = 0;
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        per_sm = blocks_cap;
        const double need = (double)per_sm * (double)(smem + 1024);
        carveout = smem_sm > 0 ? (int)ceil(100.0 * need / smem_sm) : -1;
        if (carveout > 100) carveout = 100;
    }
    cfg->threads = threads;
    cfg->smem_bytes = smem;
    cfg->scene_in_smem = 0;
    cfg->blocks = sms * per_sm;
    cfg->warps_per_sm = per_sm * nw;
    cfg->blocks_per_sm = per_sm;
    cfg->carveout = carveout;
    return cudaSuccess;
}

/* Launches a persistent batch kernel with the configuration's grid and,
 * when it caps the resident blocks, its carveout as a launch attribute
 * (kept by a captured graph's kernel node). */
template <typename... KArgs, typename... Args>
static cudaError_t launch_multi(void (*kernel)(KArgs...), const LaunchCfg& cfg, cudaStream_t st, Args... args)
{
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)cfg.blocks);
    lc.blockDim = dim3((unsigned)cfg.threads);
    lc.dynamicSmemBytes = cfg.smem_bytes;
    lc.stream = st;
    cudaLaunchAttribute at[1];
    if (cfg.carveout >= 0) {
        at[0].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        at[0].val.sharedMemCarveout = (unsigned)cfg.carveout;
        lc.attrs = at;
        lc.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&lc, kernel, args...);
}

cudaError_t launch_check_configs_multi(const BatchView& B, const LaunchCfg& cfg, const float* q, long long offset,
                                       int* res, int band_on, float band, BandQueue bq, Control* ctl,
                                       cudaStream_t st)
{
    if (B.nwork <= 0) return cudaSuccess;
    if (B.fast) return launch_multi(k_check_configs_multi<true>, cfg, st, B, q, offset, res, band_on, band, bq, ctl);
    return launch_multi(k_check_configs_multi<false>, cfg, st, B, q, offset, res, band_on, band, bq, ctl);
}

cudaError_t launch_check_edges_multi(const BatchView& B, const LaunchCfg& cfg, const float* qs, const float* qe,
                                     long long offset, int policy, unsigned* key, int band_on, float band,
                                     BandQueue bq, Control* ctl, cudaStream_t st)
{
    if (B.nwork <= 0) return cudaSuccess;
    if (policy == EDGE_EARLY_EXIT)
        return B.fast ? launch_multi(k_check_edges_multi<EDGE_EARLY_EXIT, true>, cfg, st, B, qs, qe, offset, key,
                                     band_on, band, bq, ctl)
                      : launch_multi(k_check_edges_multi<EDGE_EARLY_EXIT, false>, cfg, st, B, qs, qe, offset, key,
                                     band_on, band, bq, ctl);
    return B.fast ? launch_multi(k_check_edges_multi<EDGE_ALL_STEPS, true>, cfg, st, B, qs, qe, offset, key, band_on,
                                 band, bq, ctl)
                  : launch_multi(k_check_edges_multi<EDGE_ALL_STEPS, false>, cfg, st, B, qs, qe, offset, key, band_on,
                                 band, bq, ctl);
}

cudaError_t launch_recheck_multi(const BatchView& B, int blocks, int kind, const float* q, const float* qs,
                                 const float* qe, long long offset, int policy, int* res, unsigned* key,
                                 BandQueue bq, Control* ctl, cudaStream_t st)
{
    k_recheck_multi<<<blocks, RECHECK_THREADS, 0, st>>>(B, kind, q, qs, qe, offset, policy, res, key, bq, ctl);
    return cudaGetLastError();
}

/* Adds a request's counters to the handle's running totals. */
__global__ void k_accumulate(const Control* c, Control* total)
{
    /* atomics: requests on different streams accumulate concurrently */
    atomicAdd(&total->steps_nominal, c->steps_nominal);
    atomicAdd(&total->steps_exec, c->steps_exec);
    atomicAdd(&total->band_checks, c->band_checks);
    atomicAdd(&total->band_flips, c->band_flips);
    atomicAdd(&total->configs_exec, c->configs_exec);
    atomicAdd(&total->certified, c->certified);
    atomicAdd(&total->full_tests, c->full_tests);
    atomicAdd(&total->ovf_count, c->ovf_count);
    atomicOr(&total->flags, c->flags);
    atomicAdd(&total->next, 1ull);  /* requests completed */
}

cudaError_t launch_accumulate(const Control* c, Control* total, cudaStream_t st)
{
    k_accumulate<<<1, 1, 0, st>>>(c, total);
    return cudaGetLastError();
}

__global__ void k_fma_probe(int iters, float* out)
{
    float x[GPRM_FMA_PROBE_CHAINS];
    const float a = 1.0000001f, b = -0.9999999f;
#pragma unroll
    for (int c = 0; c < GPRM_FMA_PROBE_CHAINS; ++c) x[c] = (float)(threadIdx.x + c);
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int c = 0; c < GPRM_FMA_PROBE_CHAINS; ++c) x[c] = __fmaf_rn(x[c], a, b);
    }
    float s = 0.0f;
#pragma unroll
    for (int c = 0; c < GPRM_FMA_PROBE_CHAINS; ++c) s += x[c];
    out[(blockIdx.x * blockDim.x + threadIdx.x) & (1024 * 1024 - 1)] = s;
}

cudaError_t launch_fma_probe(int blocks, int threads, int iters, float* out, cudaStream_t st)
{
    k_fma_probe<<<blocks, threads, 0, st>>>(iters, out);
    return cudaGetLastError();
}

cudaError_t launch_fk_probe(const DevScene& sc, const float* q, float* out, cudaStream_t st)
{
    k_fk_probe<<<1, 1, 0, st>>>(sc, q, out);
    return cudaGetLastError();
}

}  // namespace gprm
