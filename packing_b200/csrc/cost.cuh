// cost.cuh -- batched tree-pair + boundary cost and gradient.
//
// One CTA evaluates one packing (instance).  Work per instance:
//   phase 0  thread per tree: pose -> (x, y, cos, sin), piece AABBs relative to
//            the tree centre, and the boundary term (pack_cuda.py:550-642).
//   phase A  every unordered pair {i, j} once (not both orders as the
//            reference's 2-threads-per-ref-tree loop does, pack_cuda.py:404-464),
//            centre cull at (2R)^2, then the 16 piece-pair AABB tests; the
//            surviving piece pairs are appended to a shared-memory work list
//            (warp ballot + one shared atomic per warp).
//   phase B  thread per listed piece pair: intersection area (or SAT
//            penetration) with the gradient of BOTH trees' poses, added into
//            per-tree int64 fixed-point accumulators (order-independent, so
//            deterministic), flushed whenever the list fills.
//   phase C  per-tree gradients out; totals by fixed-order reductions.
// Coordinates are taken relative to tree i's centre so the clipper works on
// O(1) numbers whatever the packing's extent.
#pragma once
#include "common.cuh"
#include "geometry.cuh"

#include <atomic>
#include <mutex>

struct PkCostSmem {
    float4* pose;       // [n_max] x, y, cos, sin
    float* theta;       // [n_max]
    float4* aabb;       // [4*n_max] per piece: minx, maxx, miny, maxy (centre-relative)
    unsigned* acc_lo;   // [3*n_max] fixed-point gradient, low words
    unsigned* acc_hi;   // [3*n_max] fixed-point gradient, high words
    float4* bnd;        // [n_max] boundary: cost, dh0, dh1, dh2 (unweighted)
    uint16_t* items;    // [cap_items] piece pairs: near list index | pi << 11 | pj << 13
    uint32_t* near;     // [cap_near] centre-culled pairs: i | j << 11
    int* count;         // [2] items reserved in the list; first reservation that did not fit (its base)
    double* red;        // [32]
    long long* redl;    // [32]
    float2* piece;      // [16]
    float4* piece4;     // [8] per piece: (x0, x1, x2, x3), (y0, y1, y2, y3)
    int* piece_nv;      // [4]
    unsigned int* cnt;  // [4] candidate pairs tested, near pairs, piece pairs, evaluations; then
                        // [4] kept near list: state (-1 off, 0 build next, 1 valid), length,
                        // filter flag, list distance (pk_nlist)
    int* cell_start;    // [grid_cap + 1] first sorted slot of each grid cell
    int* cell_fill;     // [grid_cap] trees per cell, then a scratch cursor
    int* sorted;        // [n_max] tree indices ordered by cell
    int* tcell;         // [n_max] cell of each tree
    int* near_cnt;      // [n_max] near pairs of each sorted position
    int* near_start;    // [n_max + 1] their offsets (exclusive scan)
    int cap_items, cap_near, grid_cap, n_cap;
};

// Cells of the broad-phase grid (each at least the interaction distance
// wide): two per tree, at least 64, at most 1024.
__host__ __device__ inline int pk_grid_cap(int n_max) { return n_max < 32 ? 64 : (n_max > 512 ? 1024 : 2 * n_max); }

// List capacities.  The near list takes 8 T pairs (2048 at most: an item names
// its pair by an 11-bit index), at least the n_max - 1 pairs of one tree for
// every n_max that pk_cost_threads gives T for.  Each warp reserves room in the
// item list for the piece pairs of 32 near pairs at a time, at most 512, and the
// list is evaluated when a warp finds none: 36 T items hold the about 7 T of a
// packing of n = T trees several times over, so they are evaluated in one go
// (the LUT's items are the near pairs themselves).
__host__ __device__ inline void pk_caps(int T, int mode, int* cap_near, int* cap_items)
{
    *cap_near = 8 * T;
    *cap_items = mode == PK_PAIR_LUT ? 0 : 36 * T;
}

// keep: room for the kept near list's state (the fused relaxation only; a
// one-shot evaluation keeps the smaller footprint, which lets the smallest
// size classes fit one more CTA per SM).
__host__ __device__ inline size_t pk_cost_smem_bytes(int n_max, int cap_near, int cap_items, bool keep = false)
{
    size_t b = 0;
    b += (size_t)n_max * 16;        // pose
    b += (size_t)n_max * 16;        // bnd
    b += (size_t)n_max * 64;        // aabb
    b += (size_t)n_max * 24;        // acc
    b += (size_t)n_max * 4;         // theta
    b += (size_t)cap_items * 2;     // items
    b += (size_t)cap_near * 4;      // near pairs
    b += (size_t)(2 * pk_grid_cap(n_max) + 1) * 4 + (size_t)n_max * 16 + 4;   // grid
    b += 8 * 16 + 16 * 8 + 16 + 16 + 16 + 32 * 8 + 32 * 8;   // piece tables, counters, reductions
    if (keep) b += 16 + 32 * 4;   // pk_nlist, pk_disp
    return (b + 15) & ~(size_t)15;   // whatever follows starts 16-byte aligned
}

__device__ inline PkCostSmem pk_cost_carve(unsigned char* base, int n_max, int cap_near, int cap_items,
                                           bool keep = false)
{
    PkCostSmem s;
    unsigned char* p = base;
    // fixed sizes first: their addresses, and the poses', are constants
    s.piece4 = (float4*)p; p += 8 * 16;
    s.piece = (float2*)p; p += 16 * 8;
    s.piece_nv = (int*)p; p += 16;
    s.count = (int*)p; p += 16;
    s.cnt = (unsigned int*)p; p += 16;
    if (keep) p += 16;   // pk_nlist
    s.red = (double*)p; p += 32 * 8;
    s.redl = (long long*)p; p += 32 * 8;
    if (keep) p += 32 * 4;   // pk_disp
    s.pose = (float4*)p; p += (size_t)n_max * 16;
    s.bnd = (float4*)p; p += (size_t)n_max * 16;
    s.aabb = (float4*)p; p += (size_t)n_max * 64;
    s.near = (uint32_t*)p; p += (size_t)cap_near * 4;
    s.items = (uint16_t*)p; p += (size_t)cap_items * 2;
    s.acc_lo = (unsigned*)p; p += (size_t)n_max * 12;
    s.acc_hi = (unsigned*)p; p += (size_t)n_max * 12;
    s.theta = (float*)p; p += (size_t)n_max * 4;
    s.grid_cap = pk_grid_cap(n_max);
    s.cell_start = (int*)p; p += (size_t)(s.grid_cap + 1) * 4;
    s.cell_fill = (int*)p; p += (size_t)s.grid_cap * 4;
    s.sorted = (int*)p; p += (size_t)n_max * 4;
    s.tcell = (int*)p; p += (size_t)n_max * 4;
    s.near_cnt = (int*)p; p += (size_t)n_max * 4;
    s.near_start = (int*)p; p += (size_t)n_max * 4 + 4;
    s.cap_items = cap_items;
    s.cap_near = cap_near;
    s.n_cap = n_max;
    return s;
}

// Arrays placed right after cnt and redl by a carve with keep; derived from
// them rather than held as pointers of their own (fewer live registers around
// the clipper).
__device__ __forceinline__ int* pk_nlist(const PkCostSmem& sm) { return (int*)(sm.cnt + 4); }
__device__ __forceinline__ float* pk_disp(const PkCostSmem& sm) { return (float*)(sm.redl + 32); }

// ---------------------------------------------------------------------------
// Convex piece intersection area with the gradient of both rigid poses.
//
// The reference clips the subject piece against the clip piece edge by edge
// (Sutherland-Hodgman, pack_cuda_primitives.py:238-296, 348-538) and back-
// propagates through every stage for the subject's vertex gradient.  Here the
// same area is assembled from the boundary of P n Q directly: each edge of P
// is clipped to the part inside Q (parametric interval against Q's half-
// planes, inside = cross >= 0 as in :263-264) and each edge of Q to the part
// inside P.  With both pieces CCW, the area is sum 1/2 cross(a', b') over
// those portions (Green's theorem).  A rigid motion of P moves only the P
// portions, so dA/d(x, y) = sum of their outward normals N = len * n_hat and
// dA/dtheta = sum cross(midpoint - centre, N) (exact for straight edges).
// Collinear edges: a P edge lying on a Q edge line is excluded; a Q edge on a
// P edge line is kept only if both run the same way, so a shared boundary
// segment is counted once and touching pieces contribute zero.
// ---------------------------------------------------------------------------
// Near-collinear edges (all four endpoints within 2e-6 tree units of the
// other edge's line) are classified from the same four numbers on both
// passes, so the two passes can never disagree about a shared boundary.
#define PK_COLLINEAR_TOL2 4e-12f   // (2e-6)^2

// (b - a) x (c - a) with fixed rounding, so that the same four points give
// the same value wherever it is evaluated.
__device__ __forceinline__ float pk_cross3_rn(float2 a, float2 b, float2 c)
{
    return __fmaf_rn(b.x - a.x, c.y - a.y, -__fmul_rn(b.y - a.y, c.x - a.x));
}

// Side values: f[k][v] = cross(Y[k+1] - Y[k], X[v] - Y[k]), X's vertices against
// Y's edge lines (>= 0 inside).
//
// A convex piece's four vertices packed in pairs for the FP32x2 instructions
// of sm_100 (FFMA2 / FMUL2: two independent FP32 operations, each rounded
// like its scalar form): x01 = (x0, x1), x23 = (x2, x3), likewise y.
struct PkQuad { float2 x01, x23, y01, y23; };

__device__ __forceinline__ float2 pk_qv(const PkQuad& q, int v)
{
    return v == 0 ? make_float2(q.x01.x, q.y01.x) : v == 1 ? make_float2(q.x01.y, q.y01.y)
         : v == 2 ? make_float2(q.x23.x, q.y23.x) : make_float2(q.x23.y, q.y23.y);
}

__device__ __forceinline__ PkQuad pk_quad(const float2 (&V)[4])
{
    PkQuad q;
    q.x01 = make_float2(V[0].x, V[1].x); q.x23 = make_float2(V[2].x, V[3].x);
    q.y01 = make_float2(V[0].y, V[1].y); q.y23 = make_float2(V[2].y, V[3].y);
    return q;
}

// X's four vertices against line k of Y, two per instruction: (f0, f1) in f01,
// (f2, f3) in f23, with the rounding of pk_cross3_rn (the vertex is taken
// relative to the line's first point before the cross product, which keeps
// small side values accurate wherever the pieces lie).
__device__ __forceinline__ void pk_side_line(const PkQuad& X, const PkQuad& Y, int k, float2& f01, float2& f23)
{
    const float2 a = pk_qv(Y, k), b = pk_qv(Y, (k + 1) & 3);
    const float ex = b.x - a.x, ey = b.y - a.y;
    const float2 ex2 = make_float2(ex, ex), ney2 = make_float2(-ey, -ey);
    const float2 nax2 = make_float2(-a.x, -a.x), nay2 = make_float2(-a.y, -a.y);   // x - a = x + (-a), exactly
    f01 = __ffma2_rn(ex2, __fadd2_rn(X.y01, nay2), __fmul2_rn(ney2, __fadd2_rn(X.x01, nax2)));
    f23 = __ffma2_rn(ex2, __fadd2_rn(X.y23, nay2), __fmul2_rn(ney2, __fadd2_rn(X.x23, nax2)));
}

// f[k][v] for the four lines of Y.
__device__ __forceinline__ void pk_side_values_q(const PkQuad& X, const PkQuad& Y, float (&f)[4][4])
{
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float2 f01, f23;
        pk_side_line(X, Y, k, f01, f23);
        f[k][0] = f01.x; f[k][1] = f01.y; f[k][2] = f23.x; f[k][3] = f23.y;
    }
}

// Whether some line of Y has every vertex of X on its outer side, by more than
// tol: f[k][v] < -tol for all v, with the side values the clipper sees.
__device__ __forceinline__ bool pk_line_separates(const PkQuad& X, const PkQuad& Y, float tol)
{
    float m = 3.4e38f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float2 f01, f23;
        pk_side_line(X, Y, k, f01, f23);
        m = fminf(m, fmaxf(fmaxf(f01.x, f01.y), fmaxf(f23.x, f23.y)));
    }
    return m < -tol;   // the degenerate fourth line of a triangle gives 0: it separates nothing
}

// Approximate a / b, as __fdividef but with subnormals taken as zero: the same
// value wherever a, b and a / b are normal, without __fdividef's scaling of
// tiny and huge divisors (3 % of the cost kernel).  A crossing parameter below
// 1e-38 is zero to everything computed from it.
__device__ __forceinline__ float pk_quotient(float a, float b)
{
    float q;
    asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(q) : "f"(a), "f"(b));
    return q;
}

// Adds the part [tin, tout] of the edge a -> b to A2 (twice the area) and to g
// (gradient of the rigid pose about centre ctr).
__device__ __forceinline__ void pk_edge_part(float2 a, float2 b, float tin, float tout, float2 ctr, float& A2, float3& g)
{
    const float dt = tout - tin;
    const float2 e = make_float2(b.x - a.x, b.y - a.y);
    A2 += dt * pk_cross(a, b);
    const float2 N = make_float2(dt * e.y, -dt * e.x);
    const float tm = 0.5f * (tin + tout);
    const float2 m = make_float2(a.x + tm * e.x - ctr.x, a.y + tm * e.y - ctr.y);
    g.x += N.x;
    g.y += N.y;
    g.z += pk_cross(m, N);
}

// One pass of the assembly: the portions of X's edges inside Y, added to A2 and
// g.  This form serves pieces with a vertex within the tolerance of a line of
// the other (rare, so out of line): per vertex, 4-bit masks of the lines it is
// outside of and near, from which collinear edges are found.  KEEP_SAME_DIR: a
// collinear edge of X is kept when it runs the same way as Y's (X = Q) or always
// dropped (X = P).  Returns (A2, g).
template <bool KEEP_SAME_DIR>
__device__ __noinline__ float4 pk_clip_near(const PkQuad XQ, bool x_tri, const PkQuad YQ, bool y_tri, float2 ctr,
                                            float A2, float3 g)
{
    const float2 X[4] = {pk_qv(XQ, 0), pk_qv(XQ, 1), pk_qv(XQ, 2), pk_qv(XQ, 3)};
    const float2 Y[4] = {pk_qv(YQ, 0), pk_qv(YQ, 1), pk_qv(YQ, 2), pk_qv(YQ, 3)};
    float f[4][4];
    pk_side_values_q(XQ, YQ, f);
    const float tiny = c_geom.coll_tiny;
    const unsigned lines = y_tri ? 0x7u : 0xFu;
    unsigned out[4], nearm[4];   // per vertex, a bit per line: outside it, near it
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        unsigned o = 0, nm = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            o |= (unsigned)(f[k][v] < 0.f) << k;
            nm |= (unsigned)(fabsf(f[k][v]) <= tiny) << k;
        }
        out[v] = o & lines;
        nearm[v] = nm & lines;
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        if (v == 3 && x_tri) break;
        const int vb = (v + 1) & 3;
        const float2 a = X[v], b = X[vb];
        unsigned skip = 0;
        bool empty = false;
        const unsigned coll = nearm[v] & nearm[vb];
        if (coll) {
            // both ends within tolerance of some line of Y: confirm collinearity
            // with the symmetric four-number test (the other pass sees the same numbers)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (!((coll >> k) & 1u)) continue;
                const float fa = f[k][v], fb = f[k][vb];
                const float2 ya = Y[k], yb = Y[(k + 1) & 3];
                const float2 ey = make_float2(yb.x - ya.x, yb.y - ya.y), ex = make_float2(b.x - a.x, b.y - a.y);
                const float ty = PK_COLLINEAR_TOL2 * __fmaf_rn(ey.x, ey.x, __fmul_rn(ey.y, ey.y));
                const float tx = PK_COLLINEAR_TOL2 * __fmaf_rn(ex.x, ex.x, __fmul_rn(ex.y, ex.y));
                const float ra = pk_cross3_rn(a, b, ya), rb = pk_cross3_rn(a, b, yb);
                if (fa * fa <= ty && fb * fb <= ty && ra * ra <= tx && rb * rb <= tx) {
                    if (!KEEP_SAME_DIR || ex.x * ey.x + ex.y * ey.y <= 0.f) empty = true;
                    skip |= 1u << k;
                }
            }
        }
        const unsigned oa = out[v] & ~skip, ob = out[vb] & ~skip;
        float tin = 0.f, tout = 1.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float fa = f[k][v], fb = f[k][vb];
            const float t = pk_quotient(fa, fa - fb);    // meaningful where the edge crosses line k
            tin = fmaxf(tin, (oa >> k) & 1u ? t : 0.f);     // entering
            tout = fminf(tout, (ob >> k) & 1u ? t : 1.f);   // leaving
        }
        const bool part = !empty && !(oa & ob) && tin < tout;
        if (part) pk_edge_part(a, b, tin, tout, ctr, A2, g);
    }
    return make_float4(A2, g.x, g.y, g.z);
}

// The pass for all other pieces.  Line by line of Y: the vertices' side values,
// their quotients along X's four edges, and per edge the largest entering and
// the smallest leaving parameter.  Whether a quotient counts is put in by
// arithmetic, with s = 1 for a vertex outside the line and 0 inside: t s is t
// or 0 (an infinite t gives NaN, which the minima and maxima ignore), t s +
// (1 - s) is t or 1.  Compares and selects share one half-rate pipe, which was
// the busiest (51 %) with them; multiplications have another to themselves.  An
// edge outside one line at both ends has tin >= tout by the same quotient.
template <bool KEEP_SAME_DIR>
__device__ __forceinline__ void pk_clip_pass(const PkQuad& X, bool x_tri, const PkQuad& Y, bool y_tri, float2 ctr,
                                             float& A2, float3& g)
{
    float tin[4] = {0.f, 0.f, 0.f, 0.f}, tout[4] = {1.f, 1.f, 1.f, 1.f};
    float mn = 3.4e38f;   // smallest |f| against Y's real lines
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float2 f01, f23;
        pk_side_line(X, Y, k, f01, f23);
        const float f[4] = {f01.x, f01.y, f23.x, f23.y};
        float s[4], r[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            s[v] = f[v] < 0.f ? 1.f : 0.f;
            r[v] = 1.f - s[v];
        }
        const float m = fminf(fminf(fabsf(f[0]), fabsf(f[1])), fminf(fabsf(f[2]), fabsf(f[3])));
        mn = fminf(mn, k == 3 && y_tri ? 3.4e38f : m);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int n = (e + 1) & 3;
            const float t = pk_quotient(f[e], f[e] - f[n]);
            tin[e] = fmaxf(tin[e], t * s[e]);
            tout[e] = fminf(tout[e], fmaf(t, s[n], r[n]));
        }
    }
    if (mn <= c_geom.coll_tiny) {
        const float4 q = pk_clip_near<KEEP_SAME_DIR>(X, x_tri, Y, y_tri, ctr, A2, g);
        A2 = q.x;
        g = make_float3(q.y, q.z, q.w);
        return;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const bool part = tin[e] < tout[e] && !(e == 3 && x_tri);
        // an empty part becomes [0, 0]: finite, so it adds zeros
        pk_edge_part(pk_qv(X, e), pk_qv(X, (e + 1) & 3), part ? tin[e] : 0.f, part ? tout[e] : 0.f, ctr, A2, g);
    }
}

// CHECK: the pieces may be separated by one of their lines (then nothing
// overlaps, and the clipper's rounding is kept from finding otherwise); without
// it the caller has tested that.
template <bool CHECK>
__device__ __forceinline__ void pk_piece_area_grad_q(const PkQuad& PQ, bool p_tri, const PkQuad& QQ, bool q_tri,
                                                     float2 d, float& area, float3& gP, float3& gQ)
{
    float A2 = 0.f;   // twice the area
    gP = make_float3(0.f, 0.f, 0.f);
    gQ = make_float3(0.f, 0.f, 0.f);
    area = 0.f;
    if (CHECK && (pk_line_separates(PQ, QQ, 0.f) || pk_line_separates(QQ, PQ, 0.f))) return;
    pk_clip_pass<false>(PQ, p_tri, QQ, q_tri, make_float2(0.f, 0.f), A2, gP);
    pk_clip_pass<true>(QQ, q_tri, PQ, p_tri, d, A2, gQ);
    area = 0.5f * A2;
    if (!(area > 0.f)) {   // empty or numerically vanishing overlap
        area = 0.f;
        gP = make_float3(0.f, 0.f, 0.f);
        gQ = make_float3(0.f, 0.f, 0.f);
    }
}

__device__ __forceinline__ void pk_piece_area_grad(const float2 (&P)[4], bool p_tri,
                                                   const float2 (&Q)[4], bool q_tri, float2 d,
                                                   float& area, float3& gP, float3& gQ)
{
    pk_piece_area_grad_q<true>(pk_quad(P), p_tri, pk_quad(Q), q_tri, d, area, gP, gQ);
}

// ---------------------------------------------------------------------------
// SAT penetration depth (sat_separation_with_grad_pose,
// pack_cuda_primitives.py:544-828) with the pose gradient of both pieces.
// Axes: P's edge normals, then Q's; a separating axis returns 0; the
// smallest overlap wins (strict <), pen1 <= pen2 selects case 1.  The
// reference evaluates each ordered pair and keeps the ref gradient; the
// other piece's gradient here is the same expression with the roles swapped
// (translation: the negative; rotation: its own extreme vertex, plus the
// axis-rotation term when the axis is one of its edges).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void pk_piece_sat_grad(const float2 (&P)[4], bool p_tri, const float2 (&Q)[4],
                                                  bool q_tri, float2 d, float& sep, float3& gP,
                                                  float3& gQ)
{
    sep = 0.f;
    gP = make_float3(0.f, 0.f, 0.f);
    gQ = make_float3(0.f, 0.f, 0.f);
    // The smallest overlap over the axes, by selects: a warp's lanes separate or
    // improve at different axes.  The extreme vertices are found once, for the axis
    // that won, from its projections computed again (the same operations).
    float best = 1.0e30f;
    bool apart = false, found = false, from1 = false, c1 = true;
    float2 bn = make_float2(0.f, 0.f);
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool tri = pass == 0 ? p_tri : q_tri;
            const float2 a = pass == 0 ? P[k] : Q[k];
            const float2 b = pass == 0 ? P[(k + 1) & 3] : Q[(k + 1) & 3];
            float2 nr = make_float2(-(b.y - a.y), b.x - a.x);
            const float len = sqrtf(nr.x * nr.x + nr.y * nr.y);
            const bool real = !(k == 3 && tri) && !(len < 1.0e-12f);
            nr.x /= len;
            nr.y /= len;
            float mn1 = P[0].x * nr.x + P[0].y * nr.y, mx1 = mn1, mn2 = Q[0].x * nr.x + Q[0].y * nr.y, mx2 = mn2;
#pragma unroll
            for (int v = 1; v < 4; ++v) {
                const float p1 = P[v].x * nr.x + P[v].y * nr.y, p2 = Q[v].x * nr.x + Q[v].y * nr.y;
                mn1 = fminf(mn1, p1); mx1 = fmaxf(mx1, p1);
                mn2 = fminf(mn2, p2); mx2 = fmaxf(mx2, p2);
            }
            apart |= real & ((mx1 < mn2) | (mx2 < mn1));   // separating axis: no overlap
            found |= real;
            const float pen1 = mx1 - mn2, pen2 = mx2 - mn1;
            const float pen = pen1 < pen2 ? pen1 : pen2;
            const bool less = real & (pen < best);
            best = less ? pen : best;
            bn.x = less ? nr.x : bn.x;
            bn.y = less ? nr.y : bn.y;
            from1 = less ? pass == 0 : from1;
            c1 = less ? pen1 <= pen2 : c1;
        }
    }
    if (apart || !found || best <= 1.0e-12f) return;
    sep = best;
    if (!(best < 1.0e30f)) return;   // a NaN angle: no axis says anything
    const float sigma = c1 ? 1.f : -1.f;
    // first vertex attaining the extreme, like the reference scans
    float2 bv = P[0], bw = Q[0];
    float pv = P[0].x * bn.x + P[0].y * bn.y, pw = Q[0].x * bn.x + Q[0].y * bn.y;
#pragma unroll
    for (int q = 1; q < 4; ++q) {
        const float p1 = P[q].x * bn.x + P[q].y * bn.y, p2 = Q[q].x * bn.x + Q[q].y * bn.y;
        const bool v1 = c1 ? p1 > pv : p1 < pv, v2 = c1 ? p2 < pw : p2 > pw;
        pv = v1 ? p1 : pv;
        bv.x = v1 ? P[q].x : bv.x;
        bv.y = v1 ? P[q].y : bv.y;
        pw = v2 ? p2 : pw;
        bw.x = v2 ? Q[q].x : bw.x;
        bw.y = v2 ? Q[q].y : bw.y;
    }
    const float2 gv = make_float2(sigma * bn.x, sigma * bn.y);
    const float2 rn = make_float2(-bn.y, bn.x);                     // d n / d theta
    const float2 vw = make_float2(bv.x - bw.x, bv.y - bw.y);
    const float axis_term = sigma * (vw.x * rn.x + vw.y * rn.y);
    const float2 rq = make_float2(bw.x - d.x, bw.y - d.y);
    gP.x = gv.x;
    gP.y = gv.y;
    gP.z = gv.x * -bv.y + gv.y * bv.x + (from1 ? axis_term : 0.f);
    gQ.x = -gv.x;
    gQ.y = -gv.y;
    gQ.z = -(gv.x * -rq.y + gv.y * rq.x) + (from1 ? 0.f : axis_term);
}

// ---------------------------------------------------------------------------
// LUT lookup with analytic gradient (lut_lookup_with_grad,
// pack_cuda_lut.py:298-415), FP32 with the reference's operation order.
// Indices are clamped into the table (the reference can read one cell out of
// range when a trimmed theta range is mirrored).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float pk_lut_lookup(const PkLut& L, float x, float y, float th, float3& g)
{
    g = make_float3(0.f, 0.f, 0.f);
    if (x < -L.x_max || x > L.x_max || y < L.y_min || y > L.y_max || th < L.t_min || th > L.t_max)
        return 0.f;
    const float xt = x >= 0.f ? x : -x;
    const float tt = x >= 0.f ? th : -th;
    const float gx = (xt - L.x_min) / (L.x_max - L.x_min) * (float)(L.nx - 1);
    const float gy = (y - L.y_min) / (L.y_max - L.y_min) * (float)(L.ny - 1);
    const float gt = (tt - L.t_min) / (L.t_max - L.t_min) * (float)(L.nt - 1);
    int ix0 = (int)floorf(gx), iy0 = (int)floorf(gy), it0 = (int)floorf(gt);
    const float fx = gx - ix0, fy = gy - iy0, ft = gt - it0;
    ix0 = min(max(ix0, 0), L.nx - 1);
    iy0 = min(max(iy0, 0), L.ny - 1);
    it0 = min(max(it0, 0), L.nt - 1);
    const int ix1 = min(ix0 + 1, L.nx - 1), iy1 = min(iy0 + 1, L.ny - 1), it1 = min(it0 + 1, L.nt - 1);
    const size_t sy = (size_t)L.nt, sx = (size_t)L.ny * L.nt;
    const float* V = L.vals;
    const float v000 = __ldg(V + ix0 * sx + iy0 * sy + it0), v001 = __ldg(V + ix0 * sx + iy0 * sy + it1);
    const float v010 = __ldg(V + ix0 * sx + iy1 * sy + it0), v011 = __ldg(V + ix0 * sx + iy1 * sy + it1);
    const float v100 = __ldg(V + ix1 * sx + iy0 * sy + it0), v101 = __ldg(V + ix1 * sx + iy0 * sy + it1);
    const float v110 = __ldg(V + ix1 * sx + iy1 * sy + it0), v111 = __ldg(V + ix1 * sx + iy1 * sy + it1);
    const float v00 = v000 * (1.0f - ft) + v001 * ft, v01 = v010 * (1.0f - ft) + v011 * ft;
    const float v10 = v100 * (1.0f - ft) + v101 * ft, v11 = v110 * (1.0f - ft) + v111 * ft;
    const float v0 = v00 * (1.0f - fy) + v01 * fy, v1 = v10 * (1.0f - fy) + v11 * fy;
    const float val = v0 * (1.0f - fx) + v1 * fx;
    const float dfx = v1 - v0;
    const float dfy = (1.0f - fx) * (v01 - v00) + fx * (v11 - v10);
    const float d0 = (v001 - v000) * (1.0f - fy) + (v011 - v010) * fy;
    const float d1 = (v101 - v100) * (1.0f - fy) + (v111 - v110) * fy;
    const float dft = d0 * (1.0f - fx) + d1 * fx;
    g.x = dfx * ((float)(L.nx - 1) / (L.x_max - L.x_min));
    g.y = dfy * ((float)(L.ny - 1) / (L.y_max - L.y_min));
    g.z = dft * ((float)(L.nt - 1) / (L.t_max - L.t_min));
    if (x < 0.f) { g.x = -g.x; g.z = -g.z; }
    return val;
}

// Adds v to the int64 at a (shared memory) with two 32-bit atomics: the low
// word's old value gives the carry, which travels with the high word.  The
// sum stays exact modulo 2^64 whatever the interleaving (the carries total
// floor((lo0 + sum lo_k) / 2^32) in any order), and a high-word add of zero
// -- small values of either sign -- is skipped.  On this GPU a 64-bit
// shared atomic costs several times two 32-bit ones.
__device__ __forceinline__ void pk_fx_add(long long* a, long long v)
{
    unsigned* w = (unsigned*)a;   // little endian: w[0] low word, w[1] high word
    const unsigned lo = (unsigned)v, hi = (unsigned)((unsigned long long)v >> 32);
    const unsigned old = atomicAdd(&w[0], lo);
    const unsigned up = hi + (unsigned)(old + lo < old);
    if (up) atomicAdd(&w[1], up);
}

// The same add on a split accumulator: low words in one array, high words
// in another, so consecutive accumulators use consecutive banks.
__device__ __forceinline__ void pk_fx_add2(unsigned* lo_w, unsigned* hi_w, long long v)
{
    const unsigned lo = (unsigned)v, hi = (unsigned)((unsigned long long)v >> 32);
    const unsigned old = atomicAdd(lo_w, lo);
    const unsigned up = hi + (unsigned)(old + lo < old);
    if (up) atomicAdd(hi_w, up);
}

__device__ __forceinline__ void pk_acc_add2(const PkCostSmem& sm, int t, float3 g)
{
    pk_fx_add2(&sm.acc_lo[3 * t + 0], &sm.acc_hi[3 * t + 0], pk_to_fx(g.x));
    pk_fx_add2(&sm.acc_lo[3 * t + 1], &sm.acc_hi[3 * t + 1], pk_to_fx(g.y));
    pk_fx_add2(&sm.acc_lo[3 * t + 2], &sm.acc_hi[3 * t + 2], pk_to_fx(g.z));
}

__device__ __forceinline__ long long pk_acc_get(const PkCostSmem& sm, int k)
{
    return (long long)(((unsigned long long)sm.acc_hi[k] << 32) | (unsigned long long)sm.acc_lo[k]);
}

__device__ __forceinline__ void pk_acc_add(long long* acc, int t, float3 g)
{
    pk_fx_add(&acc[3 * t + 0], pk_to_fx(g.x));
    pk_fx_add(&acc[3 * t + 1], pk_to_fx(g.y));
    pk_fx_add(&acc[3 * t + 2], pk_to_fx(g.z));
}

__device__ __forceinline__ void pk_load_piece(const PkCostSmem& sm, int p, float c, float s, float ox,
                                              float oy, float2 (&V)[4])
{
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const float2 l = sm.piece[p * 4 + v];
        V[v] = make_float2(c * l.x - s * l.y + ox, s * l.x + c * l.y + oy);
    }
}

// Piece p of a tree rotated by (c, s) and moved by (ox, oy), from the SoA
// table: two vertices per instruction.
__device__ __forceinline__ PkQuad pk_load_quad(const PkCostSmem& sm, int p, float c, float s, float ox, float oy)
{
    const float4 X = sm.piece4[2 * p], Y = sm.piece4[2 * p + 1];
    const float2 c2 = make_float2(c, c), s2 = make_float2(s, s), ns2 = make_float2(-s, -s);
    const float2 ox2 = make_float2(ox, ox), oy2 = make_float2(oy, oy);
    const float2 x01 = make_float2(X.x, X.y), x23 = make_float2(X.z, X.w);
    const float2 y01 = make_float2(Y.x, Y.y), y23 = make_float2(Y.z, Y.w);
    PkQuad q;
    q.x01 = __fadd2_rn(__ffma2_rn(c2, x01, __fmul2_rn(ns2, y01)), ox2);
    q.x23 = __fadd2_rn(__ffma2_rn(c2, x23, __fmul2_rn(ns2, y23)), ox2);
    q.y01 = __fadd2_rn(__ffma2_rn(s2, x01, __fmul2_rn(c2, y01)), oy2);
    q.y23 = __fadd2_rn(__ffma2_rn(s2, x23, __fmul2_rn(c2, y23)), oy2);
    return q;
}

// Centre-distance cull, rounded the same way wherever it is evaluated.  Swapping A and B
// gives the same answer: rounding is symmetric under negation.
__device__ __forceinline__ int pk_is_near(float4 A, float4 B, float cutoff)
{
    const float dx = __fsub_rn(B.x, A.x), dy = __fsub_rn(B.y, A.y);
    return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)) <= cutoff;
}

// Phase B, LUT: looks up the count near pairs of the list; returns this
// thread's fixed-point pair total.  filter: the list is a kept near list, so a
// pair is looked up only if it passes the centre cull now; the kept pairs are
// counted.
__device__ __forceinline__ long long pk_process_lut(const PkCostSmem& sm, int count, float w_pair, const PkLut& lut,
                                                    bool filter, float cutoff)
{
    long long tot = 0;
    unsigned kept = 0;
#pragma unroll 1   // one pair's eight gathers in flight per thread: two were slower
    for (int w = threadIdx.x; w < count; w += blockDim.x) {
        const uint32_t it = sm.near[w];
        const int i = it & 2047, j = (it >> 11) & 2047;
        const float4 A = sm.pose[i], B = sm.pose[j];
        if (filter) {
            if (!pk_is_near(A, B, cutoff)) continue;
            ++kept;
        }
        // ref = lower index, as the reference's triangular loop (pack_cuda_lut.py:437)
        const int r = i < j ? i : j, o = i < j ? j : i;
        const float4 R = sm.pose[r], O = sm.pose[o];
        const float dxw = O.x - R.x, dyw = O.y - R.y;
        const float dxl = R.z * dxw + R.w * dyw;
        const float dyl = -R.w * dxw + R.z * dyw;
        const float dth = pk_wrap_angle(sm.theta[o] - sm.theta[r]);
        float3 gl;
        float val = pk_lut_lookup(lut, dxl, dyl, dth, gl);
        if (lut.quadratic) {
            if (val > 0.f) {
                gl.x *= 2.0f * val; gl.y *= 2.0f * val; gl.z *= 2.0f * val;
                val = val * val;
            } else {
                val = 0.f;
                gl = make_float3(0.f, 0.f, 0.f);
            }
        }
        const float3 gr = make_float3(-gl.x * R.z + gl.y * R.w, -gl.x * R.w - gl.y * R.z,
                                      gl.x * dyl - gl.y * dxl - gl.z);
        const float3 go = make_float3(gl.x * R.z - gl.y * R.w, gl.x * R.w + gl.y * R.z, gl.z);
        const float3 gi = (r == i) ? gr : go, gj = (r == i) ? go : gr;
        if (val != 0.f || gi.x != 0.f || gi.y != 0.f || gi.z != 0.f) {
            tot += pk_to_fx(w_pair * val);
            pk_acc_add2(sm, i, make_float3(w_pair * gi.x, w_pair * gi.y, w_pair * gi.z));
            pk_acc_add2(sm, j, make_float3(w_pair * gj.x, w_pair * gj.y, w_pair * gj.z));
        }
    }
    if (filter) {
        kept = __reduce_add_sync(PK_FULL_MASK, kept);
        if ((threadIdx.x & 31) == 0 && kept) { atomicAdd(&sm.cnt[1], kept); atomicAdd(&sm.cnt[2], kept); }
    }
    return tot;
}

// Phase B, analytic modes: evaluates the count listed piece pairs; returns this
// thread's fixed-point pair total.
//
// 36 % (initial poses of a random packing) to 45 % (relaxed) of the piece pairs
// whose boxes meet are separated by one of their lines, 80 % in a nearly legal
// packing's separation cost, and a lane with such a pair idled through the
// clipper beside the others.  So each warp first tests its items (side values
// and minima only) and keeps those not separated at the front of its own part
// of the list, then evaluates these with full warps.  A warp's part is the
// items warp, warp + nwarps, ...: no barrier between the two passes, and
// consecutive items, which share trees, are spread over the warps, whose
// accumulator atomics then rarely meet.
//
// The area's test is the clipper's own (same side values).  The separation's
// axes are normalised and round differently, so there a line must clear the
// pieces by 1e-6 (side value: gap times an edge shorter than 1; coordinates are
// within 2 units, whose rounding is 3e-7) before the pair is dropped.
template <int MODE>
__device__ __forceinline__ long long pk_process_items(const PkCostSmem& sm, int count, float w_pair)
{
    long long tot = 0;
    const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float tol = MODE == PK_PAIR_AREA ? 0.f : 1e-6f;
    uint16_t* const mine = sm.items + warp;
    const int own = count > warp ? (count - warp + nw - 1) / nw : 0;   // items of this warp
    int kept = 0;
    for (int b = 0; b < own; b += 32) {
        bool keep = false;
        uint16_t it = 0;
        if (b + lane < own) {
            it = mine[(b + lane) * nw];
            const uint32_t ij = sm.near[it & 2047];
            const float4 A = sm.pose[ij & 2047], B = sm.pose[(ij >> 11) & 2047];
            const PkQuad PQ = pk_load_quad(sm, (it >> 11) & 3, A.z, A.w, 0.f, 0.f);
            const PkQuad QQ = pk_load_quad(sm, it >> 13, B.z, B.w, B.x - A.x, B.y - A.y);
            keep = !pk_line_separates(PQ, QQ, tol) && !pk_line_separates(QQ, PQ, tol);
        }
        const unsigned m = __ballot_sync(PK_FULL_MASK, keep);
        if (keep) mine[(kept + __popc(m & ((1u << lane) - 1u))) * nw] = it;
        kept += __popc(m);
    }
    __syncwarp();
    for (int b = lane; b < kept; b += 32) {
        const int it = mine[b * nw], pi = (it >> 11) & 3, pj = it >> 13;
        const uint32_t ij = sm.near[it & 2047];
        const int i = ij & 2047, j = (ij >> 11) & 2047;
        const float4 A = sm.pose[i], B = sm.pose[j];
        const float2 d = make_float2(B.x - A.x, B.y - A.y);
        float val;
        float3 gi, gj;
        const bool pt = sm.piece_nv[pi] == 3, qt = sm.piece_nv[pj] == 3;
        if (MODE == PK_PAIR_AREA) {
            const PkQuad PQ = pk_load_quad(sm, pi, A.z, A.w, 0.f, 0.f);
            const PkQuad QQ = pk_load_quad(sm, pj, B.z, B.w, d.x, d.y);
            pk_piece_area_grad_q<false>(PQ, pt, QQ, qt, d, val, gi, gj);
        } else {
            float2 P[4], Q[4];
            pk_load_piece(sm, pi, A.z, A.w, 0.f, 0.f, P);
            pk_load_piece(sm, pj, B.z, B.w, d.x, d.y, Q);
            float sp;
            pk_piece_sat_grad(P, pt, Q, qt, d, sp, gi, gj);
            const float f = 2.0f * sp;
            gi = make_float3(f * gi.x, f * gi.y, f * gi.z);
            gj = make_float3(f * gj.x, f * gj.y, f * gj.z);
            val = sp * sp;
        }
        if (val != 0.f || gi.x != 0.f || gi.y != 0.f || gi.z != 0.f) {
            tot += pk_to_fx(w_pair * val);
            pk_acc_add2(sm, i, make_float3(w_pair * gi.x, w_pair * gi.y, w_pair * gi.z));
            pk_acc_add2(sm, j, make_float3(w_pair * gj.x, w_pair * gj.y, w_pair * gj.z));
        }
    }
    return tot;
}

// The fused relaxation evaluates its items out of line: one call per flush
// saves the optimiser's registers once, and the clipper has the rest to itself.
// Inlined, they were live across it and spilled per item.  Carves the shared
// memory again, like pk_broad_phase_outlined.
template <int MODE>
__device__ __noinline__ long long pk_process_items_outlined(int n_cap, int cap_near, int cap_items, int count,
                                                            float w_pair)
{
    extern __shared__ __align__(16) unsigned char pk_smem[];
    const PkCostSmem sm = pk_cost_carve(pk_smem, n_cap, cap_near, cap_items, true);
    return pk_process_items<MODE>(sm, count, w_pair);
}

// Sorted-position ranges [b0, b1) and [b2, b3) of the half neighbourhood of
// sorted position a (grid of gx x gy cells, row-major cell order).
__device__ __forceinline__ void pk_half_neighbourhood(const PkCostSmem& sm, int a, int gx, int gy, int& b0, int& b1,
                                                      int& b2, int& b3)
{
    const int c = sm.tcell[sm.sorted[a]];
    const int cy = c / gx, cx = c - cy * gx;
    b0 = a + 1;
    b1 = sm.cell_start[cy * gx + min(cx + 2, gx)];
    if (cy + 1 < gy) {
        const int r = (cy + 1) * gx;
        b2 = sm.cell_start[r + max(cx - 1, 0)];
        b3 = sm.cell_start[r + min(cx + 2, gx)];
    } else {
        b2 = b3 = b1;
    }
}

// Processes the cn near pairs of the list: the LUT looks them up directly;
// the analytic modes expand each into the piece pairs whose boxes overlap and
// evaluate those, all in one go unless they overflow the item list.  With KEEP the list may be a kept near list
// (pk_nlist(sm)[2] set), whose pairs were within cutoff + skin when it was
// built: each pair is then first tested against the centre cutoff at the
// current poses, and the pairs that pass are counted.  The flag is read where
// it is used, so nothing extra stays live across the clipper.  Otherwise every
// listed pair is near.  All threads call it; it ends with a barrier.
template <int MODE, bool KEEP>
__device__ __forceinline__ long long pk_flush_near(const PkCostSmem& sm, int cn, const PkCostSpec& spec, int T)
{
    long long tot = 0;
    const int lane = threadIdx.x & 31;
    if (MODE == PK_PAIR_LUT) {
        const bool filter = KEEP && pk_nlist(sm)[2] != 0;
        if (threadIdx.x == 0 && !filter) sm.cnt[2] += (unsigned)cn;
        tot += pk_process_lut(sm, cn, spec.w_pair, spec.lut, filter, c_geom.cutoff_sq);
    } else {
        // Each warp expands every nwarps-th 32 pairs and reserves room for their
        // items; one that finds none stops, and goes on after the list is done.
        const bool filter = KEEP && pk_nlist(sm)[2] != 0;
        const int chunks = (cn + 31) >> 5, nw = T >> 5;
        int ch = threadIdx.x >> 5;
        unsigned near = 0;
        for (;;) {
            for (; ch < chunks; ch += nw) {
                const int w = 32 * ch + lane;
                uint32_t mask = 0;
                bool keep = false;
                if (w < cn) {
                    const uint32_t ij = sm.near[w];
                    const int i = ij & 2047, j = (ij >> 11) & 2047;
                    const float4 A = sm.pose[i], B = sm.pose[j];
                    keep = !filter || pk_is_near(A, B, c_geom.cutoff_sq);
                    if (keep) {
                        const float dx = B.x - A.x, dy = B.y - A.y;
#pragma unroll
                        for (int p = 0; p < 4; ++p) {
                            const float4 a = sm.aabb[p * sm.n_cap + i];
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                const float4 b2 = sm.aabb[q * sm.n_cap + j];
                                const bool ov = !(a.y < b2.x + dx || b2.y + dx < a.x || a.w < b2.z + dy || b2.w + dy < a.z);
                                mask |= (uint32_t)ov << (4 * p + q);
                            }
                        }
                    }
                }
                const int cnt = __popc(mask);
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(PK_FULL_MASK, incl, o);
                    if (lane >= o) incl += v;
                }
                const int wtot = __shfl_sync(PK_FULL_MASK, incl, 31);
                int wbase = 0;
                if (lane == 31 && wtot) {
                    // A reservation that does not fit stays counted, so every
                    // later one fails too and the list has no gaps: it ends where
                    // the first one failed.  (Taken back, a failed reservation
                    // could let another in behind one not yet taken back.)
                    wbase = atomicAdd(&sm.count[0], wtot);
                    if (wbase + wtot > sm.cap_items) { atomicMin(&sm.count[1], wbase); wbase = -1; }
                }
                wbase = __shfl_sync(PK_FULL_MASK, wbase, 31);
                if (wbase < 0) break;
                if (filter) near += (unsigned)__popc(__ballot_sync(PK_FULL_MASK, keep));
                int pos = wbase + incl - cnt;
                while (mask) {
                    const int b = __ffs(mask) - 1;
                    mask &= mask - 1;
                    sm.items[pos++] = (uint16_t)(w | ((b >> 2) << 11) | ((b & 3) << 13));
                }
            }
            const int more = __syncthreads_or(ch < chunks);
            const int ci = min(sm.count[0], sm.count[1]);
            if (threadIdx.x == 0) sm.cnt[2] += (unsigned)ci;
            tot += KEEP ? pk_process_items_outlined<MODE>(sm.n_cap, sm.cap_near, sm.cap_items, ci, spec.w_pair)
                        : pk_process_items<MODE>(sm, ci, spec.w_pair);
            if (!more) break;
            __syncthreads();
            if (threadIdx.x == 0) { sm.count[0] = 0; sm.count[1] = 0x7fffffff; }
            __syncthreads();
        }
        if (near && lane == 0) atomicAdd(&sm.cnt[1], near);
    }
    __syncthreads();
    if (MODE != PK_PAIR_LUT && threadIdx.x == 0) {   // the next flush appends after another barrier
        sm.count[0] = 0;
        sm.count[1] = 0x7fffffff;
    }
    return tot;
}

// Sums of the four components of bnd[0..n) in an order fixed by n alone
// (not by blockDim): lane l of warp 0 adds its contiguous chunk in double,
// then a fixed shuffle tree.  Called by warp 0 only; lane 0 gets the sums.
__device__ __forceinline__ double4 pk_canonical_sum4(int n, const float4* bnd)
{
    double4 s = make_double4(0.0, 0.0, 0.0, 0.0);
    const int k = (n + 31) >> 5;
    const int b = threadIdx.x * k, e = min(n, b + k);
    for (int t = b; t < e; ++t) {
        const float4 v = bnd[t];
        s.x += (double)v.x; s.y += (double)v.y; s.z += (double)v.z; s.w += (double)v.w;
    }
    s.x = pk_warp_sum(s.x); s.y = pk_warp_sum(s.y); s.z = pk_warp_sum(s.z); s.w = pk_warp_sum(s.w);
    return s;
}

// Images per genotype tree of a symmetric packing (spec.symmetry): 1, 2
// (SolutionCollectionSquareSymmetric180, kaggle_support.py:1272-1393) or 4
// (SolutionCollectionSquareSymmetric90, :1039-1195).
__host__ __device__ inline int pk_symmetry(const PkCostSpec& spec) { return spec.symmetry > 1 ? spec.symmetry : 1; }

// Pose of phenotype tree t = k ng + g: image k of genotype tree g, as the
// reference expands it in float32 (the angle offsets are pi / 2, pi and
// 3 pi / 2 rounded to float32 before the add):
//   180: (x, y, th), (-x, -y, th + pi)
//   90:  (x, y, th), (-y, x, th + pi/2), (-x, -y, th + pi), (y, -x, th + 3pi/2)
__device__ __forceinline__ void pk_image_pose(const float* X, int ng, int sym, int t, float& x, float& y, float& th)
{
    const int k = sym == 1 ? 0 : t / ng, g = t - k * ng;
    const float gx = X[3 * g], gy = X[3 * g + 1], gt = X[3 * g + 2];
    const float hpi = (float)(3.14159265358979323846 / 2.0), pi = (float)3.14159265358979323846,
                tpi = (float)(3.0 * 3.14159265358979323846 / 2.0);
    if (k == 0) { x = gx; y = gy; th = gt; }
    else if (sym == 2 || k == 2) { x = -gx; y = -gy; th = gt + pi; }
    else if (k == 1) { x = -gy; y = gx; th = gt + hpi; }
    else { x = gy; y = -gx; th = gt + tpi; }
}

struct PkEvalOut {
    double cost;
};

// Skin of the kept near lists (below), as a fraction of the cutoff distance.
// 0.22 relaxed 4096 x n = 200 (max_step 0.01) fastest of 0.12, 0.17, 0.22, 0.26.
#define PK_NEAR_SKIN 0.22f   // skin / cutoff distance

__device__ __forceinline__ float pk_near_skin() { return PK_NEAR_SKIN * sqrtf(c_geom.cutoff_sq); }

// Broad phase by testing every pair, for packings of at most 256 trees: thread
// per tree a, offsets 1 .. n/2 read from a position array that runs on past n
// (kept in the near list's space until that is written), one mask bit per test.
// Masks stay in the grid's cell arrays for pass 2, which expands them and tests
// nothing again.  Three barriers and about six instructions a test, against the
// grid's sorting by cell, two scans and two walks of the neighbourhoods behind a
// dozen barriers: n (n - 1) / 2 tests are the cheaper ones up to the 256 trees
// that the masks allow (one-shot area cost, grid -> this: 8192 x 40 201 -> 153 us,
// 4096 x 200 380 -> 344, 2048 x 250 231 -> 216; LUT, 8192 of 5 to 200 125 -> 102).
// Counts go to near_cnt, list offsets to near_start (in list order only if the
// list overflows), flags as in pk_broad_phase.  All threads call it, behind a
// barrier; pass 2 needs none in between.
__device__ __forceinline__ bool pk_all_pairs_fit(const PkCostSmem& sm, int n)
{
    return n <= 256 && (n + (n >> 1) + 32) * 8 <= sm.cap_near * 4;
}

template <bool KEEP>
__device__ __forceinline__ void pk_all_pairs(const PkCostSmem& sm, int n, bool build)
{
    const int T = blockDim.x, lane = threadIdx.x & 31, half = n >> 1;
    float2* pos = (float2*)sm.near;
    uint32_t* masks = (uint32_t*)sm.cell_start;   // [(half + 31) / 32][n]
    for (int t = threadIdx.x; t < n + half; t += T) {
        const float4 A = sm.pose[t < n ? t : t - n];
        pos[t] = make_float2(A.x, A.y);
    }
    if (threadIdx.x == 0) sm.near_start[n] = 0;
    float cut_list = c_geom.cutoff_sq;
    if (build) {
        const float r = sqrtf(cut_list) + pk_near_skin();
        cut_list = r * r;
    }
    for (;;) {
        __syncthreads();
        for (int a0 = 0; a0 < n; a0 += T) {
            const int a = a0 + threadIdx.x;
            int k = 0;
            if (a < n) {
                const float2 A = pos[a], nA = make_float2(-A.x, -A.y);
                for (int w = 0; 32 * w < half; ++w) {
                    const float2* o = pos + a + 1 + 32 * w;
                    const int nb = min(32, half - 32 * w);
                    uint32_t m = 0;
                    // rounded as pk_is_near rounds
#define PK_NEAR_BIT(B)                                                                       \
    {                                                                                        \
        const float2 d = __fadd2_rn(o[B], nA), q = __fmul2_rn(d, d);                         \
        if (__fadd_rn(q.x, q.y) <= cut_list) m |= 1u << (B);                                 \
    }
                    if (nb == 32) {
#pragma unroll
                        for (int b = 0; b < 32; ++b) PK_NEAR_BIT(b)
                    } else {
                        for (int b = 0; b < nb; b += 4)   // up to 3 past half: masked below
#pragma unroll
                            for (int u = 0; u < 4; ++u) PK_NEAR_BIT(b + u)
                        m &= (1u << nb) - 1u;
                    }
#undef PK_NEAR_BIT
                    if (32 * w + nb == half && 2 * half == n && a >= half) m &= ~(1u << (nb - 1));   // met twice
                    masks[w * n + a] = m;
                    k += __popc(m);
                }
                sm.near_cnt[a] = k;
            }
            int incl = k;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(PK_FULL_MASK, incl, o);
                if (lane >= o) incl += v;
            }
            int base = 0;
            if (lane == 31 && incl) base = atomicAdd(&sm.near_start[n], incl);
            base = __shfl_sync(PK_FULL_MASK, base, 31);
            if (a < n) sm.near_start[a] = base + incl - k;
        }
        if (KEEP && threadIdx.x == 0) {
            pk_nlist(sm)[2] = build;
            ((float*)pk_nlist(sm))[3] = cut_list;
        }
        __syncthreads();
        if (sm.near_start[n] <= sm.cap_near) break;
        if (!KEEP || !build) {   // several chunks: offsets in list order
            __syncthreads();
            pk_block_exclusive_scan(sm.near_cnt, sm.near_start, n, (int*)sm.redl);
            break;
        }
        // a kept list must fit in one piece: again at the cutoff, and no kept lists from now on
        build = false;
        cut_list = c_geom.cutoff_sq;
        __syncthreads();
        if (threadIdx.x == 0) { pk_nlist(sm)[0] = -1; sm.near_start[n] = 0; }
    }
    if (threadIdx.x == 0) sm.cnt[0] += (unsigned)(n * (n - 1) / 2);
}

// Broad phase on a uniform grid of cells at least the interaction distance
// wide: tree i only meets trees of the 3 x 3 cells around its own, and each
// pair is found once, from its lower index.  Builds the grid (sm.cell_start,
// sm.sorted, sm.tcell), counts each sorted position's near pairs (pass 1)
// and scans the counts into sm.near_start; returns the grid's (gx, gy), or (0, 0)
// when pk_all_pairs did it without a grid.
// build: take pairs within cutoff + skin for a kept list, falling back to the
// cutoff (and to no kept lists from then on) when they do not fit the near
// list in one piece.  Leaves pk_nlist(sm)[2] (list kept) and [3] (the
// distance pass 2 must use) for the caller, visible after its barriers.
// KEEP: the caller keeps near lists (the flags above); without it build is
// false and nothing is left in pk_nlist.  All threads call it.
template <bool KEEP>
__device__ __forceinline__ int2 pk_broad_phase(const PkCostSmem& sm, int n, bool build)
{
    if (pk_all_pairs_fit(sm, n)) {
        pk_all_pairs<KEEP>(sm, n, build);
        return make_int2(0, 0);
    }
    const int T = blockDim.x;
    const float cutoff = c_geom.cutoff_sq;
    float cut_list = cutoff;
    if (build) {
        const float r = sqrtf(cutoff) + pk_near_skin();
        cut_list = r * r;
    }
    int gx = 1, gy = 1;
    float4 bb = make_float4(-3.4e38f, -3.4e38f, -3.4e38f, -3.4e38f);   // (-min x, max x, -min y, max y)
    for (int t = threadIdx.x; t < n; t += T) {
        const float4 A = sm.pose[t];
        bb.x = fmaxf(bb.x, -A.x); bb.y = fmaxf(bb.y, A.x);
        bb.z = fmaxf(bb.z, -A.y); bb.w = fmaxf(bb.w, A.y);
    }
    bb = pk_block_max4(bb, (float*)sm.red);
    const float x0 = -bb.x, y0 = -bb.z;
    const float wx = fmaxf(bb.y - x0, 0.f), wy = fmaxf(bb.w - y0, 0.f);
    // 1 % wider than the interaction distance, so rounding in the cell
    // index never puts two interacting trees two cells apart
    float cs = sqrtf(cut_list) * 1.01f;
    for (int tries = 0; tries < 64; ++tries) {
        gx = (int)fminf(wx / cs, 2048.f) + 1;
        gy = (int)fminf(wy / cs, 2048.f) + 1;
        if (gx * gy <= sm.grid_cap) break;
        cs *= 1.25f;
    }
    if (gx * gy > sm.grid_cap) { gx = 1; gy = 1; cs = 3.4e38f; }   // non-finite extent: one cell
    const float inv = 1.0f / cs;
    const int ncell = gx * gy;
    for (int c = threadIdx.x; c < ncell; c += T) sm.cell_fill[c] = 0;
    __syncthreads();
    for (int t = threadIdx.x; t < n; t += T) {
        const float4 A = sm.pose[t];
        const int cx = min(gx - 1, max(0, (int)((A.x - x0) * inv)));
        const int cy = min(gy - 1, max(0, (int)((A.y - y0) * inv)));
        const int c = cy * gx + cx;
        sm.tcell[t] = c;
        atomicAdd(&sm.cell_fill[c], 1);
    }
    __syncthreads();
    pk_block_exclusive_scan(sm.cell_fill, sm.cell_start, ncell, (int*)sm.redl);
    for (int c = threadIdx.x; c < ncell; c += T) sm.cell_fill[c] = sm.cell_start[c];
    __syncthreads();
    for (int t = threadIdx.x; t < n; t += T) sm.sorted[atomicAdd(&sm.cell_fill[sm.tcell[t]], 1)] = t;
    __syncthreads();

    // Half neighbourhood of sorted position a in cell (cx, cy): the rest
    // of its own cell and the cell to its right (one contiguous range of
    // the sorted order), and cells cx-1..cx+1 of the row above (another).
    // Every pair of trees in touching cells is found exactly once.
    // Pass 1 counts the near pairs of each position, a scan turns the
    // counts into list offsets, and pass 2 writes them in chunks that fit
    // the near list, each chunk flushed before the next is written.
    unsigned tested = 0;
    for (int pass = 0; pass < 2; ++pass) {
        for (int a = threadIdx.x; a < n; a += T) {
            int b0, b1, b2, b3;
            pk_half_neighbourhood(sm, a, gx, gy, b0, b1, b2, b3);
            tested += (unsigned)(b1 - b0 + b3 - b2);
            const float4 A = sm.pose[sm.sorted[a]];
            int k = 0;
            for (int b = b0; b < b1; ++b) k += pk_is_near(A, sm.pose[sm.sorted[b]], cut_list);
            for (int b = b2; b < b3; ++b) k += pk_is_near(A, sm.pose[sm.sorted[b]], cut_list);
            sm.near_cnt[a] = k;
        }
        if (KEEP && threadIdx.x == 0) {
            // read by pass 2 and by the flush (after the scan's barriers)
            pk_nlist(sm)[2] = build;
            ((float*)pk_nlist(sm))[3] = cut_list;
        }
        __syncthreads();
        pk_block_exclusive_scan(sm.near_cnt, sm.near_start, n, (int*)sm.redl);
        // a kept list must fit the near list in one piece; when it does
        // not, count again at the cutoff and keep no lists from now on
        if (!KEEP || !build || sm.near_start[n] <= sm.cap_near) break;
        build = false;
        cut_list = cutoff;
        if (threadIdx.x == 0) pk_nlist(sm)[0] = -1;
    }
    atomicAdd(&sm.cnt[0], tested);
    return make_int2(gx, gy);
}

// The fused relaxation calls the broad phase and pass 2 out of line: with
// kept lists they run once per several evaluations, and their code then stays
// out of the hot loop's way.  A one-shot cost evaluation inlines them.  The
// out-of-line forms take the carve's sizes, not the caller's PkCostSmem (whose
// address would pin it to local memory), and carve the dynamic shared memory
// again: every kernel that evaluates costs places the cost arrays at its base.
__device__ __noinline__ int2 pk_broad_phase_outlined(int n_cap, int cap_near, int cap_items, int n, bool build)
{
    extern __shared__ __align__(16) unsigned char pk_smem[];
    const PkCostSmem sm = pk_cost_carve(pk_smem, n_cap, cap_near, cap_items, true);
    return pk_broad_phase<true>(sm, n, build);
}

// Pass 2: writes the near pairs of the longest run of sorted positions from
// a0 whose pairs fit the near list into sm.near, and keeps the list when
// pk_broad_phase built a kept one (the run is then every position).  Returns
// (end of the run, pairs written).  All threads call it; the pairs are
// written (behind a barrier) when it returns.
template <bool KEEP>
__device__ __forceinline__ int2 pk_write_near(const PkCostSmem& sm, int n, int a0, int gx, int gy)
{
    const int T = blockDim.x;
    int a1 = n, base = 0;
    if (gx > 0 || sm.near_start[n] > sm.cap_near) {
        // the longest run of positions from a0 whose pairs fit the list
        // (a single position's pairs always do: cap_near >= n_max)
        int lo = a0 + 1, hi = n;
        const int lim = sm.near_start[a0] + sm.cap_near;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sm.near_start[mid] <= lim) lo = mid; else hi = mid - 1;
        }
        a1 = lo;
        base = sm.near_start[a0];
    }
    const int cn = sm.near_start[a1] - base;
    if (gx == 0) {
        const uint32_t* masks = (const uint32_t*)sm.cell_start;
        for (int a = a0 + threadIdx.x; a < a1; a += T) {
            uint32_t* out = sm.near + (sm.near_start[a] - base);
            for (int w = 0; 64 * w < n - 1; ++w)   // the words pass 1 wrote: 32 w < n / 2
                for (uint32_t m = masks[w * n + a]; m; m &= m - 1) {
                    int j = a + 32 * w + __ffs(m);
                    if (j >= n) j -= n;
                    *out++ = (uint32_t)min(a, j) | ((uint32_t)max(a, j) << 11);
                }
        }
    } else {
        const float cut2 = KEEP ? ((const float*)pk_nlist(sm))[3] : c_geom.cutoff_sq;   // pass 1's distance
        for (int a = a0 + threadIdx.x; a < a1; a += T) {
            int b0, b1, b2, b3;
            pk_half_neighbourhood(sm, a, gx, gy, b0, b1, b2, b3);
            const int ia = sm.sorted[a];
            const float4 A = sm.pose[ia];
            uint32_t* out = sm.near + (sm.near_start[a] - base);
            const int kmax = sm.near_cnt[a];
            int k = 0;
            for (int b = b0; b < b3 && k < kmax; ++b) {
                if (b == b1) { b = b2; if (b >= b3) break; }
                const int ib = sm.sorted[b];
                if (pk_is_near(A, sm.pose[ib], cut2))
                    out[k++] = (uint32_t)min(ia, ib) | ((uint32_t)max(ia, ib) << 11);
            }
        }
    }
    __syncthreads();
    if (KEEP && pk_nlist(sm)[2]) {
        // the whole list is this one chunk: keep it, with the
        // positions it was built at in the grid's arrays (dead from here)
        for (int t = threadIdx.x; t < n; t += T) {
            const float4 A = sm.pose[t];
            ((float*)sm.sorted)[t] = A.x;
            ((float*)sm.tcell)[t] = A.y;
        }
        if (threadIdx.x == 0) { pk_nlist(sm)[0] = 1; pk_nlist(sm)[1] = cn; }
    } else if (threadIdx.x == 0) {
        sm.cnt[1] += (unsigned)cn;
    }
    return make_int2(a1, cn);
}

__device__ __noinline__ int2 pk_write_near_outlined(int n_cap, int cap_near, int cap_items, int n, int a0, int gx,
                                                   int gy)
{
    extern __shared__ __align__(16) unsigned char pk_smem[];
    const PkCostSmem sm = pk_cost_carve(pk_smem, n_cap, cap_near, cap_items, true);
    return pk_write_near<true>(sm, n, a0, gx, gy);
}

// The piece table in shared memory (SoA and AoS), from constant memory.
__device__ __forceinline__ void pk_load_piece_table(const PkCostSmem& sm)
{
    if (threadIdx.x < 16) {
        const float2 v = c_geom.piece[threadIdx.x >> 2][threadIdx.x & 3];
        sm.piece[threadIdx.x] = v;
        float* soa = (float*)sm.piece4;   // piece p: x at [8p + v], y at [8p + 4 + v]
        soa[8 * (threadIdx.x >> 2) + (threadIdx.x & 3)] = v.x;
        soa[8 * (threadIdx.x >> 2) + 4 + (threadIdx.x & 3)] = v.y;
    }
    if (threadIdx.x < 4) sm.piece_nv[threadIdx.x] = c_geom.piece_nv[threadIdx.x];
}

// Evaluate one instance.  X: 3n floats (global or shared), H: 3 floats or
// NULL.  G: 3n floats or NULL (written, not accumulated); GH: 3 floats or
// NULL.  Must be called by every thread of the block.
// SYM: the packing may be symmetric (spec.symmetry > 1); the plain
// instantiation keeps no symmetry state in registers.
// Kept near lists (KEEP, the fused relaxation only).  The list built by
// one evaluation holds every pair within cutoff + skin; a later evaluation
// reuses it, without building the cell grid, while no tree has moved by
// more than skin / (2 sqrt 2) per coordinate since, re-applying the exact
// centre cull to each listed pair.  Any pair near now was then within
// cutoff + skin, so the pairs evaluated are the same as a fresh grid's, and
// the fixed-point sums make the result independent of their order.
template <int MODE, bool SYM, bool KEEP = false>
__device__ double pk_eval_instance(const float* X, int ng, const float* H, const PkCostSpec& spec,
                                   float* G, float* GH, const PkCostSmem& sm)
{
    // ng genotype trees in X (3 ng floats); the cost is that of the n
    // phenotype trees, and G receives the genotype gradient
    const int sym = SYM ? pk_symmetry(spec) : 1;
    const int n = sym * ng;
    const int T = blockDim.x;
    const bool do_bnd = spec.w_boundary != 0.f && H != nullptr;
    float half = 0.f, hox = 0.f, hoy = 0.f;
    if (H) { half = H[0] * 0.5f; hox = H[1]; hoy = H[2]; }
    // piece table into shared memory first: phase 0 reads it (the fused
    // relaxation loads it once, before its first evaluation)
    if (!KEEP) {
        pk_load_piece_table(sm);
    }
    // kept list state, written by the last evaluation that built the grid
    const int nstate = KEEP ? pk_nlist(sm)[0] : -1;
    float disp = 0.f;   // largest coordinate change of this thread's trees since the list was built
    if (!KEEP) __syncthreads();
    // ---- phase 0: per tree -------------------------------------------------
    for (int t = threadIdx.x; t < n; t += T) {
        float x, y, th;
        pk_image_pose(X, ng, sym, t, x, y, th);
        if (nstate == 1) {
            // positions when the list was built, kept in the grid's dead arrays
            const float dm = fmaxf(fabsf(__fsub_rn(x, ((const float*)sm.sorted)[t])),
                                   fabsf(__fsub_rn(y, ((const float*)sm.tcell)[t])));
            disp = dm <= 1e30f ? fmaxf(disp, dm) : 3.4e38f;   // NaN or infinite: rebuild
        }
        float s, c;
        sincosf(th, &s, &c);
        sm.pose[t] = make_float4(x, y, c, s);
        sm.theta[t] = th;
        long long a0 = 0, a1 = 0, a2 = 0;
        float4 bnd = make_float4(0.f, 0.f, 0.f, 0.f);
        if (MODE == PK_PAIR_AREA || MODE == PK_PAIR_SEP) {
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                float2 V[4];
                pk_load_piece(sm, p, c, s, 0.f, 0.f, V);
                float4 bb = make_float4(V[0].x, V[0].x, V[0].y, V[0].y);
#pragma unroll
                for (int v = 1; v < 4; ++v) {
                    bb.x = fminf(bb.x, V[v].x); bb.y = fmaxf(bb.y, V[v].x);
                    bb.z = fminf(bb.z, V[v].y); bb.w = fmaxf(bb.w, V[v].y);
                }
                const float eps = 1e-6f;
                sm.aabb[p * sm.n_cap + t] = make_float4(bb.x - eps, bb.y + eps, bb.z - eps, bb.w + eps);
            }
        }
        if (do_bnd) {
            // boundary_distance_tree, pack_cuda.py:550-642
            float best = 0.f;
            int bi = 0;
            for (int v = 0; v < c_geom.n_tree; ++v) {
                const float2 l = c_geom.tree[v];
                const float vx = c * l.x - s * l.y + x - hox;
                const float vy = s * l.x + c * l.y + y - hoy;
                const float ax = fabsf(vx), ay = fabsf(vy);
                const float dx = ax > half ? ax - half : 0.f;
                const float dy = ay > half ? ay - half : 0.f;
                const float dd = dx * dx + dy * dy;
                if (dd > best) { best = dd; bi = v; }
            }
            const float2 l = c_geom.tree[bi];
            const float vx = c * l.x - s * l.y + x - hox;
            const float vy = s * l.x + c * l.y + y - hoy;
            const float ax = fabsf(vx), ay = fabsf(vy);
            const float dx = ax > half ? ax - half : 0.f;
            const float dy = ay > half ? ay - half : 0.f;
            const float gvx = dx > 0.f ? 2.0f * dx * (vx >= 0.f ? 1.f : -1.f) : 0.f;
            const float gvy = dy > 0.f ? 2.0f * dy * (vy >= 0.f ? 1.f : -1.f) : 0.f;
            const float gth = gvx * (-s * l.x - c * l.y) + gvy * (c * l.x - s * l.y);
            const float wb = spec.w_boundary;
            a0 = pk_to_fx(wb * gvx);
            a1 = pk_to_fx(wb * gvy);
            a2 = pk_to_fx(wb * gth);
            bnd = make_float4(best, -(dx + dy), -gvx, -gvy);
        }
        sm.acc_lo[3 * t] = (unsigned)a0;
        sm.acc_hi[3 * t] = (unsigned)((unsigned long long)a0 >> 32);
        sm.acc_lo[3 * t + 1] = (unsigned)a1;
        sm.acc_hi[3 * t + 1] = (unsigned)((unsigned long long)a1 >> 32);
        sm.acc_lo[3 * t + 2] = (unsigned)a2;
        sm.acc_hi[3 * t + 2] = (unsigned)((unsigned long long)a2 >> 32);
        sm.bnd[t] = bnd;
    }
    if (threadIdx.x == 0) {
        sm.count[0] = 0;
        sm.count[1] = 0x7fffffff;
        sm.cnt[3] += 1;
    }
    if (nstate == 1) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) disp = fmaxf(disp, __shfl_xor_sync(PK_FULL_MASK, disp, o));
        if ((threadIdx.x & 31) == 0) pk_disp(sm)[threadIdx.x >> 5] = disp;
    }
    __syncthreads();
    bool reuse = false;
    if (nstate == 1) {
        float dm = 0.f;
        for (int w = 0; w < (T >> 5); ++w) dm = fmaxf(dm, pk_disp(sm)[w]);
        // a pair's distance moved by at most 2 sqrt 2 dm; 1e-4 covers the rounding
        reuse = 2.8285f * dm + 1e-4f < pk_near_skin();
    }

    // ---- phases A + B: pairs -------------------------------------------------
    long long pair_tot = 0;
    if (MODE != PK_PAIR_NONE && n > 1) {
        int gx = 1, gy = 1;
        int a0 = reuse ? -1 : 0;   // -1: flush the kept list
        if (!reuse) {
            // without a kept list to reuse, build one this time (nstate >= 0)
            const int2 g = KEEP ? pk_broad_phase_outlined(sm.n_cap, sm.cap_near, sm.cap_items, n, nstate >= 0)
                                : pk_broad_phase<false>(sm, n, false);
            gx = g.x;
            gy = g.y;
        }
        while (a0 < n) {
            int cn;
            if (a0 < 0) {
                // the kept list (pk_nlist(sm)[2] is still set from when it was built)
                cn = pk_nlist(sm)[1];
                if (threadIdx.x == 0) sm.cnt[0] += (unsigned)cn;
                a0 = n;
            } else {
                const int2 r = KEEP ? pk_write_near_outlined(sm.n_cap, sm.cap_near, sm.cap_items, n, a0, gx, gy)
                                    : pk_write_near<false>(sm, n, a0, gx, gy);
                a0 = r.x;
                cn = r.y;
            }
            if (cn > 0) pair_tot += pk_flush_near<MODE, KEEP>(sm, cn, spec, T);
        }
    }

    // ---- phase C: outputs ----------------------------------------------------
    if (G) {
        // genotype gradient: the images' gradients through the symmetry's
        // rotations (backprop_phenotype, kaggle_support.py:1366-1393 and
        // :1155-1195), combined exactly in fixed point
        for (int t = threadIdx.x; t < ng; t += T) {
            long long gx = pk_acc_get(sm, 3 * t), gy = pk_acc_get(sm, 3 * t + 1), gt = pk_acc_get(sm, 3 * t + 2);
            if (sym == 2) {
                const int u = 3 * (t + ng);
                gx -= pk_acc_get(sm, u); gy -= pk_acc_get(sm, u + 1); gt += pk_acc_get(sm, u + 2);
            } else if (sym == 4) {
                const int u1 = 3 * (t + ng), u2 = 3 * (t + 2 * ng), u3 = 3 * (t + 3 * ng);
                gx = gx + pk_acc_get(sm, u1 + 1) - pk_acc_get(sm, u2) - pk_acc_get(sm, u3 + 1);
                gy = gy - pk_acc_get(sm, u1) - pk_acc_get(sm, u2 + 1) + pk_acc_get(sm, u3);
                gt = gt + pk_acc_get(sm, u1 + 2) + pk_acc_get(sm, u2 + 2) + pk_acc_get(sm, u3 + 2);
            }
            G[3 * t] = (float)((double)gx * PK_FX_INV);
            G[3 * t + 1] = (float)((double)gy * PK_FX_INV);
            G[3 * t + 2] = (float)((double)gt * PK_FX_INV);
        }
    }
    // one barrier for every total: per-warp pair partials (int64: exact in
    // any order) and the boundary sums of warp 0
    {
        const long long wsum = pk_warp_sum(pair_tot);
        if ((threadIdx.x & 31) == 0) sm.redl[threadIdx.x >> 5] = wsum;
        if (do_bnd && threadIdx.x < 32) {
            const double4 b4 = pk_canonical_sum4(n, sm.bnd);
            if (threadIdx.x == 0) { sm.red[0] = b4.x; sm.red[1] = b4.y; sm.red[2] = b4.z; sm.red[3] = b4.w; }
        }
        __syncthreads();
    }
    long long ptot = 0;
    for (int w = 0; w < (T >> 5); ++w) ptot += sm.redl[w];
    double total = (double)ptot * PK_FX_INV;
    double h0 = H ? (double)H[0] : 0.0;
    if (do_bnd) {
        total += (double)spec.w_boundary * sm.red[0];
        if (GH && threadIdx.x == 0) {
            GH[0] = (float)(spec.w_boundary * sm.red[1] + (double)spec.w_area * 2.0 * h0);
            GH[1] = (float)(spec.w_boundary * sm.red[2]);
            GH[2] = (float)(spec.w_boundary * sm.red[3]);
        }
    } else if (GH && threadIdx.x == 0) {
        GH[0] = (float)((double)spec.w_area * 2.0 * h0);
        GH[1] = 0.f;
        GH[2] = 0.f;
    }
    if (GH && spec.fixed_h && threadIdx.x == 0) { GH[0] = 0.f; GH[1] = 0.f; GH[2] = 0.f; }
    // AreaCost is zero with a fixed side, its gradient too (use_fixed_h,
    // pack_cost.py:1276-1282; every term's h gradient is zeroed, :178-189)
    if (!spec.fixed_h) total += (double)spec.w_area * h0 * h0;
    __syncthreads();
    return total;
}

// The size classes of an order that one launch covers: position b of the order
// belongs to the first class whose end lies beyond it (all ends 0: no classes).
// A parameter of a build of its own (Bounds): read by every launch they cost the
// six forked ones of a large batch 18 of 111 us, whose parameters together then no
// longer fit the SM's constant cache, and unread they cost a 64 x 20 call 0.4 of 14
// us.  Applied to the result: before the evaluation their registers made the LUT
// build spill (2000 packings of 5 to 200 trees 38.5 -> 42 us).
#define PK_MAX_BOUNDS 8
struct PkClassBounds { unsigned c[PK_MAX_BOUNDS]; };   // end << 11 | n_max

// CTA b costs instance order[b] (instance b without an order).  The LUT
// mode has no clipper: it fits 64 registers without spilling, so four CTAs of
// 256 threads share an SM and one CTA's broad phase overlaps the others'
// gathers (4096 x n = 200: 0.201 -> 0.183 ms, the same bits).
template <int MODE, bool SYM, typename... Bounds>
__global__ void __launch_bounds__(256, MODE == PK_PAIR_LUT ? 4 : 3) pk_cost_kernel(const float* __restrict__ xyt, const int* __restrict__ offsets,
                               const int* __restrict__ order, int E,
                               int n_max, const float* __restrict__ h, PkCostSpec spec,
                               float* __restrict__ cost, float* __restrict__ grad,
                               float* __restrict__ grad_h, int cap_near, int cap_items, const Bounds... cls)
{
    extern __shared__ __align__(16) unsigned char pk_smem[];
    const int e = order ? order[blockIdx.x] : blockIdx.x;

    if (e < 0 || e >= E) return;
    const int base = offsets ? offsets[e] : e * n_max;
    const int n = offsets ? offsets[e + 1] - base : n_max;
    if (n < 0 || n > n_max) {
        if (threadIdx.x == 0) cost[e] = __int_as_float(0x7fc00000);   // NaN marks a bad offset
        return;
    }
    PkCostSmem sm = pk_cost_carve(pk_smem, n_max * (SYM ? pk_symmetry(spec) : 1), cap_near, cap_items);
    if (threadIdx.x < 4) sm.cnt[threadIdx.x] = 0;
    __syncthreads();
    const double tot = pk_eval_instance<MODE, SYM>(xyt + (size_t)base * 3, n, h ? h + 3 * e : nullptr, spec,
                                              grad ? grad + (size_t)base * 3 : nullptr,
                                              grad_h ? grad_h + 3 * e : nullptr, sm);
    if (threadIdx.x == 0) {
        float c = (float)tot;
        if constexpr (sizeof...(Bounds) == 1) {
            int most = n_max;
#pragma unroll
            for (int k = PK_MAX_BOUNDS - 1; k >= 0; --k)
                if (blockIdx.x < ((cls.c[k] >> 11), ...)) most = ((int)(cls.c[k] & 2047), ...);
            if (n > most) c = __int_as_float(0x7fc00000);
        }
        cost[e] = c;
    }
}

// Multiprocessors of the current device (0 on error), asked once per device.
static int pk_sm_count()
{
    static std::atomic<int> cache[64];
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    sms = cache[dev].load(std::memory_order_relaxed);
    if (sms == 0 && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
        cache[dev].store(sms, std::memory_order_relaxed);
    return sms;
}

// Threads per CTA.  The results do not depend on them (fixed-point sums,
// reductions whose order the packing alone fixes).  A batch that fills the GPU
// gets about one thread per tree.  One that does not is as slow as its slowest
// CTA, so its CTAs grow, up to 3 x 256 threads per SM over the whole batch and
// to where more threads stop helping (n <= 24: 128, n <= 64: 192).  20
// iterations of 8 packings, us with 64 / 128 / 192 / 256 threads: n = 20 299 /
// 245 / 246 / 249, n = 50 486 / 358 / 320 / 310, n = 100 964 / 538 / 452 / 397;
// 256 packings: n = 20 358 / 309 / 281 / 286, n = 50 566 / 410 / 364 / 388,
// n = 100 1109 / 654 / 550 / 512.
static inline int pk_cost_threads(int n_max, int count)
{
    const int full = n_max <= 48 ? 64 : (n_max <= 128 ? 128 : 256);
    const int most = n_max <= 24 ? 128 : (n_max <= 64 ? 192 : 256);
    const int sms = pk_sm_count() > 0 ? pk_sm_count() : 1;
    const int per_sm = count > 0 ? (count + sms - 1) / sms : 1;   // CTAs an SM has to hold
    const int room = (768 / per_sm) & ~31;
    const int wide = room < most ? room : most;
    return wide > full ? wide : full;
}

// Raises a kernel's dynamic shared memory limit only when a launch needs more
// than any earlier one on this device, so warmed-up launches make no
// attribute call (they can then be captured into a CUDA graph).  Slots: 0-3 and
// 28-31, 40-47 the cost kernels, 4-19, 32-39 the relaxation's, 20-27 the jobs'.
static cudaError_t pk_set_smem(const void* fn, int slot, size_t smem)
{
    static size_t done[64][48];
    static unsigned gen[64];
    static std::mutex mu;
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < 0 || dev >= 64 || slot < 0 || slot >= 48) return cudaErrorInvalidValue;
    std::lock_guard<std::mutex> lock(mu);
    if (gen[dev] != g_pk_init_gen[dev]) {   // pk_init again, perhaps on a new context: nothing is raised there
        memset(done[dev], 0, sizeof(done[dev]));
        gen[dev] = g_pk_init_gen[dev];
    }
    if (smem <= done[dev][slot]) return cudaSuccess;
    err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err == cudaSuccess) done[dev][slot] = smem;
    return err;
}

// Checks the arguments of a cost launch of count instances with at most n_max
// trees, and gives its threads (threads 0: pk_cost_threads of the size bound) and
// shared memory.  *T = 0: nothing to do.
struct PkCostLaunch { int T, cap_near, cap_items; size_t smem; };

static int pk_cost_args(const float* xyt, const int* order, int count, int E, int n_max, const float* h,
                        const PkCostSpec* spec, int threads, const float* cost, PkCostLaunch* L)
{
    L->T = 0;
    int rc = pk_check_init();
    if (rc) return rc;
    if (!spec) return pk_fail(PK_EINVAL, "pk_cost: spec is NULL%s");
    if (E < 0 || n_max < 0) return pk_fail(PK_EINVAL, "pk_cost: negative size%s");
    if (count < 0 || count > E) return pk_fail(PK_EINVAL, "pk_cost: order count must be in [0, E]%s");
    if (count < E && !order) return pk_fail(PK_EINVAL, "pk_cost: a partial launch needs an order%s");
    if (E == 0 || count == 0) return PK_OK;
    if (spec->symmetry != 0 && spec->symmetry != 1 && spec->symmetry != 2 && spec->symmetry != 4)
        return pk_fail(PK_EINVAL, "pk_cost: symmetry must be 0, 1, 2 or 4%s");
    if (n_max > PK_MAX_TREES || (long long)n_max * pk_symmetry(*spec) > PK_MAX_TREES)
        return pk_fail(PK_ERANGE, "pk_cost: more than 1024 (phenotype) trees per instance%s");
    if (!cost || (!xyt && n_max > 0)) return pk_fail(PK_EINVAL, "pk_cost: xyt and cost are required%s");
    if (spec->w_boundary != 0.f && !h) return pk_fail(PK_EINVAL, "pk_cost: boundary term needs h%s");
    if (spec->w_area != 0.f && !h) return pk_fail(PK_EINVAL, "pk_cost: area term needs h%s");
    if (spec->pair_mode < PK_PAIR_NONE || spec->pair_mode > PK_PAIR_LUT)
        return pk_fail(PK_EINVAL, "pk_cost: unknown pair_mode%s");
    if (spec->pair_mode == PK_PAIR_LUT) {
        const PkLut& l = spec->lut;
        if (!l.vals || l.nx < 2 || l.ny < 2 || l.nt < 2)
            return pk_fail(PK_EINVAL, "pk_cost: LUT needs vals and at least 2 points per axis%s");
    }
    const int n = n_max * pk_symmetry(*spec);
    if (threads != 0 && (threads < 32 || threads > 256 || (threads & 31) || 8 * threads < n - 1))
        return pk_fail(PK_EINVAL, "pk_cost: threads must be 0 or a multiple of 32 in [32, 256] with "
                                  "8 * threads >= n - 1%s");
    L->T = threads != 0 ? threads : pk_cost_threads(n, count);
    pk_caps(L->T, spec->pair_mode, &L->cap_near, &L->cap_items);
    L->smem = pk_cost_smem_bytes(n, L->cap_near, L->cap_items);
    return PK_OK;
}

// count entries of the launch order (all E instances when order is NULL).
static int pk_launch_cost(const float* xyt, const int* offsets, const int* order, int count, int E, int n_max,
                          const float* h, const PkCostSpec* spec, int threads, float* cost, float* grad,
                          float* grad_h, cudaStream_t st, const PkClassBounds* classes = nullptr)
{
    PkCostLaunch L;
    const int rc = pk_cost_args(xyt, order, count, E, n_max, h, spec, threads, cost, &L);
    if (rc || L.T == 0) return rc;
    cudaError_t err = cudaSuccess;
    switch (spec->pair_mode) {
#define PK_CASE2(SLOT, KERNEL, ...)                                                                 \
    {                                                                                               \
        err = pk_set_smem((const void*)KERNEL, SLOT, L.smem);                                       \
        if (err == cudaSuccess)                                                                     \
            KERNEL<<<count, L.T, L.smem, st>>>(xyt, offsets, order, E, n_max, h, *spec, cost, grad, grad_h, L.cap_near, \
                                               __VA_ARGS__);                                        \
    }
#define PK_CASE(M)                                                                                  \
    case M:                                                                                         \
        if (classes && spec->symmetry > 1)                                                          \
            PK_CASE2(44 + M, (pk_cost_kernel<M, true, PkClassBounds>), L.cap_items, *classes)       \
        else if (classes) PK_CASE2(40 + M, (pk_cost_kernel<M, false, PkClassBounds>), L.cap_items, *classes) \
        else if (spec->symmetry > 1) PK_CASE2(28 + M, (pk_cost_kernel<M, true>), L.cap_items)       \
        else PK_CASE2(M, (pk_cost_kernel<M, false>), L.cap_items)                                   \
        if (err == cudaSuccess) err = cudaGetLastError();                                           \
        break;
        PK_CASE(PK_PAIR_NONE)
        PK_CASE(PK_PAIR_AREA)
        PK_CASE(PK_PAIR_SEP)
        PK_CASE(PK_PAIR_LUT)
#undef PK_CASE
#undef PK_CASE2
    }
    return pk_cuda_check(err, "pk_cost launch");
}

extern "C" int pk_cost(const float* xyt, const int* offsets, int E, int n_uniform, const float* h,
                       const PkCostSpec* spec, float* cost, float* grad, float* grad_h, void* stream)
{
    return pk_launch_cost(xyt, offsets, nullptr, E, E, n_uniform, h, spec, 0, cost, grad, grad_h,
                          (cudaStream_t)stream);
}

extern "C" int pk_cost_ordered(const float* xyt, const int* offsets, const int* order, int count, int E, int n_max,
                               const float* h, const PkCostSpec* spec, int threads, float* cost, float* grad,
                               float* grad_h, void* stream)
{
    if (!order) return pk_fail(PK_EINVAL, "pk_cost_ordered: order is required%s");
    return pk_launch_cost(xyt, offsets, order, count, E, n_max, h, spec, threads, cost, grad, grad_h,
                          (cudaStream_t)stream);
}

// The size classes of a largest-first order, class k on side[k], forked from and
// joined to stream, or in one launch on stream: one call instead of a launch and
// five event calls per class from Python (16 us each, 100 for a ragged batch
// whose kernels take 100).
extern "C" int pk_cost_classes(const float* xyt, const int* offsets, const int* order, const PkSizeClass* cls,
                               int ncls, int E, int n_max, const float* h, const PkCostSpec* spec, float* cost,
                               float* grad, float* grad_h, void* stream, void* const* side)
{
    if (!offsets || !order || !cls || !side || ncls < 0)
        return pk_fail(PK_EINVAL, "pk_cost_classes: offsets, order, classes and side streams are required%s");
    long long total = 0;
    int most = 0;   // trees of the largest class
    for (int k = 0; k < ncls; ++k) {
        const PkSizeClass& c = cls[k];
        if (c.start < 0 || c.count < 0 || (long long)c.start + c.count > E || c.n_max > n_max)
            return pk_fail(PK_EINVAL, "pk_cost_classes: classes must cover the order once, each within n_max%s");
        total += c.count;
        most = c.n_max > most ? c.n_max : most;
    }
    if (total != E) return pk_fail(PK_EINVAL, "pk_cost_classes: classes must cover the order once, each within n_max%s");
    cudaStream_t base = (cudaStream_t)stream;
    if (ncls == 1)
        return pk_launch_cost(xyt, offsets, order, E, E, cls[0].n_max, h, spec, cls[0].threads, cost, grad, grad_h, base);
    // One launch does without forking and joining (about 20 us), but gives every
    // packing the CTA of the largest one.  It is faster while the GPU takes the
    // batch in a few waves of such CTAs; by (E / resident CTAs), one launch
    // against forked, in us:
    //   LUT, 5 to 200 trees:  3.4  40 / 52,  5.1  58 / 55;  5 to 900:  3.4  54 / 62,  6.8  95 / 75,  14  184 / 128
    //   area, 5 to 200: 1.1  30 / 43,  4.5  75 / 72;  5 to 900: 3.4  95 / 114,  6.8  155 / 138,  14  305 / 230
    //   separation, 5 to 200:  4.5  85 / 88;  2000 of 10 trees and one of 900, LUT:  14  80 / 58
    PkClassBounds bounds = {};
    bool one = E <= 16 * pk_sm_count() && ncls <= PK_MAX_BOUNDS;
    for (int k = 0, at = 0; k < ncls && one; ++k) {
        one = cls[k].start == at;   // positions left out or named twice: class by class
        at += cls[k].count;
        bounds.c[k] = ((unsigned)at << 11) | (unsigned)(cls[k].n_max & 2047);   // n_max <= 1024 is checked below
    }
    if (one) {
        PkCostLaunch L;
        for (int k = 0; k < ncls; ++k) {   // what a class of its own refuses stays refused
            const int rc = pk_cost_args(xyt, order, cls[k].count, E, cls[k].n_max, h, spec, cls[k].threads, cost, &L);
            if (rc) return rc;
        }
        const int rc = pk_cost_args(xyt, order, E, E, most, h, spec, 0, cost, &L);
        if (rc || L.T == 0) return rc;
        const int by_regs = (spec->pair_mode == PK_PAIR_LUT ? 1024 : 768) / L.T;   // the kernel's launch bounds
        const int by_smem = (int)((size_t)228 * 1024 / (L.smem + 1024));
        if (E <= 5LL * pk_sm_count() * (by_smem < by_regs ? by_smem : by_regs))
            return pk_launch_cost(xyt, offsets, order, E, E, most, h, spec, 0, cost, grad, grad_h, base, &bounds);
    }
    cudaEvent_t fork = nullptr, join = nullptr;
    cudaError_t err = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
    if (err == cudaSuccess) err = cudaEventCreateWithFlags(&join, cudaEventDisableTiming);
    if (err == cudaSuccess) err = cudaEventRecord(fork, base);
    int rc = PK_OK;
    for (int k = 0; k < ncls && err == cudaSuccess && rc == PK_OK; ++k) {
        cudaStream_t st = (cudaStream_t)side[k];
        err = cudaStreamWaitEvent(st, fork, 0);
        if (err != cudaSuccess) break;
        rc = pk_launch_cost(xyt, offsets, order + cls[k].start, cls[k].count, E, cls[k].n_max, h, spec, cls[k].threads,
                            cost, grad, grad_h, st);
        // join even after a refused launch: a forked stream is not left behind
        err = cudaEventRecord(join, st);
        if (err == cudaSuccess) err = cudaStreamWaitEvent(base, join, 0);
    }
    if (fork) cudaEventDestroy(fork);
    if (join) cudaEventDestroy(join);
    return rc ? rc : pk_cuda_check(err, "pk_cost_classes");
}

extern "C" int pk_overlap(const float* xyt, int E, int n, int use_separation, float* cost, float* grad,
                          void* stream)
{
    PkCostSpec s;
    memset(&s, 0, sizeof(s));
    s.pair_mode = use_separation ? PK_PAIR_SEP : PK_PAIR_AREA;
    s.w_pair = 1.f;
    return pk_launch_cost(xyt, nullptr, nullptr, E, E, n, nullptr, &s, 0, cost, grad, nullptr, (cudaStream_t)stream);
}

extern "C" int pk_boundary(const float* xyt, const float* h, int E, int n, float* cost, float* grad,
                           float* grad_h, void* stream)
{
    PkCostSpec s;
    memset(&s, 0, sizeof(s));
    s.pair_mode = PK_PAIR_NONE;
    s.w_boundary = 1.f;
    return pk_launch_cost(xyt, nullptr, nullptr, E, E, n, h, &s, 0, cost, grad, grad_h, (cudaStream_t)stream);
}

extern "C" int pk_overlap_lut(const float* xyt, const int* offsets, int E, int n_uniform, const PkLut* lut,
                              float* cost, float* grad, void* stream)
{
    if (!lut) return pk_fail(PK_EINVAL, "pk_overlap_lut: lut is NULL%s");
    PkCostSpec s;
    memset(&s, 0, sizeof(s));
    s.pair_mode = PK_PAIR_LUT;
    s.w_pair = 1.f;
    s.lut = *lut;
    return pk_launch_cost(xyt, offsets, nullptr, E, E, n_uniform, nullptr, &s, 0, cost, grad, nullptr,
                          (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// LUT construction from the analytic pair cost: vals[ix, iy, it] = cost of
// a tree at the origin (theta 0) and one at (X[ix], Y[iy], T[it]) -- the
// eval_fn of CollisionCost._ensure_lut_initialized (pack_cost.py:333-377),
// which evaluates 2-tree ensembles with the kernel cost.  Thread per grid
// point; all 16 piece pairs after the centre and AABB culls.
// ---------------------------------------------------------------------------
template <int MODE>
__global__ void pk_lut_build_kernel(const float* __restrict__ X, int nx, const float* __restrict__ Y, int ny,
                                    const float* __restrict__ Tt, int nt, float* __restrict__ vals)
{
    const size_t total = (size_t)nx * ny * nt;
    for (size_t w = blockIdx.x * (size_t)blockDim.x + threadIdx.x; w < total; w += (size_t)gridDim.x * blockDim.x) {
        const int it = (int)(w % nt);
        const int iy = (int)((w / nt) % ny);
        const int ix = (int)(w / ((size_t)nt * ny));
        const float2 d = make_float2(X[ix], Y[iy]);
        float acc = 0.f;
        if (d.x * d.x + d.y * d.y <= c_geom.cutoff_sq) {
            float s, c;
            sincosf(Tt[it], &s, &c);
#pragma unroll 1
            for (int p = 0; p < 4; ++p) {
                float2 P[4];
                float4 bp = make_float4(1e30f, -1e30f, 1e30f, -1e30f);
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    P[v] = c_geom.piece[p][v];
                    bp.x = fminf(bp.x, P[v].x); bp.y = fmaxf(bp.y, P[v].x);
                    bp.z = fminf(bp.z, P[v].y); bp.w = fmaxf(bp.w, P[v].y);
                }
#pragma unroll 1
                for (int q = 0; q < 4; ++q) {
                    float2 Q[4];
                    float4 bq = make_float4(1e30f, -1e30f, 1e30f, -1e30f);
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        const float2 l = c_geom.piece[q][v];
                        Q[v] = make_float2(c * l.x - s * l.y + d.x, s * l.x + c * l.y + d.y);
                        bq.x = fminf(bq.x, Q[v].x); bq.y = fmaxf(bq.y, Q[v].x);
                        bq.z = fminf(bq.z, Q[v].y); bq.w = fmaxf(bq.w, Q[v].y);
                    }
                    if (bp.y < bq.x || bq.y < bp.x || bp.w < bq.z || bq.w < bp.z) continue;
                    float val;
                    float3 gp, gq;
                    const bool pt = c_geom.piece_nv[p] == 3, qt = c_geom.piece_nv[q] == 3;
                    if (MODE == PK_PAIR_AREA) {
                        pk_piece_area_grad(P, pt, Q, qt, d, val, gp, gq);
                    } else {
                        float sp;
                        pk_piece_sat_grad(P, pt, Q, qt, d, sp, gp, gq);
                        val = sp * sp;
                    }
                    acc += val;
                }
            }
        }
        vals[w] = acc;
    }
}

extern "C" int pk_lut_build(const float* X, int nx, const float* Y, int ny, const float* T, int nt, int pair_mode,
                            float* vals, void* stream)
{
    int rc = pk_check_init();
    if (rc) return rc;
    if (nx < 1 || ny < 1 || nt < 1) return pk_fail(PK_EINVAL, "pk_lut_build: empty grid%s");
    if (!X || !Y || !T || !vals) return pk_fail(PK_EINVAL, "pk_lut_build: NULL pointer%s");
    const size_t total = (size_t)nx * ny * nt;
    const int blocks = (int)((total + 255) / 256 < 148 * 32 ? (total + 255) / 256 : 148 * 32);
    cudaStream_t st = (cudaStream_t)stream;
    if (pair_mode == PK_PAIR_AREA)
        pk_lut_build_kernel<PK_PAIR_AREA><<<blocks, 256, 0, st>>>(X, nx, Y, ny, T, nt, vals);
    else if (pair_mode == PK_PAIR_SEP)
        pk_lut_build_kernel<PK_PAIR_SEP><<<blocks, 256, 0, st>>>(X, nx, Y, ny, T, nt, vals);
    else
        return pk_fail(PK_EINVAL, "pk_lut_build: pair_mode must be AREA or SEP%s");
    return pk_cuda_check(cudaGetLastError(), "pk_lut_build launch");
}
