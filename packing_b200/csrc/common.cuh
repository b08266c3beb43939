// common.cuh -- shared definitions for the packing_b200 CUDA library.
//
// The library is one translation unit (capi.cu includes every *.cuh), so the
// __constant__ / __device__ symbols below exist once per loaded library.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/packb200.h"

#define PK_FULL_MASK 0xffffffffu

// Tree geometry in the form the kernels read it.  Pieces are CCW; a
// triangle is padded to four vertices as [v0, v1, v2, v0], so its edge 3 is
// degenerate (zero length) and is skipped as a clipping line.
struct PkDevGeom {
    float2 piece[PK_NUM_PIECES][4];
    int piece_nv[PK_NUM_PIECES];
    float2 tree[PK_MAX_TREE_VERTS];
    int n_tree;
    float max_radius;
    float cutoff_sq;    // (2 R)^2: farther centres cannot overlap
    float coll_tiny;    // 2e-6 * longest piece edge: bound on |cross| of near-collinear points
};

// FP64 tables: the search tree, and the legality tree of the validator
// (CCW pieces padded like the FP32 ones).
struct PkDevGeom64 {
    double2 piece[PK_NUM_PIECES][4];
    int piece_nv[PK_NUM_PIECES];
    double2 tree[PK_MAX_TREE_VERTS];
    int n_tree;
    double max_radius;
    double2 legal_piece[PK_NUM_PIECES][4];
    double2 legal_tree[PK_MAX_TREE_VERTS];
    double legal_radius;
};

__constant__ PkDevGeom c_geom;
__constant__ PkDevGeom64 c_geom64;

// Fixed-point scale of the pair-gradient accumulators: sums of int64 are
// associative, so the result does not depend on the order in which threads
// add their contributions (batched == single, bit for bit).
#define PK_FX_SCALE 4294967296.0f          // 2^32
#define PK_FX_INV (1.0 / 4294967296.0)

__device__ __forceinline__ long long pk_to_fx(float v)
{
    return __float2ll_rn(v * PK_FX_SCALE);
}

__device__ __forceinline__ float pk_cross(float2 a, float2 b) { return a.x * b.y - a.y * b.x; }

// (B - A) x (C - A): >= 0 means C is on or left of the directed line A->B.
__device__ __forceinline__ float pk_cross3(float2 a, float2 b, float2 c)
{
    return (b.x - a.x) * (c.y - a.y) - (b.y - a.y) * (c.x - a.x);
}

template <typename T>
__device__ __forceinline__ T pk_warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(PK_FULL_MASK, v, o);
    return v;
}

// Block-wide maximum of four floats at once (one round trip through
// shared memory); scratch needs 4 * warps floats.  All threads get the result.
__device__ __forceinline__ float4 pk_block_max4(float4 v, float* scratch)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x = fmaxf(v.x, __shfl_xor_sync(PK_FULL_MASK, v.x, o));
        v.y = fmaxf(v.y, __shfl_xor_sync(PK_FULL_MASK, v.y, o));
        v.z = fmaxf(v.z, __shfl_xor_sync(PK_FULL_MASK, v.z, o));
        v.w = fmaxf(v.w, __shfl_xor_sync(PK_FULL_MASK, v.w, o));
    }
    __syncthreads();
    if (lane == 0) {
        scratch[4 * warp + 0] = v.x; scratch[4 * warp + 1] = v.y;
        scratch[4 * warp + 2] = v.z; scratch[4 * warp + 3] = v.w;
    }
    __syncthreads();
    float4 r = v;
    for (int w = 0; w < nw; ++w) {
        r.x = fmaxf(r.x, scratch[4 * w + 0]); r.y = fmaxf(r.y, scratch[4 * w + 1]);
        r.z = fmaxf(r.z, scratch[4 * w + 2]); r.w = fmaxf(r.w, scratch[4 * w + 3]);
    }
    __syncthreads();
    return r;
}

// Exclusive prefix sum of in[0..count) into out[0..count], out[count] = total.
// scratch needs 32 ints.  Called by all threads; ends with a barrier.
__device__ __forceinline__ void pk_block_exclusive_scan(const int* in, int* out, int count, int* scratch)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    int carry = 0;
    for (int base = 0; base < count; base += blockDim.x) {
        const int k = base + threadIdx.x;
        const int v = k < count ? in[k] : 0;
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(PK_FULL_MASK, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) scratch[warp] = incl;
        __syncthreads();
        int woff = 0, tot = 0;
        for (int w = 0; w < nw; ++w) {
            const int s = scratch[w];
            woff += w < warp ? s : 0;
            tot += s;
        }
        if (k < count) out[k] = carry + woff + incl - v;
        carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) out[count] = carry;
    __syncthreads();
}

// Elementwise arithmetic rounded after every operation (never contracted
// into an FMA), as the reference's separate tensor operations round
// (lbfgs_torch_parallel.py:546-690).
__device__ __forceinline__ float pk_rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double pk_rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float pk_radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double pk_radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float pk_rsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double pk_rsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float pk_rdiv(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double pk_rdiv(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float pk_rsqrt(float a) { return __fsqrt_rn(a); }
__device__ __forceinline__ double pk_rsqrt(double a) { return __dsqrt_rn(a); }

// Order-fixed vector reductions.  Element k belongs to group k / 128 and
// lane k % 32; thread (warp w, lane l) OWNS the elements of the groups
// g = w, w + nwarps, ... with lane l, and PK_OWN_LOOP visits exactly those.
// Vector updates written with the same ownership need no barrier before the
// next reduction.  pk_canon_sum adds each group's per-lane partial in k
// order, then the groups in order, then a fixed shuffle tree, so the sum
// depends on N alone, not on blockDim.  red: two buffers of 64 * ngroups
// entries, alternated by `flip` (one barrier per reduction: a thread can only
// write a buffer again after the next reduction's barrier, by which time every
// thread has finished reading it).  All threads call these and all get the
// result.  (The two-loop recursion's own barrier counts only some of the warps:
// between two reductions of the whole block it stays within the one buffer that
// the first of them did not use.)
#define PK_CANON_GROUP 128
#define PK_OWN_LOOP(k, N)                                                                      \
    for (int _g = (int)(threadIdx.x >> 5); _g * PK_CANON_GROUP < (N); _g += (int)(blockDim.x >> 5)) \
        _Pragma("unroll") for (int _j = 0; _j < PK_CANON_GROUP; _j += 32)                      \
            if (const int k = _g * PK_CANON_GROUP + (int)(threadIdx.x & 31) + _j; k < (N))

__host__ __device__ inline int pk_canon_groups(int N) { return (N + PK_CANON_GROUP - 1) / PK_CANON_GROUP; }

template <typename T>
__device__ __forceinline__ T* pk_canon_buf(int ng, T* red, int& flip)
{
    T* buf = red + (flip ? 64 * ng : 0);
    flip ^= 1;
    return buf;
}

// Whether two maxima get room of their own behind the buffers (8 warps' worth
// of each), so that one barrier serves them and the sums.  Only where shared
// memory is never short of it: beyond 1024 elements, or with a history whose
// coefficients lie in shared memory beside them, the last bytes can decide
// whether a launch is possible, and the maxima take a buffer in their turn.
#define PK_CANON_MAX_WARPS 8
__host__ __device__ inline bool pk_canon_joint(int N, int m) { return N <= 1024 && m <= 1024; }

// Entries of red for N elements and a history of m.
__host__ __device__ inline int pk_canon_red_len(int N, int m)
{
    return 128 * pk_canon_groups(N) + (pk_canon_joint(N, m) ? 4 * PK_CANON_MAX_WARPS : 0);
}

// Warp maximum, NaN ignored (redux.sync takes floats on sm_100a).
__device__ __forceinline__ float pk_warp_max(float v)
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ double pk_warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(PK_FULL_MASK, v, o));
    return v;
}

// The per-lane partials of ng groups added in group order.  The first eight are
// read together (a group beyond ng adds +0, which changes no sum that started
// from +0); one after the other each waited for its own load.
template <typename T>
__device__ __forceinline__ T pk_canon_groups_sum(const T* buf, int ng)
{
    const int lane = threadIdx.x & 31;
    T v[8], r = T(0);
#pragma unroll
    for (int grp = 0; grp < 8; ++grp) v[grp] = grp < ng ? buf[grp * 32 + lane] : T(0);
#pragma unroll
    for (int grp = 0; grp < 8; ++grp) r = pk_radd(r, v[grp]);
    for (int grp = 8; grp < ng; ++grp) r = pk_radd(r, buf[grp * 32 + lane]);
    return r;
}

// Barrier of the first nw warps of the block (named barrier 1; all of those
// warps, and only those, call it).
__device__ __forceinline__ void pk_warps_barrier(int nw)
{
    if (nw == 1) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"r"(32 * nw) : "memory");
}

// Second half of a canonical sum: barrier, the groups' per-lane partials in
// group order, then the shuffle tree.  buf holds ng * 32 partials.
template <typename T>
__device__ __forceinline__ T pk_canon_finish(const T* buf, int ng)
{
    __syncthreads();
    return pk_warp_sum(pk_canon_groups_sum(buf, ng));
}

// This lane's partial of one group: its (at most four) elements in k order.
template <typename T, typename Get>
__device__ __forceinline__ T pk_canon_partial(int grp, int N, Get get)
{
    T s = T(0);
#pragma unroll
    for (int j = 0; j < PK_CANON_GROUP; j += 32)
        if (const int k = grp * PK_CANON_GROUP + (int)(threadIdx.x & 31) + j; k < N) s = pk_radd(s, get(k));
    return s;
}

template <typename T, typename Get>
__device__ __forceinline__ T pk_canon_sum(int N, Get get, T* red, int& flip)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = blockDim.x >> 5;
    const int ng = pk_canon_groups(N);
    T* buf = pk_canon_buf(ng, red, flip);
    for (int grp = warp; grp < ng; grp += nw) buf[grp * 32 + lane] = pk_canon_partial<T>(grp, N, get);
    return pk_canon_finish(buf, ng);
}

// NS canonical sums (each bit-identical to its own pk_canon_sum) and NM maxima
// of absolute values (a maximum does not depend on the order; it starts from 0):
// at most two of each, in blocks of at most 8 warps.  get(k, s, m) gives the NS
// addends and NM values of element k.  joint: pk_canon_joint of the red at hand;
// one barrier then, three otherwise.
template <int NS, int NM, typename T, typename Get>
__device__ __forceinline__ void pk_canon_reduce(int N, Get get, T* red, int& flip, bool joint, T (&rs)[NS], T (&rm)[NM])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = blockDim.x >> 5;
    const int ng = pk_canon_groups(N);
    T* mbuf = red + 128 * ng + (flip ? 2 * PK_CANON_MAX_WARPS : 0);
    T* buf = pk_canon_buf(ng, red, flip);
    T m[NM];
#pragma unroll
    for (int i = 0; i < NM; ++i) m[i] = T(0);
    for (int grp = warp; grp < ng; grp += nw) {
        T s[NS];
#pragma unroll
        for (int i = 0; i < NS; ++i) s[i] = T(0);
#pragma unroll
        for (int j = 0; j < PK_CANON_GROUP; j += 32)
            if (const int k = grp * PK_CANON_GROUP + lane + j; k < N) {
                T es[NS], em[NM];
                get(k, es, em);
#pragma unroll
                for (int i = 0; i < NS; ++i) s[i] = pk_radd(s[i], es[i]);
#pragma unroll
                for (int i = 0; i < NM; ++i) m[i] = fmax(m[i], em[i]);
            }
#pragma unroll
        for (int i = 0; i < NS; ++i) buf[(i * ng + grp) * 32 + lane] = s[i];
    }
#pragma unroll
    for (int i = 0; i < NM; ++i) m[i] = pk_warp_max(m[i]);
    if (!joint) {
        __syncthreads();
        mbuf = pk_canon_buf(ng, red, flip);
    }
#pragma unroll
    for (int i = 0; i < NM; ++i)
        if (lane == 0) mbuf[PK_CANON_MAX_WARPS * i + warp] = m[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NM; ++i) rm[i] = pk_warp_max(lane < nw ? mbuf[PK_CANON_MAX_WARPS * i + lane] : T(0));
#pragma unroll
    for (int i = 0; i < NS; ++i) rs[i] = pk_warp_sum(pk_canon_groups_sum(buf + i * ng * 32, ng));
    if (!joint) __syncthreads();   // both buffers have been read
}

// Maxima of two element functions over the owned elements with one barrier.
// Starts from 0: the callers reduce absolute values.
template <typename T, typename Get>
__device__ __forceinline__ void pk_canon_max2(int N, Get get, T* red, int& flip, T& r0, T& r1)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = blockDim.x >> 5;
    T* buf = pk_canon_buf(pk_canon_groups(N), red, flip);
    T a = T(0), b = T(0);
    PK_OWN_LOOP(k, N) {
        T u, v;
        get(k, u, v);
        a = fmax(a, u);
        b = fmax(b, v);
    }
    a = pk_warp_max(a);
    b = pk_warp_max(b);
    if (lane == 0) {
        buf[warp] = a;
        buf[32 + warp] = b;
    }
    __syncthreads();
    r0 = pk_warp_max(lane < nw ? buf[lane] : T(0));
    r1 = pk_warp_max(lane < nw ? buf[32 + lane] : T(0));
}

// Bounded wrap of an angle difference into [-pi, pi], following the
// reference's subtract-2pi loop (pack_cuda_lut.py:289-293) in FP32.  Angles
// beyond +-64 pi are reduced with remainderf first so the loop stays short.
__device__ __forceinline__ float pk_wrap_angle(float t)
{
    const float PI = 3.14159265358979323846f;
    if (!(fabsf(t) < 64.0f * PI)) t = remainderf(t, 2.0f * PI);
    while (t > PI) t -= 2.0f * PI;
    while (t < -PI) t += 2.0f * PI;
    return t;
}
