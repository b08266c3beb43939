// lap.cuh -- batched linear assignment (Hungarian) and GA diversity kernels.
//
// One warp solves one N x N problem.  The reference runs the same
// shortest-augmenting-path Kuhn-Munkres on ONE thread per problem
// (lap_batch.py:62-165); here the N columns are spread over the 32 lanes so
// each Dijkstra step is a parallel slack update plus a warp argmin.  Every
// per-element float operation is the reference's, in the same order, and the
// argmin keeps the lowest column among equal slacks (the reference's strict
// '<' scan), so the assignment and the total are bit-identical to the
// sequential kernel.
#pragma once
#include "common.cuh"

#define PK_LAP_WARPS 4
// dynamic shared memory one CTA may hold on sm_100a (227 KB)
#define PK_LAP_SMEM_MAX ((size_t)227 * 1024)

// Column of slot k of this lane.  VEC: four consecutive columns per lane, so a
// row is read with one 16-byte load per four slots; otherwise column j lives in
// lane j % 32.  Either way a lane's columns ascend with k.
template <bool VEC>
__device__ __forceinline__ int pk_lap_col(int lane, int k)
{
    return VEC ? 128 * (k >> 2) + 4 * lane + (k & 3) : lane + 32 * k;
}
template <bool VEC>
__device__ __forceinline__ int pk_lap_lane(int j) { return VEC ? (j >> 2) & 31 : j & 31; }
template <bool VEC>
__device__ __forceinline__ int pk_lap_slot(int j) { return VEC ? ((j >> 7) << 2) | (j & 3) : j >> 5; }

// Minimum of a float over the warp (redux.sync takes floats on sm_100a).
__device__ __forceinline__ float pk_redux_min(float v)
{
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// a[slot] of an array held in registers.
template <int CPL, typename T>
__device__ __forceinline__ T pk_lap_pick(const T (&a)[CPL], int slot)
{
    T r = a[0];
#pragma unroll
    for (int k = 1; k < CPL; ++k) r = slot == k ? a[k] : r;
    return r;
}

// Reads this lane's columns of one cost row (columns beyond N are left alone).
template <int CPL, bool VEC>
__device__ __forceinline__ void pk_lap_row(const float* row, int N, int lane, float (&c)[CPL])
{
    if (VEC) {   // N is a multiple of 4 and the row 16-byte aligned
#pragma unroll
        for (int q = 0; q < CPL / 4; ++q)
            if (128 * q + 4 * lane < N) {
                const float4 v = *(const float4*)(row + 128 * q + 4 * lane);
                c[4 * q] = v.x; c[4 * q + 1] = v.y; c[4 * q + 2] = v.z; c[4 * q + 3] = v.w;
            }
    } else {
#pragma unroll
        for (int k = 0; k < CPL; ++k)
            if (lane + 32 * k < N) c[k] = row[lane + 32 * k];
    }
}

// Warp-cooperative Hungarian.  rowfn(row, c) reads this lane's columns of a
// cost row into c.  On success cm[k] is the row matched to the lane's k-th
// column; false if a step finds no finite slack.
//
// One problem is a chain of dependent Dijkstra steps (about 900 at N = 100,
// 2 000 in the slowest of 2048), so a step's latency and its instructions are
// what it costs.  All state is in registers: the dual of a matched row lives
// with its column (it moves when the column is rematched), the dual of row i
// in every lane, and a column's parent is the column scanned before it, so a
// step has no shared memory and no barrier: the slacks, two redux.sync minima
// (the smallest slack, then the lowest column that has it together with the
// row matched to it) and a shuffle for that row's dual.  The next row's dual
// needs no update before it is used: its column was not yet in the tree.
// PREFETCH: the next row is read as soon as it is known, before the dual
// updates, which then overlap an L2 load's latency.
template <int CPL, bool VEC, bool PREFETCH, typename RowFn>
__device__ __forceinline__ bool pk_hungarian_warp(int N, RowFn rowfn, int (&cm)[CPL])
{
    const int lane = threadIdx.x & 31;
    float v[CPL], uc[CPL], minv[CPL], c[CPL];
    int p[CPL];
    unsigned invalid = 0;
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
        v[k] = 0.f; uc[k] = 0.f; cm[k] = -1; c[k] = 0.f;
        if (pk_lap_col<VEC>(lane, k) >= N) invalid |= 1u << k;
    }
    if (PREFETCH) rowfn(0, c);
    for (int i = 0; i < N; ++i) {
        unsigned used = invalid;
        float ui = 0.f, urow = 0.f;
        int cur_row = i, cur_col = -1;
#pragma unroll
        for (int k = 0; k < CPL; ++k) { minv[k] = 1e30f; p[k] = -1; }
        for (;;) {   // each turn adds a column to the tree, so at most N turns
            if (!PREFETCH) rowfn(cur_row, c);
            // the lane's smallest slack: no branches, pairs before pairs of pairs;
            // the left one keeps a tie, and a NaN loses on either side
            float sl[CPL], su[CPL];
            unsigned ss[CPL];   // column << 16 | row matched to it (0xffff: none)
#pragma unroll
            for (int k = 0; k < CPL; ++k) {
                const bool open = !((used >> k) & 1u);
                const float red = (c[k] - urow) - v[k];
                const bool better = open && red < minv[k];
                minv[k] = better ? red : minv[k];
                p[k] = better ? cur_col : p[k];
                sl[k] = open ? minv[k] : 1e30f;
                su[k] = uc[k];
                ss[k] = ((unsigned)pk_lap_col<VEC>(lane, k) << 16) | (unsigned)(cm[k] & 0xffff);
            }
#pragma unroll
            for (int o = 1; o < CPL; o <<= 1)
#pragma unroll
                for (int k = 0; k + o < CPL; k += 2 * o) {
                    const float m = fminf(sl[k], sl[k + o]);
                    const bool right = m != sl[k];
                    sl[k] = m;
                    su[k] = right ? su[k + o] : su[k];
                    ss[k] = right ? ss[k + o] : ss[k];
                }
            // A NaN cost fails the '<' above and leaves minv untouched; a slack becomes
            // NaN when another of -inf is taken before it, and nothing chooses it then.
            const float delta = pk_redux_min(sl[0]);
            if (!(delta < 1e30f)) return false;   // no finite slack: infeasible input
            const unsigned sel = __reduce_min_sync(PK_FULL_MASK, sl[0] == delta ? ss[0] : 0xffffffffu);
            cur_row = (int)(sel & 0xffffu);
            cur_col = (int)(sel >> 16);
            const bool free_col = cur_row == 0xffff;
            const int owner = pk_lap_lane<VEC>(cur_col);
            if (PREFETCH) {
                const int nr = free_col ? i + 1 : cur_row;
                if (nr < N) rowfn(nr, c);
            }
            urow = __shfl_sync(PK_FULL_MASK, su[0], owner);
#pragma unroll
            for (int k = 0; k < CPL; ++k) {
                const bool in = (used >> k) & 1u;
                uc[k] = in ? uc[k] + delta : uc[k];
                v[k] = in ? v[k] - delta : v[k];
                minv[k] = in ? minv[k] : minv[k] - delta;
            }
            ui += delta;
            if (free_col) break;
            used |= lane == owner ? 1u << pk_lap_slot<VEC>(cur_col) : 0u;
        }
        // flip the alternating path (lap_batch.py:157-163): every column on it
        // takes the row (and that row's dual) of its parent column, the first
        // one row i
        for (int guard = 0; guard <= N; ++guard) {
            const int owner = pk_lap_lane<VEC>(cur_col), slot = pk_lap_slot<VEC>(cur_col);
            const int par = __shfl_sync(PK_FULL_MASK, pk_lap_pick<CPL>(p, slot), owner);
            int row = i;
            float du = ui;
            if (par >= 0) {
                const int pl = pk_lap_lane<VEC>(par), ps = pk_lap_slot<VEC>(par);
                row = __shfl_sync(PK_FULL_MASK, pk_lap_pick<CPL>(cm, ps), pl);
                du = __shfl_sync(PK_FULL_MASK, pk_lap_pick<CPL>(uc, ps), pl);
            }
#pragma unroll
            for (int k = 0; k < CPL; ++k)
                if (k == slot && lane == owner) { cm[k] = row; uc[k] = du; }
            if (par < 0) break;
            cur_col = par;
        }
    }
    return true;
}

// The matched costs added in row order (compute_costs, lap_batch.py:173-196):
// every lane places its columns' costs at their rows of s (N floats of this
// warp), and lane 0 adds them.  Returns lane 0's sum.
template <int CPL, bool VEC, typename CostFn>
__device__ __forceinline__ float pk_lap_total(int N, const int (&cm)[CPL], float* s, CostFn costfn)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
        const int j = pk_lap_col<VEC>(lane, k);
        if (j < N) s[cm[k]] = costfn(cm[k], j, k);
    }
    __syncwarp();
    float t = 0.f;
    if (lane == 0)
        for (int r = 0; r < N; ++r) t += s[r];
    return t;
}

// Results of problem b: row matches (-1 everywhere if infeasible), total, status.
template <int CPL, bool VEC>
__device__ __forceinline__ void pk_lap_store(bool ok, const int (&cm)[CPL], float tot, int b, int N,
                                             int* __restrict__ row_match, float* __restrict__ total,
                                             int* __restrict__ status)
{
    const int lane = threadIdx.x & 31;
    int* rm = row_match + (size_t)b * N;
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
        const int j = pk_lap_col<VEC>(lane, k);
        if (j < N) rm[ok ? cm[k] : j] = ok ? j : -1;
    }
    if (lane == 0) {
        total[b] = ok ? tot : __int_as_float(0x7fc00000);
        if (status) status[b] = ok ? 0 : 1;
    }
}

// One warp per problem, PK_LAP_WARPS problems per CTA, cost rows read from L2.
// The minimum of one CTA per SM in the launch bounds lets ptxas give every CPL
// the registers it needs.
template <int CPL, bool VEC>
__global__ void __launch_bounds__(32 * PK_LAP_WARPS, 1)
pk_hungarian_kernel(const float* __restrict__ C, int B, int N, int* __restrict__ row_match,
                    float* __restrict__ total, int* __restrict__ status)
{
    extern __shared__ __align__(16) unsigned char pk_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.x * PK_LAP_WARPS + warp;
    if (b >= B) return;
    const float* Cb = C + (size_t)b * N * N;
    int cm[CPL];
    const bool ok = pk_hungarian_warp<CPL, VEC, true>(
        N, [&](int r, float (&c)[CPL]) { pk_lap_row<CPL, VEC>(Cb + (size_t)r * N, N, lane, c); }, cm);
    float t = 0.f;
    if (ok)
        t = pk_lap_total<CPL, VEC>(N, cm, (float*)pk_smem + (size_t)warp * N,
                                   [&](int r, int j, int) { return Cb[(size_t)r * N + j]; });
    pk_lap_store<CPL, VEC>(ok, cm, t, b, N, row_match, total, status);
}

// The same solver with the problem's N x N costs copied into shared memory
// first: which row a step reads is only known when the previous step ends, so
// from L2 every step waits most of a round trip, from shared memory a few tens
// of cycles.  One warp per CTA; the CTAs beyond those resident start as others
// finish, which balances problems of very different step counts.
template <int CPL, bool VEC>
__global__ void __launch_bounds__(32)
pk_hungarian_smem_kernel(const float* __restrict__ C, int B, int N, int* __restrict__ row_match,
                         float* __restrict__ total, int* __restrict__ status)
{
    extern __shared__ __align__(16) unsigned char pk_smem[];
    const int lane = threadIdx.x;
    const int b = blockIdx.x;
    if (b >= B) return;
    const size_t nn = (size_t)N * N;
    float* Cs = (float*)pk_smem;
    float* s = Cs + ((nn + 3) & ~(size_t)3);
    const float* Cb = C + (size_t)b * nn;
    if ((((uintptr_t)Cb) & 15) == 0) {
        const size_t n4 = nn >> 2;
        const float4* src = (const float4*)Cb;
        float4* dst = (float4*)Cs;
#pragma unroll 8
        for (size_t k = lane; k < n4; k += 32) dst[k] = __ldg(src + k);
        for (size_t k = (n4 << 2) + lane; k < nn; k += 32) Cs[k] = __ldg(Cb + k);
    } else {
        for (size_t k = lane; k < nn; k += 32) Cs[k] = __ldg(Cb + k);
    }
    __syncwarp();
    int cm[CPL];
    const bool ok = pk_hungarian_warp<CPL, VEC, false>(
        N, [&](int r, float (&c)[CPL]) { pk_lap_row<CPL, VEC>(Cs + r * N, N, lane, c); }, cm);
    float t = 0.f;
    if (ok) t = pk_lap_total<CPL, VEC>(N, cm, s, [&](int r, int j, int) { return Cs[r * N + j]; });
    pk_lap_store<CPL, VEC>(ok, cm, t, b, N, row_match, total, status);
}

// Shared memory of the staged solver for N: the matrix (rounded up to whole
// float4s) and the matched costs.
static size_t pk_lap_smem_bytes(int N)
{
    return (((size_t)N * N + 3) & ~(size_t)3) * 4 + (size_t)N * 4;
}

// Problems of the staged solver that the GPU can hold at once (0: N does not fit).
template <int CPL, bool VEC>
static cudaError_t pk_lap_staged_slots(int N, long long* slots)
{
    *slots = 0;
    const size_t ssm = pk_lap_smem_bytes(N);
    if (ssm > PK_LAP_SMEM_MAX) return cudaSuccess;
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t err = pk_raise_smem((const void*)pk_hungarian_smem_kernel<CPL, VEC>, ssm);
    if (err == cudaSuccess) err = cudaGetDevice(&dev);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (err == cudaSuccess)
        err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pk_hungarian_smem_kernel<CPL, VEC>, 32, ssm);
    if (err == cudaSuccess) *slots = (long long)per_sm * sms;
    return err;
}

// The staged solver runs when every problem can be resident at once: staging
// trades concurrency for latency.  100 x 100: 600 problems (740 fit) 269 us
// staged against 322 from L2, 1000 problems 391 against 371, 2048 616 against
// 517.
template <int CPL, bool VEC>
static int pk_lap_launch(const float* C, int B, int N, int* rm, float* tot, int* status, cudaStream_t st)
{
    long long slots = 0;
    const cudaError_t err = pk_lap_staged_slots<CPL, VEC>(N, &slots);
    if (err != cudaSuccess) return pk_cuda_check(err, "pk_lap_solve occupancy");
    if (slots >= B) {
        pk_hungarian_smem_kernel<CPL, VEC><<<B, 32, pk_lap_smem_bytes(N), st>>>(C, B, N, rm, tot, status);
    } else {
        const dim3 grid((B + PK_LAP_WARPS - 1) / PK_LAP_WARPS), block(32 * PK_LAP_WARPS);
        pk_hungarian_kernel<CPL, VEC><<<grid, block, (size_t)PK_LAP_WARPS * N * 4, st>>>(C, B, N, rm, tot, status);
    }
    return pk_cuda_check(cudaGetLastError(), "pk_lap_solve launch");
}

// VEC needs 16-byte aligned rows; below four columns per lane its rounding up
// to a multiple of four would idle lanes.
static int pk_lap_dispatch(const float* C, int B, int N, int* rm, float* tot, int* status, cudaStream_t st)
{
    const bool vec = N > 96 && (N & 3) == 0 && (((uintptr_t)C) & 15) == 0;
    if (vec && N <= 128) return pk_lap_launch<4, true>(C, B, N, rm, tot, status, st);
    if (vec && N <= 256) return pk_lap_launch<8, true>(C, B, N, rm, tot, status, st);
    switch ((N + 31) / 32) {
#define PK_L(K) case K: return pk_lap_launch<K, false>(C, B, N, rm, tot, status, st);
        PK_L(1) PK_L(2) PK_L(3) PK_L(4) PK_L(5) PK_L(6) PK_L(7) PK_L(8)
#undef PK_L
    }
    return pk_fail(PK_ERANGE, "pk_lap_solve: N beyond 256%s");
}

extern "C" int pk_lap_solve(const float* C, int B, int N, int* row_match, float* total, int* status,
                            void* stream)
{
    if (B < 0 || N < 0) return pk_fail(PK_EINVAL, "pk_lap_solve: negative size%s");
    if (N > PK_MAX_LAP_N) return pk_fail(PK_ERANGE, "pk_lap_solve: N beyond 256%s");
    if (B == 0) return PK_OK;
    if (N == 0) {
        // empty assignments: totals are 0 (lap_batch.py:173-196 with N = 0)
        return pk_cuda_check(cudaMemsetAsync(total, 0, sizeof(float) * B, (cudaStream_t)stream),
                             "pk_lap_solve memset");
    }
    if (!C || !row_match || !total) return pk_fail(PK_EINVAL, "pk_lap_solve: NULL pointer%s");
    return pk_lap_dispatch(C, B, N, row_match, total, status, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// GA diversity: 8 symmetry transforms of the reference packing
// (kaggle_support.py:2061-2071), cost sqrt(dx^2 + dy^2 + wrap(dtheta)^2)
// (:2105-2112), one LAP per transform, minimum over transforms (:2126).
// The reference materialises a (8 * N_pop * N_ref, N, N) tensor and calls
// solve_lap_batch; here every problem's matrix lives only while its warp solves
// it, in shared memory or in a slab of a caller's scratch
// (pk_diversity_matrix_work).  Without scratch (pk_diversity_matrix) a CTA of 8
// warps handles one (pop, ref) pair, warp t solving transform t with its cost
// rows generated in the steps that read them.
// ---------------------------------------------------------------------------

// Transformed reference pose (kaggle_support.py:2080-2099), FP32.
__device__ __forceinline__ float3 pk_div_transform(float x, float y, float th, int t)
{
    const float PI = 3.14159265358979323846f;
    if (t >= 4) { y = -y; th = PI - th; }
    const int r = t & 3;
    const float ca[4] = {1.f, 0.f, -1.f, 0.f};
    const float sa[4] = {0.f, 1.f, 0.f, -1.f};
    const float ang[4] = {0.f, 1.5707963267948966f, 3.141592653589793f, 4.71238898038469f};
    float nx = x, ny = y;
    if (r != 0) {
        // explicit roundings: the fused and the materialised paths must agree bit for bit
        nx = __fsub_rn(__fmul_rn(x, ca[r]), __fmul_rn(y, sa[r]));
        ny = __fadd_rn(__fmul_rn(x, sa[r]), __fmul_rn(y, ca[r]));
        th = __fadd_rn(th, ang[r]);
    }
    // remainder(th + pi, 2 pi) - pi, result in [-pi, pi)
    float m = fmodf(__fadd_rn(th, PI), 2.f * PI);
    if (m < 0.f) m = __fadd_rn(m, 2.f * PI);
    return make_float3(nx, ny, __fsub_rn(m, PI));
}

// fmodf(x, 2 pi) (2 pi rounded to float), exactly: |x| < 2 pi is its own
// remainder, and for 2 pi <= |x| < 4 pi the remainder |x| - 2 pi is exact
// (Sterbenz) and takes the sign of x; anything else goes to fmodf.  The
// cost rows of the fused diversity solver are generated inside its Dijkstra
// steps, where the general fmodf was most of a step's arithmetic.
__device__ __forceinline__ float pk_fmod_2pi(float x)
{
    const float T = 2.f * 3.14159265358979323846f;
    const float ax = fabsf(x);
    if (ax < T) return x;
    if (ax < 2.f * T) return copysignf(__fsub_rn(ax, T), x);
    return fmodf(x, T);
}

__device__ __forceinline__ float pk_div_cost(float px, float py, float pt, float3 r)
{
    const float PI = 3.14159265358979323846f;
    const float dx = __fsub_rn(px, r.x), dy = __fsub_rn(py, r.y);
    float dt = pk_fmod_2pi(__fadd_rn(__fsub_rn(pt, r.z), PI));
    if (dt < 0.f) dt = __fadd_rn(dt, 2.f * PI);
    dt = __fsub_rn(dt, PI);
    return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dt, dt)));
}

// Dense cost matrices of every (transform, pop, ref) problem, in the
// reference's stacking order (transform, pop, ref) -> (N, N), for checking
// the fused kernel and for callers that want the matrices.
__global__ void pk_diversity_costs_kernel(const float* __restrict__ pop, const float* __restrict__ ref, int Np,
                                          int Nr, int n, int ntf, float* __restrict__ out)
{
    const size_t total = (size_t)ntf * Np * Nr * n * n;
    for (size_t w = blockIdx.x * (size_t)blockDim.x + threadIdx.x; w < total; w += (size_t)gridDim.x * blockDim.x) {
        const int col = (int)(w % n);
        const int row = (int)((w / n) % n);
        const size_t prob = w / ((size_t)n * n);
        const int r = (int)(prob % Nr), p = (int)((prob / Nr) % Np), t = (int)(prob / ((size_t)Np * Nr));
        const float* R = ref + ((size_t)r * n + col) * 3;
        const float* P = pop + ((size_t)p * n + row) * 3;
        out[w] = pk_div_cost(P[0], P[1], P[2], pk_div_transform(R[0], R[1], R[2], t));
    }
}

template <int CPL>
__global__ void __launch_bounds__(256)
pk_diversity_lap_kernel(const float* __restrict__ pop, const float* __restrict__ ref, int Np, int Nr, int n,
                        int ntf, float* __restrict__ out)
{
    extern __shared__ __align__(16) unsigned char pk_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pr = blockIdx.x;
    const int p = pr / Nr, r = pr % Nr;
    float* s_tot = (float*)pk_smem;                       // [8]
    float* s_pop = s_tot + 8;                             // [3n]
    float* base = s_pop + 3 * n;
    const float* P = pop + (size_t)p * n * 3;
    for (int k = threadIdx.x; k < 3 * n; k += blockDim.x) s_pop[k] = P[k];
    __syncthreads();
    if (warp < ntf) {
        float* s_cost = base + (size_t)warp * n;
        // this lane's transformed reference columns
        float3 rc[CPL];
        const float* R = ref + (size_t)r * n * 3;
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            const int j = lane + 32 * k;
            rc[k] = j < n ? pk_div_transform(R[3 * j], R[3 * j + 1], R[3 * j + 2], warp) : make_float3(0, 0, 0);
        }
        int cm[CPL];
        const bool ok = pk_hungarian_warp<CPL, false, false>(n, [&](int row, float (&c)[CPL]) {
            const float px = s_pop[3 * row], py = s_pop[3 * row + 1], pt = s_pop[3 * row + 2];
#pragma unroll
            for (int k = 0; k < CPL; ++k) c[k] = pk_div_cost(px, py, pt, rc[k]);
        }, cm);
        float t = __int_as_float(0x7fc00000);
        if (ok)
            t = pk_lap_total<CPL, false>(n, cm, s_cost, [&](int row, int, int k) {
                return pk_div_cost(s_pop[3 * row], s_pop[3 * row + 1], s_pop[3 * row + 2], rc[k]);
            });
        if (lane == 0) {
            s_tot[warp] = t;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float m = s_tot[0];
        for (int t = 1; t < ntf; ++t) m = fminf(m, s_tot[t]);
        out[pr] = m;
    }
}

// One (pair, transform) problem solved by a warp from a cost matrix it generates
// once into Cs: n^2 costs (a square root and an angle remainder each) instead of
// a row of them in every Dijkstra step, about 9 n steps at n = 100.  The steps
// then read finished rows, like the assignment solver's.  out holds the minimum
// over the transforms: totals are never negative, so their bits order as
// integers, below the NaN of an infeasible problem and the initial 0x7fffffff.
template <int CPL, bool VEC, bool PREFETCH>
__device__ __forceinline__ void pk_diversity_problem(const float* __restrict__ pop, const float* __restrict__ ref,
                                                     int Nr, int n, int ntf, int prob, float* Cs, float* s,
                                                     int* __restrict__ out)
{
    const int lane = threadIdx.x & 31;
    const int pr = prob / ntf, tf = prob - pr * ntf;
    const float* P = pop + (size_t)(pr / Nr) * n * 3;
    const float* R = ref + (size_t)(pr % Nr) * n * 3;
    float3 rc[CPL];   // this lane's transformed reference columns
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
        const int j = pk_lap_col<VEC>(lane, k);
        rc[k] = j < n ? pk_div_transform(R[3 * j], R[3 * j + 1], R[3 * j + 2], tf) : make_float3(0, 0, 0);
    }
    // every lane writes, and later reads, its own columns only: no barrier
    for (int r = 0; r < n; ++r) {
        const float px = __ldg(P + 3 * r), py = __ldg(P + 3 * r + 1), pt = __ldg(P + 3 * r + 2);
        float c[CPL];
#pragma unroll
        for (int k = 0; k < CPL; ++k) c[k] = pk_div_cost(px, py, pt, rc[k]);
        float* row = Cs + r * n;
#pragma unroll
        for (int k = 0; k < CPL; k += VEC ? 4 : 1) {
            const int j = pk_lap_col<VEC>(lane, k);
            if (VEC) { if (j < n) *(float4*)(row + j) = make_float4(c[k], c[k + 1], c[k + 2], c[k + 3]); }
            else if (j < n) row[j] = c[k];
        }
    }
    int cm[CPL];
    const bool ok = pk_hungarian_warp<CPL, VEC, PREFETCH>(
        n, [&](int r, float (&c)[CPL]) { pk_lap_row<CPL, VEC>(Cs + r * n, n, lane, c); }, cm);
    float t = __int_as_float(0x7fc00000);
    if (ok) t = pk_lap_total<CPL, VEC>(n, cm, s, [&](int r, int j, int) { return Cs[r * n + j]; });
    if (lane == 0) atomicMin(out + pr, __float_as_int(t));
}

// The matrix in shared memory, one problem per CTA of one warp: the lowest
// latency, while every problem can be resident at once.
template <int CPL, bool VEC>
__global__ void __launch_bounds__(32)
pk_diversity_staged_kernel(const float* __restrict__ pop, const float* __restrict__ ref, int Nr, int n, int ntf,
                           int* __restrict__ out)
{
    extern __shared__ __align__(16) unsigned char pk_smem[];
    float* Cs = (float*)pk_smem;
    pk_diversity_problem<CPL, VEC, false>(pop, ref, Nr, n, ntf, blockIdx.x, Cs, Cs + ((n * n + 3) & ~3), out);
}

// The matrix in the warp's own slab of a caller's scratch (slab floats apart):
// many more problems in flight than shared memory holds.  Up to 115 trees all
// slabs stay in L2; beyond, part of the rows come from HBM.  Warps take problems
// from a counter, so unequal problems even out.  128 x 8 pairs of 100 trees: 2.11
// ms with rows generated in the steps, 2.29 staged in shared memory, 1.43 from the
// scratch (16 warps per SM; 8: 1.86, 24: 1.42).  Out of L2 it is still the faster
// form, rows against scratch: 128 trees 3.30 / 2.48 ms, 200 (379 MB) 12.6 / 8.3,
// 256 (621 MB) 23.4 / 12.2, and 8 warps per SM instead of 16 are slower (200
// trees, 64 x 8 pairs: 6.4 ms against 4.6).
template <int CPL, bool VEC>
__global__ void __launch_bounds__(32 * PK_LAP_WARPS, 1)
pk_diversity_work_kernel(const float* __restrict__ pop, const float* __restrict__ ref, int Nr, int n, int ntf,
                         int problems, float* work, size_t slab, int* next, int* __restrict__ out)
{
    extern __shared__ __align__(16) unsigned char pk_smem[];
    const int warp = threadIdx.x >> 5;
    float* Cs = work + ((size_t)blockIdx.x * PK_LAP_WARPS + warp) * slab;
    float* s = (float*)pk_smem + (size_t)warp * n;
    for (;;) {
        int prob = (threadIdx.x & 31) == 0 ? atomicAdd(next, 1) : 0;
        prob = __shfl_sync(PK_FULL_MASK, prob, 0);
        if (prob >= problems) return;
        pk_diversity_problem<CPL, VEC, true>(pop, ref, Nr, n, ntf, prob, Cs, s, out);
        __syncwarp();
    }
}

// out and the problem counter before a launch of the two kernels above.
__global__ void pk_diversity_init_kernel(int* __restrict__ out, int count, int* next)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) out[k] = 0x7fffffff;
    if (next && blockIdx.x == 0 && threadIdx.x == 0) *next = 0;
}

// Shared argument checks of the diversity entry points: sizes, the (pop, ref)
// pair count of a one-CTA-per-pair grid (computed in 64 bits), and the
// pointers of a launch that has work.
static int pk_diversity_args(const char* who, const float* pop, const float* ref, int Np, int Nr, int n,
                             const float* out)
{
    if (Np < 0 || Nr < 0 || n < 0) {
        snprintf(g_pk_err, sizeof(g_pk_err), "%s: negative size", who);
        return PK_EINVAL;
    }
    if ((long long)Np * (long long)Nr > 0x7fffffffLL) {
        snprintf(g_pk_err, sizeof(g_pk_err), "%s: Np * Nr = %lld pairs exceeds the grid limit 2^31 - 1", who,
                 (long long)Np * (long long)Nr);
        return PK_ERANGE;
    }
    if ((long long)Np * Nr > 0 && (!out || (n > 0 && (!pop || !ref)))) {
        snprintf(g_pk_err, sizeof(g_pk_err), "%s: NULL pointer", who);
        return PK_EINVAL;
    }
    return PK_OK;
}

extern "C" int pk_diversity_costs(const float* pop, const float* ref, int Np, int Nr, int n, int transform,
                                  float* out, void* stream)
{
    int rc = pk_diversity_args("pk_diversity_costs", pop, ref, Np, Nr, n, out);
    if (rc) return rc;
    const int ntf = transform ? 8 : 1;
    const size_t total = (size_t)ntf * Np * Nr * n * n;
    if (total == 0) return PK_OK;
    const int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    pk_diversity_costs_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(pop, ref, Np, Nr, n, ntf, out);
    return pk_cuda_check(cudaGetLastError(), "pk_diversity_costs launch");
}

extern "C" int pk_diversity_matrix(const float* pop, const float* ref, int Np, int Nr, int n, int transform,
                                   float* out, void* stream)
{
    int rc = pk_diversity_args("pk_diversity_matrix", pop, ref, Np, Nr, n, out);
    if (rc) return rc;
    if (n > PK_MAX_LAP_N) return pk_fail(PK_ERANGE, "pk_diversity_matrix: more than 256 trees%s");
    if (Np == 0 || Nr == 0) return PK_OK;
    if (n == 0) return pk_cuda_check(cudaMemsetAsync(out, 0, sizeof(float) * (size_t)Np * Nr, (cudaStream_t)stream),
                                     "pk_diversity_matrix memset");
    const int ntf = transform ? 8 : 1;
    const int cpl = (n + 31) / 32;
    const size_t smem = 8 * 4 + (size_t)3 * n * 4 + (size_t)8 * n * 4;
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t err = cudaSuccess;
    switch (cpl) {
#define PK_D(K)                                                                                        \
    case K:                                                                                            \
        err = pk_raise_smem((const void*)pk_diversity_lap_kernel<K>, smem);                            \
        if (err == cudaSuccess) pk_diversity_lap_kernel<K><<<Np * Nr, 256, smem, st>>>(pop, ref, Np, Nr, n, ntf, out); \
        break;
        PK_D(1) PK_D(2) PK_D(3) PK_D(4) PK_D(5) PK_D(6) PK_D(7) PK_D(8)
#undef PK_D
        default: return pk_fail(PK_ERANGE, "pk_diversity_matrix: more than 256 trees%s");
    }
    if (err != cudaSuccess) return pk_cuda_check(err, "pk_diversity_matrix attribute");
    return pk_cuda_check(cudaGetLastError(), "pk_diversity_matrix launch");
}

// Scratch of pk_diversity_matrix_work: a header for the problem counter and one
// matrix slab per warp.  As many warps per SM, between 16 and 32, as keep the
// slabs within the 126 MB L2 (n <= 81: 32; 82: 28; 96 to 103: 20; from 104: 16),
// and no more than there are problems.  From 116 trees the 16 no longer fit: with
// 148 SMs 155 MB at 128 trees, 379 at 200, 621 at 256.
#define PK_DIV_HEADER 32   // floats; keeps the slabs 128-byte aligned
static size_t pk_div_slab(int n) { return ((size_t)n * n + 31) & ~(size_t)31; }

static cudaError_t pk_div_warps(int n, long long problems, long long* warps)
{
    int dev = 0, sms = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (err != cudaSuccess) return err;
    long long per_sm = (long long)(126e6 / (4.0 * (double)pk_div_slab(n) * sms)) & ~3LL;
    per_sm = per_sm < 16 ? 16 : (per_sm > 32 ? 32 : per_sm);
    long long w = per_sm * sms;
    if (w > problems) w = (problems + PK_LAP_WARPS - 1) / PK_LAP_WARPS * PK_LAP_WARPS;
    *warps = w;
    return cudaSuccess;
}

// Floats of scratch pk_diversity_matrix_work needs (0: none, or no device).
extern "C" size_t pk_diversity_work_floats(int Np, int Nr, int n, int transform)
{
    if (Np <= 0 || Nr <= 0 || n <= 0 || n > PK_MAX_LAP_N) return 0;
    long long warps = 0;
    if (pk_div_warps(n, (long long)Np * Nr * (transform ? 8 : 1), &warps) != cudaSuccess) return 0;
    return PK_DIV_HEADER + (size_t)warps * pk_div_slab(n);
}

template <int CPL, bool VEC>
static int pk_diversity_launch(const float* pop, const float* ref, int Np, int Nr, int n, int ntf, float* out,
                               float* work, size_t work_floats, cudaStream_t st)
{
    const long long problems = (long long)Np * Nr * ntf;
    const int pairs = Np * Nr;
    // Shared memory when it holds every problem at once and the matrices are
    // large: 8 pairs of 200 trees 0.95 ms against 1.44 from the scratch, but
    // 64 problems of 100 trees 0.25 against 0.23.
    cudaError_t err = cudaSuccess;
    long long slots = 0;
    const size_t ssm = pk_lap_smem_bytes(n);
    if (n > 128 && ssm <= PK_LAP_SMEM_MAX) {
        int dev = 0, sms = 0, per_sm = 0;
        err = pk_raise_smem((const void*)pk_diversity_staged_kernel<CPL, VEC>, ssm);
        if (err == cudaSuccess) err = cudaGetDevice(&dev);
        if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (err == cudaSuccess)
            err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pk_diversity_staged_kernel<CPL, VEC>, 32, ssm);
        slots = (long long)per_sm * sms;
    }
    long long warps = 0;
    if (err == cudaSuccess && slots < problems) err = pk_div_warps(n, problems, &warps);
    if (err != cudaSuccess) return pk_cuda_check(err, "pk_diversity_matrix_work occupancy");
    const size_t slab = pk_div_slab(n);
    if (slots < problems && work_floats < PK_DIV_HEADER + (size_t)warps * slab)
        return pk_fail(PK_EINVAL, "pk_diversity_matrix_work: work holds fewer floats than pk_diversity_work_floats%s");
    int* next = slots < problems ? (int*)work : nullptr;
    pk_diversity_init_kernel<<<(pairs + 255) / 256 < 592 ? (pairs + 255) / 256 : 592, 256, 0, st>>>((int*)out, pairs,
                                                                                                    next);
    if (slots >= problems)
        pk_diversity_staged_kernel<CPL, VEC><<<(int)problems, 32, ssm, st>>>(pop, ref, Nr, n, ntf, (int*)out);
    else
        pk_diversity_work_kernel<CPL, VEC><<<(int)(warps / PK_LAP_WARPS), 32 * PK_LAP_WARPS,
                                             (size_t)PK_LAP_WARPS * n * 4, st>>>(
            pop, ref, Nr, n, ntf, (int)problems, work + PK_DIV_HEADER, slab, next, (int*)out);
    return pk_cuda_check(cudaGetLastError(), "pk_diversity_matrix_work launch");
}

extern "C" int pk_diversity_matrix_work(const float* pop, const float* ref, int Np, int Nr, int n, int transform,
                                        float* out, float* work, size_t work_floats, void* stream)
{
    int rc = pk_diversity_args("pk_diversity_matrix_work", pop, ref, Np, Nr, n, out);
    if (rc) return rc;
    if (n > PK_MAX_LAP_N) return pk_fail(PK_ERANGE, "pk_diversity_matrix_work: more than 256 trees%s");
    const int ntf = transform ? 8 : 1;
    cudaStream_t st = (cudaStream_t)stream;
    // a 31-bit problem counter; beyond it (and for empty packings) the form without scratch
    if (Np == 0 || Nr == 0 || n == 0 || (long long)Np * Nr * ntf > 0x7fff0000LL)
        return pk_diversity_matrix(pop, ref, Np, Nr, n, transform, out, stream);
    if (!work || ((uintptr_t)work & 127)) return pk_fail(PK_EINVAL, "pk_diversity_matrix_work: work must be 128-byte aligned%s");
    if (n > 96 && (n & 3) == 0)
        return n <= 128 ? pk_diversity_launch<4, true>(pop, ref, Np, Nr, n, ntf, out, work, work_floats, st)
                        : pk_diversity_launch<8, true>(pop, ref, Np, Nr, n, ntf, out, work, work_floats, st);
    switch ((n + 31) / 32) {
#define PK_D(K) case K: return pk_diversity_launch<K, false>(pop, ref, Np, Nr, n, ntf, out, work, work_floats, st);
        PK_D(1) PK_D(2) PK_D(3) PK_D(4) PK_D(5) PK_D(6) PK_D(7) PK_D(8)
#undef PK_D
    }
    return pk_fail(PK_ERANGE, "pk_diversity_matrix_work: more than 256 trees%s");
}

// diversity_shortcut_kernel (lap_batch.py:216-331): transform of the
// reference by (cos_a, sin_a, mirror), then for every population tree the
// nearest transformed reference tree; sum of those distances.  One CTA per
// (pop, ref) pair; the sum runs over trees in index order like the reference.
__global__ void pk_diversity_shortcut_kernel(const float* __restrict__ pop, const float* __restrict__ ref, int Np,
                                             int Nr, int n, float cos_a, float sin_a, int mirror,
                                             float* __restrict__ out)
{
    extern __shared__ __align__(16) unsigned char pk_smem[];
    float* rx = (float*)pk_smem;
    float* ry = rx + n;
    float* rt = ry + n;
    float* part = rt + n;
    const float PI = 3.14159265358979323846f, TWO_PI = 2.0f * PI;
    const int b = blockIdx.x;
    const int pi = b / Nr, ri = b % Nr;
    const float* P = pop + (size_t)pi * n * 3;
    const float* R = ref + (size_t)ri * n * 3;
    const float rot = atan2f(sin_a, cos_a);
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        float x = R[3 * k], y = R[3 * k + 1], t = R[3 * k + 2];
        if (mirror) { y = -y; t = PI - t; }
        const float xr = x * cos_a - y * sin_a, yr = x * sin_a + y * cos_a;
        float tr = t + rot;
        tr = fmodf(tr + PI, TWO_PI);
        if (tr < 0) tr += TWO_PI;
        tr -= PI;
        rx[k] = xr; ry[k] = yr; rt[k] = tr;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const float px = P[3 * k], py = P[3 * k + 1], pt = P[3 * k + 2];
        float best = 1e30f;
        for (int j = 0; j < n; ++j) {
            const float dx = px - rx[j], dy = py - ry[j];
            float dt = pt - rt[j];
            dt = fmodf(dt + PI, TWO_PI);
            if (dt < 0) dt += TWO_PI;
            dt -= PI;
            const float sq = dx * dx + dy * dy + dt * dt;
            if (sq < best) best = sq;
        }
        part[k] = sqrtf(best);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int k = 0; k < n; ++k) t += part[k];
        out[b] = t;
    }
}

extern "C" int pk_diversity_shortcut(const float* pop, const float* ref, int Np, int Nr, int n, float cos_a,
                                     float sin_a, int mirror, float* out, void* stream)
{
    int rc = pk_diversity_args("pk_diversity_shortcut", pop, ref, Np, Nr, n, out);
    if (rc) return rc;
    if (n > 3072) return pk_fail(PK_ERANGE, "pk_diversity_shortcut: more than 3072 trees (48 KB of shared memory)%s");
    if (Np == 0 || Nr == 0) return PK_OK;
    if (n == 0) return pk_cuda_check(cudaMemsetAsync(out, 0, sizeof(float) * (size_t)Np * Nr, (cudaStream_t)stream),
                                     "pk_diversity_shortcut memset");
    const int T = n < 32 ? 32 : (n > 256 ? 256 : ((n + 31) / 32) * 32);
    pk_diversity_shortcut_kernel<<<Np * Nr, T, (size_t)4 * n * 4, (cudaStream_t)stream>>>(pop, ref, Np, Nr, n, cos_a,
                                                                                         sin_a, mirror, out);
    return pk_cuda_check(cudaGetLastError(), "pk_diversity_shortcut launch");
}
