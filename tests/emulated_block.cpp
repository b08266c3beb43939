// One thread block on the CPU, for the L-BFGS kernels' reductions.
//
// Every thread of the block is a fiber that runs until it waits at a barrier or
// a warp operation.  Which warp runs next is the caller's priority list, so a
// warp can be held back as long as the barriers it shares with others allow: a
// kernel whose result changes with the list reads shared memory that another
// warp may already have written again.
//
// KERNELS_INC is the text of the reductions and of the L-BFGS kernels, with the
// two inline-PTX functions (warp maximum, named barrier) calling the ones here.
#include <math.h>
#include <stddef.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <ucontext.h>

#include <algorithm>
#include <initializer_list>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __constant__
#define __shared__
#define __forceinline__ inline
#define __noinline__
#define __align__(n) __attribute__((aligned(n)))

struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct double2 { double x, y; };
struct Dim { unsigned x; };
static Dim threadIdx, blockDim, blockIdx, gridDim;
static unsigned char pk_smem[1 << 18] __align__(16);
using std::max;
using std::min;

static float __fadd_rn(float a, float b) { return a + b; }
static float __fsub_rn(float a, float b) { return a - b; }
static float __fmul_rn(float a, float b) { return a * b; }
static float __fdiv_rn(float a, float b) { return a / b; }
static float __fsqrt_rn(float a) { return sqrtf(a); }
static double __dadd_rn(double a, double b) { return a + b; }
static double __dsub_rn(double a, double b) { return a - b; }
static double __dmul_rn(double a, double b) { return a * b; }
static double __ddiv_rn(double a, double b) { return a / b; }
static double __dsqrt_rn(double a) { return sqrt(a); }
static long long __float2ll_rn(float a) { return llrintf(a); }

// ---- the block ---------------------------------------------------------------
struct Fiber { ucontext_t ctx; std::vector<char> stack; bool done, waiting; };
struct Wait { int arrived = 0; std::vector<int> who; };   // a barrier or a warp operation
static std::vector<Fiber> fibers;
static std::vector<Wait> warp_wait, block_wait;
static std::vector<double> warp_val;   // [2][threads]: a lane's operand, two operations deep
static std::vector<int> warp_op;       // operations a lane has begun
static ucontext_t scheduler;
static int current;
static void (*body)();

static void wait_at(Wait& w, int count)
{
    w.who.push_back(current);
    if (++w.arrived == count) {
        for (int f : w.who) fibers[f].waiting = false;
        w.who.clear();
        w.arrived = 0;
    } else {
        fibers[current].waiting = true;
    }
    const int me = current;
    swapcontext(&fibers[me].ctx, &scheduler);   // resumed once released
    current = me;
    threadIdx.x = me;
}
static void __syncthreads() { wait_at(block_wait[0], blockDim.x); }
static void block_barrier(int id, int threads) { wait_at(block_wait[id], threads); }
static void __syncwarp() { wait_at(warp_wait[current / 32], 32); }

static double* exchange(double v)
{
    double* slot = &warp_val[(size_t)(warp_op[current]++ & 1) * blockDim.x];
    slot[current] = v;
    __syncwarp();
    return slot + current / 32 * 32;
}
template <typename T>
static T __shfl_xor_sync(unsigned, T v, int o) { const int l = current & 31; return (T)exchange(v)[l ^ o]; }
template <typename T>
static T __shfl_up_sync(unsigned, T v, int o) { const int l = current & 31; return (T)exchange(v)[l >= o ? l - o : l]; }
static float warp_max(float v) { const double* e = exchange(v); return (float)*std::max_element(e, e + 32); }
static int atomicOr(int* a, int v) { const int old = *a; *a |= v; return old; }

static void entry() { threadIdx.x = current; body(); fibers[current].done = true; swapcontext(&fibers[current].ctx, &scheduler); }

// Runs the block: always the first warp of the list that can go on.  False if
// no fiber can (a barrier that not all of its threads reach).
static bool run_block(int threads, const std::vector<int>& order, void (*kernel)())
{
    blockDim.x = threads;
    body = kernel;
    fibers.assign(threads, Fiber());
    warp_wait.assign(threads / 32, Wait());
    block_wait.assign(16, Wait());
    warp_val.assign(2 * threads, 0.0);
    warp_op.assign(threads, 0);
    for (int t = 0; t < threads; ++t) {
        Fiber& f = fibers[t];
        f.stack.resize(1 << 16);
        f.done = f.waiting = false;
        getcontext(&f.ctx);
        f.ctx.uc_stack.ss_sp = f.stack.data();
        f.ctx.uc_stack.ss_size = f.stack.size();
        f.ctx.uc_link = nullptr;
        makecontext(&f.ctx, entry, 0);
    }
    for (;;) {
        int next = -1;
        bool left = false;
        for (int w : order)
            for (int t = 32 * w; t < 32 * w + 32 && next < 0; ++t) {
                left |= !fibers[t].done;
                if (!fibers[t].done && !fibers[t].waiting) next = t;
            }
        if (next < 0) return !left;
        current = next;
        swapcontext(&scheduler, &fibers[next].ctx);
    }
}

// What the threads got from their reductions (all threads must get the same).
static std::vector<std::vector<double>> recorded;
static void record(std::initializer_list<double> v) { recorded[current].insert(recorded[current].end(), v); }

#include KERNELS_INC

// ---- five iterations of a small quadratic on one block -------------------------
template <typename F>
struct Run {
    int N, m, threads;
    std::vector<F> x, g, d, pg, S, Y, ro, scalars;
    int hlen = 0, hstart = 0, evals = 0, active = 0, any[2] = {0, 0};
    PkLbfgsState<F> s;
    Run(int N_, int m_, int threads_) : N(N_), m(m_), threads(threads_), x(N_), g(N_), d(N_), pg(N_),
                                        S((size_t)m_ * N_), Y((size_t)m_ * N_), ro(m_), scalars(5)
    {
        for (int k = 0; k < N; ++k) x[k] = (F)sin(1.0 + 0.7 * k);
    }
};
static Run<float>* rf;
static Run<double>* rd;
static int cur_iter;
static PkLbfgsParams prm;
static void kernel_f() { pk_lbfgs_iterate_kernel<float>(rf->s, cur_iter, prm); }
static void kernel_d() { pk_lbfgs_iterate_kernel<double>(rd->s, cur_iter, prm); }

template <typename F>
static bool iterate(Run<F>& r, const std::vector<int>& order, void (*kernel)(), std::vector<F>& result)
{
    F* sc = r.scalars.data();   // loss, ploss, loss0, H, t
    r.s.x = r.x.data(); r.s.g = r.g.data(); r.s.loss = sc; r.s.d = r.d.data(); r.s.pg = r.pg.data();
    r.s.ploss = sc + 1; r.s.loss0 = sc + 2; r.s.S = r.S.data(); r.s.Y = r.Y.data(); r.s.ro = r.ro.data();
    r.s.H = sc + 3; r.s.t = sc + 4; r.s.hlen = &r.hlen; r.s.hstart = &r.hstart; r.s.evals = &r.evals;
    r.s.active = &r.active; r.s.any_active = r.any; r.s.M = 1; r.s.N = r.N; r.s.m = r.m;
    blockIdx.x = 0;
    gridDim.x = 1;
    result.clear();
    for (cur_iter = 1; cur_iter <= 5; ++cur_iter) {
        F loss = 0;
        for (int k = 0; k < r.N; ++k) {
            const F c = (F)(1 + (k * 37 % 11));
            r.g[k] = c * r.x[k];
            loss += c * r.x[k] * r.x[k] / 2;
        }
        sc[0] = loss;
        memset(pk_smem, 0xff, sizeof(pk_smem));   // NaN where nothing was written
        recorded.assign(r.threads, std::vector<double>());
        if (!run_block(r.threads, order, kernel)) return false;
        for (int t = 0; t < r.threads; ++t)
            for (double v : recorded[t]) result.push_back((F)v);
        for (int k = 0; k < r.N; ++k) r.x[k] += r.scalars[4] * r.d[k];
        result.insert(result.end(), r.d.begin(), r.d.end());
        result.insert(result.end(), r.ro.begin(), r.ro.end());
        result.insert(result.end(), r.scalars.begin(), r.scalars.end());
    }
    return true;
}

template <typename F>
static bool with_order(int N, int m, int threads, const std::vector<int>& order, std::vector<F>& out);
template <>
bool with_order<float>(int N, int m, int threads, const std::vector<int>& order, std::vector<float>& out)
{
    Run<float> r(N, m, threads);
    rf = &r;
    return iterate(r, order, kernel_f, out);
}
template <>
bool with_order<double>(int N, int m, int threads, const std::vector<int>& order, std::vector<double>& out)
{
    Run<double> r(N, m, threads);
    rd = &r;
    return iterate(r, order, kernel_d, out);
}

// The lists: in order, reversed, and each warp first and last among the others.
template <typename F>
static int check(int N, int m, int threads)
{
    const int nw = threads / 32;
    std::vector<int> order(nw);
    for (int w = 0; w < nw; ++w) order[w] = w;
    std::vector<F> want, got;
    if (!with_order<F>(N, m, threads, order, want)) { printf("N = %d, %d threads: a barrier is left waiting\n", N, threads); return 1; }
    for (F v : want) if (!(v == v)) { printf("N = %d, %d threads: NaN\n", N, threads); return 1; }
    int bad = 0;
    for (int k = 0; k <= 2 * nw; ++k) {
        std::vector<int> list(order);
        if (k == 0) std::reverse(list.begin(), list.end());
        else if (k <= nw) std::swap(list[k - 1], list[nw - 1]);
        else std::swap(list[k - nw - 1], list[0]);
        const bool ok = with_order<F>(N, m, threads, list, got);
        if (!ok || memcmp(got.data(), want.data(), want.size() * sizeof(F)) != 0) {
            printf("N = %d, m = %d, %d threads, %zu bytes: differs with the warps run as", N, m, threads, sizeof(F));
            for (int w : list) printf(" %d", w);
            printf("\n");
            ++bad;
        }
    }
    return bad;
}

int main(int argc, char** argv)
{
    if (argc != 4) return 2;
    const int N = atoi(argv[1]), m = atoi(argv[2]), threads = atoi(argv[3]);
    prm.lr = 1.0; prm.max_step = 0.5; prm.has_max_step = 1; prm.max_eval = 1000;
    return check<float>(N, m, threads) + check<double>(N, m, threads) ? 1 : 0;
}
